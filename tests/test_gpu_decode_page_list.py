"""The page kernel's list of pages (csrc/decode_pages.cu): more rows than shares and fewer, sequences
without pages between others, more sequences than a launch covers, lengths that grew under a captured
graph.  Checked against float64 on what is stored."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_decode_pages import _errors

pytestmark = pytest.mark.gpu


def _context(lens, h, group, vb=3, dt="float16", max_tokens=None):
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv, make_q

    ctx = KVContext(n_seqs=len(lens), n_kv_heads=h, n_q_heads=h * group, value_bits=vb, kv_dtype=dt,
                    max_tokens_per_seq=max_tokens or max(lens), seed=3, outlier_frac=0.02)
    made = {}
    for seq, n in enumerate(lens):
        if n:
            key = (seq % 7, n)
            if key not in made:
                made[key] = [torch.from_numpy(x)[None].to(getattr(torch, dt)).cuda()
                             for x in make_kv(80 + seq % 7, h, n, dtype=np.float32)]
            ctx.append(0, *made[key], seq_begin=seq)
    q = torch.from_numpy(make_q(5, h * group))[None].repeat(len(lens), 1, 1).cuda()
    return ctx, q


class _Only:
    """A context seen through a list of its sequences."""

    def __init__(self, ctx, seqs):
        self.ctx, self.seqs, self.geom = ctx, seqs, ctx.geom

    def dequant(self, layer, seq, a, b):
        return self.ctx.dequant(layer, self.seqs[seq], a, b)

    def export_block(self, layer, seq, b):
        return self.ctx.export_block(layer, self.seqs[seq], b)

    def cold_blocks(self, n):
        return self.ctx.cold_blocks(n)


@pytest.mark.parametrize("lens,h,group", [
    ([513], 1, 5),                                     # one page, one group of the GPU
    ([513, 0, 768, 769, 300, 20000], 2, 7),            # short rows beside a long one
    ([0, 0, 40], 2, 6),                                # no page at all
    ([1100] * 40, 8, 9),                               # 1 920 pages in 640 rows: shares across rows
])
def test_shares_of_the_list(lens, h, group):
    ctx, q = _context(lens, h, group)
    out = ctx.decode(0, q)
    pick = sorted({0, len(lens) - 1, len(lens) // 2, *range(min(len(lens), 6))})
    err, bound = _errors(_Only(ctx, pick), q[pick], [lens[i] for i in pick], out[pick])
    assert (err <= bound).all(), (err / bound).max().item()
    if group == 9:  # equal tokens: equal but for the order of the sums, wherever the shares fall
        same = out[::7]
        assert float((same - same[0]).abs().max()) <= 1e-5 * float(same[0].abs().max())


def test_more_sequences_than_a_launch_covers():
    lens = [0] * 2100
    for i in (0, 7, 2046, 2047, 2048, 2099):
        lens[i] = 530 + i % 100
    ctx, q = _context(lens, 1, 5)
    out = ctx.decode(0, q)
    pick = [i for i, n in enumerate(lens) if n]
    err, bound = _errors(_Only(ctx, pick), q[pick], [lens[i] for i in pick], out[pick])
    assert (err <= bound).all(), (err / bound).max().item()
    assert not out[[1, 2045, 2098]].any()


def test_graph_replayed_on_longer_sequences():
    """The split counts are the host's, the lengths the device's: a captured decode attends whatever is
    stored when it is replayed."""
    import torch

    from turboquant_pro_b200.synth import make_kv

    lens, more = [700, 600], [7000, 600]
    ctx, q = _context(lens, 2, 7, max_tokens=9000)
    out = torch.empty_like(q)
    ctx.decode(0, q, out=out)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.decode(0, q, out=out)
    for seq in range(2):
        k, v = make_kv(90 + seq, 2, more[seq], dtype=np.float32)
        ctx.append(0, *(torch.from_numpy(x)[None].half().cuda() for x in (k, v)), seq_begin=seq)
    graph.replay()
    torch.cuda.synchronize()
    err, bound = _errors(ctx, q, [a + b for a, b in zip(lens, more)], out)
    assert (err <= bound).all(), (err / bound).max().item()


@pytest.mark.parametrize("q_scale,v_scale", [(1e25, 1.0), (1e-30, 1.0), (1.0, 1e-18), (1.0, 1e15)])
def test_operands_far_from_one(q_scale, v_scale):
    """The operands' halves are scaled by powers of two, page by page: no magnitude that float32 holds
    leaves the fp16 range."""
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv, make_q

    n, h, group = 700, 2, 5
    ctx = KVContext(n_seqs=1, n_kv_heads=h, n_q_heads=h * group, value_bits=4, kv_dtype="float32",
                    max_tokens_per_seq=n, seed=3, outlier_frac=0.0)
    k, v = (torch.from_numpy(x)[None].cuda() for x in make_kv(81, h, n, dtype=np.float32))
    ctx.append(0, k, v * v_scale)
    q = torch.from_numpy(make_q(5, h * group))[None].cuda() * q_scale
    out = ctx.decode(0, q)[0].double().view(h, group, 128)
    kd, vd = (x.double() for x in ctx.dequant(0, 0, 0, n))
    s = torch.einsum("hgd,htd->hgt", q[0].double().view(h, group, 128), kd) / 128**0.5
    ref = torch.einsum("hgt,htd->hgd", s.softmax(-1), vd)
    # float32 sums of 128 and 700 terms: 2^-24 of the largest times the root of their number, and room
    assert float((out - ref).norm() / ref.norm()) <= 1e-5
