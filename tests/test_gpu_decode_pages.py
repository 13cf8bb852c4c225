"""The float32 page kernel (groups the tensor-core kernel has no tile for) and the ring writer at their
edges: head tiles with idle heads, one page and none, windows that are no multiple of a round, a spilled
page, partial block ranges, ragged batches; rows off the 16-byte grid.  (The group of three is served by
the general-shape kernel, through the same merge.)"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stored(ctx, seq, n, mode="nf4_asym"):
    """Keys and values of a sequence in float64 as the kernels take them: at an outlier the dense
    value plus the correction stored in fp16."""
    import torch

    from oracle import tq_oracle as orc

    kd, vd = (x.double().cpu().numpy() for x in ctx.dequant(0, seq, 0, n))
    h, s = kd.shape[0], ctx.geom.block_tokens
    for b in range(ctx.cold_blocks(n)):
        blk = ctx.export_block(0, seq, b)
        if blk["outlier_idx"] is None or not len(blk["outlier_idx"]):
            continue
        dense = orc.dequant_keys(orc.unpack_key_codes(blk["key_indices"], h * s * 128).reshape(h, s, 128),
                                 blk["nf4_scale"][0], blk["nf4_mean"][0], mode=mode).astype(np.float32)
        at = blk["outlier_idx"]
        full = dense.astype(np.float64).reshape(-1)
        full[at] += (blk["outlier_val"].astype(np.float32) - dense.reshape(-1)[at]).astype(np.float16)
        kd[:, b * s:(b + 1) * s] = full.reshape(h, s, 128)
    return torch.from_numpy(kd).cuda(), torch.from_numpy(vd).cuda()


def _errors(ctx, q, lens, out, mode="nf4_asym"):
    """Per sequence and query head: the output's distance from float64 on what is stored, over its
    norm, and the bound it has to meet."""
    import torch

    h, group = ctx.geom.n_kv_heads, ctx.geom.n_q_heads // ctx.geom.n_kv_heads
    err, bound = [], []
    for seq, n in enumerate(lens):
        if n == 0:
            assert not out[seq].any()
            continue
        kd, vd = _stored(ctx, seq, n, mode)
        qd = q[seq].double().view(h, group, 128)
        s = torch.einsum("hgd,htd->hgt", qd, kd) / 128 ** 0.5
        want = torch.einsum("hgt,htd->hgd", s.softmax(-1), vd).reshape(h * group, 128)
        # A score is a float32 sum of 128 products in chains of eight to sixteen: within 16 half units
        # of the sum of magnitudes, twice (numerator and denominator) in the output; the exponentials
        # and the other sums stay below 2e-5.
        mags = torch.einsum("hgd,htd->hgt", qd.abs(), kd.abs()).amax(-1).reshape(-1) / 128 ** 0.5
        err.append((out[seq] - want).norm(dim=1) / want.norm(dim=1))
        bound.append(2e-5 + 32 * 2.0 ** -24 * mags)
    return torch.cat(err), torch.cat(bound)


@pytest.mark.parametrize("group,vb,dt", [(3, 3, "float16"), (5, 4, "bfloat16"), (6, 3, "float32"),
                                         (7, 3, "bfloat16"), (7, 4, "float16"), (9, 3, "float16"),
                                         (16, 4, "float16")])
@pytest.mark.parametrize("n", [1, 17, 129, 512, 513, 1400, 5000])
@pytest.mark.parametrize("layout,frac", [("plain", 0.02), ("off_grid", 0.0)])
def test_page_kernel_against_float64(group, vb, dt, n, layout, frac):
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv, make_q

    h = 2
    ctx = KVContext(n_seqs=2, n_kv_heads=h, n_q_heads=h * group, value_bits=vb, kv_dtype=dt,
                    max_tokens_per_seq=n, seed=3, outlier_frac=frac)
    for seq in range(2):
        k, v = make_kv(40 + seq, h, n, dtype=np.float32)
        if n > 600 and frac:
            k[5:12, 1] = 200.0  # more outliers than the overflow list takes
        kt, vt = (torch.from_numpy(x).to(getattr(torch, dt)).cuda() for x in (k, v))
        if layout == "off_grid":
            wide = torch.zeros((2, n, h, 131), dtype=kt.dtype, device="cuda")
            wide[0, ..., 1:129], wide[1, ..., 1:129] = kt, vt
            kt, vt = wide[0, ..., 1:129], wide[1, ..., 1:129]
        m = n // 3
        for a, b in ((0, m), (m, n)):
            if b > a:
                ctx.append(0, kt[None, a:b], vt[None, a:b], seq_begin=seq)
    q = torch.from_numpy(np.stack([make_q(s, h * group) for s in range(2)])).cuda()
    out = ctx.decode(0, q)
    assert ctx.last_kernel() == "general" and ctx.status() == 0
    err, bound = _errors(ctx, q, [n, n], out)
    assert (err <= bound).all(), (err / bound).max().item()
    if n == 5000:  # two halves of the blocks, merged
        nb = ctx.cold_blocks(n)
        parts = torch.stack([ctx.decode_partial(0, q, 0, nb // 2, False),
                             ctx.decode_partial(0, q, nb // 2, nb, True)])
        both = ctx.lse_combine(parts.reshape(2, -1, 130)).view_as(out)
        err, bound = _errors(ctx, q, [n, n], both)
        assert (err <= bound).all(), (err / bound).max().item()


@pytest.mark.parametrize("group,q_dtype", [(5, "float32"), (7, "float16"), (7, "bfloat16"),
                                           (8, "float32"), (11, "float32")])
@pytest.mark.parametrize("mode", ["nf4_asym", "nf4", "uniform"])
def test_page_kernel_on_a_ragged_batch(group, q_dtype, mode):
    """Sequences of no, few and many pages side by side, every key grid, 16-bit queries, and the form
    whose partials lie inside the library; groups of eight as far as the general kernel is asked for."""
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv, make_q

    h, lens = 2, [700, 0, 40, 5000, 1300]
    ctx = KVContext(n_seqs=len(lens), n_kv_heads=h, n_q_heads=h * group, value_bits=3 + group % 2,
                    kv_dtype="float16", max_tokens_per_seq=max(lens), seed=3, key_mode=mode,
                    outlier_frac=0.02)
    for seq, n in enumerate(lens):
        if n:
            k, v = make_kv(60 + seq, h, n, dtype=np.float16)
            if seq == 4:
                k[5:12, 1] = 90.0  # more outliers than the overflow list takes
            ctx.append(0, *(torch.from_numpy(x)[None].cuda() for x in (k, v)), seq_begin=seq)
    q = torch.from_numpy(np.stack([make_q(s, h * group) for s in range(len(lens))])).cuda()
    q = q.to(getattr(torch, q_dtype))
    ctx.set_kernel("general")
    outs = [ctx.decode(0, q), ctx.decode_static_scratch(0, q)]
    assert ctx.last_kernel() == "general" and ctx.status() == 0
    for out in outs:
        err, bound = _errors(ctx, q, lens, out, mode)
        assert (err <= bound).all(), (err / bound).max().item()
