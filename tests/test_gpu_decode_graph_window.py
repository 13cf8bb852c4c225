"""Decodes captured while every sequence fits the uncompressed window, replayed after blocks were compressed."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_decode_pages import _errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,dt", [(7, "float16"), (3, "float32")])  # page kernel, general kernel
@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("start", [0, 40, 512])
def test_captured_below_the_window(group, dt, static, start):
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv, make_q

    h, n = 2, 3000
    ctx = KVContext(n_seqs=2, n_kv_heads=h, n_q_heads=h * group, value_bits=3, kv_dtype=dt,
                    max_tokens_per_seq=n, seed=3, outlier_frac=0.0)
    ctx.set_kernel("general")
    tokens = [[torch.from_numpy(x).to(getattr(torch, dt))[None].cuda()
               for x in make_kv(70 + s, h, n, dtype=np.float32)] for s in range(2)]
    q = torch.from_numpy(np.stack([make_q(s, h * group) for s in range(2)])).cuda()
    out = torch.empty_like(q)
    decode = ctx.decode_static_scratch if static else ctx.decode
    for s in range(2):
        if start:
            ctx.append(0, *(x[:, :start] for x in tokens[s]), seq_begin=s)
    decode(0, q, out=out)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        decode(0, q, out=out)
    for s, end in enumerate((n, 700)):
        ctx.append(0, *(x[:, start:end] for x in tokens[s]), seq_begin=s)
        assert ctx.cold_blocks(end) > 0
    graph.replay()
    torch.cuda.synchronize()
    err, bound = _errors(ctx, q, [n, 700], out)
    assert (err <= bound).all(), (err / bound).max().item()
