"""An append recorded in a CUDA graph stores what the same append stores when it is launched directly:
the value encoder starts while the key encoder drains, in a graph as on a stream."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dt", [(1400, "bfloat16"), (700, "float32")])
def test_captured_append(n, dt):
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv

    stores = []
    for captured in (False, True):
        ctx = KVContext(n_layers=2, n_seqs=2, n_kv_heads=2, n_q_heads=4, kv_dtype=dt, max_tokens_per_seq=4 * n,
                        seed=3)
        k, v = (torch.stack([torch.from_numpy(x)] * 2).to(getattr(torch, dt)).cuda()
                for x in make_kv(7, 2, n, dtype=np.float32))
        for layer in range(2):
            ctx.append(layer, k, v)
        torch.cuda.synchronize()
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                for layer in range(2):
                    ctx.append(layer, k, v)
            graph.replay()
        else:
            for layer in range(2):
                ctx.append(layer, k, v)
        torch.cuda.synchronize()
        assert not ctx.status()
        stores.append([x.cpu() for layer in range(2) for seq in range(2) for x in ctx.dequant(layer, seq, 0, 2 * n)])
    for a, b in zip(*stores):
        assert torch.equal(a, b)
