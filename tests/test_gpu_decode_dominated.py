"""The page kernel where one token takes nearly all of the softmax and has no value: what is left of the
output comes from probabilities of 1e-11 and less.  Against float64 on what is stored."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_decode_pages import _errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,vb", [(5, 3), (7, 4), (12, 3)])
@pytest.mark.parametrize("nats", [16, 24, 32])
@pytest.mark.parametrize("at", [100, 1100])  # in the first page and in the last one
def test_dominating_token_without_a_value(group, vb, nats, at):
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv, make_q

    h, n = 2, 1600
    k, v = make_kv(83, h, n, dtype=np.float32)
    q = make_q(6, h * group).reshape(h, group, 128)
    k *= 0.1
    for i in range(h):  # a key that every head of the group scores `nats`
        k[at, i] = np.linalg.lstsq(q[i].astype(np.float64), np.full(group, nats * 128 ** 0.5), rcond=None)[0]
    v[at] = 0
    ctx = KVContext(n_seqs=1, n_kv_heads=h, n_q_heads=h * group, value_bits=vb, kv_dtype="float32",
                    max_tokens_per_seq=n, seed=3, outlier_frac=0.0)
    ctx.append(0, *(torch.from_numpy(x)[None].cuda() for x in (k, v)))
    qt = torch.from_numpy(q.reshape(1, h * group, 128)).cuda()
    out = ctx.decode(0, qt)
    assert ctx.last_kernel() == "general" and ctx.status() == 0
    err, bound = _errors(ctx, qt, [n], out)
    assert (err <= bound).all(), (err / bound).max().item()
