"""The float32 page kernel (groups the tensor-core kernel has no tile for) and the ring writer at their
edges: head tiles with idle heads, one page and none, windows that are no multiple of a round, a spilled
page, partial block ranges; rows off the 16-byte grid."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
    want = []
    for seq in range(2):
        kd, vd = (x.double() for x in ctx.dequant(0, seq, 0, n))
        s = torch.einsum("hgd,htd->hgt", q[seq].double().view(h, group, 128), kd) / 128 ** 0.5
        want.append(torch.einsum("hgt,htd->hgd", s.softmax(-1), vd).reshape(h * group, 128))
    want = torch.stack(want)
    # Without outliers: float32 products and sums over 128 channels, scores of some tens in the
    # exponent.  With them, the corrections are stored in fp16: half a unit in the eleventh bit of
    # q * delta / sqrt(128), up to 4 * 200 / 11.3 * 2^-12 = 0.017 in a score.
    tol = 2e-2 if frac else 2e-5
    assert ((out - want).norm() / want.norm()).item() < tol
    if n == 5000:  # two halves of the blocks, merged
        nb = ctx.cold_blocks(n)
        parts = torch.stack([ctx.decode_partial(0, q, 0, nb // 2, False),
                             ctx.decode_partial(0, q, nb // 2, nb, True)])
        both = ctx.lse_combine(parts.reshape(2, -1, 130)).view_as(out)
        assert ((both - want).norm() / want.norm()).item() < tol
