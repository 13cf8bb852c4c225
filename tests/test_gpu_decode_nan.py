"""Pages whose scores and values are not numbers, beside a window of ordinary tokens: the merge must not
take their partial for one that holds nothing."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group,dt", [(7, "float16"), (12, "bfloat16"), (3, "float32")])
@pytest.mark.parametrize("static", [False, True])
def test_nan_pages_are_not_empty_ones(group, dt, static):
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.synth import make_kv, make_q

    h, n = 2, 512 + 3 * 256
    ctx = KVContext(n_seqs=2, n_kv_heads=h, n_q_heads=h * group, value_bits=3, kv_dtype=dt,
                    max_tokens_per_seq=n, seed=3, outlier_frac=0.0)
    ctx.set_kernel("general")
    for seq in range(2):
        k, v = make_kv(90 + seq, h, n, dtype=np.float32)
        if seq == 0:  # head 0: every page, so that no partial of a page has a score
            k[:3 * 256, 0, 7] = np.nan
            v[:3 * 256, 0, 7] = np.nan
        ctx.append(0, *(torch.from_numpy(x).to(getattr(torch, dt))[None].cuda() for x in (k, v)), seq_begin=seq)
    assert ctx.cold_blocks(n) == 3
    q = torch.from_numpy(np.stack([make_q(s, h * group) for s in range(2)])).cuda()
    out = (ctx.decode_static_scratch if static else ctx.decode)(0, q).view(2, h, group, 128)
    assert torch.isnan(out[0, 0]).all()
    assert torch.isfinite(out[0, 1]).all() and torch.isfinite(out[1]).all()
