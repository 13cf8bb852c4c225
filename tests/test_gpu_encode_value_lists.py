"""The value encoder's lists of products near a boundary (csrc/encode_values.cu) when every product is
on one, against the encoder on mma.sync."""

import pytest
from test_gpu_encode_values import _values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,scale", [("float16", float("inf")), ("bfloat16", 1e-18), ("float32", 1e-18)])
@pytest.mark.parametrize("vb", [3, 4])
def test_every_product_listed(dt, scale, vb):
    """Rows whose norm cannot be divided out: 16 entries a lane and group, lists that are full from the
    first group on, and warps that wait for room while others read the same counts."""
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    v = torch.randn((1, 1400, 3, 128), generator=gen, device="cuda")
    if scale == float("inf"):
        v[..., 17] = scale
    else:
        v *= scale
    a, b = _values(v.to(getattr(torch, dt)), (700, 700), 3, vb, 512, dt)
    assert a == b


@pytest.mark.parametrize("dt,vb", [("float16", 3), ("bfloat16", 4), ("float32", 4)])
def test_a_tile_that_is_not_encoded_is_stored_as_zeros(dt, vb):
    """The test hook withholds the products of the first CTA's second tile; the waits for them run out, the
    status word says so, and that tile and the CTA's later ones are rows of zeros, the others as ever."""
    import torch

    from turboquant_pro_b200 import KVContext

    h, blocks, n = 8, 20, 512 + 20 * 256
    gen = torch.Generator(device="cuda")
    gen.manual_seed(10)
    x = torch.randn((1, n, h, 128), generator=gen, device="cuda").to(getattr(torch, dt))
    good, ctx = (KVContext(n_layers=1, n_seqs=1, n_kv_heads=h, n_q_heads=h, value_bits=vb,
                           hot_window=512, max_tokens_per_seq=n, kv_dtype=dt, seed=5)
                 for _ in range(2))
    good.append(0, x, x)
    want_k, want = good.dequant(0, 0, 0, n)
    ctx._regions["pages"].fill_(0x5A)  # what an earlier user of the pages left there
    ctx.debug_wait(wait_limit=512, withhold_tile=(1 << 20) + 1)
    ctx.append(0, x, x)
    assert ctx.status() == 2 and ctx.status() == 0
    ctx.debug_wait()
    k, v = ctx.dequant(0, 0, 0, n)
    assert torch.equal(k, want_k)
    tile = 64 if dt == "float32" else 128
    parts, ctas = 256 // tile, torch.cuda.get_device_properties(0).multi_processor_count
    lost = torch.zeros((h, n), dtype=torch.bool, device="cuda")
    for w in range(ctas, h * blocks * parts, ctas):
        head, t = w // (blocks * parts), w % (blocks * parts) * tile
        lost[head, t:t + tile] = True
    assert lost.any() and not v[lost].any() and torch.equal(v[~lost], want[~lost])
    for head, t in lost.nonzero()[::tile].tolist():
        codes = ctx.export_block(0, 0, t // 256)["value_indices"]
        row = 128 * vb // 8
        at = (head * 256 + t % 256) * row
        assert not codes.reshape(-1)[at:at + row].any()
    ctx.clear(0, 0)
    ctx.append(0, x, x)
    assert ctx.status() == 0 and torch.equal(ctx.dequant(0, 0, 0, n)[1], want)


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("vb", [3, 4])
def test_sums_that_cancel_near_a_boundary(dt, vb):
    """Rows that put one channel on a boundary by two large parts of opposite sign: where the tensor cores'
    sums are least exact and a wrong code is nearest."""
    import numpy as np
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200.context import value_codebook

    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    h, n = 4, 4096
    pi = torch.from_numpy(np.asarray(KVContext(
        n_layers=1, n_seqs=1, n_kv_heads=1, n_q_heads=1, value_bits=vb, hot_window=512,
        max_tokens_per_seq=600, kv_dtype=dt, seed=3).pi, dtype=np.float32)).cuda().double()
    bounds = torch.from_numpy(np.asarray(value_codebook(128, vb)[1])).cuda().double()
    row = pi[torch.randint(0, 128, (n, h), device="cuda", generator=gen)]
    first = torch.arange(128, device="cuda") < 64
    n1 = (row * row * first).sum(-1)
    n2 = (row * row * ~first).sum(-1)
    b = bounds[torch.randint(0, len(bounds), (n, h), device="cuda", generator=gen)]
    # (n1 - s n2) / sqrt(n1 + s^2 n2) = b, for s of the sign that cancels
    lo, hi = torch.full_like(n1, -50.0), torch.full_like(n1, 50.0)
    for _ in range(60):
        mid = (lo + hi) / 2
        above = (n1 - mid * n2) / (n1 + mid * mid * n2).sqrt() > b
        lo, hi = torch.where(above, mid, lo), torch.where(above, hi, mid)
    v = torch.where(first, row, -lo[..., None] * row).to(getattr(torch, dt))[None]
    a, b = _values(v, (n,), h, vb, 512, dt)
    assert a == b
