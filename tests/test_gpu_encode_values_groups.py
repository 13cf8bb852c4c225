"""The value encoder of 16-token groups on tcgen05.mma (csrc/encode.cu), which serves blocks that are no multiple
of 128 tokens, against the one on mma.sync, bit for bit: 96- and 160-token blocks."""

import pytest
from test_gpu_encode_values import _values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [192, 320])
@pytest.mark.parametrize("dt,vb,key_mode", [("float16", 3, None), ("bfloat16", 4, None), ("float32", 3, None),
                                            ("float32", 4, None), ("float16", 4, "polar"),
                                            ("float16", 3, "polar")])
@pytest.mark.parametrize("aligned", [True, False])
def test_groups_write_the_same_pages(window, dt, vb, key_mode, aligned):
    """Every element type, code width and row alignment, and keys in PolarQuant form; the tokens include zero
    rows, whose products sit on a boundary in every channel: three in one group, whole groups (more at once
    than the list of deferred products holds), one that goes through the ring first."""
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(12)
    v = torch.randn((1, 1100, 2, 128), generator=gen, device="cuda")
    for lo, hi in ((5, 8), (32, 80), (200, 201), (720, 722)):
        v[:, lo:hi] = 0
    a, b = _values(v.to(getattr(torch, dt)), (700, 400), 2, vb, window, dt, aligned, key_mode)
    assert a == b


@pytest.mark.parametrize("window", [192, 320])
@pytest.mark.parametrize("dt,vb,aligned", [("float16", 3, True), ("bfloat16", 4, True), ("float32", 4, False)])
def test_groups_fill_the_pipeline(window, dt, vb, aligned):
    """More than four groups of 16 tokens for each of the six parts of a CTA: the pipeline of three groups in
    flight runs full and drains; the second call also takes rows from the ring."""
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(13)
    b, h, n = 2, 8, 4200
    assert b * h * ((n - window) // 16) > 4 * 6 * 148
    v = torch.randn((b, n, h, 128), generator=gen, device="cuda").to(getattr(torch, dt))
    v[:, 2000:2100] = 0
    x, y = _values(v, (900, n - 900), h, vb, window, dt, aligned)
    assert x == y
