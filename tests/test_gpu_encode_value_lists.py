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
