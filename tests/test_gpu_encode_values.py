"""The value encoder for blocks of 128 and 256 tokens (csrc/encode_values.cu) against the one on
mma.sync, bit for bit: where tiles, ring and caller's rows meet, and rows off the ordinary."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _values(v, chunks, h, vb, window, dt, aligned=True, key_mode=None):
    """The value containers of every block after appends of ``chunks`` tokens, by both encoders."""
    import torch

    from turboquant_pro_b200 import KVContext
    from turboquant_pro_b200._lib import load

    lib = load()
    b, n = v.shape[0], v.shape[1]
    if not aligned:
        wide = torch.zeros((b, n, h, 129), dtype=v.dtype, device="cuda")
        wide[..., 1:] = v
        v = wide[..., 1:]
    out = []
    try:
        for kind in (0, 1):
            assert lib.tq_set_value_encoder(kind) == 0
            extra = {} if key_mode is None else dict(key_mode=key_mode, key_bits=vb, outlier_frac=0.0)
            ctx = KVContext(n_layers=1, n_seqs=b, n_kv_heads=h, n_q_heads=h, value_bits=vb,
                            hot_window=window, max_tokens_per_seq=n, kv_dtype=dt, seed=3, **extra)
            t = 0
            for c in chunks:
                ctx.append(0, v[:, t:t + c], v[:, t:t + c])
                t += c
            assert t == n and ctx.status() & 2 == 0
            blocks = ctx.lengths(0, 0)[1] // (window // 2)
            assert blocks > 0
            got = []
            for s in range(b):
                for i in range(blocks):
                    e = ctx.export_block(0, s, i)
                    names = ["value_indices", "value_norms"]
                    if key_mode == "polar":
                        names += ["key_indices"]
                    got += [np.asarray(e[x]).tobytes() for x in names]
            out.append(got)
    finally:
        assert lib.tq_set_value_encoder(-1) == 0
    return out


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("vb", [3, 4])
@pytest.mark.parametrize("window,chunks,aligned", [
    (512, (513,), True),                      # one block, one CTA's tile after the other
    (512, (300, 1, 290, 700, 129), True),     # tiles cut between ring and rows, the ring wrapping
    (256, (257, 100, 31, 700), True),         # 128-token blocks
    (512, (700, 500), False),                 # rows off the 16-byte grid
])
def test_tiles_equal_groups(dt, vb, window, chunks, aligned):
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    h = 3
    v = torch.randn((2, sum(chunks), h, 128), generator=gen, device="cuda")
    v = (v * torch.exp(torch.randn((h, 128), generator=gen, device="cuda"))).to(getattr(torch, dt))
    a, b = _values(v, chunks, h, vb, window, dt, aligned)
    assert a == b


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("vb", [3, 4])
def test_rows_off_the_ordinary(dt, vb):
    """Zero rows (every product on a boundary), single entries (products beyond the outermost
    boundary, and sums that reach 1), rows of Pi, denormals, the largest numbers, infinities, NaN."""
    import torch

    from turboquant_pro_b200 import KVContext

    gen = torch.Generator(device="cuda")
    gen.manual_seed(6)
    h, n = 2, 1100
    v = torch.randn((1, n, h, 128), generator=gen, device="cuda")
    pi = KVContext(n_layers=1, n_seqs=1, n_kv_heads=1, n_q_heads=1, value_bits=vb, hot_window=512,
                   max_tokens_per_seq=600, kv_dtype=dt, seed=3).pi
    pi = torch.from_numpy(np.asarray(pi, dtype=np.float32)).cuda()
    v[0, 0:40] = 0.0
    v[0, 20:30] *= -1.0                        # (zeros with a sign)
    for t in range(128):                       # one entry, both signs
        v[0, 64 + t, 0], v[0, 64 + t, 1] = 0.0, 0.0
        v[0, 64 + t, 0, t], v[0, 64 + t, 1, t] = 1.0, -3.0
    v[0, 200:328, 0] = pi                      # y = 1 in one channel
    v[0, 200:328, 1] = pi.T
    tiny, huge = {"float16": (6e-8, 6e4), "bfloat16": (1e-39, 3e38), "float32": (1e-42, 3e38)}[dt]
    v[0, 330:340] *= tiny
    v[0, 340:350] *= huge / 8
    v[0, 350:360] *= {"float16": 1e-5}.get(dt, 1e-20)
    v[0, 360:370, :, 5] = float("inf")
    v[0, 370:380, :, 7] = float("nan")
    v[0, 380:390] = 1.0
    a, b = _values(v.to(getattr(torch, dt)), (n,), h, vb, 512, dt)
    assert a == b


@pytest.mark.parametrize("dt,vb", [("float16", 3), ("bfloat16", 4), ("float32", 4)])
def test_many_tiles_per_cta(dt, vb):
    """More than eight tiles a CTA: the ring of slots wraps, the lists fill and drain."""
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)
    h, n = 32, 6000
    v = torch.randn((1, n, h, 128), generator=gen, device="cuda").to(getattr(torch, dt))
    v[:, 1000:1100] = 0
    v[:, 2000:2040] = float("inf")             # every channel of every head on the lists
    a, b = _values(v, (n,), h, vb, 512, dt)
    assert a == b


def test_polar_keys_take_the_same_tiles():
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(8)
    v = torch.randn((1, 1300, 2, 128), generator=gen, device="cuda").half()
    a, b = _values(v, (700, 600), 2, 4, 512, "float16", key_mode="polar")
    assert a == b


@pytest.mark.parametrize("vb,outer", [(3, 0.3), (4, 0.25)])
def test_codebook_wider_than_the_table(vb, outer, monkeypatch):
    """A caller's codebook whose boundaries crowd in the middle leaves no range in which 32 bins part all of
    them: the table must not be used with the outer ones beyond its range."""
    import torch

    from turboquant_pro_b200 import context

    n = 2**vb
    inner = 0.004 * (np.arange(n - 3) - (n - 4) / 2)
    bounds = np.concatenate([[-outer], inner, [outer]]).astype(np.float32)
    cents = np.concatenate([[-0.4], (bounds[1:] + bounds[:-1]) / 2, [0.4]]).astype(np.float32)
    monkeypatch.setattr(context, "value_codebook", lambda head_dim, bits: (cents, bounds))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(6)
    v = torch.randn((1, 1500, 2, 128), generator=gen, device="cuda").half()
    a, b = _values(v, (1500,), 2, vb, 512, "float16")
    assert a == b
