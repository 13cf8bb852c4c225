"""The key encoder for 256-token blocks, bit for bit against the CPU oracle at the places where it
can go wrong: every outlier count it takes (and one it leaves to the general encoder), tokens split
between the hot ring and the caller's tensor, equal magnitudes, channels whose levels round together
(constants, a large zero-point over a small range), every grid and element type."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, W, S = 2, 512, 256


def _tokens(rng, n, dt):
    """(n, H, 128) float32 holding values of `dt`, with the awkward channels named above."""
    import torch

    x = rng.standard_normal((n, H, 128)).astype(np.float32) * np.exp(rng.normal(0, 1, (1, H, 128)))
    x[:, :, 3] *= 20.0
    x[:, 0, 8] = 0.0                                              # all zero
    x[:, 0, 9] = 1.25                                             # constant
    x[:, 0, 10] = 300.0 + 0.25 * rng.integers(0, 2, n)            # two values far from zero
    x[:, 0, 11] = rng.integers(-3, 4, n)                          # many equal magnitudes
    x[:, 0, 12] = 1.0e-6 * rng.standard_normal(n)
    x[:, 1, 13] = np.linspace(-1.0, 1.0, n)                       # all large ones side by side
    x[:, 1, 14] = 40.0 + rng.standard_normal(n)
    x[::7, 1, 15] = -0.0
    x[5:9, 1, :] = 9.0                                            # more outliers than fixed slots
    return torch.from_numpy(x.astype(np.float32)).to(getattr(torch, dt))


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("mode", ["nf4_asym", "nf4", "uniform"])
@pytest.mark.parametrize("frac,k", [(0.0, 0), (0.003, 1), (0.02, 5), (0.032, 8), (0.036, 9)])
def test_key_blocks_equal_the_oracle(dt, mode, frac, k):
    import torch

    from oracle import tq_oracle as orc
    from turboquant_pro_b200 import KVContext

    assert orc.outlier_count(S, frac) == k or frac == 0.0
    n = 1100
    t = _tokens(np.random.default_rng(11), n, dt)
    ctx = KVContext(n_layers=1, n_seqs=1, n_kv_heads=H, n_q_heads=H, value_bits=3, hot_window=W,
                    max_tokens_per_seq=n, kv_dtype=dt, outlier_frac=frac, key_mode=mode, seed=5)
    kt = t[None].cuda()
    for a, b in ((0, 37), (37, 650), (650, n)):  # blocks from the ring, the tensor and both
        ctx.append(0, kt[:, a:b], kt[:, a:b])
    assert ctx.status() == 0
    x = t.float().numpy()
    for blk in range(ctx.lengths(0, 0)[1] // S):
        want = orc.encode_keys(x[blk * S:(blk + 1) * S].transpose(1, 0, 2), frac, mode)
        got = ctx.export_block(0, 0, blk)
        assert np.array_equal(got["nf4_scale"][0].view(np.uint32), want["scale"].view(np.uint32))
        assert np.array_equal(got["nf4_mean"][0], want["mean"])
        assert np.array_equal(got["key_indices"], orc.pack_key_codes(want["codes"]))
        if k:
            assert np.array_equal(got["outlier_idx"], want["out_idx"])
            assert np.array_equal(got["outlier_val"].view(np.uint16), want["out_val"].view(np.uint16))


def _blocks(t, mode, frac, dt):
    """The exported cold blocks of tokens appended in one go."""
    from turboquant_pro_b200 import KVContext

    ctx = KVContext(n_layers=1, n_seqs=1, n_kv_heads=H, n_q_heads=H, value_bits=3, hot_window=W,
                    max_tokens_per_seq=8 * t.shape[0], kv_dtype=dt, outlier_frac=frac,
                    key_mode=mode, seed=5)  # (room for many equal magnitudes)
    kt = t[None].cuda()
    ctx.append(0, kt, kt)
    assert ctx.status() == 0
    return [ctx.export_block(0, 0, b) for b in range(ctx.lengths(0, 0)[1] // S)]


def _outliers(x, k):
    """(flat indices, fp16 bits) of a block ``(S, H, 128)``: every token whose magnitude reaches the
    channel's k-th largest; a NaN is below every magnitude and never one."""
    mag = np.where(np.isnan(x), -1.0, np.abs(x)).transpose(1, 0, 2)
    kth = np.sort(mag, axis=1)[:, -k, :]
    flat = np.flatnonzero((mag >= kth[:, None, :]) & (mag >= 0.0))
    with np.errstate(over="ignore"):
        return flat, x.transpose(1, 0, 2).reshape(-1)[flat].astype(np.float16).view(np.uint16)


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("mode", ["nf4_asym", "nf4", "uniform"])
@pytest.mark.parametrize("frac,k", [(0.003, 1), (0.02, 5), (0.032, 8)])
def test_nan_keys_are_never_outliers(dt, mode, frac, k):
    import torch

    n = W + 2 * S
    x = np.random.default_rng(2).standard_normal((n, H, 128)).astype(np.float32)
    x[7, 0, 5] = np.nan                       # beside ordinary tokens
    x[7, 1, :] = np.nan                       # a whole row
    x[::3, 0, 6] = np.nan
    x[:, 0, 7] = 0.0                          # the k-th magnitude is zero
    x[2::5, 0, 7] = np.nan
    x[:, 1, 8] = np.nan                       # fewer than k numbers
    x[[3, 90, 300], 1, 8] = [1.0, -2.0, 0.5]
    t = torch.from_numpy(x).to(getattr(torch, dt))
    x = t.float().numpy()
    for blk, got in enumerate(_blocks(t, mode, frac, dt)[:2]):
        idx, val = _outliers(x[blk * S:(blk + 1) * S], k)
        assert np.array_equal(got["outlier_idx"], idx)
        assert np.array_equal(got["outlier_val"].view(np.uint16), val)


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("mode", ["nf4_asym", "nf4", "uniform"])
def test_keys_at_and_beyond_the_top_of_the_range(dt, mode):
    """Against the general encoder, which takes the same tokens with nine outliers a channel (the
    codes, scales and zero-points do not depend on their number)."""
    import torch

    n = W + 2 * S
    rng = np.random.default_rng(3)
    x = rng.standard_normal((n, H, 128))
    sign = rng.choice([-1.0, 1.0], n)
    x[9, 0, 4] = np.inf
    x[9, 0, 7] = -np.inf
    x[[9, 30], 0, 10] = [np.inf, -np.inf]
    x[:, 0, 12] = np.inf * sign
    x[5, 0, 14] = np.inf
    x[8, 0, 14] = np.nan
    x[8, 0, 16] = np.nan
    x[40, 0, 20] = 3.3e38                        # above the largest border of the table
    x[40, 0, 23] = -3.3e38
    x[:, 0, 26] = 3.35e38 * sign
    x[:, 0, 28] = 2.5e38 * rng.uniform(-1, 1, n)
    x[:, 0, 31] = 1.0e38 + 1.0e36 * rng.standard_normal(n)
    x[:, 0, 33] = 3.0e38
    x[:, 0, 34] = -1.0e38 * rng.uniform(0, 3.3, n)
    x[:, 0, 36] = 2.0 ** 126 * rng.uniform(0.99, 1.01, n) * sign
    x[:, 0, 38] = 2.0 ** 125 * rng.uniform(-1, 1, n)
    x[:, 0, 40] = 6.5e4 * rng.uniform(-1, 1, n)  # (the top of fp16)
    x[:, 0, 41] = 1.0e-40 * rng.standard_normal(n)
    with np.errstate(over="ignore"):
        t = torch.from_numpy(x.astype(np.float32)).to(getattr(torch, dt))
    x = t.float().numpy()
    for blk, (got, want) in enumerate(zip(_blocks(t, mode, 0.02, dt)[:2],
                                          _blocks(t, mode, 0.036, dt)[:2], strict=True)):
        codes = [b["key_indices"].reshape(H, S, 64) for b in (got, want)]
        assert not np.argwhere((codes[0] != codes[1]).any(axis=1)).tolist()
        assert np.array_equal(got["nf4_scale"], want["nf4_scale"])
        assert np.array_equal(got["nf4_mean"], want["nf4_mean"], equal_nan=True)
        idx, val = _outliers(x[blk * S:(blk + 1) * S], 5)
        assert np.array_equal(got["outlier_idx"], idx)
        assert np.array_equal(got["outlier_val"].view(np.uint16), val)


@pytest.mark.parametrize("dt", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("mode", ["nf4_asym", "nf4", "uniform"])
def test_channels_of_nan_have_the_general_encoder_s_extremes(dt, mode):
    import torch

    n = W + 2 * S
    x = np.random.default_rng(4).standard_normal((n, H, 128)).astype(np.float32)
    x[:, 0, 2] = np.nan
    x[:, 1, 5] = np.nan
    x[70, 1, 5] = -3.0                           # a single number
    x[:64, 0, 9] = np.nan                        # the tokens of some threads
    x[0, 0, 11] = np.nan                         # a first token
    t = torch.from_numpy(x).to(getattr(torch, dt))
    for got, want in zip(_blocks(t, mode, 0.02, dt)[:2], _blocks(t, mode, 0.036, dt)[:2], strict=True):
        assert np.array_equal(got["key_indices"], want["key_indices"])
        assert np.array_equal(got["nf4_scale"], want["nf4_scale"])
        assert np.array_equal(got["nf4_mean"], want["nf4_mean"], equal_nan=True)


@pytest.mark.parametrize("dt", ["float16", "float32"])
def test_a_block_that_does_not_arrive_is_stored_empty(dt):
    """The test hook withholds one row of the first block; the wait for it runs out, the status word
    says so, and the cache holds zeros in that block's place."""
    import torch

    from turboquant_pro_b200 import KVContext

    n = W + 2 * S
    x = np.random.default_rng(6).standard_normal((n, H, 128)).astype(np.float32)
    kt = torch.from_numpy(x).to(getattr(torch, dt))[None].cuda()
    good, ctx = (KVContext(n_layers=1, n_seqs=1, n_kv_heads=H, n_q_heads=H, value_bits=3,
                           hot_window=W, max_tokens_per_seq=n, kv_dtype=dt, seed=5)
                 for _ in range(2))
    good.append(0, kt, kt)
    want_k, want_v = good.dequant(0, 0, 0, n)
    ctx._regions["pages"].fill_(0x5A)  # what an earlier user of the pages left there
    ctx.debug_wait(wait_limit=256, withhold_tile=17)
    ctx.append(0, kt, kt)
    assert ctx.status() == 2 and ctx.status() == 0
    ctx.debug_wait()
    k, v = ctx.dequant(0, 0, 0, n)
    assert not k[0, :S].any()
    assert torch.equal(k[0, S:], want_k[0, S:]) and torch.equal(k[1], want_k[1])
    assert torch.equal(v, want_v)
    blk = ctx.export_block(0, 0, 0)
    assert (blk["outlier_idx"] >= S * 128).all() and not blk["nf4_scale"][0, 0].any()
    q = torch.randn((1, H, 128), device="cuda")
    s = torch.einsum("hd,htd->ht", q[0].double(), k.double()) / 128 ** 0.5
    want = torch.einsum("ht,htd->hd", s.softmax(-1), v.double())
    for kernel in ("auto", "general"):
        ctx.set_kernel(kernel)
        # (the scores' outlier corrections are stored in fp16: about 3e-4 of a score of one)
        assert ((ctx.decode(0, q)[0] - want).norm() / want.norm()).item() < 5e-3
    ctx.clear(0, 0)
    ctx.append(0, kt, kt)
    assert ctx.status() == 0 and torch.equal(ctx.dequant(0, 0, 0, n)[0], want_k)
