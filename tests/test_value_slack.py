"""How far the value encoder's products may be from the reference's sums, and its slack: products nearer to a
boundary than the slack are computed again, so the slack has to cover the distance with room."""

import numpy as np
import pytest

D, STEP = 128, 16
# |exact - reference's sequential float32 sum|: 127 roundings of a running sum below 1, 128 of quotients and products
REFERENCE = 127 * 2.0**-25 + 2.0**-23
# eight steps of 16 terms and the sum before, each cut off 24 bits below the largest of the 17
CUT = 8 * 17 * 2.0**-24
# what the parts of the rotation leave out (of float32 rows likewise): two of fp16, three of bfloat16
PARTS = {0: 2 * 2.0**-23, 1: 2.0**-23, 2: 2.0**-26}


def _lib():
    import __graft_entry__ as ge

    ge._load_build_module().build()
    from turboquant_pro_b200 import _lib

    return _lib.load()


def _round(x, bits):
    m, e = np.frexp(x)
    return np.ldexp(np.round(m * 2.0**bits), e - bits)


def _split(x, bits):
    parts = []
    for _ in range(3 if bits == 8 else 2):
        parts.append(_round(x - sum(parts), bits))
    return parts


def _cut_sum(acc, terms):
    """Sum of ``acc`` and the last axis, every addend cut off at 2^-23 of the largest one's power of two."""
    all_ = np.concatenate([acc[..., None], terms], -1)
    unit = np.exp2(np.floor(np.log2(np.maximum(np.abs(all_).max(-1, keepdims=True), 1e-300))) - 23)
    return (np.trunc(all_ / unit) * unit).sum(-1)


@pytest.mark.parametrize("dt", [0, 1, 2])
def test_slack_is_two_and_a_half_times_the_bound(dt):
    bound = REFERENCE + CUT + PARTS[dt]
    assert _lib().tq_debug_value_slack() >= 2.45 * bound


@pytest.mark.parametrize("dt", [0, 1, 2])
def test_bound_holds_for_sums_that_are_cut_off(dt):
    """The products as the encoder forms them, by tensor cores that cut off: rows whose partial sums come
    near 1 and cancel, rows along one row of the rotation, ordinary rows."""
    from oracle import tq_oracle as orc

    rng = np.random.default_rng(3)
    pi = np.asarray(orc.rotation(D, 3)[0], np.float64)
    bits = 8 if dt == 2 else 11
    c = rng.integers(0, D, 600)
    sign = np.where(np.arange(D) < rng.choice([16, 32, 64, 96], (600, 1)), 1.0, -rng.uniform(0, 2, (600, 1)))
    sign[:100], sign[100:300] = 1.0, sign[100:300] + 0.02 * rng.standard_normal((200, D))
    x = np.concatenate([pi[c] * sign, rng.standard_normal((200, D))])
    if dt != 0:
        x = _round(x, bits)  # (float32 rows are split, others are operands as they are)
    x = x.astype(np.float32).astype(np.float64)
    u = x / np.linalg.norm(x, axis=1, keepdims=True)
    exact = u @ pi.T
    p_hi, *p_low = _split(pi.astype(np.float32).astype(np.float64), bits)
    x_hi, x_lo = _split(u, bits) if dt == 0 else (u, None)
    acc = np.zeros_like(exact)
    small = [(x_hi, p_low[0])] + ([(x_lo, p_hi)] if dt == 0 else [])
    for parts in ([(x_hi, p) for p in p_low[1:]], small, [(x_hi, p_hi)]):
        for k in range(0, D, STEP):
            for xs, ps in parts:
                acc = _cut_sum(acc, xs[:, None, k:k + STEP] * ps[None, :, k:k + STEP])
    assert np.abs(acc - exact).max() <= CUT + PARTS[dt]
