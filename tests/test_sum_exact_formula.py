"""The float64 defect pass adds a float and its rounding error in double by
adding units in the last place to the double's bits (fl_common.cuh,
sum_exact); restated here in integers and checked against the addition."""
import numpy as np


def sum_exact(a, b):
    """(sum, taken): the integer form where its conditions hold."""
    ua, ub = a.view(np.uint32).astype(np.int64), b.view(np.uint32).astype(np.int64)
    ea, eb = ua >> 23 & 0xFF, ub >> 23 & 0xFF
    sh = 29 - (ea - eb)
    mb = (ub & 0x7FFFFF) | 0x800000
    down, up = np.clip(-sh, 0, 31), np.clip(sh, 0, 31)
    fast = (ea != 0xFF) & (eb != 0) & (sh <= 5) & (sh > -23) & ((mb & ((1 << down) - 1)) == 0)
    k = np.where(sh >= 0, mb << np.minimum(up, 5), mb >> down)
    minus = ((ua ^ ub) >> 31 & 1) == 1
    k = np.where(minus & ((ua & 0x7FFFFF) == 0), 2 * k, k)
    bits = ((ua >> 31 & 1).astype(np.uint64) << np.uint64(63)) | ((ea + 896) << 52 | (ua & 0x7FFFFF) << 29).astype(np.uint64)
    return (bits + np.where(minus, -k, k).astype(np.uint64)).view(np.float64), fast


def test_sum_exact_equals_the_addition():
    rng = np.random.default_rng(7)
    n = 400000
    x = (rng.uniform(-1, 1, n) * 2.0 ** rng.integers(-40, 40, n)).astype(np.float32)
    y = (rng.uniform(-1, 1, n) * 2.0 ** rng.integers(-40, 40, n)).astype(np.float32)
    x[::5] = np.float32(2.0) ** rng.integers(-20, 20, x[::5].size).astype(np.float32)  # powers of two, and just off
    y[::7] = (1 + np.float32(2.0 ** -23) * rng.integers(0, 3, y[::7].size)).astype(np.float32)
    p = x.astype(np.float64) * y.astype(np.float64)  # exact: 48 bits
    a = p.astype(np.float32)
    b = (p - a.astype(np.float64)).astype(np.float32)  # exact: the rounding error
    got, fast = sum_exact(a, b)
    want = a.astype(np.float64) + b.astype(np.float64)
    assert np.array_equal(got[fast], want[fast])
    assert fast.mean() > 0.7  # the others take the addition itself
    # and what is not a rounding error: the form is taken only where it is exact
    c = (rng.uniform(-1, 1, n) * 2.0 ** rng.integers(-60, 60, n)).astype(np.float32)
    got, fast = sum_exact(a, c)
    assert np.array_equal(got[fast], (a.astype(np.float64) + c.astype(np.float64))[fast])
