"""The warp pass's branchless square root (sqrt_mid in warp_pass.cuh), restated
in NumPy: for any approximate reciprocal root within 2 ulp (CUDA's documented
bound for rsqrtf), the Newton step and Tuckerman's test give the rounded root."""
import numpy as np

F = np.float32


def _fma(a, b, c):
    # exact here: the products have 48 bits, the sums cancel to far fewer than 53
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def _sqrt_mid(x, y):
    s = (x * y).astype(F)
    s = _fma(_fma(-s, s, x), (F(0.5) * y).astype(F), s)
    r = _fma(-s, s, x)
    up, dn = np.nextafter(s, F(np.inf)), np.nextafter(s, F(0))
    return np.where(r > s * (up - s), up, np.where(r <= -(s * (s - dn)), dn, s)).astype(F)


def test_root_is_the_rounded_one_for_any_reciprocal_root_within_2_ulp():
    rng = np.random.default_rng(5)
    x = np.concatenate([
        np.exp(rng.uniform(np.log(1e-18), np.log(1e18), 400000)),
        (rng.integers(1, 1 << 12, 100000).astype(np.float64)) ** 2,                 # exact roots
        1.0 + np.arange(-2000, 2000) * 2.0 ** -24, 4.0 + np.arange(-2000, 2000) * 2.0 ** -23,  # around powers
    ]).astype(F)
    y0 = (1.0 / np.sqrt(x.astype(np.float64))).astype(F)
    exact = np.sqrt(x)  # IEEE: the rounded root
    for ulps in (-2, -1, 0, 1, 2):
        y = (y0.view(np.int32) + np.int32(ulps)).view(F)
        assert np.array_equal(_sqrt_mid(x, y), exact), ulps
