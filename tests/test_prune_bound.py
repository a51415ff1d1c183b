"""The box test's error bound, checked on CPU.

The count pass rules a (32 queries x 32 candidates) tile out when the squared
distance of the two boxes of FP32 local coordinates, accumulated in FP32 with
one rounding per subtraction and per fused multiply-add, exceeds
pruneT = RU32((T + 2M)(1 + 2^-20)) (filter_bounds in sj_api.cpp; M is the
filter's margin).  No pair of a ruled-out tile may satisfy the FP64 predicate.
Boxes of single points are the tightest case; pairs within 1e-5 relative of the
radius, in every rounding situation that random offsets give, far from the
origin and with long non-indexed dimensions among them.
"""
import math

import numpy as np
import pytest

from test_filter_bounds import bounds, threshold


def _fma32(a, b, c):
    # a * b is exact in 64 bits for 32-bit factors; the sum is rounded twice
    # (64 then 32 bits), at most one unit of the last 32-bit place off
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


@pytest.mark.parametrize("D,k,eps,far,long_dim", [
    (2, 2, 0.0015, 0.0, 1.0), (3, 3, 0.02, 2.5e4, 1.0), (4, 3, 0.01, 0.0, 0.3), (6, 6, 0.03, 0.0, 1.0),
    (8, 4, 0.05, 0.0, 1.0), (16, 6, 0.05, 10.0, 2.0), (5, 2, 0.15, 0.0, 40.0)])
def test_no_hit_in_a_ruled_out_pair(D, k, eps, far, long_dim):
    r = np.random.default_rng(D * 100 + k)
    n = 200_000
    lo = np.full(D, far)
    hi = lo + np.where(np.arange(D) < k, 1.0, long_dim)
    origin = np.where(np.arange(D) < k, lo + 0.5 * eps, 0.5 * (lo + hi))   # first cell's centre
    q = lo + r.random((n, D)) * np.where(np.arange(D) < k, eps, long_dim)
    u = r.standard_normal((n, D))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    c = q + u * eps * (1.0 + r.uniform(-1e-5, 1e-5, (n, 1)))
    c = np.clip(c, np.where(np.arange(D) < k, lo - eps, lo), np.where(np.arange(D) < k, lo + 2 * eps, hi))
    T = threshold(eps)
    margin = float(bounds(D, k, eps, lo, hi)[0])
    prune = np.nextafter(np.float32((T + 2.0 * margin) * (1.0 + math.ldexp(1.0, -20))), np.float32(np.inf))
    a, b = (q - origin).astype(np.float32), (c - origin).astype(np.float32)
    d2 = np.zeros(n, np.float32)
    for l in range(D):
        gap = np.maximum(np.float32(0), np.maximum(b[:, l] - a[:, l], a[:, l] - b[:, l]))
        d2 = _fma32(gap, gap, d2)
    # the predicate's value up to a few units of the last 64-bit place
    exact = ((c - q) ** 2).sum(1)
    hit = exact <= T * (1.0 + 1e-14)
    assert not np.any(hit & (d2 > prune))
    assert np.any(hit) and np.any(~hit)
    # and the test is worth its name: pairs clearly outside are ruled out where the margin is small
    if margin < 1e-3 * T:
        assert np.any(d2 * 1.01 > prune)
