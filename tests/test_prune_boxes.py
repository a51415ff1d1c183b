"""The engine's own bounds (csrc/sj_host.h, compiled alone) and the box test with them, on CPU.

  * margin, band and pruneT agree with the restatement of test_filter_bounds.py;
  * boxes of 32 points each, at distances from touching to twice the radius: no
    pair of a ruled-out tile satisfies the FP64 predicate, and where the margin is
    small every pair of boxes 1.02 radii or more apart is ruled out;
  * pairs at the radius, up to one part in 1e6 beyond: none that is a hit is ruled out;
  * outside the range in which FP32 squares hold, nothing is ruled out.
"""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from test_filter_bounds import bounds, threshold
from test_prune_bound import _fma32

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "self-join-hpbdc2019_b200", "csrc")
F32_INF = np.float32(np.inf)


class Bounds(C.Structure):
    _fields_ = [("margin", C.c_double), ("delta", C.c_float), ("pruneT", C.c_float)]


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    d = tmp_path_factory.mktemp("bounds")
    (d / "b.cpp").write_text('#include "sj_host.h"\n'
                             'extern "C" sj_filter_bounds bounds_of(int D, int k, double eps, double T, const double *lo,\n'
                             '                                      const double *hi)\n'
                             '{ return sj_filter_bounds_of(D, k, eps, T, lo, hi); }\n')
    lib = str(d / "b.so")
    subprocess.check_call(["g++", "-std=c++17", "-O3", "-shared", "-fPIC", "-I", CSRC, str(d / "b.cpp"), "-o", lib])
    f = C.CDLL(lib).bounds_of
    f.restype = Bounds

    def call(D, k, eps, lo, hi):
        ptr = [np.ascontiguousarray(v, np.float64) for v in (lo, hi)]
        return f(D, k, C.c_double(eps), C.c_double(threshold(eps)), *[v.ctypes.data_as(C.c_void_p) for v in ptr])

    return call


CONFIGS = [(2, 2, 0.0015, 0.0, 1.0), (3, 3, 0.02, 2.5e4, 1.0), (4, 3, 0.01, 0.0, 0.3), (6, 6, 0.03, 0.0, 1.0),
           (8, 4, 0.05, 0.0, 1.0), (16, 6, 0.05, 10.0, 2.0), (5, 2, 0.15, 0.0, 40.0)]


def _range(D, k, far, long_dim):
    lo = np.full(D, far)
    return lo, lo + np.where(np.arange(D) < k, 1.0, long_dim)


@pytest.mark.parametrize("D,k,eps,far,long_dim", CONFIGS)
def test_bounds_as_restated(engine, D, k, eps, far, long_dim):
    lo, hi = _range(D, k, far, long_dim)
    b = engine(D, k, eps, lo, hi)
    _, margin, delta = bounds(D, k, eps, lo, hi)
    prune = np.nextafter(np.float32((threshold(eps) + 2.0 * margin) * (1.0 + math.ldexp(1.0, -20))), F32_INF)
    # the compiler may contract the sums of squares: a few units of the last 64-bit place
    assert abs(b.margin - margin) <= 1e-14 * margin
    assert abs(float(b.delta) - delta) <= 2.0 ** -22 * delta
    assert abs(float(b.pruneT) - float(prune)) <= 2.0 ** -22 * float(prune)


def _box_d2(a, b):
    """Squared distance of the boxes of FP32 points a, b: (tiles, points, D), as the kernel forms it."""
    d2 = np.zeros(len(a), np.float32)
    for l in range(a.shape[2]):
        gap = np.maximum(np.float32(0), np.maximum(b[:, :, l].min(1) - a[:, :, l].max(1),
                                                   a[:, :, l].min(1) - b[:, :, l].max(1)))
        d2 = _fma32(gap, gap, d2)
    return d2


@pytest.mark.parametrize("D,k,eps,far,long_dim", CONFIGS)
def test_boxes_of_several_points(engine, D, k, eps, far, long_dim):
    r = np.random.default_rng(D * 10 + k)
    lo, hi = _range(D, k, far, long_dim)
    b = engine(D, k, eps, lo, hi)
    prune, T = np.float32(b.pruneT), threshold(eps)
    tiles, pts = 4000, 32
    origin = np.where(np.arange(D) < k, lo + 0.5 * eps, 0.5 * (lo + hi))   # first cell's centre
    spread = eps * 10.0 ** r.uniform(-4, -0.7, (tiles, 1, 1))
    qc = lo + r.random((tiles, 1, D)) * np.where(np.arange(D) < k, eps, long_dim)
    u = r.standard_normal((tiles, 1, D))
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    cc = qc + u * eps * r.uniform(0.0, 2.0 + 20 * spread / eps)
    q = qc + spread * r.uniform(-0.5, 0.5, (tiles, pts, D))
    c = cc + spread * r.uniform(-0.5, 0.5, (tiles, pts, D))
    q = np.clip(q, lo, np.where(np.arange(D) < k, lo + eps, hi))
    c = np.clip(c, np.where(np.arange(D) < k, lo - eps, lo), np.where(np.arange(D) < k, lo + 2 * eps, hi))
    out = _box_d2((q - origin).astype(np.float32), (c - origin).astype(np.float32)) > prune
    d2 = np.zeros((tiles, pts, pts))
    gap2 = np.zeros(tiles)
    for l in range(D):
        d2 += (q[:, :, None, l] - c[:, None, :, l]) ** 2
        gap2 += np.maximum(0.0, np.maximum(c[:, :, l].min(1) - q[:, :, l].max(1),
                                           q[:, :, l].min(1) - c[:, :, l].max(1))) ** 2
    hit = (d2 <= T * (1.0 + 1e-14)).any((1, 2))
    assert np.any(hit) and not np.any(hit & out)
    apart = gap2 >= 1.02 ** 2 * T
    assert np.sum(apart) > 100
    if b.margin < 1e-3 * T:   # T + 2M, and the FP32 rounding of coordinates and sum below M: at most 1.004 T
        assert np.all(out[apart])


@pytest.mark.parametrize("D,k,eps,far,long_dim", CONFIGS)
def test_pairs_just_at_the_radius(engine, D, k, eps, far, long_dim):
    r = np.random.default_rng(D * 10 + k + 1)
    lo, hi = _range(D, k, far, long_dim)
    prune, T = np.float32(engine(D, k, eps, lo, hi).pruneT), threshold(eps)
    n = 100_000
    origin = np.where(np.arange(D) < k, lo + 0.5 * eps, 0.5 * (lo + hi))
    q = lo + r.random((n, D)) * np.where(np.arange(D) < k, eps, long_dim)
    u = r.standard_normal((n, D))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    c = q + u * eps * (1.0 + r.uniform(-1e-6, 1e-6, (n, 1)))
    hit = ((c - q) ** 2).sum(1) <= T * (1.0 + 1e-14)
    out = _box_d2((q - origin).astype(np.float32)[:, None], (c - origin).astype(np.float32)[:, None]) > prune
    assert np.any(hit) and np.any(~hit) and not np.any(hit & out)


@pytest.mark.parametrize("eps", [1e-16, 1e16])
def test_nothing_is_ruled_out_outside_the_range(engine, eps):
    assert engine(2, 2, eps, np.zeros(2), np.full(2, 100 * eps)).pruneT == F32_INF


def test_nothing_is_ruled_out_where_the_margin_overflows(engine):
    assert engine(2, 1, 1.0, np.zeros(2), np.array([10.0, 1e30])).pruneT == F32_INF
