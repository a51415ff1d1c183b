"""The count pass's tile paths and the fused emission at their edges, against the oracle (GPU).

  * cells of 31 / 32 / 33 points (warp-per-task kernel up to 32 queries, the CTA
    kernel above), 127 / 128 / 129 (a run of the in-cell order), 511 / 512 / 513
    and 1025 (query tiles), 4097 (several runs and tiles), in every padded width;
  * points at the radius (both precisions must agree with the FP64 predicate
    where boxes are ruled out next to hits);
  * a mean occupancy just below and above 16 (the in-cell order's threshold);
  * device delivery: the keys that the emission writes.

Whole pair sets are compared (count and set hash, or the sorted list), so there
is no tolerance.
"""
import numpy as np
import pytest

import oracle
import sjoin
from conftest import shell_points

pytestmark = pytest.mark.gpu


def _check(pts, eps, k, mode, prec, **kw):
    ok, ov = oracle.OracleIndex(pts, eps, k).pairs()
    with sjoin.SelfJoin(pts.shape[1], eps, indexed_dims=k, mode=mode, precision=prec, **kw) as sj:
        sj.set_points(pts)
        sj.build_index()
        st = sj.join(sjoin.DELIVER_NONE)
        deg = sj.degrees()
    assert st.total_pairs == len(ok)
    assert st.pair_hash == oracle.hash_pairs(ok, ov)
    assert np.array_equal(deg, np.bincount(ok, minlength=len(pts)))


@pytest.mark.parametrize("prec", [sjoin.PREC_FP64, sjoin.PREC_FP32_REFINE])
@pytest.mark.parametrize("n", [31, 32, 33, 127, 128, 129, 511, 512, 513, 1025, 4097])
def test_cell_sizes(n, prec):
    # one full cell and a sparse one beside it, so that a task has a remainder
    r = np.random.default_rng(n)
    a = r.random((n, 3)) * 0.0999
    b = r.random((19, 3)) * 0.0999 + np.array([0.1, 0.0, 0.0])
    pts = np.vstack([a, b])
    for mode in (3, 6, 10):
        _check(pts, 0.1, 3, mode, prec)


@pytest.mark.parametrize("prec", [sjoin.PREC_FP64, sjoin.PREC_FP32_REFINE])
@pytest.mark.parametrize("dim,k", [(1, 1), (2, 2), (3, 2), (4, 4), (6, 5), (8, 4), (11, 3), (16, 6)])
def test_widths(dim, k, prec):
    r = np.random.default_rng(dim)
    pts = np.clip(r.exponential(0.06, (2500, dim)), 0.0, 1.0)
    eps = 0.05 * np.sqrt(dim)
    for mode in (4, 9, 10):
        _check(pts, eps, k, mode, prec)


@pytest.mark.parametrize("dim", [2, 4, 6])
def test_points_at_the_radius(dim):
    eps = 0.3
    pts = shell_points(1500, dim, eps, dim) * np.where(np.arange(dim) < 2, 1.0, 0.5)
    for prec in (sjoin.PREC_FP64, sjoin.PREC_FP32_REFINE):
        _check(shell_points(1500, dim, eps, dim), eps, dim, 10, prec)
        _check(pts, eps, dim, 6, prec)


@pytest.mark.parametrize("per_cell", [15, 16, 17])
def test_occupancy_threshold(per_cell):
    # a 12 x 12 grid of cells with the same number of points in each
    r = np.random.default_rng(per_cell)
    c = np.stack(np.meshgrid(np.arange(12), np.arange(12), indexing="ij"), -1).reshape(-1, 1, 2)
    pts = ((c + 0.02 + 0.96 * r.random((144, per_cell, 2))) * 0.08).reshape(-1, 2)
    for mode in (3, 5, 10):
        _check(pts, 0.08, 2, mode, sjoin.PREC_FP64, capacity=65536)


def test_device_delivery_keys_and_values():
    torch = pytest.importorskip("torch")
    r = np.random.default_rng(5)
    pts = np.clip(r.exponential(0.025, (6000, 4)), 0.0, 1.0)
    ok, ov = oracle.OracleIndex(pts, 0.02, 4).pairs()

    class Dev:
        def __init__(self, ptr, n):
            self.__cuda_array_interface__ = dict(shape=(n,), typestr="<i4", data=(ptr, False), version=3)

    ks, vs = [], []

    def cb(_i, kptr, vptr, cnt):
        if cnt:
            ks.append(torch.as_tensor(Dev(kptr, cnt), device="cuda").cpu().numpy().copy())
            vs.append(torch.as_tensor(Dev(vptr, cnt), device="cuda").cpu().numpy().copy())

    with sjoin.SelfJoin(4, 0.02, mode=10, precision=1, capacity=65536) as sj:
        sj.set_points(pts)
        sj.build_index()
        sj.join(sjoin.DELIVER_DEVICE, cb)
    assert all(np.all(np.diff(k) >= 0) for k in ks)
    ck, cv = sjoin.canonical(np.concatenate(ks), np.concatenate(vs))
    assert np.array_equal(ck, ok) and np.array_equal(cv, ov)


@pytest.mark.parametrize("dim,k", [(5, 5), (6, 6), (7, 7), (9, 9), (11, 10)])
@pytest.mark.parametrize("mode", [3, 4, 6])
def test_neighbour_walk_depths(dim, k, mode):
    # up to six indexed dimensions are walked breadth first, the ones above depth first
    r = np.random.default_rng(dim)
    pts = np.clip(r.exponential(0.05, (900, dim)), 0.0, 1.0)
    eps = 0.08
    ix = oracle.OracleIndex(pts, eps, k)
    ok, ov = ix.pairs()
    with sjoin.SelfJoin(dim, eps, indexed_dims=k, mode=mode) as sj:
        sj.set_points(pts)
        sj.build_index()
        st = sj.join(sjoin.DELIVER_NONE)
    assert st.total_pairs == len(ok) and st.pair_hash == oracle.hash_pairs(ok, ov)
    assert st.full_stencil_calcs == int(ix.cell_candidates().sum())


@pytest.mark.parametrize("mode,prec", [(3, 0), (10, 1)])
def test_csr_of_one_batch(mode, prec):
    # one batch: the emission writes straight into the caller's rows
    torch = pytest.importorskip("torch")
    r = np.random.default_rng(9)
    pts = r.random((5000, 3))
    n, eps = len(pts), 0.07
    ok, ov = oracle.OracleIndex(pts, eps, 3).pairs()
    deg = np.bincount(ok, minlength=n)
    with sjoin.SelfJoin(3, eps, mode=mode, precision=prec) as sj:
        sj.set_points(pts)
        sj.build_index()
        row = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda")
        small = torch.full((len(ok) - 1,), -7, dtype=torch.int32, device="cuda")
        with pytest.raises(sjoin.SJError) as e:
            sj.neighbor_csr(row.data_ptr(), small.data_ptr(), len(ok) - 1)
        assert e.value.status == sjoin.SJ_ERR_BAD_INPUT
        assert bool((small == -7).all())          # refused before anything is written
        want = np.concatenate([[0], np.cumsum(deg)])
        assert np.array_equal(row.cpu().numpy(), want)   # the sizes are there all the same
        cols = torch.full((len(ok) + 3,), -7, dtype=torch.int32, device="cuda")
        assert sj.neighbor_csr(row.data_ptr(), cols.data_ptr(), len(ok) + 3) == len(ok)
        st = sj.stats()
        assert st.num_batches == 1 and st.total_pairs == len(ok)
        _, hits, _ = sj.cell_features(with_hits=True)
        assert int(hits.sum()) == len(ok)
    c = cols.cpu().numpy()
    assert np.all(c[len(ok):] == -7)
    keys = np.repeat(np.arange(n), deg)
    assert np.array_equal(c[:len(ok)][np.lexsort((c[:len(ok)], keys))], ov)
    assert np.array_equal(row.cpu().numpy(), want)


def test_many_small_units():
    # more than a million emission units of a few pairs each: warps take several
    # at a time and step over the dead ones
    pts = np.random.default_rng(5).random((750_000, 2))
    _check(pts, 0.0006, 2, 6, sjoin.PREC_FP32_REFINE)
