"""The device CSR table by the number of its batches, against the oracle (GPU).

  * one batch, emitted straight into the caller's arrays, on cells dense enough
    for the spatial order of their points; the same points as a host list;
  * several batches, whose plan is made once: the launches above those of the
    same join without a table are the appends and a fixed few;
  * too small an array: refused, with the table's size in the statistics;
  * planned as one batch and counted as several (an untrained network predicts
    next to nothing), up to more than 2^32 pairs in that one batch.

Whole rows are compared, so there is no tolerance.
"""
import numpy as np
import pytest

import oracle
import sjoin
from conftest import exp_points

pytestmark = pytest.mark.gpu


def _table(sj, n, total):
    torch = pytest.importorskip("torch")
    row = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda")
    cols = torch.full((total,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()   # the engine writes on its own stream
    assert sj.neighbor_csr(row.data_ptr(), cols.data_ptr(), total) == total
    return row.cpu().numpy(), cols.cpu().numpy()


def _check(row, cols, ok, ov, n):
    deg = np.bincount(ok, minlength=n)
    assert np.array_equal(row, np.concatenate([[0], np.cumsum(deg)]))
    keys = np.repeat(np.arange(n, dtype=np.int32), deg)
    order = np.lexsort((cols, keys))
    assert np.array_equal(cols[order], ov)


@pytest.mark.parametrize("prec", [sjoin.PREC_FP64, sjoin.PREC_FP32_REFINE])
@pytest.mark.parametrize("mode", [3, 5, 6, 10])
def test_one_batch_on_dense_cells(mode, prec):
    # the densest cells hold some hundred points: runs of the in-cell order and several tiles
    pts = exp_points(4000, 2, 31)
    ok, ov = oracle.OracleIndex(pts, 0.01, 2).pairs()
    with sjoin.SelfJoin(2, 0.01, mode=mode, precision=prec) as sj:
        sj.set_points(pts)
        sj.build_index()
        row, cols = _table(sj, len(pts), len(ok))
        st = sj.stats()
        assert st.num_batches == 1 and st.total_pairs == len(ok) and st.pair_hash == oracle.hash_pairs(ok, ov)
        ks, vs = [], []

        def take(_batch, key, val):
            ks.append(key.copy())
            vs.append(val.copy())

        sj.join(sjoin.DELIVER_HOST, take)
    _check(row, cols, ok, ov, len(pts))
    ck, cv = sjoin.canonical(np.concatenate(ks), np.concatenate(vs))
    assert np.array_equal(ck, ok) and np.array_equal(cv, ov)


def _launches(call):
    before = sjoin.kernel_launch_count()
    call()
    return sjoin.kernel_launch_count() - before


@pytest.mark.parametrize("untrained", [False, True])
@pytest.mark.parametrize("mode", [3, 10])
def test_several_batches_are_planned_once(mode, untrained):
    pts = exp_points(6000, 2, 32)
    ok, ov = oracle.OracleIndex(pts, 0.01, 2).pairs()
    assert len(ok) > 3 * 65536
    kw = dict(scheduler=sjoin.SCHED_LEARNED, alpha=0.0) if untrained else {}
    with sjoin.SelfJoin(2, 0.01, mode=mode, capacity=65536, **kw) as sj:
        if untrained:
            sj.set_estimator(sjoin.mlp_init(3))
        sj.set_points(pts)
        sj.build_index()
        sj.join(sjoin.DELIVER_DEVICE)
        joined = _launches(lambda: sj.join(sjoin.DELIVER_DEVICE))
        ref = sj.stats()
        if untrained:   # one batch by the plan, several by the count
            assert ref.estimated_pairs <= 65536 and ref.overflow_retries == 1
        got = {}
        table = _launches(lambda: got.update(t=_table(sj, len(pts), len(ok))))
        st = sj.stats()
    _check(*got["t"], ok, ov, len(pts))
    assert (st.num_batches, st.overflow_retries) == (ref.num_batches, ref.overflow_retries)
    # beside the appends: the sizing count pass (at most two kernels), the rows' scan and check
    assert table - joined - st.num_batches <= 12


def test_more_than_32_bits_of_pairs_in_the_planned_batch():
    torch = pytest.importorskip("torch")
    n = 66_000   # all within the radius of each other: n^2 > 2^32 pairs
    pts = 0.01 * np.random.default_rng(3).random((n, 2))
    with sjoin.SelfJoin(2, 0.05, mode=10, precision=sjoin.PREC_FP32_REFINE, scheduler=sjoin.SCHED_LEARNED,
                        capacity=2_000_000_000) as sj:
        sj.set_estimator(sjoin.mlp_init(3))
        sj.set_points(pts)
        sj.build_index()
        row = torch.full((n + 1,), -1, dtype=torch.int64, device="cuda")
        cols = torch.full((n * n,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert sj.neighbor_csr(row.data_ptr(), cols.data_ptr(), n * n) == n * n
        st = sj.stats()
    assert st.estimated_pairs <= 2_000_000_000 and st.overflow_retries >= 1 and st.num_batches >= 3
    assert torch.equal(row.cpu(), torch.arange(n + 1, dtype=torch.int64) * n)
    every = torch.arange(n, dtype=torch.int32, device="cuda")
    for i in range(0, n, 6000):   # every row holds every point once
        rows, _ = torch.sort(cols.view(n, n)[i:i + 6000], dim=1)
        assert torch.equal(rows, every.expand_as(rows))


@pytest.mark.parametrize("capacity", [0, 65536])
def test_refused_table_reports_its_size(capacity):
    torch = pytest.importorskip("torch")
    pts = exp_points(4000, 2, 33)
    ok, _ = oracle.OracleIndex(pts, 0.01, 2).pairs()
    row = torch.zeros(len(pts) + 1, dtype=torch.int64, device="cuda")
    cols = torch.zeros(len(ok) - 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with sjoin.SelfJoin(2, 0.01, mode=9, precision=sjoin.PREC_FP32_REFINE, capacity=capacity) as sj:
        sj.set_points(pts)
        sj.build_index()
        sj.degrees()
        ref = sj.stats()
        sj.set_points(pts)   # statistics start anew
        sj.build_index()
        with pytest.raises(sjoin.SJError) as e:
            sj.neighbor_csr(row.data_ptr(), cols.data_ptr(), len(ok) - 1)
        st = sj.stats()
    assert e.value.status == sjoin.SJ_ERR_BAD_INPUT
    assert row[-1].item() == len(ok) and not torch.any(cols)
    assert (st.total_pairs, st.distance_calcs) == (len(ok), ref.distance_calcs)
    assert st.refined_pairs <= st.distance_calcs
