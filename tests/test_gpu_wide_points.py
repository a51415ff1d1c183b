"""Sparse cells of wide points: the count pass that tests the last dimensions first (GPU).

Points of 9 to 16 dimensions in cells of 1 to 7 points (queries one by one below
six, by their box above; an odd one has no partner), with pairs on both sides of
the radius whose distance lies in the first dimensions alone, in the last alone
or in all of them.  Whole pair sets against the oracle: no tolerance.
"""
import numpy as np
import pytest

import oracle
import sjoin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [sjoin.PREC_FP64, sjoin.PREC_FP32_REFINE])
@pytest.mark.parametrize("dim", [8, 9, 12, 13, 16])
@pytest.mark.parametrize("where", ["first", "last", "all"])
def test_pairs_in_a_part_of_the_dimensions(dim, where, prec):
    r = np.random.default_rng(dim)
    k, eps = 3, 0.1
    pts = []
    for size in range(1, 8):   # clusters of a few points around a centre, in one cell or two
        for _ in range(40):
            c = 0.15 + 0.7 * r.random(dim)
            step = r.standard_normal((size, dim))
            if where == "first":
                step[:, 4:] = 0.0
            elif where == "last":
                step[:, :dim - 8 if dim > 8 else 4] = 0.0
            step /= np.linalg.norm(step, axis=1, keepdims=True)
            far = r.choice([0.0, 0.5, 1.0 - 1e-9, 1.0, 1.0 + 1e-9, 1.5], (size, 1))
            pts.append(np.vstack([c, c + eps * far * step]))
    pts = np.vstack(pts)
    ok, ov = oracle.OracleIndex(pts, eps, k).pairs()
    assert len(ok) > len(pts)   # pairs beyond the points themselves
    for mode in (3, 6, 10):
        with sjoin.SelfJoin(dim, eps, indexed_dims=k, mode=mode, precision=prec) as sj:
            sj.set_points(pts)
            sj.build_index()
            st = sj.join(sjoin.DELIVER_NONE)
            deg = sj.degrees()
        assert (st.total_pairs, st.pair_hash) == (len(ok), oracle.hash_pairs(ok, ov))
        assert np.array_equal(deg, np.bincount(ok, minlength=len(pts)))
