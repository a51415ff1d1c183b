"""The scan of a batch's key counts where its 16-byte accesses end, against the oracle (GPU).

Point counts around the smallest of the two-kernel form (16,384 elements go to
one block), with every remainder of a thread's eight elements that matters and
whole tiles of 2,048.  Whole pair sets and row lengths are compared, so there is
no tolerance.
"""
import numpy as np
import pytest

import oracle
import sjoin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16383, 16384, 16385, 16388, 16391, 16392, 16393, 18431, 18432, 18433, 20481])
def test_counts_at_tile_edges(n):
    pts = np.random.default_rng(n).random((n, 2))
    eps = 0.012
    ok, ov = oracle.OracleIndex(pts, eps, 2).pairs()
    with sjoin.SelfJoin(2, eps, mode=5) as sj:
        sj.set_points(pts)
        sj.build_index()
        for _ in range(2):   # the second join finds the counts that the first one's scan cleared
            st = sj.join(sjoin.DELIVER_NONE)
            assert (st.total_pairs, st.pair_hash) == (len(ok), oracle.hash_pairs(ok, ov))
        deg = sj.degrees()
    assert np.array_equal(deg, np.bincount(ok, minlength=n))
