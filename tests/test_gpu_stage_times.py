"""Stage times that are read later are those of the call that they belong to (GPU).

Through the raw ABI: the Python wrapper reads the statistics after every join.
"""
import ctypes as C

import numpy as np
import pytest

import sjoin

pytestmark = pytest.mark.gpu


def test_degrees_after_a_join_whose_times_were_not_read():
    lib = sjoin.load()
    pts = np.random.default_rng(4).random((20000, 2))
    deg = np.zeros(len(pts), np.uint32)
    with sjoin.SelfJoin(2, 0.01) as sj:
        sj.set_points(pts)
        sj.build_index()
        st = sj.join(sjoin.DELIVER_NONE)
        assert st.ms_estimate > 0 and st.ms_total > 0
        assert lib.sj_join(sj._h, sjoin.DELIVER_NONE, sjoin.BATCH_CB(lambda b, u: 0), None) == 0
        assert lib.sj_degrees(sj._h, deg.ctypes.data_as(C.c_void_p)) == 0
        both = sj.stats()   # the degree count has no estimate; its total is the join's
        again = sj.stats()
    assert both.ms_estimate == 0 and both.ms_total > 0
    assert int(deg.sum()) == both.total_pairs
    assert again.as_dict() == both.as_dict()
