"""The cost order: heaviest cells first, however little they differ (GPU).

Eight cells of 400 points that are all within the radius of each other, one batch
each, and beside every one a cell of 1 to 8 points out of reach: the evaluations,
and so the predicted costs, differ by 0.05 % from one cell to the next, rising
with the cell id.
"""
import numpy as np
import pytest

import sjoin

pytestmark = pytest.mark.gpu


def test_batches_come_heaviest_first():
    eps, cells, per = 0.01, 8, 400
    r = np.random.default_rng(6)
    pts, owner = [np.array([[0.0, 0.0]])], [-1]   # the grid starts at this point less eps
    for i in range(cells):
        x0 = 0.05 + 3 * i * eps   # the cell's low corner (grid lines are multiples of eps)
        pts.append(np.column_stack([x0 + eps * (0.1 + 0.2 * r.random(per)), eps * (0.1 + 0.2 * r.random(per))]))
        owner += [i] * per
        pts.append(np.column_stack([x0 + eps * (1.8 + 0.1 * r.random(i + 1)), eps * (0.1 + 0.2 * r.random(i + 1))]))
        owner += [-1] * (i + 1)
    pts, owner = np.vstack(pts), np.array(owner)
    order = []

    def take(_batch, key, _val):
        order.extend(c for c in dict.fromkeys(owner[key].tolist()) if c >= 0 and c not in order)

    with sjoin.SelfJoin(2, eps, mode=9, capacity=200_000) as sj:
        sj.set_points(pts)
        sj.build_index()
        st = sj.join(sjoin.DELIVER_HOST, take)
    assert st.num_batches >= cells and st.overflow_retries == 0
    assert order == list(range(cells))[::-1]
