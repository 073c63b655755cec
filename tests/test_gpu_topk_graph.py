"""The query graph of plain top-k belongs to one index: after that index is destroyed, another one built
in its place (often at the same address) answers from its own arrays."""
import numpy as np
import pytest

import gat_b200 as G
from gat_b200 import data as D

pytestmark = pytest.mark.gpu


def test_plain_after_index_replaced(gpu_ctx):
    q = D.walks(D.lengths(5, 0, 0, 0, 10, 60, 3), 4)
    for n in (2000, 300, 2500, 200):
        t = D.walks(D.lengths(n, 0, 0, 0, 1, 60, n), n)
        db = G.TrajectorySet(gpu_ctx, t)
        g = G.Grid(gpu_ctx, db, D.BOX, 0.01, 2, 512)
        ids, dist, _ = g.topk(q, 16, 5e-4)
        ids1, dist1, _ = g.topk(q, 16, 5e-4, "plain")
        assert np.array_equal(ids, ids1) and np.array_equal(dist, dist1)
        g.close()
        db.close()
