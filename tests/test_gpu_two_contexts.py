"""Contexts used from several threads at once."""
import threading

import numpy as np
import pytest

import gat_b200 as G
from gat_b200 import data as D

pytestmark = pytest.mark.gpu


def test_topk_over_sets_of_unlike_lengths():
    """The top-k order needs shared memory by the longest walk of its set: contexts over sets of 200 to 4,096 points
    at most, each in a thread of its own, launch the same kernels with different amounts."""
    work, errors = [], []
    for longest, seed in ((200, 51), (1024, 52), (2048, 53), (4096, 54)):
        ctx = G.Context(0)
        lens = np.full(40, 30, np.int32)
        lens[0] = longest
        t = D.walks(lens, seed)
        grid = G.Grid(ctx, G.TrajectorySet(ctx, t), D.BOX, 0.01, 2, 512)
        q = t.subset([3, 5, 7, 11, 13])
        work.append((grid, q, grid.topk(q, 4, 5e-4, "batched")[:2]))

    def run(grid, q, want):
        try:
            for _ in range(4000):
                got = grid.topk(q, 4, 5e-4, "batched")
                assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        except Exception as e:  # a launch that failed, or other results
            errors.append(e)

    threads = [threading.Thread(target=run, args=w) for w in work]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
