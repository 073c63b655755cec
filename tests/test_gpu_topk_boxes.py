"""Top-k candidates whose box is just within or just beyond the match tolerance of the query's (the
distance is then taken by formula), and sets larger than one sort tile: every distance of the full
ranking equals the oracle's."""
import numpy as np
import pytest

import gat_b200 as G
from gat_b200 import data as D
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _set(parts):
    return G.Trajectories(np.array([len(p) for p in parts], np.int32), np.concatenate([p[:, 0] for p in parts]).astype(np.float32),
                          np.concatenate([p[:, 1] for p in parts]).astype(np.float32))


@pytest.mark.parametrize("execution", ["batched", "plain"])
def test_boxes_at_the_tolerance(gpu_ctx, execution):
    eps = 5e-4
    rng = np.random.default_rng(1)
    base = np.array([121.5, 31.2]) + np.cumsum(rng.normal(0, 1e-4, (150, 2)), 0)
    w = base.max(0) - base.min(0)
    parts = [base]
    for axis in (0, 1):
        for side in (-1, 1):
            for f in np.concatenate([np.linspace(0.9, 1.1, 21), [0.9999, 1.0, 1.0001, 0.0, 3.0]]):
                d = np.zeros(2)
                d[axis] = side * (w[axis] + f * eps)  # edge to edge: f * eps apart
                n = int(rng.integers(1, 150))
                parts.append(np.concatenate([base[:n] + d, base[-1:] + d]))
    t = _set(parts)
    g = G.Grid(gpu_ctx, G.TrajectorySet(gpu_ctx, t), D.BOX, 0.0025, 2, 512)
    q = t.subset([1, 2, 40, 80, 100])
    ids, dist, _ = g.topk(q, t.n, eps, execution)
    for i in range(q.n):
        a = np.stack(q.points(i + 1), 1)
        want = np.array([po.edr(a, np.stack(t.points(j), 1), eps) for j in range(1, t.n + 1)])
        order = np.lexsort((np.arange(1, t.n + 1), want))
        assert np.array_equal(ids[i], order + 1) and np.array_equal(dist[i], want[order])


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 9001])
def test_sort_tiles(gpu_ctx, n):
    t = D.walks(D.lengths(n, 0, 0, 0, 1, 30, n), n)
    g = G.Grid(gpu_ctx, G.TrajectorySet(gpu_ctx, t), D.BOX, 0.01, 2, 512)
    q = D.walks(D.lengths(6, 0, 0, 0, 1, 40, 3), 4)
    k = min(n, 20)
    ids, dist, _ = g.topk(q, k, 5e-3)
    ids1, dist1, _ = g.topk(q, k, 5e-3, "plain")
    for i in range(q.n):
        a = np.stack(q.points(i + 1), 1)
        la = np.full(n, len(a), np.int32)
        want = po.edr_batch(la, np.tile(a, (n, 1)), t.lengths, np.stack([t.lon, t.lat], 1), 5e-3)
        order = np.lexsort((np.arange(1, n + 1), want))[:k]
        for got_i, got_d in ((ids[i], dist[i]), (ids1[i], dist1[i])):
            assert np.array_equal(got_i, order + 1) and np.array_equal(got_d, want[order])
