"""Id-set range queries over point groups against the point scan (GAT_TUNE_RANGE_SHAPE = 1, the general
path) and the oracle, over the forms a query and a set can take: rectangles on cell borders, of no size,
inverted, beyond the grid, infinite or NaN; clustered sets that outgrow a team's set; trees that are one
leaf or as deep as the grid; batch sizes on both sides of every switch."""
import numpy as np
import pytest

import gat_b200 as G
from gat_b200 import _lib as L
from gat_b200 import data as D
from gat_b200.api import Index
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _general(ctx, ix, q, result="ids"):
    ctx.set_tuning(L.GAT_TUNE_RANGE_SHAPE, 1)
    try:
        return ix.range_query(q, result, capacity=4_000_000)
    finally:
        ctx.set_tuning(L.GAT_TUNE_RANGE_SHAPE, 0)


def _same_plain_and_points(ctx, ix, q):
    """Plain id sets, batched and plain point lists of few queries."""
    a, b = _general(ctx, ix, q), ix.range_query(q, "ids", "plain", capacity=4_000_000)
    assert np.array_equal(a.offsets, b.offsets) and np.array_equal(a.tids, b.tids)
    a = _general(ctx, ix, q, "points")
    for execution, part in (("batched", len(q)), ("plain", min(len(q), 12))):
        b = ix.range_query(q[:part], "points", execution, capacity=4_000_000)
        e = a.offsets[part]
        assert np.array_equal(a.offsets[:part + 1], b.offsets)
        assert np.array_equal(a.tids[:e], b.tids) and np.array_equal(a.pidx[:e], b.pidx)


def _same(ctx, ix, q):
    a, b = _general(ctx, ix, q), ix.range_query(q, capacity=4_000_000)
    assert np.array_equal(a.offsets, b.offsets) and np.array_equal(a.tids, b.tids)
    return b


def _odd_rectangles(t, cell, seed):
    """Rectangles whose edges lie on cell borders, on points, or nowhere sensible."""
    rng = np.random.default_rng(seed)
    x0, y0, x1, y1 = D.BOX
    c = np.float32(cell)
    k = rng.integers(0, int(1 / cell), (300, 4))
    gx = np.float32(x0) + c * np.minimum(k[:, 0], k[:, 1]).astype(np.float32)
    hx = np.float32(x0) + c * (np.maximum(k[:, 0], k[:, 1]) + rng.integers(0, 2, 300)).astype(np.float32)
    gy = np.float32(y1) - c * np.maximum(k[:, 2], k[:, 3]).astype(np.float32)
    hy = np.float32(y1) - c * np.minimum(k[:, 2], k[:, 3]).astype(np.float32)
    p = rng.integers(0, t.lon.size, (300, 2))
    ax, ay = t.lon[p], t.lat[p]
    point = np.stack([ax[:, 0], ay[:, 0], ax[:, 0], ay[:, 0]], 1)
    span = np.stack([ax.min(1), ay.min(1), ax.max(1), ay.max(1)], 1)
    inf, nan = np.inf, np.nan
    wild = np.array([[x0, y0, x1, y1], [x0 - 5, y0 - 5, x1 + 5, y1 + 5], [x1, y1, x0, y0], [-inf, -inf, inf, inf],
                     [121.4, 31.0, inf, inf], [-inf, 31.0, 121.2, 31.1], [nan, y0, x1, y1], [x0, nan, x1, y1], [x0, y0, nan, y1],
                     [x0, y0, x1, nan], [nan] * 4, [121.5, 31.2, 121.4, 31.3], [10, 10, 11, 11], [121.999, 30.69, 122.5, 30.71],
                     [120.9, 31.69, 121.001, 31.8], [121.3, 30.0, 121.31, 33.0]], np.float32)
    return np.concatenate([np.stack([gx, gy, hx, hy], 1), point, span, wild]).astype(np.float32)


@pytest.mark.parametrize("cell,cap", [(0.01, 512), (0.01, 1), (0.02, 10_000_000), (0.003, 64)])
def test_odd_rectangles(gpu_ctx, cell, cap):
    t = D.walks(D.lengths(3000, 0, 0, 0, 1, 200, 31), 31)
    db = G.TrajectorySet(gpu_ctx, t)
    q = _odd_rectangles(t, cell, 5)
    finite = np.isfinite(q).all(1)
    g, f = G.Grid(gpu_ctx, db, D.BOX, cell, 2, cap), G.FSG(gpu_ctx, db, D.BOX, cell)
    for ix, o in ((g, po.OracleGrid(t, D.BOX, cell, 2, cap)), (f, po.OracleFSG(t, D.BOX, cell))):
        r = _same(gpu_ctx, ix, q[finite])
        off, ids = o.range(q[finite], 0)
        assert np.array_equal(r.offsets, off) and np.array_equal(r.tids, ids)
    few = np.concatenate([q[:20], q[300:320], q[600:620], q[900:903], q[-5:]])
    for ix in (g, f, G.MortonGrid(g), G.STIG(gpu_ctx, db, 64)):
        _same_plain_and_points(gpu_ctx, ix, few)
    _same(gpu_ctx, g, q)  # NaN and infinite rectangles too: the two paths agree
    _same(gpu_ctx, f, q[~np.isinf(q).any(1)])
    _same(gpu_ctx, G.MortonGrid(g), q)
    for block in (2, 64, 5000):
        s = G.STIG(gpu_ctx, db, block)
        _same(gpu_ctx, s, q)
        off, ids = po.OracleSTIG(t, block).range(q[finite], 0)
        r = s.range_query(q[finite])
        assert np.array_equal(r.offsets, off) and np.array_equal(r.tids, ids)


@pytest.mark.parametrize("nq", [1, 31, 444, 445, 1024, 1025, 3001])
def test_batch_sizes(gpu_ctx, nq):
    t = D.walks(D.lengths(20_000, 0, 0, 0, 20, 200, 32), 32)
    db = G.TrajectorySet(gpu_ctx, t)
    q = D.boxes(nq, 1, 0.001, 0.3, 33)
    g = G.Grid(gpu_ctx, db, D.BOX, 0.005, 2, 512)
    for ix in (g, G.FSG(gpu_ctx, db, D.BOX, 0.005), G.MortonGrid(g), G.STIG(gpu_ctx, db, 1000)):
        _same(gpu_ctx, ix, q)
        _same_plain_and_points(gpu_ctx, ix, q[:100])


def test_clustered_set(gpu_ctx):
    """Most walks in one corner, ids in two far ranges: the expected sizes are wrong, so queries outgrow
    every team in turn, and a result's ids crowd in few buckets."""
    t = D.walks(D.lengths(12_000, 0, 0, 0, 20, 120, 34), 34)
    off = t.offsets
    for i in range(t.n):
        s, e = off[i], off[i + 1]
        if i < 2500 or i >= 9000:  # pulled into a 0.02 degree square
            t.lon[s:e] = np.float32(121.3) + (t.lon[s:e] - np.float32(121.0)) * np.float32(0.02)
            t.lat[s:e] = np.float32(31.1) + (t.lat[s:e] - np.float32(30.7)) * np.float32(0.02)
    db = G.TrajectorySet(gpu_ctx, t)
    rng = np.random.default_rng(6)
    c = rng.uniform([121.295, 31.095], [121.325, 31.125], (900, 2))
    h = np.exp(rng.uniform(np.log(0.0005), np.log(0.02), (900, 2)))
    q = np.concatenate([np.concatenate([c - h, c + h], 1), D.boxes(600, 1, 0.001, 0.05, 35)]).astype(np.float32)
    g = G.Grid(gpu_ctx, db, D.BOX, 0.002, 2, 512)
    for ix in (g, G.FSG(gpu_ctx, db, D.BOX, 0.002), G.MortonGrid(g), G.STIG(gpu_ctx, db, 1024)):
        r = _same(gpu_ctx, ix, q)
        assert int(np.diff(r.offsets).max()) > 4096  # beyond the largest set
        _same(gpu_ctx, ix, q[:200])
        _same_plain_and_points(gpu_ctx, ix, np.concatenate([q[900:930], q[:8], q[930:940]]))


def test_tiny_sets_and_fine_cells(gpu_ctx):
    for n, lo, hi, cell in ((1, 1, 1, 0.01), (2, 300, 300, 0.5), (40, 2000, 4000, 0.0005)):
        t = D.walks(D.lengths(n, 0, 0, 0, lo, hi, 36), 36)
        db = G.TrajectorySet(gpu_ctx, t)
        q = np.concatenate([D.boxes(500, 1, 0.0005, 0.5, 37), _odd_rectangles(t, 0.01, 38)[:600]])
        g = G.Grid(gpu_ctx, db, D.BOX, cell, 2, 512)
        for ix in (g, G.FSG(gpu_ctx, db, D.BOX, cell), G.MortonGrid(g), G.STIG(gpu_ctx, db, 16)):
            _same(gpu_ctx, ix, q)


def test_snapshot_keeps_groups(gpu_ctx, tmp_path):
    t = D.walks(D.lengths(4000, 0, 0, 0, 20, 200, 39), 39)
    db = G.TrajectorySet(gpu_ctx, t)
    q = D.boxes(700, 1, 0.001, 0.1, 40)
    for ix in (G.Grid(gpu_ctx, db, D.BOX, 0.005, 2, 512), G.FSG(gpu_ctx, db, D.BOX, 0.005), G.STIG(gpu_ctx, db, 500)):
        ix.save(str(tmp_path / "i.bin"))
        back = Index.load(gpu_ctx, db, str(tmp_path / "i.bin"))
        assert back.info()["device_bytes"] == ix.info()["device_bytes"]
        a, b = ix.range_query(q), back.range_query(q)
        assert np.array_equal(a.offsets, b.offsets) and np.array_equal(a.tids, b.tids)


@pytest.mark.parametrize("nq", [1024, 1025, 1185, 9473])
def test_point_lists_of_long_batches(gpu_ctx, nq):
    """Both gathers of a batch's point lists: a CTA a query, and a warp a query in one and in two turns."""
    t = D.walks(D.lengths(3_000, 0, 0, 0, 20, 200, 36), 36)
    g = G.Grid(gpu_ctx, G.TrajectorySet(gpu_ctx, t), D.BOX, 0.005, 2, 512)
    q = D.boxes(nq, 1, 0.001, 0.05, 37)
    a = _general(gpu_ctx, g, q, "points")
    b = g.range_query(q, "points", "batched", capacity=4_000_000)
    assert np.array_equal(a.offsets, b.offsets)
    assert np.array_equal(a.tids, b.tids) and np.array_equal(a.pidx, b.pidx)


@pytest.mark.parametrize("walks", [64, 65, 224, 225])
def test_long_point_lists(gpu_ctx, walks):
    """Lists of 64 points a walk on both sides of what the two passes hold (4,096 and 14,336)."""
    t = D.walks(D.lengths(walks, 0, 0, 0, 64, 64, 38), 38)
    g = G.Grid(gpu_ctx, G.TrajectorySet(gpu_ctx, t), D.BOX, 0.005, 2, 64)
    box = np.array([[t.lon.min(), t.lat.min(), t.lon.max(), t.lat.max()]], np.float32)
    q = np.concatenate([box, D.boxes(30, 1, 0.1, 0.6, 39), box])
    for ix in (g, G.FSG(gpu_ctx, g.db, D.BOX, 0.005), G.MortonGrid(g)):
        a = _general(gpu_ctx, ix, q, "points")
        b = ix.range_query(q, "points", "batched", capacity=4_000_000)
        assert a.offsets[1] > 0
        assert np.array_equal(a.offsets, b.offsets)
        assert np.array_equal(a.tids, b.tids) and np.array_equal(a.pidx, b.pidx)


def test_point_lists_of_walks_that_outgrow(gpu_ctx):
    """Rectangles whose border crosses more leaves than the walk's ranges hold, and more nodes than its frontier,
    with few points and with many; beside ordinary ones."""
    t = D.walks(D.lengths(2_000, 0, 0, 0, 20, 200, 61), 61)
    g = G.Grid(gpu_ctx, G.TrajectorySet(gpu_ctx, t), D.BOX, 0.0005, 2, 1)
    x0, y0, x1, y1 = D.BOX
    wide = [[x0 - 1, y0 + 0.001 * k, x1 + 1, y0 + 0.001 * k + 0.0007] for k in range(0, 900, 30)]
    large = [[x0 + 0.01 * k, y0 + 0.01 * k, x1 - 0.01 * k, y1 - 0.01 * k] for k in range(1, 25)]
    q = np.concatenate([np.array(wide + large, np.float32), D.boxes(100, 1, 0.001, 0.1, 62)])
    off, tid, pidx = po.OracleGrid(t, D.BOX, 0.0005, 2, 1).range(q, 1)
    for ix in (g, G.MortonGrid(g)):
        r = ix.range_query(q, "points", "batched", capacity=4_000_000)
        assert np.array_equal(r.offsets, off) and np.array_equal(r.tids, tid) and np.array_equal(r.pidx, pidx)


@pytest.mark.parametrize("walks,cell,block", [(3000, 0.01, 64), (225, 0.005, 5000), (1, 0.5, 2)])
def test_point_lists_of_every_index(gpu_ctx, walks, cell, block):
    """Point lists against the oracle: those of an FSG and a STIG take the point scan whatever the knob says, so one
    path cannot be held against the other there."""
    t = D.walks(D.lengths(walks, 0, 0, 0, 1, 200, 63), 63)
    q = _odd_rectangles(t, cell, 64)
    q = np.concatenate([q[np.isfinite(q).all(1)][::3], D.boxes(40, 1, 0.001, 0.4, 65)])
    db = G.TrajectorySet(gpu_ctx, t)
    g = G.Grid(gpu_ctx, db, D.BOX, cell, 2, 64)
    grid = po.OracleGrid(t, D.BOX, cell, 2, 64)
    for ix, o in ((g, grid), (G.MortonGrid(g), grid), (G.FSG(gpu_ctx, db, D.BOX, cell), po.OracleFSG(t, D.BOX, cell)),
                  (G.STIG(gpu_ctx, db, block), po.OracleSTIG(t, block))):
        off, tid, pidx = o.range(q, 1)
        for execution, part in (("batched", len(q)), ("plain", 20)):
            r = ix.range_query(q[:part], "points", execution, capacity=8_000_000)
            e = off[part]
            assert np.array_equal(r.offsets, off[:part + 1])
            assert np.array_equal(r.tids, tid[:e]) and np.array_equal(r.pidx, pidx[:e])


@pytest.mark.parametrize("walks,points", [(3, 1000), (20, 400), (33, 130), (1100, 4)])
def test_clustered_point_keys(gpu_ctx, walks, points):
    """Lists around 1,024 points and above whose keys crowd in few buckets (walks of many points, ids far apart) or
    in none, in both passes."""
    rng = np.random.default_rng(69)
    lens = np.full(9000, 1, np.int32)
    ids = np.sort(rng.choice(9000, walks, replace=False))
    lens[ids] = points
    t = D.walks(lens, 69)
    off = t.offsets
    for i in ids:  # inside one square
        s, e = off[i], off[i + 1]
        t.lon[s:e] = rng.uniform(121.3, 121.34, e - s)
        t.lat[s:e] = rng.uniform(31.1, 31.14, e - s)
    g = G.Grid(gpu_ctx, G.TrajectorySet(gpu_ctx, t), D.BOX, 0.005, 2, 64)
    k = rng.uniform(0, 0.02, (40, 2))
    q = np.concatenate([121.3 + k[:, :1], 31.1 + k[:, 1:], 121.34 - k[:, 1:], 31.14 - k[:, :1]], 1).astype(np.float32)
    q = np.concatenate([q, np.array([[121.3, 31.1, 121.34, 31.14], [121.0, 30.7, 122.0, 31.7]], np.float32)])
    off, tid, pidx = po.OracleGrid(t, D.BOX, 0.005, 2, 64).range(q, 1)
    for ix in (g, G.MortonGrid(g)):
        r = ix.range_query(q, "points", "batched", capacity=4_000_000)
        assert np.array_equal(r.offsets, off) and np.array_equal(r.tids, tid) and np.array_equal(r.pidx, pidx)


@pytest.mark.parametrize("walks", [300, 6000])
def test_scattered_points(gpu_ctx, walks):
    """Points far from one another, most of them a group of its own: long candidate lists are handed to the CTA and
    to the point scan, in batches on both sides of the one-CTA-each size and in plain execution."""
    rng = np.random.default_rng(66)
    t = D.walks(D.lengths(walks, 0, 0, 0, 20, 80, 66), 66)
    t.lon[:] = rng.uniform(121.01, 121.99, t.lon.size)
    t.lat[:] = rng.uniform(30.71, 31.69, t.lat.size)
    db = G.TrajectorySet(gpu_ctx, t)
    c = rng.uniform([121.05, 30.75], [121.95, 31.65], (500, 2))
    h = np.exp(rng.uniform(np.log(0.002), np.log(0.45), (500, 1)))
    q = np.concatenate([c - h, c + h], 1).astype(np.float32)
    q[::50] = [121.0, 30.7, 122.0, 31.7]
    g = G.Grid(gpu_ctx, db, D.BOX, 0.001, 2, 16)
    for ix in (g, G.FSG(gpu_ctx, db, D.BOX, 0.001), G.MortonGrid(g), G.STIG(gpu_ctx, db, 32)):
        a = _same(gpu_ctx, ix, q)
        _same(gpu_ctx, ix, q[:16])
        for lo, hi in ((0, 1), (1, 2), (5, 25), (40, 60)):
            b = ix.range_query(q[lo:hi], "ids", "plain", capacity=4_000_000)
            assert np.array_equal(b.offsets, a.offsets[lo:hi + 1] - a.offsets[lo])
            assert np.array_equal(b.tids, a.tids[a.offsets[lo]:a.offsets[hi]])


def test_walks_that_outgrow(gpu_ctx):
    """Id sets of rectangles over more rows of cells, blocks and nodes than a team has room for, of few ids and of
    more than a set holds, beside ordinary ones."""
    t = D.walks(D.lengths(9_000, 0, 0, 0, 20, 60, 67), 67)
    db = G.TrajectorySet(gpu_ctx, t)
    x0, y0, x1, y1 = D.BOX
    tall = [[x0 + 0.009 * k, y0 - 1, x0 + 0.009 * k + 0.004, y1 + 1] for k in range(100)]
    wide = [[x0 - 1, y0 + 0.009 * k, x1 + 1, y0 + 0.009 * k + 0.004] for k in range(100)]
    large = [[x0 + 0.01 * k, y0 + 0.01 * k, x1 - 0.01 * k, y1 - 0.01 * k] for k in range(20)]
    q = np.concatenate([np.array(tall + wide + large, np.float32), D.boxes(300, 1, 0.001, 0.05, 68)])
    g = G.Grid(gpu_ctx, db, D.BOX, 0.0004, 2, 1)
    for ix in (g, G.FSG(gpu_ctx, db, D.BOX, 0.0004), G.MortonGrid(g), G.STIG(gpu_ctx, db, 16)):
        a = _same(gpu_ctx, ix, q)
        assert int(np.diff(a.offsets).max()) > 4096
        _same(gpu_ctx, ix, q[95:105])
        b = ix.range_query(q[98:102], "ids", "plain", capacity=4_000_000)
        assert np.array_equal(b.tids, a.tids[a.offsets[98]:a.offsets[102]])
