"""The packed row tiles of the EDR kernel at the sizes and inputs where they can go wrong, against the
oracle: tile and chunk edges, pairs whose first match comes late or never (distances taken by
formula), the longest supported sides (the ends of the 16-bit range), NaN and infinite points."""
import numpy as np
import pytest

import gat_b200 as G
from gat_b200 import data as D
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu
EPS = 5e-4


def _cat(parts):
    return np.array([len(p) for p in parts], np.int32), np.concatenate(parts).astype(np.float32)


def _check(ctx, A, B, rows, eps=EPS):
    la, a = _cat(A)
    lb, b = _cat(B)
    ctx.set_edr_rows(rows)
    try:
        got = G.edr_pairs(ctx, la, a, lb, b, eps)
    finally:
        ctx.set_edr_rows(0)
    assert np.array_equal(got, po.edr_batch(la, a, lb, b, eps))


def _walks(lens, seed):
    t = D.walks(np.asarray(lens, np.int32), seed)
    off = t.offsets
    return [np.stack([t.lon[off[i]:off[i + 1]], t.lat[off[i]:off[i + 1]]], 1) for i in range(t.n)]


@pytest.mark.parametrize("rows", [0, 2, 4, 8])
def test_edges(gpu_ctx, rows):
    """Heights 64 / 128 / 256 and the last tile's 64 / 128 / 256; chunks of 32 columns, 63 columns of skew."""
    short = [1, 2, 63, 64, 65, 127, 128, 129, 191, 192, 193, 255, 256, 257, 320, 321, 385, 513]
    extra = [0, 1, 31, 32, 33, 62, 63, 64, 95, 96, 97, 130]
    ls = np.array([(s, s + e) for s in short for e in extra], np.int32)
    a, b = D.pairs(ls[:, 0], ls[:, 1], 7)
    oa, ob = np.cumsum(ls[:, 0])[:-1], np.cumsum(ls[:, 1])[:-1]
    _check(gpu_ctx, np.split(a, oa), np.split(b, ob), rows)
    _check(gpu_ctx, np.split(b, ob), np.split(a, oa), rows, 5e-3)


@pytest.mark.parametrize("rows", [0, 2, 8])
def test_first_match_late_or_never(gpu_ctx, rows):
    """A pair meets only from some row and column on (or in one point, or never)."""
    rng = np.random.default_rng(3)
    A = _walks(rng.integers(1, 700, 160), 5)
    B = []
    for i, x in enumerate(A):
        y = (np.repeat(x, rng.integers(1, 3), 0) + rng.normal(0, 2e-4, (1, 2))).astype(np.float32)
        r, c = int(rng.integers(0, len(x))), int(rng.integers(0, len(y)))
        if i % 4 == 0:
            y += 3  # never
        elif i % 4 == 1:
            y[:c] += 3  # columns meet from c on
        elif i % 4 == 2:
            x[:r] -= 3  # rows meet from r on
        else:
            z = y[c].copy()
            y += 3
            y[c] = z  # one point
        B.append(y)
    _check(gpu_ctx, A, B, rows)
    _check(gpu_ctx, B, A, rows)


def test_longest_sides(gpu_ctx):
    """16,384 points on both sides: identical (0), apart (formula), apart but for the last points."""
    (x,) = _walks([16384], 11)
    far = x + np.float32(4)
    near_end = far.copy()
    near_end[-40:] = x[-40:]
    _check(gpu_ctx, [x, x, x, x[:16383]], [x, far, near_end, far], 0)


def test_not_finite(gpu_ctx):
    """NaN matches nothing; an infinite difference (or inf - inf) is no match."""
    A = _walks([70, 130, 300, 64, 65], 13)
    B = [x.copy() for x in A]
    A[0][5] = np.nan
    B[1][40, 0] = np.nan
    A[2][100:140] = np.inf
    B[2][90:150] = np.inf
    A[3][:] = np.nan
    B[4][3] = -np.inf
    _check(gpu_ctx, A, B, 0)
    _check(gpu_ctx, B, A, 8)


def _restart_at_the_end():
    """16,384 points a side (eps = 1): the last row's fall restarts on the last column but one, and the last
    row meets the last column there."""
    n = 16384
    cols = np.full((n, 2), 1000.0)
    cols[n - 5:n - 1] = [(0.25 * k, -0.25 * k) for k in range(4)]
    cols[n - 1] = (-0.375, 1.3)
    # row r meets columns n - 4 + s .. n - 4 + e, by r mod 8; 4 and 7 meet none
    meets = {1: (2, 2), 2: (0, 0), 3: (0, 0), 5: (0, 0), 6: (0, 1), 0: (0, 2)}
    rows = np.array([(0.25 * meets[r % 8][1] - 0.875, -0.875 - 0.25 * meets[r % 8][0]) if r % 8 in meets else (-1000.0, -1000.0)
                     for r in range(1, n + 1)])
    rows[0] = (0.25 * 3 - 0.875, -0.875 - 0.25 * 2)
    rows[n - 1] = (-0.375, 0.4)
    return rows.astype(np.float32), cols.astype(np.float32)


@pytest.mark.parametrize("rows", [2, 4, 8])
def test_last_row_of_the_longest_side(gpu_ctx, rows):
    """Row 16,384 holds the one value that fills its half word to the top: at column 0 (the last point against the
    first ones), where its fall restarts at the end, and beside pairs of 16,383 points."""
    a, b = _restart_at_the_end()
    (x,) = _walks([16384], 17)
    far = x + np.float32(4)
    corner = far.copy()
    corner[[0, 1, 2, 31, 32, 16380, 16383]] = x[[-1, -1, -2, -1, -3, -1, -2]]
    A = [a, b, x, corner, a[1:], x[1:]]
    B = [b, a, corner, x, b[1:], corner[:-1]]
    _check(gpu_ctx, A[:2] + A[4:5], B[:2] + B[4:5], rows, 1.0)
    _check(gpu_ctx, A[2:4] + A[5:], B[2:4] + B[5:], rows)
    la = np.array([16384], np.int32)
    gpu_ctx.set_edr_rows(rows)
    try:
        assert G.edr_pairs(gpu_ctx, la, a, la, b, 1.0)[0] == 32766
    finally:
        gpu_ctx.set_edr_rows(0)


@pytest.mark.parametrize("n", [1, 64, 65])
def test_few_pairs_of_a_short_side(gpu_ctx, n):
    """Sides of up to 16 points against long ones: the tuner may take column tiles up to 64 pairs. The same pairs again
    take what it chose."""
    rng = np.random.default_rng(n)
    short = rng.integers(1, 17, n).astype(np.int32)
    long = np.maximum(short, np.exp(rng.uniform(0, np.log(16384), n)).astype(np.int32))
    long[0] = 16384
    a, b = D.pairs(short, long, 19)
    want = po.edr_batch(short, a, long, b, 5e-3)
    for _ in range(2):
        assert np.array_equal(G.edr_pairs(gpu_ctx, short, a, long, b, 5e-3), want)
        assert np.array_equal(G.edr_pairs(gpu_ctx, long, b, short, a, 5e-3), po.edr_batch(long, b, short, a, 5e-3))
