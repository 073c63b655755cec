"""The workloads whose speed is tracked: range queries, EDR distances and top-k similarity.

Every case is one call (or one short burst of requests) of the kind a program using gat_b200
makes over a trajectory set and indexes that it keeps resident: random walks of the five
configured workloads in the one-degree box, rectangles and query walks of their distributions.

A case holds plain values only:

  op = "range"  `nq` rectangles with sides log-uniform in [side_lo, side_hi] degrees over a set of
                `n` walks of U[len_lo, len_hi] points, answered by one `index` ("grid", "morton",
                "stig", "fsg") as trajectory ids or (trajectory, point) lists (`result`), batched or
                one query per launch sequence (`exec`), over device arrays (`api` =
                "device") or host arrays ("host") of the caller
  op = "edr"    `nq` pairs, both lengths log-uniform in [len_lo, len_hi]
  op = "topk"   the `k` most similar walks for `nq` queries drawn from a set of `n` walks with
                lognormal(ln 200, 0.6) lengths in [32, 1024]
  op = "serve"  a burst of `nq` requests through the server: 70% rectangles spread over the grid,
                STIG and FSG indexes, 30% top-k queries of log-uniform [16, len_hi] points
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import gat_b200 as G
from gat_b200 import _lib as L
from gat_b200 import data

EPS = 5e-4  # match tolerance of the EDR configurations, degrees per axis
TOPK_CELL = 0.0025  # 256 x 256 virtual cells after a shift of 2
LEAF_CAP = 512
STIG_BLOCK = 10240


def _range(name, n, nq, index, result, exec, api, length=(50, 350), side=(0.001, 0.05), cell=0.001):
    return {"name": name, "op": "range", "n": n, "nq": nq, "index": index, "result": result, "exec": exec, "api": api,
            "len_lo": length[0], "len_hi": length[1], "side_lo": side[0], "side_hi": side[1], "cell": cell}


def listed():
    return [
        # one square asked of a small resident set: the latency of the smallest call
        _range("range_one", 10_000, 1, "grid", "ids", "plain", "device", (20, 200), (0.01, 0.01), 0.01),
        # configuration 1: 1,000 squares, every point in them, from and to host arrays
        _range("range_points_1k", 10_000, 1_000, "grid", "points", "batched", "host", (20, 200), (0.01, 0.01), 0.01),
        # a serving-sized batch over a mid-sized set
        _range("range_batch_64", 300_000, 64, "grid", "ids", "batched", "device"),
        # configuration 3: the analytic batch over the full set
        _range("range_grid_100k", 1_000_000, 100_000, "grid", "ids", "batched", "device"),
        # the other two indexes, batches in between, sizes off the powers of two
        _range("range_fsg_20k", 300_000, 20_011, "fsg", "ids", "batched", "device"),
        _range("range_stig_5k", 60_000, 5_003, "stig", "ids", "batched", "device"),
        # a few short pairs from host arrays: the latency of a distance call
        {"name": "edr_16_short", "op": "edr", "nq": 16, "len_lo": 20, "len_hi": 200, "api": "host"},
        # configuration 4: pairs of very uneven lengths in one launch
        {"name": "edr_4096", "op": "edr", "nq": 4096, "len_lo": 16, "len_hi": 4096, "api": "device"},
        # a few very long pairs, up to the longest supported side: each pair's critical path counts
        {"name": "edr_24_long", "op": "edr", "nq": 24, "len_lo": 2000, "len_hi": 16384, "api": "device"},
        # configuration 2: one similarity query at a time, and a batch of them from host arrays
        {"name": "topk_one", "op": "topk", "n": 100_000, "nq": 1, "k": 32, "exec": "plain", "api": "device"},
        {"name": "topk_64", "op": "topk", "n": 100_000, "nq": 64, "k": 32, "exec": "batched", "api": "host"},
        # configuration 5, scaled to a burst: mixed requests batched as they arrive
        {"name": "serve_192", "op": "serve", "n": 100_000, "nq": 192, "k": 64, "len_hi": 1024},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    op = rng.choice(["range", "range", "range", "edr", "edr", "topk"])
    if op == "range":
        index = rng.choice(["grid", "grid", "fsg", "morton", "stig"])
        n = _log(rng, 10_000, 60_000 if index == "stig" else 500_000)
        result = rng.choice(["ids", "ids", "points"])
        ex = rng.choice(["batched", "batched", "batched", "plain"])
        nq = _log(rng, 1, 24) if ex == "plain" else _log(rng, 1, 50_000 if result == "ids" else 2_000)
        lo = math.exp(rng.uniform(math.log(0.001), math.log(0.02)))
        side = (lo, min(0.05, lo * math.exp(rng.uniform(0.0, math.log(50.0)))))
        length = rng.choice([(20, 200), (50, 350)])
        # no more candidate points (or points returned) than the listed batches
        inside = n * 0.5 * sum(length) * _log_mean(*side) ** 2
        nq = max(1, min(nq, int((2.5e9 if result == "ids" else 3e7) / inside)))
        c = _range("", n, nq, index, result, ex, rng.choice(["device", "host"]), length, side, rng.choice([0.001, 0.0025]))
    elif op == "edr":
        lo = _log(rng, 2, 2000)
        hi = _log(rng, lo, 16384)
        # no more cells than the 4,096-pair configuration
        mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo
        c = {"op": "edr", "nq": _log(rng, 1, max(1, min(4096, int(1.5e9 / (mean * mean))))), "len_lo": lo, "len_hi": hi,
             "api": rng.choice(["device", "host"])}
    else:
        ex = rng.choice(["plain", "batched"])
        c = {"op": "topk", "n": _log(rng, 10_000, 100_000), "nq": _log(rng, 1, 8 if ex == "plain" else 64),
             "k": rng.randint(8, 64), "exec": ex, "api": rng.choice(["device", "host"])}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- inputs
def _set(case, seed):
    n = case["n"]
    if case["op"] == "range":
        lens = data.lengths(n, L.GAT_LEN_UNIFORM, 0, 0, case["len_lo"], case["len_hi"], seed)
    else:
        lens = data.lengths(n, L.GAT_LEN_LOGNORMAL, math.log(200.0), 0.6, 32, 1024, seed)
    return data.walks(lens, seed)


def _boxes(case, n, seed):
    lo, hi = case.get("side_lo", 0.001), case.get("side_hi", 0.05)
    return data.boxes(n, L.GAT_SIDE_LOGUNIFORM if hi > lo else L.GAT_SIDE_FIXED, lo, hi, seed)


def _pairs(case, seed):
    n = case["nq"]
    la = data.lengths(n, L.GAT_LEN_LOGUNIFORM, 0, 0, case["len_lo"], case["len_hi"], seed)
    lb = data.lengths(n, L.GAT_LEN_LOGUNIFORM, 0, 0, case["len_lo"], case["len_hi"], seed + 1)
    a, b = data.pairs(la, lb, seed)
    return la, a, lb, b


def _starts(lens):
    off = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=off[1:])
    return off


def _queries(case, t, seed):
    """Query walks drawn from the set, as configuration 2 draws them."""
    return t.subset(data.sample_ids(case["nq"], t.n, seed))


def _log_mean(lo, hi):
    return (hi - lo) / math.log(hi / lo) if hi > lo else float(lo)


def _capacity(case):
    """Result entries a program sets aside: every rectangle at its largest for a few, twice the mean
    for many (a walk of a few hundred steps is about 0.0025 degrees wide)."""
    n, nq, m, hi = case["n"], case["nq"], _log_mean(case["side_lo"], case["side_hi"]), case["side_hi"]
    if case["result"] == "points":
        total = n * 0.5 * (case["len_lo"] + case["len_hi"])
        mean, most = total * m * m, 1.5 * total * hi * hi + 2048
    else:
        mean, most = n * (m + 0.0025) ** 2, 1.5 * n * (hi + 0.0025) ** 2 + 64
    return int(min(nq * most, 2 * nq * mean + 8 * most))


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    s = {"case": case, "ctx": G.Context(torch.cuda.current_device())}
    ctx, op = s["ctx"], case["op"]
    if op == "range":
        t = _set(case, seed)
        s["db"] = G.TrajectorySet(ctx, t)
        if case["index"] == "stig":
            s["ix"] = G.STIG(ctx, s["db"], STIG_BLOCK)
        elif case["index"] == "fsg":
            s["ix"] = G.FSG(ctx, s["db"], G.BOX, case["cell"])
        else:
            s["ix"] = s["grid"] = G.Grid(ctx, s["db"], G.BOX, case["cell"], 2, LEAF_CAP)
            if case["index"] == "morton":
                s["ix"] = G.MortonGrid(s["grid"])
        s["q"], cap = _boxes(case, case["nq"], seed), _capacity(case)
        s["off"], s["tid"] = np.zeros(case["nq"] + 1, np.int64), np.zeros(cap, np.int32)
        s["pidx"] = np.zeros(cap if case["result"] == "points" else 0, np.int32)
        if case["api"] == "device":
            for key in ("q", "off", "tid", "pidx"):
                s[key] = _cuda(s[key])
    elif op == "edr":
        la, a, lb, b = _pairs(case, seed)
        s["pairs"] = (la, a, lb, b)
        if case["api"] == "device":
            s["pairs"] = (_cuda(la), _cuda(_starts(la)), _cuda(a), _cuda(lb), _cuda(_starts(lb)), _cuda(b))
            s["out"] = torch.empty(case["nq"], dtype=torch.int32, device="cuda")
    else:
        t = _set(case, seed)
        s["db"] = G.TrajectorySet(ctx, t)
        s["ix"] = G.Grid(ctx, s["db"], G.BOX, TOPK_CELL, 2, LEAF_CAP)
        if op == "topk":
            q = s["q"] = _queries(case, t, seed)
            if case["api"] == "device":
                s["max_len"] = int(q.lengths.max())
                s["q"] = (_cuda(q.lengths), _cuda(_starts(q.lengths)), _cuda(np.stack([q.lon, q.lat], 1)))
                s["ids"] = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
                s["dist"] = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
        else:
            s["stig"] = G.STIG(ctx, s["db"], STIG_BLOCK)
            s["fsg"] = G.FSG(ctx, s["db"], G.BOX, TOPK_CELL)
            s["server"] = G.Server(ctx, s["ix"], s["stig"], s["fsg"])
            n_topk = case["nq"] * 3 // 10
            walk = data.walks(data.lengths(n_topk, L.GAT_LEN_LOGUNIFORM, 0, 0, 16, case["len_hi"], seed + 2), seed + 2)
            box = _boxes(case, case["nq"] - n_topk, seed)
            kinds = (L.GAT_INDEX_GRID, L.GAT_INDEX_STIG, L.GAT_INDEX_FSG)
            reqs = [("range", box[i], kinds[i % 3]) for i in range(len(box))]
            for i in range(n_topk):  # spread evenly among the rectangles
                reqs.insert(int((i + 0.5) * len(box) / n_topk) + i, ("topk", walk.points(i + 1), 8 + i * 7 % (case["k"] - 7)))
            s["reqs"], s["width"] = reqs, int(1.5 * case["n"] * 0.0525 ** 2) + 64
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- one pass
def _ptr(t):
    return C.c_void_p(t.data_ptr())


_RESULT = {"ids": L.GAT_RESULT_IDS, "points": L.GAT_RESULT_POINTS}
_EXEC = {"batched": L.GAT_EXEC_BATCHED, "plain": L.GAT_EXEC_PLAIN}


def run(state):
    case, ctx = state["case"], state["ctx"]
    op = case["op"]
    if op == "range":
        off, tid, pidx, need = state["off"], state["tid"], state["pidx"], C.c_int64(0)
        points, kind, ex = case["result"] == "points", _RESULT[case["result"]], _EXEC[case["exec"]]
        if case["api"] == "host":
            rc = L.lib.gat_range_query(ctx.h, state["ix"].h, state["q"].ctypes.data, case["nq"], kind, ex,
                                       off.ctypes.data_as(L.P_i64), tid.ctypes.data_as(L.P_i32),
                                       pidx.ctypes.data_as(L.P_i32) if points else None, len(tid), C.byref(need))
        else:
            rc = L.lib.gat_range_query_dev(ctx.h, state["ix"].h, _ptr(state["q"]), case["nq"], kind, ex, _ptr(off), _ptr(tid),
                                           _ptr(pidx) if points else None, tid.numel(), C.byref(need))
        ctx.check(rc, "range query")
        return (off, tid, pidx) if points else (off, tid)
    if op == "edr":
        if case["api"] == "host":
            return G.edr_pairs(ctx, *state["pairs"], EPS)
        la, oa, a, lb, ob, b = state["pairs"]
        ctx.check(L.lib.gat_edr_pairs_dev(ctx.h, case["nq"], _ptr(la), _ptr(oa), _ptr(a), _ptr(lb), _ptr(ob), _ptr(b), EPS,
                                          _ptr(state["out"])), "gat_edr_pairs_dev")
        return state["out"]
    if op == "topk":
        if case["api"] == "host":
            ids, dist, _ = state["ix"].topk(state["q"], case["k"], EPS, case["exec"])
            return ids, dist
        ql, qo, qx = state["q"]
        ctx.check(L.lib.gat_topk_dev(ctx.h, state["ix"].h, case["nq"], _ptr(ql), _ptr(qo), _ptr(qx), state["max_len"],
                                     case["k"], EPS, _EXEC[case["exec"]], _ptr(state["ids"]), _ptr(state["dist"]), None),
                  "gat_topk_dev")
        return state["ids"], state["dist"]
    server, n, k = state["server"], len(state["reqs"]), case["k"]
    rids = [server.submit_range(x, kind) if what == "range" else server.submit_topk(x[0], x[1], kind, EPS)
            for what, x, kind in state["reqs"]]
    # one row per request: a range request's id set, or a top-k request's ids and distances
    ids, dist = np.zeros((n, state["width"]), np.int32), np.zeros((n, k), np.int32)
    for i, ((what, _, kind), rid) in enumerate(zip(state["reqs"], rids)):
        if server.wait(rid) != L.GAT_OK:
            raise RuntimeError(f"request {rid} failed")
        if what == "range":
            r = server.range_result(rid)
            ids[i, :len(r)] = r
        else:
            ids[i, :kind], dist[i, :kind] = server.topk_result(rid, kind)
        server.release(rid)
    return ids, dist


# ---------------------------------------------------------------- what a pass cannot do without
def _range_work(n, nq, mean_len, side, index_bytes, out_bytes, points):
    """The candidates' coordinates and ids once each (where rectangles overlap they share them), the
    rectangles, the offsets and the results."""
    total = n * mean_len
    inside = total * side * side  # points in one rectangle of the unit box
    covered = total * (1.0 - math.exp(-nq * side * side))
    walks = min(float(n), n * (side + 0.0025) ** 2)  # a walk of a few hundred steps is about 0.0025 degrees wide
    results = nq * (inside if points else min(inside, walks))
    return index_bytes * covered + 24.0 * nq + out_bytes * results, 4.0 * nq * inside


def work(case):
    op = case["op"]
    if op == "range":
        points = case["result"] == "points"
        b, f = _range_work(case["n"], case["nq"], 0.5 * (case["len_lo"] + case["len_hi"]),
                           _log_mean(case["side_lo"], case["side_hi"]), 12.0, 8.0 if points else 4.0, points)
        return {"bytes": b, "flops": f}
    if op == "edr":
        m = _log_mean(case["len_lo"], case["len_hi"])
        # per cell: two subtractions, two compares, and the three-way choice of the recurrence
        return {"bytes": case["nq"] * (16.0 * m + 28.0), "flops": 12.0 * case["nq"] * m * m}
    if op == "topk":
        # the frequency vectors and bounds of every walk, then at least the k winners' distances
        m = 200.0 * math.exp(0.18)
        return {"bytes": case["n"] * (8.0 * 4.0 + 12.0) + case["nq"] * (8.0 * m + case["k"] * (8.0 * m + 8.0)),
                "flops": 12.0 * case["nq"] * case["k"] * m * m}
    n_topk = case["nq"] * 3 // 10
    m = 200.0 * math.exp(0.18)
    b, f = _range_work(case["n"], case["nq"] - n_topk, m, _log_mean(0.001, 0.05), 12.0, 4.0, False)
    ql, k = _log_mean(16, case["len_hi"]), 0.5 * (8 + case["k"])
    return {"bytes": b + case["n"] * 44.0 + n_topk * (8.0 * ql + k * (8.0 * m + 8.0)), "flops": f + 12.0 * n_topk * k * ql * m}


# ---------------------------------------------------------------- the values themselves
def _edr_one(a, b, u):
    """The recurrence over one pair, by anti-diagonals: with m, u, l the diagonal, upper and left
    operands, the cell is m when it is below both, else l when it is below both, else u."""
    if len(b) < len(a):
        a, b = b, a  # rows are the shorter side
    n, m = len(a), len(b)
    match = (np.abs(a[:, None, 0] - b[None, :, 0]) < u) & (np.abs(a[:, None, 1] - b[None, :, 1]) < u)
    big = np.int64(1) << 40
    prev2, prev = np.full(n + 1, big), np.full(n + 1, big)  # diagonals d - 2 and d - 1, by row
    prev2[0] = 0
    prev[0], prev[1] = 1, 1
    for d in range(2, n + m + 1):
        cur = np.full(n + 1, big)
        if d <= m:
            cur[0] = d
        if d <= n:
            cur[d] = d
        r = np.arange(max(1, d - m), min(n, d - 1) + 1)
        if len(r):
            dg = prev2[r - 1] + np.where(match[r - 1, d - r - 1], 0, 1)
            up, left = prev[r - 1] + 1, prev[r] + 1
            cur[r] = np.where((dg < up) & (dg < left), dg, np.where((left < up) & (left < dg), left, up))
        prev2, prev = prev, cur
    return int(prev[n])


def exact(case, seed):
    if case["op"] == "edr":
        la, a, lb, b = _pairs(case, seed)
        if float((la.astype(np.int64) * lb).sum()) > 2e8 or float((la.astype(np.int64) + lb).sum()) > 2e5:
            return None
        oa, ob = _starts(la), _starts(lb)
        # the test is |float difference| < eps with eps in double
        out = [_edr_one(a[oa[i]:oa[i + 1]], b[ob[i]:ob[i + 1]], np.float64(EPS)) for i in range(case["nq"])]
        return np.asarray(out, np.int32)
    if case["op"] == "range":
        t, q = _set(case, seed), _boxes(case, case["nq"], seed)
        width = float(np.minimum(q[:, 2], 122.0).mean() - np.maximum(q[:, 0], 121.0).mean())
        if t.lon.size > 2e7 or case["nq"] * t.lon.size * max(width, 0.0) > 4e8:
            return None
        order = np.argsort(t.lon, kind="stable")
        x, y = t.lon[order], t.lat[order]
        off = _starts(t.lengths)
        tid = np.repeat(np.arange(1, t.n + 1, dtype=np.int32), t.lengths)[order]
        pidx = (order - off[tid - 1]).astype(np.int32)
        offsets, tids, pids = np.zeros(case["nq"] + 1, np.int64), [], []
        for i, (x0, y0, x1, y1) in enumerate(q):
            s, e = np.searchsorted(x, x0, "left"), np.searchsorted(x, x1, "right")
            h = s + np.flatnonzero((y[s:e] >= y0) & (y[s:e] <= y1))
            if case["result"] == "points":
                h = h[np.lexsort((pidx[h], tid[h]))]
                tids.append(tid[h])
                pids.append(pidx[h])
            else:
                tids.append(np.unique(tid[h]))
            offsets[i + 1] = offsets[i] + len(tids[-1])
        got = [np.zeros(_capacity(case), np.int32) for _ in range(2 if case["result"] == "points" else 1)]
        for buf, parts in zip(got, (tids, pids)):
            buf[:offsets[-1]] = np.concatenate(parts)
        return (offsets, *got)
    return None
