"""Measured cases: what a user of the FRW library has it do, through the
Python package (frw.Layout, frw.Batch, frw.ControlVariate, frw.Layout3).

Layouts come from the library's seeded generators at the density of the
benchmark's (one rect per 100 x 100 units, boxes likewise); a state's seed
moves the layout, the points and the walks' random numbers.  Kinds of case:

walk     walks from one conductor, result rows on the host (Layout.walk) or,
         with "device", added into the caller's device arrays
         (Layout.walk_device), as a multi-GPU sum or a chained run does
trace    per-walk records (Layout.walk_trace: randomWalkCudaWrapper's outputs)
create   a layout from host rects, a run of walks on it, its release: a
         program that meets every layout once
query    maximal empty squares and containing conductors of points, in host
         or in device memory
batch    many layouts of uneven size in one launch (frw.Batch)
cv       a control variate trained and used for one estimate
walk3, query3, create3   the same over 3-D box conductors; create3 runs the
         rows of several targets in one launch, as a capacitance matrix does
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "engineer-thesis_b200"))
import frw  # noqa: E402

# perimeter walks: the reference's start on the scaled surface, or the
# uniform start on the offset surface that gives capacitances
REFERENCE, CAPACITANCE = "reference", "capacitance"


def listed():
    return [
        # getAvgPathLen's usual call on a hand-made layout: 1000 walks on 100 rects; launches and latency
        dict(name="walk 1e3 on 100 rects", kind="walk", rects=100, walks=1000, estimate=REFERENCE),
        # the smallest benchmark configuration: one capacitance row, 1e5 walks on 100 rects
        dict(name="capacitance 1e5 on 100", kind="walk", rects=100, walks=100_000, estimate=CAPACITANCE),
        # an ordinary run: the capacitance row of a 10^4-rect layer, rows left on the device
        dict(name="capacitance 1e7 on 1e4", kind="walk", rects=10_000, walks=10_000_000, estimate=CAPACITANCE,
             device=True),
        # the headline: 1e8 walks with the reference's walk definition on a resident 10^6-rect layer
        dict(name="walk 1e8 on 1e6", kind="walk", rects=1_000_000, walks=100_000_000, estimate=REFERENCE,
             device=True),
        # per-walk outputs of an odd number of walks, copied to the host
        dict(name="trace 1000003 on 1e4", kind="trace", rects=10_000, walks=1_000_003, estimate=CAPACITANCE),
        # end to end from host rects: upload, tree and cell lists, walks, rows back, release
        dict(name="create 1e6, walk 1e7", kind="create", rects=1_000_000, walks=10_000_000, estimate=REFERENCE),
        # batched collision queries with points anywhere in the largest layer
        dict(name="query 1e7 on 1e6", kind="query", rects=1_000_000, points=10_000_000, device=True),
        # 64 layouts of 100 to 1e5 rects in one launch, walks by rect count
        dict(name="batch of 64, 2e7 walks", kind="batch", rects=100_000, layouts=64, walks=20_000_000),
        # the control variate of a target on the largest layer: training, exact mean and an estimate
        dict(name="control variate on 1e6", kind="cv", rects=1_000_000, walks=20_000_000, grid=16384,
             train=1_000_000, epochs=4),
        # the 3-D benchmark: capacitance row of a box among 10^4
        dict(name="walk3 1e7 on 1e4", kind="walk3", boxes=10_000, walks=10_000_000, device=True),
        # 3-D clearance queries with points anywhere
        dict(name="query3 1e7 on 1e4", kind="query3", boxes=10_000, points=10_000_000, device=True),
        # a 3-D layout met once: grid build and four rows of its capacitance matrix
        dict(name="create3 1e5, 4 targets", kind="create3", boxes=100_000, walks=500_000, targets=4),
    ]


def _log(rng, lo, hi):
    """An integer log-uniform in [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["walk", "walk", "trace", "create", "query", "query", "batch", "cv", "walk3", "query3",
                       "create3"])
    c = dict(kind=kind)
    if kind in ("walk", "trace", "create"):
        c["rects"] = _log(rng, 100, 1_000_000)
        c["walks"] = _log(rng, 1000, {"walk": 30_000_000, "trace": 2_000_000, "create": 10_000_000}[kind])
        c["estimate"] = rng.choice([REFERENCE, CAPACITANCE])
        if kind == "walk":
            c["device"] = rng.random() < 0.5
            option = rng.choice(["", "", "strata", "grid", "exact"])
            if option == "strata":
                c["strata"] = 1 << rng.randrange(4, 13)
            elif option == "grid" and c["estimate"] == CAPACITANCE:
                c["grid"] = 1 << rng.randrange(6, 15)
            elif option == "exact":
                c["exact_perimeter"] = True
    elif kind == "query":
        c["rects"] = _log(rng, 100, 1_000_000)
        c["device"] = rng.random() < 0.6
        c["points"] = _log(rng, 100, 10_000_000 if c["device"] else 300_000)
    elif kind == "batch":
        c["rects"] = _log(rng, 1000, 100_000)
        c["layouts"] = rng.randrange(2, 65)
        c["walks"] = _log(rng, 10_000, 20_000_000)
    elif kind == "cv":
        c["rects"] = _log(rng, 1000, 1_000_000)
        c["walks"] = _log(rng, 1_000_000, 20_000_000)
        c["grid"] = 1 << rng.randrange(10, 15)
        c["train"] = _log(rng, 100_000, 1_000_000)
        c["epochs"] = rng.randrange(1, 5)
    else:
        c["boxes"] = _log(rng, 100, 100_000)
        if kind == "query3":
            c["device"] = rng.random() < 0.6
            c["points"] = _log(rng, 100, 10_000_000 if c["device"] else 300_000)
        else:
            c["walks"] = _log(rng, 1000, 10_000_000 if kind == "walk3" else 500_000)
            if kind == "walk3":
                c["device"] = rng.random() < 0.5
                if rng.random() < 0.3:
                    c["strata"] = 1 << rng.randrange(4, 13)
            else:
                c["targets"] = rng.randrange(1, 9)
    return c


# ---- what a user's program has in hand before the call ----


def _rects(seed, n):
    return frw.generate_layout(seed * 7919 + n, n, 100.0 * math.sqrt(n))


def _boxes(seed, n):
    return frw.generate_layout3(seed * 7919 + n, n, math.ceil(20.0 * math.sqrt(n)), 400.0, 5, 50, 5, 20, 2)


def _target(seed, n, k=0):
    return (seed * 48271 + k * 69621 + 11) % n


def _opts(case):
    if case.get("estimate") == REFERENCE:
        return frw.opts(start_strata=case.get("strata", 0), exact_perimeter=case.get("exact_perimeter", False))
    return frw.capacitance_opts(1.0, start_strata=case.get("strata", 0), start_grid=case.get("grid", 0),
                                exact_perimeter=case.get("exact_perimeter", False))


def _batch_sizes(case):
    """Rect counts log-uniform from 100 to the case's largest, in a fixed uneven order."""
    m = case["layouts"]
    lo, hi = math.log(100), math.log(case["rects"])
    at = [(k * 37) % m / max(m - 1, 1) for k in range(m)]
    n = [int(round(math.exp(lo + (hi - lo) * t))) for t in at]
    total = sum(n)
    return n, [max(1, case["walks"] * k // total) for k in n]


def _points(seed, n, lo, hi):
    """Uniform points of the layer, as FP64 device rows."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((n, len(lo)), generator=g, device="cuda", dtype=torch.float64)
    lo, hi = (torch.tensor(np.asarray(v), device="cuda") for v in (lo, hi))
    return lo + u * (hi - lo)


def _device_rows(n):
    return dict(rows=torch.zeros(n + 4, dtype=torch.int64, device="cuda"),
                sums=torch.zeros(2 * n, dtype=torch.float64, device="cuda"),
                status=torch.zeros(1, dtype=torch.int32, device="cuda"))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind, seed=seed)
    if kind in ("walk3", "query3", "create3"):
        s["host"] = _boxes(seed, case["boxes"])
        s["n"] = case["boxes"]
        s["o"] = frw.opts3(start_strata=case.get("strata", 0))
        if kind == "create3":
            s["targets"] = [_target(seed, case["boxes"], k) for k in range(case["targets"])]
            return s
        s["L"] = frw.Layout3.from_boxes(s["host"])
    elif kind == "batch":
        n, w = _batch_sizes(case)
        s["L"] = [frw.Layout.from_rects(_rects(seed + k, m)) for k, m in enumerate(n)]
        s["B"] = frw.Batch(s["L"], [_target(seed, m, k) for k, m in enumerate(n)], w, frw.capacitance_opts(1.0))
        return s
    else:
        s["host"] = _rects(seed, case["rects"])
        s["n"] = case["rects"]
        s["o"] = _opts(case)
        if kind == "create":
            s["target"] = _target(seed, s["n"])
            return s
        s["L"] = frw.Layout.from_rects(s["host"])
    s["target"] = _target(seed, s["n"])
    if kind in ("query", "query3"):
        b, d = s["L"].bounds, len(s["L"].bounds) // 2
        p = _points(seed, case["points"], b[:d], b[d:])
        if case.get("device"):
            s["points"] = p
            dims = (case["points"], 4) if kind == "query" else (case["points"],)
            s["out"] = torch.empty(dims, dtype=torch.float64, device="cuda")
            s["hit"] = torch.empty(case["points"], dtype=torch.int64, device="cuda")
        else:
            s["points"] = p.cpu().numpy()
    elif case.get("device"):
        s.update(_device_rows(s["n"]))
    elif kind == "cv":
        s["cv_opts"] = frw.cv_opts(train_walks=case["train"], train_seed=seed + 0x7E57, epochs=case["epochs"])
    torch.cuda.synchronize()  # the layouts and arrays are ready before they are used on the library's streams
    return s


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _row(r):
    """A result with its rows at their whole capacity (the result's arrays are
    the filled fronts of these; zero past the conductors reached)."""
    rows = {k: getattr(r, k).base for k in ("conductor", "hits", "cap", "cap_se", "sum_w", "sum_w2")}
    rows["hits"] = rows["hits"].view(np.int64)
    return dict(rows, counts=[r.walks, r.escaped, r.aborted, r.hops_total], gauss=r.gauss, other=r.fraction_other)


def _row_table(rs):
    """The rows of several results, one after another."""
    rows = [_row(r) for r in rs]
    out = {k: np.stack([r[k] for r in rows]) for k in
           ("gauss", "conductor", "hits", "cap", "cap_se", "sum_w", "sum_w2")}
    out["counts"] = np.array([r["counts"] for r in rows], dtype=np.int64)
    out["other"] = np.array([r["other"] for r in rows])
    return out


def run(s):
    case, kind, seed = s["case"], s["kind"], s["seed"]
    if kind in ("walk", "walk3"):
        if not case.get("device"):
            return _row(s["L"].walk(s["target"], case["walks"], seed, s["o"]))
        n, rows, sums = s["n"], s["rows"], s["sums"]
        rows.zero_()
        sums.zero_()
        s["L"].walk_device(s["target"], case["walks"], seed, s["o"], rows[:n], sums[:n], sums[n:], rows[n:],
                           s["status"], _stream())
        return rows, sums, s["status"]
    if kind == "trace":
        return s["L"].walk_trace(s["target"], 0, case["walks"], seed, s["o"])
    if kind == "create":
        with frw.Layout.from_rects(s["host"]) as L:
            return _row(L.walk(s["target"], case["walks"], seed, s["o"]))
    if kind in ("query", "query3"):
        if not case.get("device"):
            return s["L"].query(s["points"])
        s["L"].query_device(s["points"], s["out"], s["hit"], _stream())
        return s["out"], s["hit"]
    if kind == "batch":
        return _row_table(s["B"].run(seed, capacity=1024))
    if kind == "cv":
        cv = frw.ControlVariate(s["L"], s["target"], s["o"], s["cv_opts"])
        r, i = cv.walk(case["walks"], seed), cv.info
        out = [cv.params(), i.mean_term, i.train_loss, r.plain, r.plain_se, r.cv, r.cv_se]
        cv.close()
        return out
    with frw.Layout3.from_boxes(s["host"]) as L3:  # create3
        return _row_table(L3.walk_batch(s["targets"], case["walks"], seed, s["o"], capacity=4096))


# ---- work a pass cannot do without ----
# A walk takes about this many queries (the seeded layouts' means), each with
# the gaps to one rect or box, the square or cube it allows, a bin of the
# Green's function and the next point: some 60 FP64 operations.
HOPS = {REFERENCE: 10.5, CAPACITANCE: 6.4, "3d": 11.9}
QUERY_FLOPS = 60


def work(case):
    kind = case["kind"]
    if kind == "query":
        return dict(bytes=case["points"] * 56 + case["rects"] * 16, flops=case["points"] * QUERY_FLOPS)
    if kind == "query3":
        return dict(bytes=case["points"] * 40 + case["boxes"] * 24, flops=case["points"] * 12)
    if kind == "batch":
        n, w = _batch_sizes(case)
        return dict(bytes=sum(n) * 16, flops=sum(w) * HOPS[CAPACITANCE] * QUERY_FLOPS)
    if kind in ("walk3", "create3"):
        rows = case["boxes"] * 24 * (case.get("targets", 1) if kind == "create3" or case.get("device") else 0)
        return dict(bytes=case["boxes"] * 24 + rows,
                    flops=case["walks"] * case.get("targets", 1) * HOPS["3d"] * QUERY_FLOPS)
    out = case["rects"] * 24 if case.get("device") else case["walks"] * 24 if kind == "trace" else 0
    flops = case["walks"] * HOPS[case.get("estimate", CAPACITANCE)] * QUERY_FLOPS
    if kind == "cv":  # 16 -> 64 -> 64 -> 1: forward and backward of every training row, forward of every grid point
        mac = 16 * 64 + 64 * 64 + 64
        flops += case["train"] * (HOPS[CAPACITANCE] * QUERY_FLOPS + case["epochs"] * 6 * mac)
        flops += case["grid"] * 200 * 2 * mac
    return dict(bytes=case["rects"] * 16 + out, flops=flops)


# ---- values in 64 bits, without the library ----


def _exact_query(points, rects, bounds):
    """The expand-and-bisect square of every point and the lowest rect that
    contains it, every box tested against every rect."""
    dev = points.device
    b = [float(v) for v in bounds]
    px, py = points[:, 0], points[:, 1]
    n = len(points)
    chunk = max(1, 200_000_000 // len(rects))

    def touches(x0, y0, x1, y1):
        out = torch.zeros(len(x0), dtype=torch.bool, device=dev)
        for i in range(0, len(x0), chunk):
            k = slice(i, i + chunk)
            m = rects[:, 2][None] >= x0[k, None]
            m &= rects[:, 0][None] <= x1[k, None]
            m &= rects[:, 3][None] >= y0[k, None]
            m &= rects[:, 1][None] <= y1[k, None]
            out[k] = m.any(1)
        return out | ~((y0 >= b[1]) & (x0 >= b[0]) & (y1 <= b[3]) & (x1 <= b[2]))

    sq = torch.stack([px - 1, py - 1, px + 1, py + 1], 1)
    two = torch.stack([px - 2, py - 2, px + 2, py + 2], 1)
    done = touches(*sq.T)
    at2 = ~done & touches(*two.T)
    sq[at2] = two[at2]
    live = torch.nonzero(~(done | at2)).reshape(-1)
    o = sq[live]
    dist = torch.full((len(live),), 0.05 * max(b[2] - b[0], b[3] - b[1]), dtype=torch.float64, device=dev)
    least = float(np.float32(0.095))
    reached = torch.zeros(len(live), dtype=torch.bool, device=dev)
    for _ in range(400):
        if not len(live):
            break
        c = touches(*o.T)
        reached |= c
        halve = reached & (dist > least)
        go = c | ~reached | halve  # a free box stops once dist is small
        stop = ~go
        sq[live[stop]] = o[stop]
        live, o, dist, reached, c, halve = (v[go] for v in (live, o, dist, reached, c, halve))
        dist = torch.where(halve, dist * 0.5, dist)
        step = torch.where(c, dist, -dist)[:, None]
        o = torch.cat([o[:, :2] + step, o[:, 2:] - step], 1)
    hit = torch.full((n,), -1, dtype=torch.int64, device=dev)
    for i in range(0, n, chunk):
        x, y = px[i:i + chunk, None], py[i:i + chunk, None]
        m = (rects[:, 0][None] <= x) & (rects[:, 2][None] >= x) & (rects[:, 1][None] <= y) & (rects[:, 3][None] >= y)
        hit[i:i + chunk] = torch.where(m.any(1), m.to(torch.uint8).argmax(1), hit[i:i + chunk])
    return sq, hit


def _exact_query3(points, boxes):
    """L-infinity distance to the nearest box and the lowest box at it."""
    n = len(points)
    d = torch.empty(n, dtype=torch.float64, device=points.device)
    k = torch.empty(n, dtype=torch.int64, device=points.device)
    chunk = max(1, 100_000_000 // len(boxes))
    for i in range(0, n, chunk):
        g = torch.zeros((len(points[i:i + chunk]), len(boxes)), dtype=torch.float64, device=points.device)
        for a in range(3):
            p = points[i:i + chunk, a, None]
            torch.maximum(g, boxes[:, a][None] - p, out=g)
            torch.maximum(g, p - boxes[:, 3 + a][None], out=g)
        v = g.min(1).values
        d[i:i + chunk] = v
        k[i:i + chunk] = (g == v[:, None]).to(torch.uint8).argmax(1)
    return d, k


def exact(case, seed):
    """Queries against every rect or box while that stays within seconds.  A
    walk's counts are whole numbers and its sums those of the same walks;
    replaying its draws and queries one by one takes minutes to hours."""
    if case["kind"] not in ("query", "query3"):
        return None
    flat = case["kind"] == "query"
    n = case["rects" if flat else "boxes"]
    if case["points"] * n > (3e9 if flat else 2e10):
        return None
    s = prepare(case, seed)
    host = torch.from_numpy(s["host"].astype(np.float64)).cuda()
    p = torch.as_tensor(s["points"], device="cuda")
    return _exact_query(p, host, s["L"].bounds) if flat else _exact_query3(p, host)
