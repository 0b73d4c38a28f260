"""Timed cases of the miner: whole calls through the package's public entry points.

A case is one call as a program makes it: a mine of one dataset (resident, or read from host memory), of a batch of
jobs, of a CSV file, one that keeps its instance tables, or one gradient of the cost model.  Datasets come from the
package's generator at the densities of its configurations; sizes run from a couple of thousand points to the 20
million of the benchmark, odd ones among them.
"""
import math
import os
import sys
import tempfile

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "gpu-colocationmininig_gb300"))

import colo  # noqa: E402
from colo import gen  # noqa: E402

FIELDS = ("cand", "ub", "passed", "rows", "num", "pi", "prevalent", "argmin")
EXACT_POINTS = 25_000   # datasets up to this many points are mined again in plain numpy by exact()


def listed():
    return [
        # the smallest call: one district's points, where launches and waits are all there is
        {"name": "tiny_2k", "kind": "mine", "n": 2003, "features": 9, "density": "town", "form": "batched",
         "reach": 1.0, "thr": 0.2, "max_size": 6},
        # the small plain configuration's size (20,000 points, 10 equal features)
        {"name": "small_20k", "kind": "mine", "n": 20000, "features": 10, "density": "small", "form": "batched",
         "reach": 1.0, "thr": 0.3, "max_size": 4},
        # an ordinary city: odd sizes, a second mask word, no size cap
        {"name": "ragged_300k", "kind": "mine", "n": 300007, "features": 37, "density": "town", "form": "batched",
         "reach": 1.3, "thr": 0.15, "max_size": 0},
        # the million-point configuration with the cost model, as the headline form runs it
        {"name": "mid_1m", "kind": "mine", "n": 1000000, "features": 40, "density": "town", "form": "learned",
         "reach": 1.0, "thr": 0.2, "max_size": 6},
        # the benchmark's workload: 20 million points, 100 features
        {"name": "large_20m", "kind": "mine", "n": 20000000, "features": 100, "density": "region", "form": "learned",
         "reach": 1.0, "thr": 0.15, "max_size": 0},
        # a short distance over a wide extent: more than 2^32 grid cells (64-bit cell keys)
        {"name": "sparse_2m", "kind": "mine", "n": 2000003, "features": 60, "density": "wide", "form": "batched",
         "reach": 1.0, "thr": 0.1, "max_size": 0},
        # dense clusters without a size cap: tens of millions of instance-table rows
        {"name": "dense_200k", "kind": "mine", "n": 200000, "features": 200, "density": "dense", "form": "learned",
         "reach": 1.0, "thr": 0.1, "max_size": 0},
        # points that stay in host memory and are read by each mine
        {"name": "host_4m", "kind": "host", "n": 4000000, "features": 100, "density": "region", "form": "learned",
         "reach": 1.0, "thr": 0.15, "max_size": 0},
        # a caller that reads the instance tables too
        {"name": "tables_700k", "kind": "tables", "n": 700001, "features": 40, "density": "town", "form": "batched",
         "reach": 1.0, "thr": 0.2, "max_size": 6},
        # what the command-line program does: a CSV file in, patterns out
        {"name": "csv_1m", "kind": "csv", "n": 1000000, "features": 40, "density": "town", "form": "batched",
         "reach": 1.0, "thr": 0.2, "max_size": 6},
        # many independent jobs of ragged sizes in one call
        {"name": "batch_128", "kind": "batch", "jobs": 128, "form": "learned"},
        # one gradient of the cost model over the rows it was trained on
        {"name": "model_205k", "kind": "model", "n": 205545},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mine", "mine", "mine", "mine", "host", "tables", "csv", "batch", "model"])
    if kind == "model":
        return {"kind": kind, "n": _log_uniform(rng, 100, 250_000)}
    form = rng.choice(["batched", "learned"])
    if kind == "batch":
        return {"kind": kind, "jobs": _log_uniform(rng, 2, 128), "form": form}
    density = rng.choice(["town", "town", "region", "region", "wide", "dense"]) if kind == "mine" else \
        rng.choice(["town", "region"])
    top = {"mine": 20_000_000, "host": 6_000_000, "tables": 1_000_000, "csv": 1_500_000}[kind]
    lo, hi, most = {"town": (1_000, 2_000_000, 64), "region": (20_000, 20_000_000, 160),
                    "wide": (50_000, 4_000_000, 100), "dense": (60_000, 200_000, 220)}[density]
    n = _log_uniform(rng, lo, min(hi, top))
    features = max(8, min(most, _log_uniform(rng, 8, most), n // 100))
    if density == "dense":   # rows grow with the power of a feature's points in a cluster: as many features as listed
        features = rng.randrange(200, 221)
    return {"kind": kind, "n": n, "features": features,
            "density": density, "form": form,
            "reach": 1.0 if density == "dense" else round(rng.uniform(0.6, 1.4), 3),
            "thr": rng.choice([0.1, 0.15, 0.2, 0.3]), "max_size": rng.choice([0, 0, 4, 6])}


def _points(case, seed):
    """(workload, distance): the case's points, at the density of one of the generator's configurations."""
    base = {"small": 0, "town": 1, "region": 3, "wide": 3, "dense": 4}[case["density"]]
    spec, R, _, _ = gen.spec_config(base, seed)
    scale = case["n"] / spec.n
    if base:
        spec.n, spec.nfeat = case["n"], case["features"]
        spec.width *= math.sqrt(scale)
        spec.nhot = max(1, round(spec.nhot * scale))
        spec.ndense = max(1, round(spec.ndense * scale)) if spec.ndense else 0
        spec.pat_max = min(spec.pat_max, spec.nfeat)
    if case["density"] == "wide":
        # the whole domain whatever the size, and a reach that makes more than 2^32 cells of it
        spec.width, R = 1e6, 14.0
        spec.pat_sigma = 0.3 * R
    R = float(np.float32(R * case["reach"]))
    return gen.generate(spec, "case", R, case["thr"], case["max_size"]), R


_ctx = None


def _context():
    """The program's context: one for all its datasets, with the trained cost model installed."""
    global _ctx
    if _ctx is None:
        _ctx = colo.Context(0)
        _ctx.set_model(colo.load_model())
    return _ctx


def _params(case, R, thr, max_size):
    return colo.default_params(R, thr, colo.MODE_LEARNED if case["form"] == "learned" else colo.MODE_BATCHED,
                               max_size=max_size, keep_tables=case["kind"] == "tables")


def _model_rows(case, seed):
    """Feature rows in the ranges that mining meets (log counts and their ratios), and log1p(rows) targets."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, 12.0, (case["n"], colo.MODEL_FEATURES)).astype(np.float32)
    x[:, 0] = rng.integers(2, 8, case["n"]) / 8
    return colo.init_model(seed), x, (0.5 * x[:, 1] + 0.5 * x[:, 9]).astype(np.float32)


def prepare(case, seed):
    ctx = _context()
    state = {"kind": case["kind"], "ctx": ctx, "room": _room(case)}
    if case["kind"] == "model":
        state["args"] = _model_rows(case, seed)
        return state
    if case["kind"] == "batch":
        jobs = gen.config2_jobs(case["jobs"], seed)
        state["ds"] = [ctx.dataset(j.x, j.y, j.fid, j.bounds) for j in jobs]
        state["params"] = [_params(case, j.R, j.thr, j.max_size) for j in jobs]
        return state
    wl, R = _points(case, seed)
    ds = ctx.dataset(wl.x, wl.y, wl.fid, wl.bounds)
    state["params"] = _params(case, R, case["thr"], case["max_size"])
    if case["kind"] == "csv":
        state["dir"] = tempfile.TemporaryDirectory(prefix="colo_case_")
        state["path"] = os.path.join(state["dir"].name, "points.csv")
        ds.write_csv(state["path"])
        return state
    if case["kind"] != "host":
        ds.upload()
    state["ds"] = ds
    return state


def _room(case):
    """Values that a result buffer holds: (per candidate, per member of a candidate, in instance tables).  Every seed
    has its own number of candidates above the pairs; a program that keeps result buffers sizes them once."""
    if case["kind"] == "model":
        return None
    jobs, features = (case["jobs"], 32) if case["kind"] == "batch" else (1, case["features"])
    pairs = jobs * features * (features - 1) // 2
    return 2 * pairs + 4096, 6 * pairs + 16384, (2 * case["n"] + 65536 if case["kind"] == "tables" else 0)


def _whole(parts, size, dtype):
    """The parts end to end at the front of a zeroed buffer."""
    out, at = np.zeros(size, dtype), 0
    for p in parts:
        out[at:at + p.size] = p.ravel()   # raises when the buffer is too small
        at += p.size
    return out


def _flat(results, room):
    """Every candidate of every level and job: each field end to end (a mine has too many levels for one array each)."""
    per_candidate, per_member, in_tables = room
    levels = [lev for r in results for lev in r.levels]
    out = {}
    for f in FIELDS:
        parts = [getattr(lev, f) for lev in levels]
        dtype = parts[0].dtype if parts else np.uint32
        out[f] = _whole(parts, per_member if f in ("cand", "ub", "num") else per_candidate, dtype)
    if in_tables:
        out["tables"] = _whole([t for lev in levels for t in lev.tables.values()], in_tables, np.uint32)
    return out


def run(state):
    ctx = state["ctx"]
    if state["kind"] == "model":
        grad, loss = ctx.model_grad(*state["args"])
        return {"grad": grad, "loss": loss}
    if state["kind"] == "batch":
        results = ctx.mine_batch(state["ds"], state["params"])
    elif state["kind"] == "csv":
        results = [ctx.mine(colo.Dataset.from_csv(ctx, state["path"], device=True), state["params"])]
    else:
        results = [ctx.mine(state["ds"], state["params"])]
    return _flat(results, state["room"])


def work(case):
    """Bytes: the points read once, the pairs' results written once (larger patterns depend on the data)."""
    if case["kind"] == "model":
        weights = colo.MODEL_FEATURES * 64 + 64 * 64 + 64
        return {"bytes": 4 * (case["n"] * (colo.MODEL_FEATURES + 1) + 2 * colo.MODEL_PARAMS),
                "flops": 6 * weights * case["n"]}
    if case["kind"] == "batch":   # 2,000 to 400,000 points a job (log-uniform), 8 to 32 features
        return {"bytes": case["jobs"] * (8 * 75_000 + 58 * 190), "flops": 0}
    pairs = case["features"] * (case["features"] - 1) // 2
    return {"bytes": (26 if case["kind"] == "csv" else 8) * case["n"] + 58 * pairs, "flops": 0}


# ---- the same in plain numpy, 64 bits ---------------------------------------------------------------------------


def exact(case, seed):
    if case["kind"] == "model":
        return _model_exact(*_model_rows(case, seed))
    if case["kind"] != "mine" or case["n"] > EXACT_POINTS or case["density"] not in ("town", "small"):
        return None
    wl, R = _points(case, seed)
    out = dict.fromkeys(FIELDS)
    pi = _mine_pi(wl, np.float32(R), np.float32(case["thr"]), case["max_size"])
    out["pi"] = _whole([pi], _room(case)[0], np.float64)
    return out


def _model_exact(params, x, t):
    p, x, t = params.astype(np.float64), x.astype(np.float64), t.astype(np.float64)
    x = np.hstack([x, np.zeros((len(x), 8))])
    at = np.cumsum([32 * 64, 64, 64 * 64, 64, 64])
    w1, b1, w2, b2, w3, b3 = np.split(p, at)
    w1, w2 = w1.reshape(32, 64), w2.reshape(64, 64)
    h1 = np.maximum(x @ w1 + b1, 0)
    h2 = np.maximum(h1 @ w2 + b2, 0)
    d = h2 @ w3 + b3 - t
    g = d / len(x)
    d2 = np.outer(g, w3) * (h2 > 0)
    d1 = (d2 @ w2.T) * (h1 > 0)
    grad = np.concatenate([(x.T @ d1).ravel(), d1.sum(0), (h1.T @ d2).ravel(), d2.sum(0), h2.T @ g, [g.sum()]])
    return {"grad": grad, "loss": float(0.5 * np.mean(d * d))}


def _expand(start, count):
    """Indices start[i] .. start[i] + count[i] - 1 end to end, and each one's i."""
    owner = np.repeat(np.arange(len(count)), count)
    first = np.cumsum(count) - count
    return np.arange(int(count.sum())) - first[owner] + start[owner], owner


def _mine_pi(wl, R, thr, max_size):
    """PI of every candidate of every level (-1: stopped by the filter): the level-wise miner over the reference's
    grid, quad filter, participation windows and join order, for grids of at least three columns."""
    x, y, fid, F = wl.x, wl.y, wl.fid, wl.nfeat
    start = np.searchsorted(fid, np.arange(F + 1))
    count = np.diff(start)
    b = wl.bounds
    gx = int(np.ceil((b[2] - b[0]) / R))
    gy = int(np.ceil(((b[3] + R) - b[1]) / R))
    cx, cy = ((x - b[0]) / R).astype(np.int64), ((y - b[1]) / R).astype(np.int64)
    key = cy * gx + cx
    order = np.argsort(key, kind="stable")
    skey = key[order]
    # neighbours b of a with a higher feature, by (a, b)
    pa, pb = [], []
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            ok = (cx + dx >= 0) & (cx + dx < gx) & (cy + dy >= 0) & (cy + dy < gy)
            a = np.flatnonzero(ok)
            k = key[a] + dy * gx + dx
            lo = np.searchsorted(skey, k)
            at, own = _expand(lo, np.searchsorted(skey, k, side="right") - lo)
            pa.append(a[own])
            pb.append(order[at])
    pa, pb = np.concatenate(pa), np.concatenate(pb)

    def within(i, j):
        d2 = (x[j] - x[i]).astype(np.float64) ** 2 + (y[j] - y[i]).astype(np.float64) ** 2
        return d2.astype(np.float32) <= R * R

    keep = fid[pb] > fid[pa]
    pa, pb = pa[keep], pb[keep]
    keep = within(pa, pb)
    pa, pb = pa[keep], pb[keep]
    by = np.lexsort((pb, fid[pb], pa))
    pa, pb = pa[by], pb[by]
    code = pa * F + fid[pb]     # ascending: the neighbours of point p with feature f are one range
    # points of each feature per grid cell, and the features of each 2x2 block
    cells = np.zeros((F, gy, gx), np.int32)
    np.add.at(cells, (fid, cy, cx), 1)
    has = cells > 0
    quad = has[:, :-1, :-1] | has[:, :-1, 1:] | has[:, 1:, :-1] | has[:, 1:, 1:]

    def passes(c):
        full = np.logical_and.reduce(quad[list(c[:8])])
        u = np.zeros((gy, gx), bool)
        u[:-1, :-1] |= full
        u[:-1, 1:] |= full
        u[1:, :-1] |= full
        u[1:, 1:] |= full
        ub = [int(cells[f][u].sum()) if i < 8 else 0 for i, f in enumerate(c)]
        return min(np.float32(v / float(np.float32(count[f]))) for v, f in zip(ub, c)) >= thr

    def ratio(c, table):
        k = len(c)
        bits = []
        for j, f in enumerate(c):
            m = np.zeros(count[f], bool)
            m[table[:, j] - start[f]] = True
            bits.append(m)
        win = [int(m[:-1].sum()) for m in bits]
        last = [int(m[-1]) for m in bits]
        if k == 2:
            first = int(bits[1][0])
            num = [win[0], int(bits[1].sum()) - first + (1 if first or last[0] else 0)]
        else:
            num = [win[0]] + [last[t - 1] + win[t] for t in range(1, k)]
        return min([1.0] + [v / count[f] for v, f in zip(num, c)])

    cands = [(i, j) for i in range(F) for j in range(i + 1, F)]
    tables = {(f,): np.arange(start[f], start[f + 1])[:, None] for f in range(F)}
    pi = []
    while cands:
        k = len(cands[0])
        new, prevalent = {}, []
        for c in cands:
            if not passes(c):
                pi.append(-1.0)
                continue
            t = tables[c[:-1]]
            want = t[:, 0] * F + c[-1]
            lo = np.searchsorted(code, want)
            at, own = _expand(lo, np.searchsorted(code, want, side="right") - lo)
            rows = np.column_stack([t[own], pb[at]])
            ok = np.ones(len(rows), bool)
            for j in range(1, k - 1):
                ok &= within(rows[:, j], rows[:, k - 1])
            rows = rows[ok]
            pi.append(ratio(c, rows))
            if not np.float32(pi[-1]) < thr:
                prevalent.append(c)
                new[c] = rows
        tables = new
        cands, have = [], set(prevalent)
        if (max_size and k + 1 > max_size) or k + 1 > F:
            break
        for i, p in enumerate(prevalent):
            for q in prevalent[i + 1:]:
                if p[:-1] != q[:-1]:
                    break
                c = p + q[-1:]
                if any(c[:d] + c[d + 1:] not in have for d in range(k - 2, -1, -1)):
                    break
                cands.append(c)
    return np.array(pi, np.float64)
