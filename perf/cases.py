"""The work a program built on pmdd_b200 has the GPU do, as cases to be timed.

Each case is one call, or one short sequence of calls, into the package's public entry
points, from host data to sorted frontiers on the host:

* ``dd``     -- one decision diagram through ``enumerate_dd`` (upload included), the
                call the command line makes: knapsack, set packing, methods 1 and 3,
                with and without state dominance;
* ``tsp``    -- TSP instances given by their cost matrices (``ResidentSet.from_tsp`` once,
                then ``enumerate``);
* ``stream`` -- many knapsack and set-packing diagrams advanced together from a resident
                set, the batched workload;
* ``build``  -- knapsack instances whose diagrams are built on the device and enumerated
                in the same pass (``ResidentSet.from_knapsack``);
* ``served`` -- a mixed request list submitted to the serving loop and polled until done;
* ``filter`` -- the standalone Pareto filter of one point set.

The instances are those of ``pmdd_b200.instances`` (profits, weights and costs U[1,1000],
set-packing objectives U[1,100] with 20 constraints), sized as the repository's benchmark
and tests size them.  Frontiers come back in no fixed order, so every pass sorts them the
way the command line does before it writes them, into rows of a fixed number (zeros behind
the frontier, its length beside it).
"""
from __future__ import annotations

import concurrent.futures as cf

import numpy as np

import pmdd_b200 as P
from pmdd_b200 import instances

SETPACKING_ROWS = 20


def listed():
    return [
        # the smallest solve a caller makes: launches, copies and the host step decide
        {"name": "kp3_n20", "kind": "dd", "ptype": 1, "nobjs": 3, "n": 20, "method": 1, "sd": 0},
        # many thin layers: a hundred dependent steps with a few thousand candidates each
        {"name": "sp3_n100", "kind": "dd", "ptype": 2, "nobjs": 3, "n": 100, "method": 1, "sd": 0},
        # set packing with label pruning between the nodes of a layer, odd size
        {"name": "sp3_n91_sd", "kind": "dd", "ptype": 2, "nobjs": 3, "n": 91, "method": 1, "sd": 1},
        # seven objectives: high-dimensional filters of middling size
        {"name": "kp7_n25", "kind": "dd", "ptype": 1, "nobjs": 7, "n": 25, "method": 1, "sd": 0},
        # the large single instance, top-down: most destinations outgrow shared memory
        {"name": "kp4_n60", "kind": "dd", "ptype": 1, "nobjs": 4, "n": 60, "method": 1, "sd": 0},
        # the same instance from both ends, joined at the cutset
        {"name": "kp4_n60_m3", "kind": "dd", "ptype": 1, "nobjs": 4, "n": 60, "method": 3, "sd": 0},
        # three-objective TSP by the coupled method, the served mix's largest city count
        {"name": "tsp3_n13_m3", "kind": "tsp", "nobjs": 3, "n": 13, "method": 3, "count": 1},
        # five-objective TSP, top-down: few very large destinations of high dimension
        {"name": "tsp5_n13", "kind": "tsp", "nobjs": 5, "n": 13, "method": 1, "count": 1},
        # the batched stream, a quarter of the benchmark's list (two knapsacks per set packing)
        {"name": "stream_192", "kind": "stream", "count": 192},
        # a caller with many fresh knapsacks: diagrams built on the device, then solved
        {"name": "build_kp3_64", "kind": "build", "nobjs": 3, "count": 64},
        # the serving loop on a burst of the mixed request list
        {"name": "served_48", "kind": "served", "count": 48},
        # the standalone filter of one large candidate set
        {"name": "filter4_32768", "kind": "filter", "nobjs": 4, "n": 32768},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["dd", "dd", "dd", "dd", "tsp", "tsp", "stream", "build", "served", "filter", "filter"])
    if kind == "dd":
        if rng.random() < 0.6:
            d = rng.choice([3, 3, 4, 5, 7])
            n = rng.randint(20, {3: 60, 4: 60, 5: 32, 7: 25}[d])
            return {"kind": "dd", "ptype": 1, "nobjs": d, "n": n, "method": rng.choice([1, 3]),
                    "sd": 1 if d == 3 and rng.random() < 0.3 else 0}
        d = rng.choice([3, 3, 4])
        return {"kind": "dd", "ptype": 2, "nobjs": d, "n": rng.randint(60, 100 if d == 3 else 80),
                "method": rng.choice([1, 3]), "sd": rng.choice([0, 0, 1])}
    if kind == "tsp":
        d = rng.choice([3, 3, 4, 5])
        return {"kind": "tsp", "nobjs": d, "n": rng.randint(9, 13 if d < 5 else 12), "method": rng.choice([1, 3]),
                "count": rng.choice([1, 1, 7])}
    if kind == "stream":
        return {"kind": "stream", "count": _log_int(rng, 9, 192)}
    if kind == "build":
        return {"kind": "build", "nobjs": rng.choice([3, 3, 4]), "count": _log_int(rng, 3, 32)}
    if kind == "served":
        return {"kind": "served", "count": _log_int(rng, 8, 48)}
    d = rng.choice([2, 3, 4, 5, 7])
    return {"kind": "filter", "nobjs": d, "n": _log_int(rng, 100, 65537 if d < 5 else 16385)}


# ------------------------------------------------------------------ instances
def _dd_text(ptype, nobjs, n, seed):
    if ptype == 1:
        return instances.knapsack_text(n, nobjs, seed)
    return instances.setpacking_text(n, SETPACKING_ROWS, nobjs, seed)


def _build_all(specs):
    with cf.ThreadPoolExecutor(8) as ex:
        return list(ex.map(lambda s: P.DecisionDiagram.from_text(*s), specs))


def _stream_specs(count, seed):
    """Two knapsacks (n ~ U{20..60}) for every set packing (n ~ U{60..100})."""
    kp = count - count // 3
    return [(text, ptype, 3) for ptype, text, _ in instances.stream_mix(kp, count - kp, 3, seed0=1000 * seed)]


def _build_instances(case, seed):
    """Knapsacks with n ~ U{20..60} (n ~ U{20..40} above three objectives)."""
    rng = np.random.default_rng(20_000 + seed)
    hi = 61 if case["nobjs"] == 3 else 41
    return [instances.knapsack_arrays(int(rng.integers(20, hi)), case["nobjs"], 1000 * seed + i)
            for i in range(case["count"])]


def _filter_points(case, seed):
    """Points of a shell around a concave front, as the candidates of a destination lie."""
    rng = np.random.default_rng(30_000 + seed)
    g = np.abs(rng.standard_normal((case["n"], case["nobjs"])))
    g /= np.linalg.norm(g, axis=1, keepdims=True)
    r = 50_000 * (1 - 0.3 * rng.random(case["n"]))
    return np.rint(g * r[:, None]).astype(np.int32)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": dict(case)}
    if kind == "dd":
        text = _dd_text(case["ptype"], case["nobjs"], case["n"], 1000 * seed)
        s["dd"] = P.DecisionDiagram.from_text(text, case["ptype"], case["nobjs"])
    elif kind == "tsp":
        costs = [instances.tsp_arrays(case["n"], case["nobjs"], 1000 * seed + i) for i in range(case["count"])]
        s["set"] = P.ResidentSet.from_tsp(costs)
    elif kind == "stream":
        s["set"] = P.ResidentSet(_build_all(_stream_specs(case["count"], seed)))
    elif kind == "build":
        s["instances"] = _build_instances(case, seed)
    elif kind == "served":
        mix = instances.served_mix(case["count"], seed)
        dds = iter(_build_all([(text, p, 3) for p, text, _, _ in mix if p != 3]))
        s["requests"] = [(p, instances.tsp_arrays_from_tag(tag) if p == 3 else next(dds), method)
                         for p, text, method, tag in mix]
        s["server"] = P.Server(budget_bytes=16 << 30)
        for n in sorted({r[1].shape[1] for r in s["requests"] if r[0] == 3}):
            s["server"].prepare_tsp(n)
    else:
        s["points"] = _filter_points(case, seed)
    return s


# ----------------------------------------------------------------- one pass
def _rows(case):
    """Rows that hold every frontier of the case's ranges."""
    if case["kind"] == "filter":
        return case["n"]
    if case["kind"] in ("stream", "served", "build"):
        return 4096 * case["count"]
    return (16384 if case["nobjs"] <= 3 else 131072) * case.get("count", 1)


def _padded(case, pts, count):
    out = np.zeros((_rows(case), pts.shape[1]), dtype=pts.dtype)
    out[:len(pts)] = pts
    return {"points": out, "count": np.asarray(count, dtype=np.int64)}


def _sorted_one(case, pts):
    return _padded(case, P.sort_lexicographic_ascending(pts), [len(pts)])


def _sorted_set(case, frontiers):
    """The frontiers of several instances as one sorted array and their lengths."""
    count = [len(f) for f in frontiers]
    pts = np.concatenate(frontiers)
    owner = np.repeat(np.arange(len(frontiers)), count)
    return _padded(case, pts[np.lexsort(tuple(pts.T[::-1]) + (owner,))], count)


def _serve(server, requests):
    for i, (ptype, what, method) in enumerate(requests):
        if ptype == 3:
            server.submit_tsp(what, i, method=method)
        else:
            server.submit(what, i, method=method)
    got = [None] * len(requests)
    left = len(requests)
    while left:
        server.run()
        while (r := server.poll()) is not None:
            if r.status != 0:
                raise RuntimeError(f"request {r.req_id}: {r.error}")
            got[r.req_id] = r.frontier
            left -= 1
    return got


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dd":
        pts = P.enumerate_dd(state["dd"], method=case["method"], state_dominance=case["sd"])
        return _sorted_one(case, pts)
    if kind == "tsp":
        return _sorted_set(case, state["set"].enumerate(method=case["method"]))
    if kind == "stream":
        return _sorted_set(case, state["set"].enumerate(method=1))
    if kind == "build":
        built = P.ResidentSet.from_knapsack(state["instances"])
        out = _sorted_set(case, built.enumerate(method=1))
        built.close()
        return out
    if kind == "served":
        return _sorted_set(case, _serve(state["server"], state["requests"]))
    return _sorted_one(case, P.pareto_filter(state["points"]))


# --------------------------------------------------------------- what it needs
def _dd_work(dds, method, sd):
    """(bytes, ops) of enumerating each diagram: its arcs read once, every layer's
    candidate points read and surviving points written once, one addition per candidate
    coordinate and join-product coordinate."""
    b = f = 0
    for dd in dds:
        st = {}
        P.enumerate_dd(dd, method=method, state_dominance=sd, stats=st)
        d = dd.nobjs
        b += 8 * dd.num_arcs + 4 * d * (st["work_candidates_total"] + st["work_frontier_survivors_total"])
        f += d * (st["work_candidates_total"] + st["work_join_products_total"])
    return b, f


def work(case):
    """Bytes and operations of one pass on the instances of one fixed seed."""
    kind = case["kind"]
    seed = 1
    if kind == "dd":
        b, f = _dd_work([prepare(case, seed)["dd"]], case["method"], case["sd"])
    elif kind in ("tsp", "stream"):
        s = prepare(case, seed)["set"]
        st = {}
        s.enumerate(method=case.get("method", 1), stats=st)
        arcs = sum(s.dd_info(i)["num_arcs"] for i in range(s.count))
        d = case.get("nobjs", 3)
        b = 8 * arcs + 4 * d * (st["work_candidates_total"] + st["work_frontier_survivors_total"])
        f = d * (st["work_candidates_total"] + st["work_join_products_total"])
    elif kind == "build":
        s = P.ResidentSet.from_knapsack(_build_instances(case, seed))
        st = {}
        s.enumerate(method=1, stats=st)
        d = case["nobjs"]
        # the diagrams' arcs are written once and read once
        b = 16 * sum(s.dd_info(i)["num_arcs"] for i in range(s.count))
        b += 4 * d * (st["work_candidates_total"] + st["work_frontier_survivors_total"])
        f = d * st["work_candidates_total"]
    elif kind == "served":
        b = f = 0
        for ptype, text, method, _ in instances.served_mix(case["count"], seed):
            got = _dd_work([P.DecisionDiagram.from_text(text, ptype, 3)], method, 0)
            b, f = b + got[0], f + got[1]
    else:
        n, d = case["n"], case["nobjs"]
        b, f = 8 * n * d, n * d
    return {"bytes": b, "flops": f}


# -------------------------------------------------------------------- exact
def _maxima(pts):
    """Maximal points under componentwise >=, one copy of each, in decreasing order of
    the objective sum block by block: a point's dominators never have a smaller sum."""
    pts = np.unique(pts, axis=0)
    pts = pts[np.argsort(-pts.sum(axis=1), kind="stable")]
    keep = pts[:0]
    for i in range(0, len(pts), 256):
        b = pts[i:i + 256]
        for j in range(0, len(keep), 4096):
            b = b[~(keep[None, j:j + 4096] >= b[:, None]).all(axis=2).any(axis=1)]
        ge = (b[None] >= b[:, None]).all(axis=2)
        np.fill_diagonal(ge, False)
        keep = np.concatenate([keep, b[~ge.any(axis=1)]])
    return keep


def _exact_rows(case, pts):
    return _padded(case, pts[np.lexsort(pts.T[::-1])], [len(pts)])


def _exact_knapsack(profits, weights, cap):
    """Item by item over (used capacity, profits) labels, dominated labels dropped."""
    d, n = profits.shape
    labels = np.zeros((1, d + 1), dtype=np.int64)  # minus the used capacity, profits
    for i in range(n):
        add = labels + np.concatenate([[-weights[i]], profits[:, i]]).astype(np.int64)
        labels = _maxima(np.concatenate([labels, add[add[:, 0] >= -cap]]))
    return _maxima(labels[:, 1:])


def exact(case, seed):
    if case["kind"] == "filter" and case["n"] <= 32768:
        return _exact_rows(case, _maxima(_filter_points(case, seed).astype(np.int64)))
    if case["kind"] == "dd" and case["ptype"] == 1 and case["n"] <= 20 and case["nobjs"] <= 3:
        return _exact_rows(case, _exact_knapsack(*instances.knapsack_arrays(case["n"], case["nobjs"], 1000 * seed)))
    return None
