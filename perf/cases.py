"""Performance cases: the searches a user of this package runs, through its public calls.

A case is one user-visible pass, from host instance arrays to host results (``noalloc``:
device buffers to device buffers, as that call is defined).  Kinds:

``solve``     ``Context.solve_batch`` of one instance with ``beams`` seeded beams that share
              one bound group: a single search, or the ranks of a multi-start as beams.
``rounds``    ``Context.solve_iterations``: the multi-start driver, bound carried over.
``batch``     ``Context.solve_batch`` of many instances of uneven sizes and beam widths.
``served``    a burst of requests to a running ``Server``: all submitted, then all awaited.
``noalloc``   ``bsj_solve_noalloc``: one search on the caller's buffers and stream.

Instances have the shape of the Lawrence / Taillard families: every job visits every
machine once in a random order, durations U[1, 99].  A case fixes sizes, modes and widths;
the seed fixes machine orders, durations and search seeds.  Every output is a whole
number: makespans, schedules and counters of exact searches.
"""
import ctypes
import math

import numpy as np
import torch

from beamsearch_jssp_gpu_gb300 import BeamSpec, Context, Server
from beamsearch_jssp_gpu_gb300 import _native as nat

NO_BOUND = 500000

# a program keeps one context and one server for all of its searches
_kept = {}


def _context():
    if "ctx" not in _kept:
        _kept["ctx"] = Context(0)
    return _kept["ctx"]


def _server():
    if "srv" not in _kept:
        _kept["srv"] = Server(0, max_inflight=96)
    return _kept["srv"]


def listed():
    return [
        # the smallest call: BS-ICH on a 10x5 instance at the CPU solver's own widths
        {"name": "ich_10x5_K64", "kind": "solve", "mode": "ich", "n": 10, "m": 5, "K": 64, "beams": 1},
        # an interactive solve of a Lawrence-size instance: launches and latency
        {"name": "v2_15x15_K256", "kind": "solve", "mode": "v2", "n": 15, "m": 15, "K": 256, "beams": 1},
        # run_gpu_beam_search_v1 as its caller does: one instance, one beam, K=1024
        {"name": "v1_20x15_K1024", "kind": "solve", "mode": "v1", "n": 20, "m": 15, "K": 1024, "beams": 1},
        # the top of the beam-width sweep, v1's stored child slots included
        {"name": "v1_20x15_K16384", "kind": "solve", "mode": "v1", "n": 20, "m": 15, "K": 16384, "beams": 1},
        # an operator that owns its memory and stream: device buffers in and out
        {"name": "noalloc_30x20_K1000", "kind": "noalloc", "mode": "v2", "n": 30, "m": 20, "K": 1000},
        # the multi-start driver: 3 ranks, 4 rounds, an odd size and width
        {"name": "rounds_37x11_K1500", "kind": "rounds", "mode": "clean", "n": 37, "m": 11, "K": 1500, "beams": 3,
         "rounds": 4},
        # one wide search of a Taillard-size instance
        {"name": "v2_50x20_K4096", "kind": "solve", "mode": "v2", "n": 50, "m": 20, "K": 4096, "beams": 1},
        # eight ranks as beams of one launch: the benchmark's workload
        {"name": "v2_50x20_K4096_b8", "kind": "solve", "mode": "v2", "n": 50, "m": 20, "K": 4096, "beams": 8},
        # the same at the largest benchmarked instance
        {"name": "v2_100x20_K4096_b8", "kind": "solve", "mode": "v2", "n": 100, "m": 20, "K": 4096, "beams": 8},
        # exact BS-PMS, eight ranks
        {"name": "pms_30x20_K1024_b8", "kind": "solve", "mode": "pms", "n": 30, "m": 20, "K": 1024, "beams": 8},
        # many instances of uneven size in one call
        {"name": "batch_96", "kind": "batch", "count": 96, "mix": 1},
        # requests that overlap on a running server, mixed sizes, widths and branching
        {"name": "served_40", "kind": "served", "count": 40, "mix": 1},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "rounds", "noalloc", "batch", "served"])
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 8, 96), "mix": rng.randrange(2, 1 << 20)}
    if kind == "served":
        return {"kind": kind, "count": _log_int(rng, 4, 40), "mix": rng.randrange(2, 1 << 20)}
    if kind == "noalloc":
        # the scratch array bounds beam width times operations
        n, m = _log_int(rng, 6, 60), rng.randrange(4, 21)
        per = 2 * (4 * m + 6 * n + 48) + 12 * n + 4 * n * m + 64
        return {"kind": kind, "mode": rng.choice(["v2", "clean"]), "n": n, "m": m,
                "K": _log_int(rng, 32, min(8192, (48 << 20) // per))}
    if kind == "rounds":
        n, m = _log_int(rng, 6, 60), rng.randrange(3, 21)
        return {"kind": kind, "mode": rng.choice(["v1", "v2", "clean"]), "n": n, "m": m, "K": _log_int(rng, 32, 4096),
                "beams": rng.randrange(2, 9), "rounds": rng.randrange(2, 5)}
    mode = rng.choice(["v1", "v2", "v2", "clean", "clean", "ich", "pms"])
    if mode == "ich":
        return {"kind": kind, "mode": mode, "n": _log_int(rng, 5, 20), "m": rng.randrange(2, 16),
                "K": _log_int(rng, 16, 256), "beams": rng.randrange(1, 5)}
    if mode == "pms":
        return {"kind": kind, "mode": mode, "n": _log_int(rng, 5, 30), "m": rng.randrange(2, 21),
                "K": _log_int(rng, 16, 1024), "beams": rng.randrange(1, 9)}
    n, m, beams = _log_int(rng, 5, 100), rng.randrange(2, 21), rng.choice([1, 1, 1, 2, 3, 4, 8])
    top = 16384 if beams * n <= 200 else 4096
    return {"kind": kind, "mode": mode, "n": n, "m": m, "K": _log_int(rng, 32, top), "beams": beams}


def _instances(sizes, seed):
    """Machine orders and durations of instances of the given sizes."""
    g = np.random.default_rng(seed)
    out = []
    for n, m in sizes:
        mc = np.argsort(g.random((n, m)), axis=1).astype(np.int32)
        out.append((mc, g.integers(1, 100, (n, m), dtype=np.int32)))
    return out, g


def _mixed(case):
    """(n, m, mode, K) of every search of a ``batch`` or ``served`` case."""
    g = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        if case["kind"] == "batch":
            out.append((int(g.choice([10, 15, 20, 30, 50, 100])), int(g.choice([5, 10, 15, 20])), "v2",
                        int(g.choice([256, 512, 1024, 4096]))))
            continue
        n, m = int(g.choice([15, 20, 30, 50, 100])), int(g.choice([15, 20]))
        mode = str(g.choice(["v2", "clean", "v2", "clean", "pms"]))
        if mode == "pms":   # exact branching: its heap is serial, so requests of it stay small
            out.append((min(n, 30), m, mode, 256))
        else:
            out.append((n, m, mode, int(g.choice([256, 1024, 4096]))))
    return out


def _warm_server(srv, shapes):
    """Before traffic a server builds the plans of the shapes it expects, once."""
    ready = _kept.setdefault("ready", {})
    want = {}
    for s in shapes:
        want[s] = want.get(s, 0) + 1
    target = srv.stats()["plans_prepared"]
    for s in sorted(want):
        n, m, mode, K = s
        more = want[s] - ready.get(s, 0)
        if more > 0:
            (inst,), _ = _instances([(n, m)], 0)
            srv.prepare(inst[0], inst[1], mode, K, copies=more)
            ready[s] = want[s]
            target += more
    while srv.stats()["plans_prepared"] < target:
        pass


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "served"):
        shapes = _mixed(case)
        insts, g = _instances([(n, m) for n, m, _, _ in shapes], seed)
        seeds = [int(x) for x in g.integers(0, 1 << 30, len(shapes))]
        if kind == "served":
            srv = _server()
            _warm_server(srv, shapes)
            reqs = [(mc, du, s[2], s[3], sd) for (mc, du), s, sd in zip(insts, shapes, seeds)]
            return {"case": case, "srv": srv, "reqs": reqs}
        beams = [BeamSpec(s[2], s[3], NO_BOUND, sd, i, -1) for i, (s, sd) in enumerate(zip(shapes, seeds))]
        return {"case": case, "ctx": _context(), "insts": insts, "beams": beams}
    insts, g = _instances([(case["n"], case["m"])], seed)
    if kind == "noalloc":
        mc, du = (torch.from_numpy(x).cuda() for x in insts[0])
        out = torch.empty(2 + case["n"] * case["m"], dtype=torch.int32, device="cuda")
        return {"case": case, "lib": nat.load(), "machine": mc, "duration": du, "out": out,
                "seed": int(g.integers(0, 1 << 30))}
    if kind == "rounds":
        return {"case": case, "ctx": _context(), "inst": insts[0],
                "seeds": g.integers(0, 1 << 30, (case["rounds"], case["beams"]))}
    seeds = [int(x) for x in g.integers(0, 1 << 30, case["beams"])]
    beams = [BeamSpec(case["mode"], case["K"], NO_BOUND, sd, 0, 0) for sd in seeds]
    return {"case": case, "ctx": _context(), "insts": insts, "beams": beams}


def _arrays(results):
    """Result dicts as arrays: one value per search, and all schedules end to end."""
    keys = [k for k in ("makespan", "found", "expanded", "slots", "levels", "group_best") if k in results[0]]
    out = {k: np.array([int(r[k]) for r in results], dtype=np.int64) for k in keys}
    out["schedules"] = np.concatenate([r["seq"] for r in results])
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "served":
        srv = state["srv"]
        tickets = [srv.submit(*r) for r in state["reqs"]]
        return _arrays([srv.wait(t) for t in tickets])
    if kind == "noalloc":
        p = ctypes.c_void_p
        rc = state["lib"].bsj_solve_noalloc(
            case["n"], case["m"], p(state["machine"].data_ptr()), p(state["duration"].data_ptr()),
            nat.MODES[case["mode"]], case["K"], NO_BOUND, state["seed"], p(state["out"].data_ptr()),
            p(torch.cuda.current_stream().cuda_stream))
        if rc != nat.BSJ_OK:
            raise nat.BsjError(rc, "bsj_solve_noalloc")
        return state["out"]
    if kind == "rounds":
        best, seq, per_round = state["ctx"].solve_iterations(*state["inst"], case["mode"], case["K"], state["seeds"])
        return {"best": best, "schedule": seq, "per_round": per_round}
    return _arrays(state["ctx"].solve_batch(state["insts"], state["beams"]))


def work(case):
    """Bytes: every instance read and every result written once, and one 4-byte lineage word
    per survivor and level, which the schedule is read back from.  Operations: a survivor's
    ready operations are tested for the pivot machine (or branched on) at every level."""
    if case["kind"] in ("batch", "served"):
        searches = [(n, m, K) for n, m, _, K in _mixed(case)]
    else:
        searches = [(case["n"], case["m"], case["K"])] * (case.get("beams", 1) * case.get("rounds", 1))
    b = sum(8 * n * m + 4 * n * m + 4 * n * m * K for n, m, K in searches)
    return {"bytes": b, "flops": sum(n * m * K * n for n, m, K in searches)}


def exact(case, seed):
    """Whole numbers only: there is no rounding to measure."""
    return None
