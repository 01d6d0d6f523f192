"""The work that users of this library have it do, as cases that can be timed.

A case is a dict of plain values.  ``prepare`` makes what a program has in
hand before the call (its preference lists, its batch or server handle),
``run`` is one pass through the public Python API, ``work`` the bytes a pass
cannot do without.  All outputs are whole numbers: the man-optimal matching of
an instance is unique, so they are right or wrong, never close.

The paths, and the ranges they are used over:

  solve   one instance on the device, n from 64 to 30000, over the workload
          families: uniform, congested (the men share one list), correlated
          (a common score plus noise), and the reference's own PERFECT,
          CONGESTED, RANDOM(g) and SOLO
  host    the same from numpy arrays: both lists are in host memory and the
          matching comes back to it
  batch   many independent instances of uneven size in one call
  serve   a burst of requests through the serving loop, until all have their
          matching
  invert  the women's int32 rank matrix alone (the reference's init study)
  check   the stability checker on a finished matching
"""
from __future__ import annotations

import atexit
import math

import numpy as np
import torch

import pactae_b200 as pb

# workload families: generator kind and parameter
KINDS = {
    "uniform": (pb.SMP_GEN_UNIFORM, 0),
    "congested": (pb.SMP_GEN_CONGESTED, 0),
    "correlated": (pb.SMP_GEN_CORRELATED, 500),  # noise sigma 0.05
    "perfect": (pb.SMP_GEN_PERFECT, 0),
    "ref_congested": (pb.SMP_GEN_REF_CONGESTED, 0),
    "random5": (pb.SMP_GEN_GROUPED, 5),
    "solo": (pb.SMP_GEN_SOLO, 0),
}
MIX = ("uniform", "congested", "correlated")  # by the kind number of a seeded mix

_held: dict = {}


def _context() -> pb.Context:
    """The process's solver context: a program makes one and keeps it."""
    if "ctx" not in _held:
        _held["ctx"] = pb.Context()
    return _held["ctx"]


def _server() -> pb.Server:
    """The process's serving loop, started once."""
    if "server" not in _held:
        _held["server"] = pb.Server()
    return _held["server"]


@atexit.register
def _close() -> None:
    for name in ("server", "ctx"):
        if name in _held:
            _held.pop(name).close()


def listed() -> list[dict]:
    return [
        # the smallest call: a handful of people, where only latency counts
        {"name": "solve_uniform_97", "path": "solve", "kind": "uniform", "n": 97},
        # the reference's CPU-sized instance
        {"name": "solve_uniform_2000", "path": "solve", "kind": "uniform", "n": 2000},
        # the headline instance: 7.2 GB of lists
        {"name": "solve_uniform_30000", "path": "solve", "kind": "uniform", "n": 30000},
        # contention: every man has the same list
        {"name": "solve_congested_30000", "path": "solve", "kind": "congested", "n": 30000},
        # contention: common scores with noise, men go deep into their lists
        {"name": "solve_correlated_30000", "path": "solve", "kind": "correlated", "n": 30000},
        # the reference's RANDOM(5) family, at an odd size
        {"name": "solve_random5_15013", "path": "solve", "kind": "random5", "n": 15013},
        # the reference's SOLO family: one displacement chain, an odd size (the women numbered at random)
        {"name": "solve_solo_10007", "path": "solve", "kind": "solo", "n": 10007},
        # lists in host memory, an odd size, end to end
        {"name": "host_uniform_16411", "path": "host", "kind": "uniform", "n": 16411},
        # the uneven mix of many instances, n log-uniform in [16, 4096]
        {"name": "batch_mix_1024", "path": "batch", "count": 1024, "n_lo": 16, "n_hi": 4096, "mix": 5},
        # a burst of requests, n log-uniform in [64, 16384]
        {"name": "serve_burst_48", "path": "serve", "count": 48, "n_lo": 64, "n_hi": 16384, "mix": 6},
        # the rank matrix of one side, an odd size
        {"name": "invert_20011", "path": "invert", "kind": "uniform", "n": 20011},
        # a matching verified: blocking pairs and proposals counted
        {"name": "check_correlated_12007", "path": "check", "kind": "correlated", "n": 12007},
    ]


def _log_uniform(rng, lo: int, hi: int) -> int:
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    path = rng.choice(("solve", "solve", "solve", "host", "batch", "serve", "invert", "check"))
    if path == "batch":
        n_hi = _log_uniform(rng, 256, 4096)
        return {"path": path, "count": _log_uniform(rng, 32, 1024), "n_lo": 16, "n_hi": n_hi,
                "mix": rng.randrange(1 << 20)}
    if path == "serve":
        n_hi = _log_uniform(rng, 1024, 16384)
        return {"path": path, "count": _log_uniform(rng, 8, 48), "n_lo": 64, "n_hi": n_hi,
                "mix": rng.randrange(1 << 20)}
    if path == "invert":
        return {"path": path, "kind": "uniform", "n": _log_uniform(rng, 256, 20011)}
    if path == "check":
        return {"path": path, "kind": rng.choice(("uniform", "correlated")), "n": _log_uniform(rng, 256, 12007)}
    if path == "host":
        return {"path": path, "kind": rng.choice(("uniform", "uniform", "congested", "correlated")),
                "n": _log_uniform(rng, 64, 12007)}
    kind = rng.choice(("uniform", "uniform", "congested", "correlated", "perfect", "ref_congested", "random5", "solo"))
    top = {"random5": 15013, "solo": 10007}.get(kind, 30000)
    return {"path": path, "kind": kind, "n": _log_uniform(rng, 64, top)}


def _mix(case: dict) -> list[tuple[int, str]]:
    """The sizes and families of a batch's or a burst's instances."""
    metas = [pb.batch_instance(case["mix"], b, case["n_lo"], case["n_hi"]) for b in range(case["count"])]
    return [(n, MIX[kind]) for n, kind in metas]


def _lists(kind: str, n: int, seed: int, salt: int = 0, device: bool = True):
    code, param = KINDS[kind]
    pref_m, pref_w = _context().generate(code, n, seed, salt=salt, param=param, device=device)
    if kind == "solo":  # its matching is the same for every seed: number the women at random
        gen = torch.Generator(device="cuda").manual_seed(seed)
        number = torch.randperm(n, generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
        pref_m = number[pref_m.to(torch.int64)]
        pref_w = pref_w[torch.argsort(number)]
    return pref_m, pref_w


def prepare(case: dict, seed: int) -> dict:
    path = case["path"]
    state = {"path": path}
    if path in ("batch", "serve"):
        state["instances"] = [
            (*_lists(kind, n, seed, salt=b), torch.empty(n, dtype=torch.int32, device="cuda"))
            for b, (n, kind) in enumerate(_mix(case))
        ]
        if path == "batch":
            state["batch"] = pb.Batch(_context(), state["instances"])
        else:
            state["server"] = _server()
        return state
    state["ctx"] = _context()
    state["pref_m"], state["pref_w"] = _lists(case["kind"], case["n"], seed, device=path != "host")
    if path == "check":
        state["match"], _ = state["ctx"].solve(state["pref_m"], state["pref_w"])
    return state


def run(state: dict):
    path = state["path"]
    if path in ("solve", "host"):
        match, stats = state["ctx"].solve(state["pref_m"], state["pref_w"])
        return {"match": match, "proposals": stats["proposals"]}
    if path == "batch":
        status, proposals, _ = state["batch"].run()
        return {"match": _joined(state), "status": np.array(status), "proposals": np.array(proposals)}
    if path == "serve":
        server = state["server"]
        tickets = [server.submit(pm, pw, mt) for pm, pw, mt in state["instances"]]
        results = [server.poll(t) for t in tickets]
        return {"match": _joined(state), "status": np.array([r["status"] for r in results]),
                "proposals": np.array([r["proposals"] for r in results])}
    if path == "invert":
        return state["ctx"].invert(state["pref_w"])
    blocking, proposals = state["ctx"].check(state["pref_m"], state["pref_w"], state["match"])
    return {"blocking": blocking, "proposals": proposals}


def _joined(state: dict) -> torch.Tensor:
    """The matchings of all instances, one after another."""
    return torch.cat([mt for _, _, mt in state["instances"]])


def work(case: dict) -> dict:
    """Each preference list read once, each output written once."""
    if case["path"] in ("batch", "serve"):
        return {"bytes": sum(8 * n * n + 4 * n for n, _ in _mix(case)), "flops": 0}
    n = case["n"]
    return {"bytes": 8 * n * n + 4 * n, "flops": 0}


def exact(case: dict, seed: int):
    """The same outputs from plain Python or torch, where that is quick."""
    path = case["path"]
    if path == "invert":
        pref_w = _lists(case["kind"], case["n"], seed)[1].to(torch.int64)
        ranks = torch.arange(case["n"], device="cuda").expand_as(pref_w)
        return torch.empty_like(pref_w).scatter_(1, pref_w, ranks).to(torch.int32)
    if path in ("solve", "host") and case["kind"] == "uniform" and case["n"] <= 2500:
        pref_m, pref_w = _lists(case["kind"], case["n"], seed, device=False)
        match, proposals = _gale_shapley(pref_m, pref_w)
        return {"match": torch.from_numpy(match).cuda() if path == "solve" else match, "proposals": proposals}
    return None


def _gale_shapley(pref_m: np.ndarray, pref_w: np.ndarray) -> tuple[np.ndarray, int]:
    n = pref_m.shape[0]
    rank = np.empty_like(pref_w)
    np.put_along_axis(rank, pref_w, np.arange(n, dtype=np.int32)[None, :], axis=1)
    husband = [-1] * n
    at = [0] * n
    free = list(range(n))
    proposals = 0
    while free:
        m = free.pop()
        while True:
            w = int(pref_m[m, at[m]])
            at[m] += 1
            proposals += 1
            h = husband[w]
            if h < 0 or rank[w, m] < rank[w, h]:
                husband[w] = m
                if h >= 0:
                    free.append(h)
                break
    match = np.empty(n, dtype=np.int32)
    for w, m in enumerate(husband):
        match[m] = w
    return match, proposals
