"""Performance cases: label-propagation solves as user programs call them.

Every case is one call (or one short sequence of calls) through the public
Python entry points of ``glp_b200``, on graphs from the package's own
samplers.  All outputs are whole numbers (labels, change counts, vertex ids),
so two builds have to agree on them exactly.

* ``solve``: a resident ``Graph`` handle and one ``run`` of a method, labels
  left in the caller's device tensor;
* ``batch``: many small graphs packed in a ``Batch``, one ``run``;
* ``build``: ``Graph.from_edges`` on an edge list in device memory, then a
  short classic solve on the graph it built;
* ``oneshot``: ``run_method`` on a CSR in host memory: handle, solve, labels
  back on the host.

``work`` counts each input read once and each output written once.  The
solves are iterative: one that counts every vertex in each of its steps reads
the columns once per step, so a graph larger than the L2 cannot reach that
figure.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from glp_b200 import _lib, graphs
from glp_b200.batch import Batch
from glp_b200.engine import Graph, make_params, run_method

METHODS = {"classic": _lib.METHOD_CLASSIC, "layered": _lib.METHOD_LAYERED, "slpa": _lib.METHOD_SLPA,
           "user": _lib.METHOD_USER, "seeded": _lib.METHOD_SEEDED}
HOOKS = {"classic": _lib.HOOKS_CLASSIC, "layered": _lib.HOOKS_LAYERED, "degree": _lib.HOOKS_WEIGHTED_DEGREE}
GAMMAS = (1.0, 1 / 2, 1 / 4, 1 / 8, 1 / 16)  # the five layers of the layered solve


def _rmat(scale: int, edge_factor: int) -> dict:
    return {"graph": "rmat", "scale": scale, "edge_factor": edge_factor}


def _planted(n: int, k: int, intra: float, inter: float) -> dict:
    return {"graph": "planted", "n": n, "k": k, "intra": intra, "inter": inter}


def _overlap(n: int, k: int, deg: float) -> dict:
    return {"graph": "overlap", "n": n, "k": k, "overlap": 0.1, "deg": deg}


def _solve(method: str, graph: dict, niter: int, **options) -> dict:
    return {"call": "solve", "method": method, **graph, "niter": niter, "weighted": False, "sorted": True, **options}


def listed() -> list[dict]:
    return [
        # a small social graph solved again and again while it is explored:
        # every step is microseconds of work
        {"name": "classic-rmat16", **_solve("classic", _rmat(16, 16), 20)},
        # the headline workload: communities of a large skewed graph
        {"name": "classic-rmat24", **_solve("classic", _rmat(24, 16), 20)},
        # a large graph without hubs and with clear communities
        {"name": "classic-planted10m", **_solve("classic", _planted(10_000_000, 1000, 18.0, 2.0), 20)},
        # interaction counts as edge weights, on a skewed graph
        {"name": "classic-weighted-rmat22", **_solve("classic", _rmat(22, 16), 20, weighted=True)},
        # multi-resolution communities (graph reordering): five layers
        {"name": "layered-rmat22", **_solve("layered", _rmat(22, 16), 10)},
        # the same over edge weights; vertex ids as they came, not degree-sorted
        {"name": "layered-weighted-planted", **_solve("layered", _planted(2_000_003, 200, 18.0, 2.0), 10,
                                                       weighted=True, sorted=False)},
        # overlapping communities with speaker memory
        {"name": "slpa-overlap2m", **_solve("slpa", _overlap(2_000_000, 2000, 24.0), 20)},
        # semi-supervised labelling: a few known vertices on a skewed graph
        {"name": "seeded-rmat20", **_solve("seeded", _rmat(20, 16), 10, seed_share=0.02)},
        # a user's own score: FP64 degree-normalised votes through the hooks
        {"name": "user-degree-rmat20", **_solve("user", _rmat(20, 16), 10, hooks="degree")},
        # many small graphs at once (ego networks, molecules, per-user graphs)
        {"name": "batch-256", "call": "batch", "count": 256, "mix": 1, "niter": 20},
        # raw edges of the day's log to a graph and its first communities
        {"name": "build-rmat22", "call": "build", **_rmat(22, 16), "keep_ids": False, "niter": 3},
        # the command line's whole job: a CSR on the host in, labels out
        {"name": "oneshot-planted200k", "call": "oneshot", "method": "classic", **_planted(200_003, 100, 18.0, 2.0),
         "niter": 20, "weighted": False},
    ]


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_rmat(rng, scales: tuple[int, int], samples: int) -> dict:
    """A scale of the range and an edge factor (odd ones too), at most 2^samples edge samples."""
    scale = rng.randint(*scales)
    return _rmat(scale, int(round(_log_uniform(rng, 4, min(48, 2 ** (samples - scale))))))


def _draw_planted(rng, n_max: int) -> dict:
    n = int(_log_uniform(rng, 3000, n_max))
    deg = _log_uniform(rng, 8.0, 20.0)
    intra = round(deg * rng.uniform(0.7, 0.95), 2)
    return _planted(n, max(4, int(n / _log_uniform(rng, 200, 10000))), intra, round(deg - intra, 2))


def draw(rng) -> dict:
    kind = rng.choice(("classic", "classic", "weighted", "layered", "layered", "slpa", "seeded", "user", "batch",
                       "build", "oneshot"))
    srt = rng.random() < 0.7
    if kind == "classic":
        g = _draw_rmat(rng, (12, 23), 28) if rng.random() < 0.5 else _draw_planted(rng, 8_000_000)
        return _solve("classic", g, rng.randint(5, 20), sorted=srt)
    if kind == "weighted":
        g = _draw_rmat(rng, (12, 21), 26) if rng.random() < 0.5 else _draw_planted(rng, 3_000_000)
        return _solve("classic", g, rng.randint(5, 20), weighted=True, sorted=srt)
    if kind == "layered":
        weighted = rng.random() < 0.4
        g = (_draw_rmat(rng, (12, 21), 25 if weighted else 26) if rng.random() < 0.5
             else _draw_planted(rng, 2_000_000))
        return _solve("layered", g, rng.randint(3, 10), weighted=weighted, sorted=srt)
    if kind == "slpa":
        n = int(_log_uniform(rng, 5000, 2_000_000))
        return _solve("slpa", _overlap(n, max(4, n // rng.randint(300, 2000)), round(rng.uniform(8.0, 24.0), 1)),
                      rng.randint(5, 20), sorted=srt)
    if kind == "seeded":
        g = _draw_rmat(rng, (12, 20), 24) if rng.random() < 0.5 else _draw_planted(rng, 1_500_000)
        return _solve("seeded", g, rng.randint(3, 10), weighted=rng.random() < 0.3, sorted=srt,
                      seed_share=round(_log_uniform(rng, 0.002, 0.2), 4))
    if kind == "user":
        hooks = rng.choice(sorted(HOOKS))
        top = 21 if hooks == "layered" else 24  # five layers
        g = _draw_rmat(rng, (12, top - 4), top) if rng.random() < 0.5 else _draw_planted(rng, 2 ** (top - 4))
        return _solve("user", g, rng.randint(3, 10), weighted=rng.random() < 0.3, sorted=srt, hooks=hooks)
    if kind == "batch":
        return {"call": "batch", "count": int(_log_uniform(rng, 4, 220)), "mix": rng.randint(2, 1000),
                "niter": rng.randint(5, 20)}
    if kind == "build":
        g = _draw_rmat(rng, (12, 22), 26) if rng.random() < 0.5 else _draw_planted(rng, 4_000_000)
        return {"call": "build", **g, "keep_ids": rng.random() < 0.3, "niter": rng.randint(1, 3)}
    g = _draw_rmat(rng, (12, 16), 20) if rng.random() < 0.5 else _draw_planted(rng, 200_000)
    return {"call": "oneshot", "method": rng.choice(("classic", "layered", "slpa")), **g, "niter": rng.randint(5, 20),
            "weighted": rng.random() < 0.3}


def _edges(case: dict, seed: int):
    """The case's edge sample on the device, and its vertex count."""
    if case["graph"] == "rmat":
        return (*graphs.sample_rmat(case["scale"], case["edge_factor"], seed, device="cuda"), 1 << case["scale"])
    if case["graph"] == "planted":
        return (*graphs.sample_planted(case["n"], case["k"], case["intra"], case["inter"], seed, device="cuda"),
                case["n"])
    return (*graphs.sample_overlap(case["n"], case["k"], case["overlap"], case["deg"], seed, device="cuda"),
            case["n"])


def _csr(case: dict, seed: int) -> graphs.CSR:
    src, dst, n = _edges(case, seed)
    g = graphs.build_csr(src, dst, n, relabel=case.get("sorted", True))
    return graphs.add_weights(g, 16, seed) if case["weighted"] else g


def prepare(case: dict, seed: int) -> dict:
    call = case["call"]
    state = {"call": call, "niter": case["niter"]}
    if call == "solve":
        g = _csr(case, seed)
        state.update(method=METHODS[case["method"]], handle=Graph(g),
                     labels=torch.empty(g.n, dtype=torch.int32, device="cuda"))
        options = {"gammas": GAMMAS}
        if case["method"] == "slpa":
            options.update(slpa_T=case["niter"], seed=seed)
        if case["method"] == "user":
            options.update(hooks=HOOKS[case["hooks"]])
        if case["method"] == "seeded":
            state["handle"].set_seeds(np.random.default_rng(seed).random(g.n) < case["seed_share"])
        state["params"] = make_params(**options)
    elif call == "batch":
        # the mix fixes every graph's size, the seed its edges
        batch = Batch([graphs.planted(s["n"], s["k"], s["intra"], s["inter"], seed * 1000 + i, device="cuda")
                       for i, s in enumerate(graphs.batch_specs(case["count"], case["mix"]))])
        state.update(batch=batch, labels=torch.empty(batch.n, dtype=torch.int32, device="cuda"))
    elif call == "build":
        src, dst, n = _edges(case, seed)
        state.update(src=src, dst=dst, n=n, keep_ids=case["keep_ids"],
                     labels=torch.empty(n, dtype=torch.int32, device="cuda"))
    else:
        state.update(method=METHODS[case["method"]], csr=_csr(case, seed).to("cpu"),
                     params=make_params(gammas=GAMMAS, slpa_T=case["niter"], seed=seed))
    return state


def run(state: dict) -> dict:
    call, niter = state["call"], state["niter"]
    if call == "solve":
        r = state["handle"].run(state["method"], niter, state["params"], labels_out=state["labels"])
        return {"labels": r.labels, "changed": r.changed}
    if call == "batch":
        labels, changed = state["batch"].run(niter, labels_out=state["labels"])
        return {"labels": labels, "changed": changed}
    if call == "build":
        g, old_id = Graph.from_edges(state["src"], state["dst"], state["n"], keep_ids=state["keep_ids"])
        with g:
            r = g.run(_lib.METHOD_CLASSIC, niter, labels_out=state["labels"])
        return {"labels": r.labels, "changed": r.changed, "old_id": old_id}
    r = run_method(state["method"], state["csr"], niter, state["params"])
    out = {"labels": r.labels, "changed": r.changed}
    if r.vol is not None:  # layered
        out["vol"] = r.vol
    if r.slpa_comm is not None:
        out.update(comm=r.slpa_comm, ncomm=r.slpa_ncomm, mem=r.slpa_mem)
    return out


def _size(case: dict) -> tuple[float, float]:
    """(vertices, CSR entries) to be expected: both directions of every edge sample."""
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        return n, 2.0 * case["edge_factor"] * n
    return case["n"], case["n"] * (case["intra"] + case["inter"] if case["graph"] == "planted" else case["deg"])


def work(case: dict) -> dict:
    if case["call"] == "batch":  # log-uniform sizes 1000..200000 and mean degrees 4..64
        n = case["count"] * (200000 - 1000) / math.log(200.0)
        m = n * (64 - 4) / math.log(16.0)
    else:
        n, m = _size(case)
    total = 4 * (n + 1) + 4 * m + 4 * n  # offsets and columns in, labels out
    if case.get("weighted"):
        total += 4 * m
    if case["call"] == "build":
        total = 4 * m + 8 * n  # both ends of m / 2 edges in, labels and old ids out
    if case.get("method") == "seeded":
        total += n
    return {"bytes": total, "flops": 0}


def exact(case: dict, seed: int):
    """None: the outputs are whole numbers, equal bit for bit or wrong."""
    return None
