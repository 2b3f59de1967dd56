"""The launches that graphs above a million vertices take, against the oracle
after every iteration.  A core graph with every degree class is padded with
disjoint triangles (which make the plan a large graph's at little cost, and
settle in three steps) or with isolated vertices (which grow the label arrays
alone)."""
import functools

import numpy as np
import pytest
import torch

from glp_b200 import _lib
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import from_numpy
from oracle import oracle as O

pytestmark = pytest.mark.gpu

UNMERGED, RINGS = 360_000, 700_000  # triangles: more than 2^20, 2^21 vertices


@functools.lru_cache(maxsize=None)
def _core(order, seed=4):
    """Symmetric, rows strictly ascending: 2300 vertices of degree about 257..400
    (more than a merged plan has), sixteen of 1100..9000, one of 26000, and 30,000
    of up to 60 in groups whose labels repeat."""
    rng = np.random.default_rng(seed)
    dense, sparse = 2300, 30000
    mids = [1100, 1500, 2047, 2049, 2600, 3300, 4096, 4097, 5200, 6000, 7000, 8192, 8193, 8700, 9000, 12300]
    hubs = dense + sparse
    n = hubs + len(mids) + 1
    us = [np.repeat(np.arange(dense), 250), dense + np.repeat(np.arange(sparse), rng.integers(1, 26, sparse))]
    vs = [rng.integers(0, dense // 4, len(us[0])) + us[0] // (dense // 4) * (dense // 4) % dense,
          dense + (us[1] - dense) // 60 * 60 + rng.integers(0, 60, len(us[1]))]
    for i, d in enumerate([*mids, 26000]):
        us.append(np.full(d, hubs + i))
        vs.append(dense + rng.choice(sparse, d, replace=False))
    u, v = np.concatenate(us), np.concatenate(vs)
    keep = (u != v) & (v < n)
    u, v = u[keep], v[keep]
    key = np.unique(np.concatenate([u * n + v, v * n + u]))
    rank = rng.permutation(n)
    if order == "sorted":
        rank[np.argsort(-np.bincount(key // n, minlength=n), kind="stable")] = np.arange(n)
    key = np.sort(rank[key // n] * n + rank[key % n])
    return np.bincount(key // n, minlength=n), key % n


def _graph(order, triangles=0, isolated=0):
    deg, cols = _core(order)
    n = len(deg)
    ends = n + (3 * np.arange(triangles)[:, None] + [1, 2, 0, 2, 0, 1]).ravel()
    deg = np.concatenate([deg, np.full(3 * triangles, 2), np.zeros(isolated, np.int64)])
    if order == "sorted":  # the core's own vertices of degree 1 and 0 end up behind the triangles
        order_ = np.argsort(-deg, kind="stable")
        rank = np.empty(len(deg), np.int64)
        rank[order_] = np.arange(len(deg))
        row = np.repeat(np.arange(len(deg)), deg)
        key = np.sort(rank[row] * len(deg) + rank[np.concatenate([cols, ends])])
        deg, cols = deg[order_], key % len(deg)
    else:
        cols = np.concatenate([cols, ends])
    return (np.concatenate([[0], np.cumsum(deg)]).astype(np.int32), cols.astype(np.int32))


def _weights(off, cols):
    """0..3, and 1 in rows of two, so that the triangles settle."""
    w = np.random.default_rng(5).integers(0, 4, len(cols)).astype(np.int32)
    w[np.repeat(np.diff(off) == 2, np.diff(off))] = 1
    return w


@functools.lru_cache(maxsize=2)
def _padded(order, triangles):
    return _graph(order, triangles)


def _trace(off, cols, w, method, niter, seeds=None, **opts):
    trace = []
    with Graph(from_numpy(off, cols, w)) as g:
        if seeds is not None:
            g.set_seeds(seeds)
        g.run(method, niter, make_params(**opts), callback=lambda it, lab: trace.append(lab) and False)
    return np.array(trace)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("order,triangles", [("sorted", RINGS), ("mixed", RINGS), ("sorted", UNMERGED)])
def test_layered_per_iteration(order, triangles, weighted):
    off, cols = _padded(order, triangles)
    w = _weights(off, cols) if weighted else None
    got = _trace(off, cols, w, _lib.METHOD_LAYERED, 3, dstar=[2, 9])
    _, _, want = O.layered_run(off, cols, [2, 9], 3, w=w, trace=True)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("triangles", [0, UNMERGED])
def test_layered_pairs_beyond_the_cache(triangles):
    """(label, volume) pairs past a quarter of the L2: degrees 17..32 gather the
    labels alone."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    off, cols = _graph("sorted", triangles, isolated=l2 // 32 + 1000)
    got = _trace(off, cols, None, _lib.METHOD_LAYERED, 2, dstar=[2, 17])
    _, _, want = O.layered_run(off, cols, [2, 17], 2, trace=True)
    np.testing.assert_array_equal(got, want)


def test_weighted_layered_pairs_beyond_the_whole_cache():
    """(label, volume) pairs past the L2: the small tiers follow the big tier."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    off, cols = _graph("sorted", isolated=l2 // 8 + 1000)
    w = _weights(off, cols)
    with Graph(from_numpy(off, cols, w)) as g:
        got = g.run(_lib.METHOD_LAYERED, 3, make_params(dstar=[3]))
    want, vol = O.layered_run(off, cols, [3], 3, w=w)[:2]
    np.testing.assert_array_equal(got.labels, want)
    np.testing.assert_array_equal(got.vol, vol)


METHODS = {"classic": (_lib.METHOD_CLASSIC, dict(cycle_stop=-1)), "wide": (_lib.METHOD_LAYERED, dict(dstar=[65536])),
           "seeded": (_lib.METHOD_SEEDED, {})}


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("method", sorted(METHODS))
def test_unmerged_tiers_per_iteration(method, order, weighted):
    """Three small tiers and a launch per big range: full-count steps of each
    score, and (classic) majority and frontier steps with their three lists."""
    off, cols = _padded(order, UNMERGED)
    w = _weights(off, cols) if weighted else None
    m, opts = METHODS[method]
    niter = 10 if method == "classic" else 4
    seeds = None
    if method == "seeded":
        seeds = np.random.default_rng(6).random(len(off) - 1) < 0.05
    got = _trace(off, cols, w, m, niter, seeds, **opts)
    if method == "classic":
        _, want = O.classic_run(off, cols, niter, w=w, trace=True)
        n = len(off) - 1
        changed = [np.count_nonzero(want[it] != want[it - 1]) for it in (1, 2)]
        assert n < 20 * changed[0] < 10 * n and 20 * changed[1] < n  # a majority step, then frontier steps
    elif method == "wide":
        _, _, want = O.layered_run(off, cols, opts["dstar"], niter, w=w, trace=True)
    else:
        _, want = O.seeded_run(off, cols, seeds, niter, w=w, trace=True)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("order", ["sorted", "mixed"])
def test_tiny_max_selects_the_small_tiers(order):
    """A graph below 2^20 vertices counts degrees 1..32 in one launch, except
    where tiny_max is given: then the tiers are those of glp_graph_plan."""
    off, cols = _graph(order, triangles=50)
    with Graph(from_numpy(off, cols)) as g:
        res = {t: g.run(_lib.METHOD_CLASSIC, 3, make_params(tiny_max=t, serial_step=1, majority_permille=1,
                                                            frontier_permille=-1), profile=True)
               for t in (0, 4, 8, -1)}
    for t, r in res.items():
        np.testing.assert_array_equal(r.labels, res[0].labels)
        tiny, group16, group32 = r.step_tier_ms[2][:3]
        assert group32 > 0
        assert (tiny > 0) == (t > 0) and (group16 > 0) == (t != 0), (t, tiny, group16)


@pytest.mark.parametrize("weighted", [False, True])
def test_classic_labels_beyond_the_cache(weighted):
    """Labels past a quarter of the L2: the hubs are counted after the big tier."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    off, cols = _graph("sorted", isolated=l2 // 16 + 1000)
    w = _weights(off, cols) if weighted else None
    with Graph(from_numpy(off, cols, w)) as g:
        for niter in (2, 5):
            got = g.run(_lib.METHOD_CLASSIC, niter, make_params(majority_permille=1, frontier_permille=-1))
            np.testing.assert_array_equal(got.labels, O.classic_run(off, cols, niter, w=w))
