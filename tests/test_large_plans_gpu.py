"""The launches that graphs above a million vertices take, against the oracle
after every iteration.  A core graph with every degree class is padded with
disjoint edges (which make the plan a large graph's at little cost) or with
isolated vertices (which grow the label arrays alone)."""
import functools

import numpy as np
import pytest
import torch

from glp_b200 import _lib
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import from_numpy
from oracle import oracle as O

pytestmark = pytest.mark.gpu

UNMERGED, RINGS = 560_000, 1_060_000  # disjoint edges: more than 2^20, 2^21 vertices


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
    if order == "sorted":
        rank = np.empty(n, np.int64)
        rank[np.argsort(-np.bincount(key // n, minlength=n), kind="stable")] = np.arange(n)
        key = np.sort(rank[key // n] * n + rank[key % n])
    return np.bincount(key // n, minlength=n), key % n


def _graph(order, pairs=0, isolated=0):
    deg, cols = _core(order)
    n = len(deg)
    ends = n + (np.arange(2 * pairs) ^ 1)
    deg = np.concatenate([deg, np.ones(2 * pairs, np.int64), np.zeros(isolated, np.int64)])
    if order == "sorted":  # the core's own vertices of degree 1 and 0 end up behind the pairs
        order_ = np.argsort(-deg, kind="stable")
        rank = np.empty(len(deg), np.int64)
        rank[order_] = np.arange(len(deg))
        row = np.repeat(np.arange(len(deg)), deg)
        key = np.sort(rank[row] * len(deg) + rank[np.concatenate([cols, ends])])
        deg, cols = deg[order_], key % len(deg)
    else:
        cols = np.concatenate([cols, ends])
    return (np.concatenate([[0], np.cumsum(deg)]).astype(np.int32), cols.astype(np.int32))


def _weights(cols, wmax=3):
    return np.random.default_rng(5).integers(0, wmax + 1, len(cols)).astype(np.int32)


@functools.lru_cache(maxsize=2)
def _padded(order, pairs):
    return _graph(order, pairs)


def _trace(off, cols, w, method, niter, seeds=None, **opts):
    trace = []
    with Graph(from_numpy(off, cols, w)) as g:
        if seeds is not None:
            g.set_seeds(seeds)
        g.run(method, niter, make_params(**opts), callback=lambda it, lab: trace.append(lab) and False)
    return np.array(trace)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("order,pairs", [("sorted", RINGS), ("mixed", RINGS), ("sorted", UNMERGED)])
def test_layered_per_iteration(order, pairs, weighted):
    off, cols = _padded(order, pairs)
    w = _weights(cols) if weighted else None
    got = _trace(off, cols, w, _lib.METHOD_LAYERED, 3, dstar=[2, 9])
    _, _, want = O.layered_run(off, cols, [2, 9], 3, w=w, trace=True)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("pairs", [0, UNMERGED])
def test_layered_pairs_beyond_the_cache(pairs):
    """(label, volume) pairs past a quarter of the L2: degrees 17..32 gather the
    labels alone."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    off, cols = _graph("sorted", pairs, isolated=l2 // 32 + 1000)
    got = _trace(off, cols, None, _lib.METHOD_LAYERED, 2, dstar=[2, 17])
    _, _, want = O.layered_run(off, cols, [2, 17], 2, trace=True)
    np.testing.assert_array_equal(got, want)


def test_weighted_layered_pairs_beyond_the_whole_cache():
    """(label, volume) pairs past the L2: the small tiers follow the big tier."""
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    off, cols = _graph("sorted", isolated=l2 // 8 + 1000)
    w = _weights(cols)
    with Graph(from_numpy(off, cols, w)) as g:
        got = g.run(_lib.METHOD_LAYERED, 3, make_params(dstar=[3]))
    want, vol = O.layered_run(off, cols, [3], 3, w=w)[:2]
    np.testing.assert_array_equal(got.labels, want)
    np.testing.assert_array_equal(got.vol, vol)
