"""Seeded LP (method 5) on the degree tiers, per iteration against the oracle:
rows at every tier's edges and hubs, seeds and unlabelled regions in each,
weights with zeros (a labelled neighbour of weight 0 still is a candidate)."""
import numpy as np
import pytest

from glp_b200 import _lib
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import from_numpy
from oracle import oracle as O
from tests.graphs_fixtures import degree_ladder, rmat_np

pytestmark = pytest.mark.gpu

LADDER = [1, 8, 9, 16, 17, 32, 33, 128, 129, 256, 257, 1024, 1025, 2049, 4097, 8193, 12289, 24577]
TIERS = {"default": {}, "small_hubs": dict(mid_max=64, big_max=256, hub_chunk=256)}


@pytest.mark.parametrize("share", [0.0005, 0.3])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("tiers", sorted(TIERS))
@pytest.mark.parametrize("graph", ["ladder", "rmat13"])
def test_seeded_tiers_per_iteration(graph, tiers, weighted, share):
    off, cols = degree_ladder(LADDER) if graph == "ladder" else rmat_np(13, seed=8)[:2]
    n = len(off) - 1
    rng = np.random.default_rng(7)
    w = rng.integers(0, 3, size=len(cols)).astype(np.int32) if weighted else None
    seeds = rng.random(n) < share
    seeds[:len(LADDER):3] = True  # seeds among the large rows too
    trace = []
    with Graph(from_numpy(off, cols, w)) as g:
        g.set_seeds(seeds)
        res = g.run(_lib.METHOD_SEEDED, 6, make_params(**TIERS[tiers]),
                    callback=lambda it, lab: trace.append(lab) and False)
    _, want = O.seeded_run(off, cols, seeds, 6, w=w, trace=True)
    prev = np.where(seeds, np.arange(n), -1)
    for it in range(6):
        np.testing.assert_array_equal(trace[it], want[it], err_msg=f"iteration {it}")
        assert res.changed[it] == np.count_nonzero(want[it] != prev)
        prev = want[it]
