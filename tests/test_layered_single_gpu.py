"""Layered LP's table-free labels (volume 1 among the step's labels, rows that
list no neighbour twice): every tier and the hubs, weighted and not, against
the oracle after every iteration; and rows with repeated neighbours, where a
label of volume 1 occurs more than once and must be counted."""
import numpy as np
import pytest

from glp_b200 import _lib, graphs
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import from_numpy
from oracle import oracle as O
from tests.graphs_fixtures import csr_from_adj, degree_ladder, rmat_np

pytestmark = pytest.mark.gpu

TIERS = {"default": {}, "small_hubs": dict(mid_max=64, big_max=256, hub_chunk=256)}


def _repeated():
    """Every neighbour up to three times, degrees to 900: not strictly ascending."""
    rng = np.random.default_rng(2)
    return csr_from_adj([sorted(np.repeat(rng.integers(0, 3000, d), rng.integers(1, 4, d)).tolist())
                         for d in rng.choice([3, 20, 60, 150, 300], 3000)])


GRAPHS = {"ladder": lambda: degree_ladder([40, 64, 65, 200, 256, 257, 700, 1500, 3000, 5000, 12289, 24577]),
          "rmat13": lambda: rmat_np(13, seed=4)[:2], "repeated": _repeated}


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("tiers", sorted(TIERS))
@pytest.mark.parametrize("graph", sorted(GRAPHS))
def test_layered_per_iteration(graph, tiers, weighted):
    off, cols = GRAPHS[graph]()
    w = np.random.default_rng(5).integers(0, 4, len(cols)).astype(np.int32) if weighted else None
    trace = []
    with Graph(from_numpy(off, cols, w)) as g:
        res = g.run(_lib.METHOD_LAYERED, 4, make_params(dstar=[2, 9], **TIERS[tiers]),
                    callback=lambda it, lab: trace.append(lab) and False)
    _, vol, want = O.layered_run(off, cols, [2, 9], 4, w=w, trace=True)
    np.testing.assert_array_equal(np.array(trace), want)
    np.testing.assert_array_equal(res.vol, vol)
