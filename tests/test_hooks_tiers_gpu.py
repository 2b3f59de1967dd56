"""Method 4 at the edges of the hook kernel's row classes (eight lanes, a warp
with one chunk, a warp with a table, a block with a shared table, a block with
a spill table): FP64 frequencies against a plain restatement that sums them
in the documented order, so labels must be equal after every iteration."""
import numpy as np
import pytest

from glp_b200 import _lib, graphs
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import from_numpy
from tests.graphs_fixtures import degree_ladder, star, undirected

pytestmark = pytest.mark.gpu


def _restate(off, cols, w, lab):
    deg = np.diff(off).astype(np.float64)
    new = lab.copy()
    for v in np.nonzero(np.diff(off))[0]:
        acc = {}
        for c0 in range(off[v], off[v + 1], 32):
            chunk = {}
            for j in range(c0, min(c0 + 32, off[v + 1])):
                u = cols[j]
                chunk[lab[u]] = chunk.get(lab[u], 0.0) + (1.0 if w is None else float(w[j])) / deg[u]
            for l, s in chunk.items():
                acc[l] = acc.get(l, 0.0) + s
        new[v] = max(acc.items(), key=lambda kv: (kv[1], kv[0]))[0]
    return new


def _hot_rows():
    """Rows of every class whose neighbours carry two labels after a step:
    many lanes and many warps add to one label's frequency."""
    degs = [8, 9, 32, 33, 128, 129, 300, 1279, 1280, 2047, 2048, 2500]
    leaves = max(degs)
    edges = [(c, len(degs) + i) for c, d in enumerate(degs) for i in range(d)]
    return undirected(len(degs) + leaves, edges)


CASES = {
    "ladder": lambda: degree_ladder([1, 7, 8, 9, 31, 32, 33, 127, 128, 129, 255, 256, 257, 1279, 1280, 1281, 2047, 2048, 2049]),
    "hot": _hot_rows,
    "star": lambda: star(1500),
    # the hub rows' shared table closes at 4608 labels: at its edge and beyond it
    "hub_open": lambda: degree_ladder([4607, 4608, 4609, 6143, 6144, 6145]),
    "hub_spill": lambda: degree_ladder([7000, 9217, 20000]),
    "tiny": lambda: undirected(3, [(0, 1)]),
}


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("case", sorted(CASES))
def test_degree_votes_per_iteration(case, weighted):
    off, cols = CASES[case]()
    w = graphs.add_weights(from_numpy(off, cols), 16, seed=3).weights.numpy() if weighted else None
    trace = []
    with Graph(from_numpy(off, cols, w)) as g:
        res = g.run(_lib.METHOD_USER, 4, make_params(hooks=_lib.HOOKS_WEIGHTED_DEGREE),
                    callback=lambda it, lab: trace.append(lab) and False)
    lab = np.arange(len(off) - 1, dtype=np.int32)
    for it in range(4):
        new = _restate(off, cols, w, lab)
        np.testing.assert_array_equal(trace[it], new, err_msg=f"iteration {it}")
        assert res.changed[it] == np.count_nonzero(new != lab)
        lab = new
