"""Degrees 1..32 (one thread per vertex, sorted labels): every degree, in runs
of equal degree and mixed within a warp, each score, against the oracle after
every iteration; and labels past the range of 32-bit sort keys."""
import numpy as np
import pytest

from glp_b200 import _lib
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import from_numpy
from oracle import oracle as O
from tests.graphs_fixtures import csr_from_adj

pytestmark = pytest.mark.gpu

METHODS = {"classic": (_lib.METHOD_CLASSIC, {}), "layered": (_lib.METHOD_LAYERED, dict(dstar=[2, 17])),
           "wide": (_lib.METHOD_LAYERED, dict(dstar=[65536]))}


def _rows(order, n=2000, seed=3):
    """A directed CSR with 1..32 distinct neighbours per vertex, from few
    targets so that labels repeat."""
    rng = np.random.default_rng(seed)
    deg = rng.integers(1, 33, n)
    if order == "sorted":
        deg = -np.sort(-deg)
    return csr_from_adj([sorted(rng.choice(60, d, replace=False).tolist()) for d in deg])


@pytest.mark.parametrize("wmax", [0, 3, 70000])
@pytest.mark.parametrize("order", ["sorted", "mixed"])
@pytest.mark.parametrize("method", sorted(METHODS))
def test_small_degrees_per_iteration(method, order, wmax):
    off, cols = _rows(order)
    w = np.random.default_rng(5).integers(0, wmax + 1, len(cols)).astype(np.int32) if wmax else None
    m, opts = METHODS[method]
    trace = []
    with Graph(from_numpy(off, cols, w)) as g:
        g.run(m, 4, make_params(**opts), callback=lambda it, lab: trace.append(lab) and False)
    if method == "classic":
        _, want = O.classic_run(off, cols, 4, w=w, trace=True)
    else:
        _, _, want = O.layered_run(off, cols, opts["dstar"], 4, w=w, trace=True)
    np.testing.assert_array_equal(np.array(trace), want)


@pytest.mark.parametrize("method", ["classic", "layered"])
def test_labels_beyond_32_bit_sort_keys(method):
    """The same rows at the end of 2^27 + 2000 vertices: every label is shifted
    by 2^27, which keeps their order, and the vertices before are isolated."""
    off, cols = _rows("sorted")
    w = np.random.default_rng(5).integers(1, 4, len(cols)).astype(np.int32)
    shift = 1 << 27
    m, opts = METHODS[method]
    with Graph(from_numpy(off, cols, w)) as g:
        want = g.run(m, 3, make_params(**opts))
    with Graph(from_numpy(np.concatenate([np.zeros(shift, np.int32), off]), cols + shift, w)) as g:
        got = g.run(m, 3, make_params(**opts))
    np.testing.assert_array_equal(got.labels[shift:], want.labels + shift)
    np.testing.assert_array_equal(got.changed, want.changed)
