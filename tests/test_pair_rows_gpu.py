"""Degrees 33..64 (two threads per vertex, sorted halves): every degree, few and
many distinct labels, runs that cross the halves, in classic, SLPA and seeded
runs and in batches, against the oracle after every iteration."""
import numpy as np
import pytest

from glp_b200 import _lib
from glp_b200.batch import Batch
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import from_numpy
from oracle import oracle as O
from tests.graphs_fixtures import csr_from_adj

pytestmark = pytest.mark.gpu


def _rows(targets, n=900, lo=31, hi=67):
    """A directed CSR with lo..hi-1 distinct neighbours per vertex among `targets` vertices."""
    rng = np.random.default_rng(targets)
    return csr_from_adj([sorted(rng.choice(targets, d, replace=False).tolist()) for d in rng.integers(lo, hi, n)])


@pytest.mark.parametrize("targets", [70, 900])
@pytest.mark.parametrize("majority", [1, 1000])
def test_pair_rows_per_iteration(targets, majority):
    off, cols = _rows(targets)
    n = len(off) - 1
    seeds = np.random.default_rng(1).random(n) < 0.1
    p = make_params(majority_permille=majority, slpa_T=6, seed=3)
    with Graph(from_numpy(off, cols)) as g:
        trace = []
        g.run(_lib.METHOD_CLASSIC, 6, p, callback=lambda it, lab: trace.append(lab) and False)
        np.testing.assert_array_equal(np.array(trace), O.classic_run(off, cols, 6, trace=True)[1])
        np.testing.assert_array_equal(g.run(_lib.METHOD_SLPA, 6, p).labels,
                                      O.slpa_run(off, cols, 6, 6, 3, 0.1)["labels"])
        g.set_seeds(seeds)
        np.testing.assert_array_equal(g.run(_lib.METHOD_SEEDED, 5).labels, O.seeded_run(off, cols, seeds, 5))


@pytest.mark.parametrize("frontier", [-1, 1000])
def test_pair_rows_in_batches(frontier):
    graphs = [_rows(70, 300), _rows(200, 500, 20, 40), _rows(400, 401, 33, 65)]
    with Batch([from_numpy(*g) for g in graphs]) as b:
        labels, _ = b.run(7, make_params(frontier_permille=frontier))
        for got, g in zip(b.split(labels), graphs):
            np.testing.assert_array_equal(got, O.classic_run(*g, 7))
