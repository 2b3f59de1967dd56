"""The sort, the duplicate filter and the column writer of glp_graph_from_edges
at the sizes where they change course: tile edges, one hash bucket and many, a
bucket that has to be split, hot keys, every combination of the flags, against
numpy."""
import numpy as np
import pytest
import torch

from glp_b200.engine import Graph

pytestmark = pytest.mark.gpu


def _numpy_csr(src, dst, n, directed, keep_ids):
    s, d = src.astype(np.int64), dst.astype(np.int64)
    s, d = s[s != d], d[s != d]
    if not directed:
        s, d = np.concatenate([s, d]), np.concatenate([d, s])
    k = np.unique(s << 32 | d)
    old = np.arange(n)
    if not keep_ids:
        old = np.lexsort((old, -np.bincount(k >> 32, minlength=n)))
        new = np.empty(n, np.int64)
        new[old] = np.arange(n)
        k = np.sort(new[k >> 32] << 32 | new[k & 0xFFFFFFFF])
    off = np.concatenate([[0], np.cumsum(np.bincount(k >> 32, minlength=n))])
    return off, k & 0xFFFFFFFF, old


def _mix64(z):  # the bucket hash (SplitMix64's finaliser)
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _one_bucket(n=1 << 18):
    """About 9000 distinct edges whose hashes share their top six bits."""
    rng = np.random.default_rng(3)
    u, v = np.sort(rng.integers(0, n, (2, 600_000)), axis=0)
    keep = (u < v) & (_mix64((u.astype(np.uint64) << np.uint64(18)) | v.astype(np.uint64)) >> np.uint64(58) == 0)
    return np.tile(u[keep], 2), np.tile(v[keep], 2), n


def _random(count, n, seed=1):
    rng = np.random.default_rng(seed)
    return rng.integers(0, n, count), rng.integers(0, n, count), n


SETS = {
    "one": lambda: (np.array([0]), np.array([1]), 2),
    "loops": lambda: (np.array([0, 0]), np.array([0, 0]), 1),
    "hot": lambda: (np.zeros(30000, int), np.arange(30000) % 7, 9),
    "tile-1": lambda: _random(8191, 5000),
    "tile": lambda: _random(8192, 5000),
    "tile+1": lambda: _random(8193, 300),
    "buckets": lambda: _random(300_000, 65537),
    "bucket-split": _one_bucket,
}


@pytest.mark.parametrize("keep_ids", [False, True])
@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("name", sorted(SETS))
def test_from_edges_equals_numpy(name, directed, keep_ids):
    src, dst, n = SETS[name]()
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    off, cols, old = _numpy_csr(src, dst, n, directed, keep_ids)
    g, got_old = Graph.from_edges(torch.from_numpy(src).cuda(), torch.from_numpy(dst).cuda(), n, directed=directed,
                                  keep_ids=keep_ids)
    with g:
        csr = g.export()
    np.testing.assert_array_equal(csr.offsets.numpy(), off)
    np.testing.assert_array_equal(csr.cols.numpy(), cols)
    np.testing.assert_array_equal(got_old, old)
