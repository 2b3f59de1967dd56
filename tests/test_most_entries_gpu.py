"""A CSR of 2^31 - 1 entries, the most there can be: kernels that walk a row by
rounds pass its end, and 2^31, in the last rows."""
import pytest
import torch

from glp_b200 import _lib
from glp_b200.engine import Graph, make_params
from glp_b200.graphs import CSR

pytestmark = pytest.mark.gpu

N, D = 1 << 21, 1024


@pytest.fixture(scope="module")
def graph():
    """Row v: D consecutive vertices from v * 977 mod (N - D) on (one less in the
    last row); every row strictly ascending."""
    m = N * D - 1
    free, _ = torch.cuda.mem_get_info()
    if free < 60 << 30:
        pytest.skip("needs 60 GB of device memory")
    base = (torch.arange(N, device="cuda") * 977 % (N - D)).int()
    cols = (base[:, None] + torch.arange(D, device="cuda", dtype=torch.int32)).view(-1)[:m]
    off = torch.arange(N + 1, device="cuda") * D
    off[-1] = m
    with Graph(CSR(off.int(), cols, None)) as g:
        del cols
        torch.cuda.empty_cache()
        yield g, base.long()


def _window_max(x, base):
    """Per row, the largest of x over its columns."""
    first = x[:N].unfold(0, D, 1).max(1).values  # D columns from b on
    out = first[base]
    out[-1] = x[base[-1]:base[-1] + D - 1].max()
    return out


@pytest.mark.parametrize("method", ["classic", "layered"])
def test_last_rows(graph, method):
    g, base = graph
    # a row's neighbours hold distinct labels in the first step: the last wins
    l1 = base + D - 1
    l1[-1] -= 1
    if method == "classic":  # the second step: distinct labels again (a window holds no two of one residue)
        want = _window_max(l1, base)
        got = g.run(_lib.METHOD_CLASSIC, 2, make_params())
    else:  # score 2 - vol[label]: the largest label among those that the fewest hold
        vol = torch.bincount(l1, minlength=N)
        want = _window_max((2 - vol[l1]) * (1 << 32) + l1, base) & 0xFFFFFFFF
        got = g.run(_lib.METHOD_LAYERED, 2, make_params(dstar=[2]))
    assert torch.equal(torch.as_tensor(got.labels).cuda().long(), want)
    assert got.changed[0] == int((l1 != torch.arange(N, device="cuda")).sum())
