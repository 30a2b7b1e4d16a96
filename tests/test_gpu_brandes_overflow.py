"""Exact betweenness where path counts leave the doubles' range: a fan of
layers, each wired to the next completely, from whose root 16^(d-1) paths reach
a node of layer d -- infinitely many in the last layer of 257.  The pairs that
end there add nothing, and every other value is that of the plain formula
sigma_v / sigma_w (1 + delta_w); nothing becomes NaN.  The oracle's Brandes is
that formula in doubles, at the tolerance of the other exact tests."""
import numpy as np
import pytest

from conftest import port_graph

pytestmark = pytest.mark.gpu

LAYERS, WIDTH = 257, 16


def fan():
    prev, pairs = np.zeros(1, np.int64), []
    for d in range(LAYERS):
        cur = 1 + d * WIDTH + np.arange(WIDTH)
        pairs.append(np.stack(np.meshgrid(prev, cur, indexing="ij"), -1).reshape(-1, 2))
        prev = cur
    return np.concatenate(pairs)


def chain(first, count):  # from the root past the fan's last layer: that one is not the deepest
    ids = np.concatenate([[0], first + np.arange(count)])
    return np.stack([ids[:-1], ids[1:]], 1)


def isolated(n):  # the state no longer fits in shared memory
    return np.array([[n - 2, n - 1]])


N = 1 + LAYERS * WIDTH
CASES = {
    "last_layer": ([fan()], False),
    "last_layer_directed": ([fan()], True),
    "not_the_deepest": ([fan(), chain(N, 300)], True),
    "in_global_memory": ([fan(), isolated(20000)], True),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_infinite_counts_at_the_ends_add_nothing(sb, port, name):
    parts, directed = CASES[name]
    hg = sb.HostGraph.from_pairs(np.concatenate(parts).astype(np.uint32), directed)
    want = port_graph(port, hg.csr()).brandes()
    assert np.isfinite(want).all() and want.max() > 0
    got = sb.Graph.from_host(hg).exact_betweenness()
    np.testing.assert_allclose(got, want, rtol=1e-10, atol=1e-15)
