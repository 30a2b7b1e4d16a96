"""Exact betweenness where the kernel's form changes: state and sums in shared
memory, state only, all in global memory (with the node counts of the
borders), one source per CTA at each CTA size, rows of a few lanes and rows
scanned by a whole warp, and searches of many levels; directed and not.  The
oracle's Brandes at the tolerance of the small graphs (sums of doubles of at
most n^2 terms: 1e-10 relative is far above their rounding)."""
import numpy as np
import pytest

from conftest import port_graph

pytestmark = pytest.mark.gpu


def star(n):
    return np.stack([np.zeros(n - 1), np.arange(1, n)], 1)


def ring(n):
    return np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)


CASES = {
    "pair": lambda sb: (ring(2), False),
    "star31": lambda sb: (star(31), False),
    "star1200": lambda sb: (star(1200), False),
    "ring257": lambda sb: (ring(257), False),
    "ring257_directed": lambda sb: (ring(257), True),
    "ba3100": lambda sb: (sb.barabasi_albert(3100, 3, 5), False),    # 3 CTAs an SM
    "ba5900": lambda sb: (sb.barabasi_albert(5900, 2, 6), False),    # 1 CTA an SM
    "ba11546": lambda sb: (sb.barabasi_albert(11546, 1, 7), False),  # sums in shared memory
    "ba11547": lambda sb: (sb.barabasi_albert(11547, 1, 7), False),  # and beyond it
    "rmat14_directed": lambda sb: (sb.rmat(14, 4, 8, True), True),
    "ba19164": lambda sb: (sb.barabasi_albert(19164, 1, 9), False),  # state in shared memory
    "ba19165": lambda sb: (sb.barabasi_albert(19165, 1, 9), False),  # and beyond it
    "rmat15_directed": lambda sb: (sb.rmat(15, 2, 10, True), True),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_matches_oracle(sb, port, name):
    pairs, directed = CASES[name](sb)
    hg = sb.HostGraph.from_pairs(pairs.astype(np.uint32), directed)
    g = sb.Graph.from_host(hg)
    got = g.exact_betweenness()
    np.testing.assert_allclose(got, port_graph(port, hg.csr()).brandes(), rtol=1e-10, atol=1e-15)
    np.testing.assert_array_equal(got, g.exact_betweenness())


def plain_brandes(rows):
    """Brandes over forward rows, one source at a time."""
    n = len(rows)
    bc = np.zeros(n)
    for s in range(n):
        dist, sigma, order = {s: 0}, {s: 1.0}, [s]
        for v in order:
            for w in rows[v]:
                if w not in dist:
                    dist[w], sigma[w] = dist[v] + 1, 0.0
                    order.append(w)
                if dist[w] == dist[v] + 1:
                    sigma[w] += sigma[v]
        delta = dict.fromkeys(order, 0.0)
        for v in reversed(order):
            for w in rows[v]:
                if dist[w] == dist[v] + 1:
                    delta[v] += sigma[v] / sigma[w] * (1.0 + delta[w])
            if v != s:
                bc[v] += delta[v]
    return bc


@pytest.mark.parametrize("n", [60, 20000])
def test_one_way_rows_of_an_undirected_upload(sb, n):
    """Uploaded rows are taken as they are: an entry without its counterpart on
    the other node's row is an edge one way.  A ring of 60 nodes with such
    entries; the other nodes have none."""
    r = np.random.RandomState(n)
    rows = [[(i - 1) % 60, (i + 1) % 60] for i in range(60)]
    for i in r.randint(0, 60, 20):
        rows[i].append((int(i) + 7) % 60)
    rows = [sorted(set(x)) for x in rows]
    off = np.zeros(n + 1, np.uint64)
    off[1:61] = np.cumsum([len(x) for x in rows])
    off[61:] = off[60]
    adj = np.concatenate(rows).astype(np.uint32)
    csr = sb.CSR(n, False, off, adj, off, adj, np.zeros(n, np.uint32), 1, 60)
    got = sb.Graph.upload(csr).exact_betweenness()
    want = np.zeros(n)
    want[:60] = plain_brandes(rows) / (n * (n - 1.0))
    np.testing.assert_allclose(got, want, rtol=1e-10, atol=1e-15)
