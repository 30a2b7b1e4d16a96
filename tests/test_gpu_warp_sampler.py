"""The warp sampler (one warp a sample, a hash table of the visited nodes in
shared memory) against the oracle, sample by sample, at the sizes where it
can go wrong: frontiers and tables that overflow (those samples are left to
the CTA sampler in the middle of their search), more meeting edges, path-map
nodes and paths than it keeps near, rows without entries, self-loops, and
tables that forget older levels.  The results are whole numbers and must be
equal (Sp_sampler::random_path, silvan/src/Sp_sampler.cpp:41-238)."""
import numpy as np
import pytest

from conftest import port_graph

pytestmark = pytest.mark.gpu


def star(n):  # one frontier of n - 1 entries: beyond 4096 it is left at once
    return np.stack([np.zeros(n - 1), np.arange(1, n)], 1), False


def bipartite(a, b):  # a * b meeting edges at one level, a or b predecessors a node
    u, v = np.meshgrid(np.arange(a), np.arange(b))
    return np.stack([u.ravel(), a + v.ravel()], 1), False


def path(n):  # n levels of one node
    return np.stack([np.arange(n - 1), np.arange(1, n)], 1), False


def random_graph(n, m, directed, seed):  # isolated nodes, sinks and self-loops among it
    r = np.random.RandomState(seed)
    e = r.randint(0, n, (m, 2))
    e[:n // 20, 1] = e[:n // 20, 0]
    e[:, 1] = np.where(r.rand(m) < 0.3, e[:, 1] % 11, e[:, 1])
    return np.vstack([e, [[0, n - 1]]]), directed


def lattice(side):  # the table is rebuilt from the last levels many times
    i = np.arange(side * side).reshape(side, side)
    return np.vstack([np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1),
                      np.stack([i[:-1].ravel(), i[1:].ravel()], 1)]), False


GRAPHS = {
    "star40": star(40), "star4097": star(4097), "star4200": star(4200),
    "bipartite9x7": bipartite(9, 7), "bipartite40x33": bipartite(40, 33),
    "bipartite90x80": bipartite(90, 80), "path2": path(2), "path33": path(33),
    "path700": path(700), "sparse": random_graph(2500, 3000, False, 1),
    "sinks": random_graph(2500, 5000, True, 2), "table_full": random_graph(6000, 30000, False, 3),
    "table_full_directed": random_graph(6000, 40000, True, 4), "lattice80": lattice(80),
    "lattice301": lattice(301),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("alpha", [2.3, -1.0])
def test_replay_matches_oracle(sb, port, name, alpha):
    if name.startswith("lattice") and alpha > 0:
        pytest.skip("a lattice asks for astronomically many paths")
    pairs, directed = GRAPHS[name]
    hg = sb.HostGraph.from_pairs(pairs.astype(np.uint32), directed)
    csr = hg.csr()
    count = 60 if name in ("path700", "lattice301") else 600
    a = sb.Graph.from_host(hg).replay(3, 5, count, alpha)
    b = port_graph(port, csr).replay(3, 5, count, alpha)
    assert (a["status"] == 0).all()
    for f in ("path_length", "num_paths", "vis_edges", "offsets", "nodes", "counts"):
        np.testing.assert_array_equal(a[f], getattr(b, f), err_msg=f)


@pytest.mark.parametrize("name", ["lattice80", "bipartite40x33", "sinks"])
def test_weighted_run_matches_oracle(sb, port, name):
    """Sigma-weighted predecessors, found by the whole warp on the level above."""
    pairs, directed = GRAPHS[name]
    hg = sb.HostGraph.from_pairs(pairs.astype(np.uint32), directed)
    csr = hg.csr()
    kw = dict(alpha=0.0, alpha_given=True, seed=8)
    job = sb.Probabilistic(sb.Graph.from_host(hg), 0.05, 0.1, backtrack="sigma", **kw)
    res = job.run()
    o = port_graph(port, csr).run(csr.diameter, 0.05, 0.1, weighted=True, **kw)
    for f in ("num_samples", "vis_edges", "first_pass_samples"):
        assert res[f] == o[f], f
    c = job.counters()
    for f in ("approx", "wimpy", "mcrade"):
        np.testing.assert_array_equal(c[f], o[f], err_msg=f)


def test_one_way_rows_of_an_undirected_upload(sb, port):
    """Uploaded rows are taken as they are.  An entry without its counterpart
    (v on u's row, u not on v's) rules the warp sampler out: the graph is
    drawn by the general search, which reads forward rows as the oracle does
    and reports SILVAN_E_STATE for a walk that needs the rank of a predecessor
    missing from the reverse row."""
    n = 60
    ring = [[(i - 1) % n, (i + 1) % n] for i in range(n)]
    ring[7].append(30)
    ring[41].append(12)
    rows = [np.unique(r) for r in ring]
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum([len(r) for r in rows])
    adj = np.concatenate(rows).astype(np.uint32)
    cc = np.zeros(n, np.uint32)
    csr = sb.CSR(n, False, off, adj, off, adj, cc, 1, n)
    a = sb.Graph.upload(csr).replay(3, 0, 400, -1.0)
    b = port_graph(port, csr).replay(3, 0, 400, -1.0)
    np.testing.assert_array_equal(a["vis_edges"], b.vis_edges)
    ok = a["status"] == 0
    assert ok.sum() >= 390 and (a["status"][~ok] == -10).all()
    for i in np.flatnonzero(ok):
        p, q = slice(*a["offsets"][i:i + 2]), slice(*b.offsets[i:i + 2])
        assert a["path_length"][i] == b.path_length[i] and a["num_paths"][i] == b.num_paths[i]
        np.testing.assert_array_equal(a["nodes"][p], b.nodes[q])
        np.testing.assert_array_equal(a["counts"][p], b.counts[q])
