"""Component numbers and the diameter bound on the device at the sizes where the
kernels change their way: rows longer than all warps share, one level per node,
levels of more nodes than warps, chunks of entries that begin and end inside
rows, runs of empty rows, components of one node.  Whole numbers, equal to the
host's (silvan/src/Graph.cpp:109-316)."""
import numpy as np
import pytest

from test_gpu_ingest import assert_same_graph

pytestmark = pytest.mark.gpu


def star(n, hub=0):
    ids = np.setdiff1d(np.arange(n), [hub])
    return np.stack([np.full(n - 1, hub), ids], 1)


def path(n, step=1):
    i = np.arange(0, (n - 1) * step, step)
    return np.stack([i, i + step], 1)


def mixed(n, m, seed, hubs):
    r = np.random.RandomState(seed)
    e = r.randint(0, n, (m, 2))
    for h in range(hubs):  # rows of thousands of entries, both ways
        e = np.vstack([e, np.stack([np.full(n // 3, h * 7), r.randint(0, n, n // 3)], 1)])
        e = np.vstack([e, np.stack([r.randint(0, n, n // 3), np.full(n // 3, h * 7 + 1)], 1)])
    return e


GRAPHS = {
    "pair": path(2), "path33": path(33), "path3000": path(3000), "spaced": path(70, 4001),
    "star2049": star(2050), "star2048": star(2049, 2048), "star9000": star(9000, 77),
    "two_stars": np.vstack([star(5000), star(4000) + 6000]),
    "sparse": mixed(20000, 9000, 1, 0), "hubs": mixed(15000, 20000, 2, 3),
    "entries1024": path(513), "dense": mixed(600, 100000, 3, 0),
    "far": np.array([[0, 1], [300000, 300001], [300001, 300002], [150000, 150000]]),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("directed", [False, True])
def test_components_match_the_host(sb, tmp_path, name, directed):
    path_ = str(tmp_path / "g.txt")
    sb.write_edge_list(path_, GRAPHS[name].astype(np.uint32))
    assert_same_graph(sb.Graph.load(path_, directed).csr(),
                      sb.HostGraph.load(path_, directed).csr())
