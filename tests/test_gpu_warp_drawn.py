"""Which samples the warp sampler draws and which it leaves.  Both samplers give
the same samples, so a run that equals the oracle's does not say who drew them:
here each job has an engine of its own (a slot count that no other test asks
for), whose first launch tries the warps on every graph, and the counts of
silvan_job_sampler_info say that the warps drew (left < tried) and, on graphs
beyond one of their limits, that they gave samples up (left > 0): levels, paths
of a sample, entries of a frontier, nodes in the table.  All results are the
oracle's bit for bit (Sp_sampler::random_path, silvan/src/Sp_sampler.cpp:41-238)."""
import itertools

import numpy as np
import pytest

from test_gpu_modes import assert_same_run
from test_gpu_warp_sampler import GRAPHS, bipartite, path
from conftest import port_graph

pytestmark = pytest.mark.gpu

fresh_slots = itertools.count(33)


def layered(*widths):  # consecutive layers wired completely
    first = np.cumsum([0] + list(widths))
    e = []
    for i in range(len(widths) - 1):
        a, b = np.meshgrid(np.arange(first[i], first[i + 1]), np.arange(first[i + 1], first[i + 2]))
        e.append(np.stack([a.ravel(), b.ravel()], 1))
    return np.concatenate(e), False


def ring(n):
    i = np.arange(n)
    return np.stack([i, (i + 1) % n], 1), False


ONE_PATH = dict(alpha=0.0, alpha_given=True)
SMALL = {  # drawn by the warps to the last sample
    "bipartite9x7": (GRAPHS["bipartite9x7"], {}),
    "path33": (path(33), {}), "path700": (path(700), ONE_PATH),
    "layered28": (layered(40, 28, 28, 40), {}),   # 784 paths: 1,803 are drawn
}
BEYOND = {  # some of the samples are beyond a limit
    "layered32": (layered(40, 32, 32, 40), {}),   # 1,024 paths: 2,355 of 2,048 are drawn
    "bipartite64x4200": (bipartite(64, 4200), {}),  # 4,200 entries from an end itself
    "layered90": (layered(60, 90, 90, 60), ONE_PATH),  # 8,100 meeting edges
    "table_full": (GRAPHS["table_full"], {}),
    "table_full_directed": (GRAPHS["table_full_directed"], {}),
}


def run_fresh(sb, pairs, directed, slots=None, **kw):
    hg = sb.HostGraph.from_pairs(pairs.astype(np.uint32), directed)
    job = sb.Probabilistic(sb.Graph.from_host(hg), 0.1, 0.1, seed=6,
                           slots=slots or next(fresh_slots), **kw)
    return hg.csr(), job, job.run()


@pytest.mark.parametrize("name", sorted(SMALL) + sorted(BEYOND))
def test_samples_are_tried(sb, port, name):
    (pairs, directed), kw = {**SMALL, **BEYOND}[name]
    csr, job, res = run_fresh(sb, pairs, directed, **kw)
    assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, 0.1, 0.1, seed=6, **kw))
    got = job.sampler_info()
    assert got["warps"] > 0 and got["warp_tried"] > 0
    if name in SMALL:
        assert got["warp_left"] == 0
    else:
        assert 0 < got["warp_left"] < got["warp_tried"]


def test_searches_of_more_levels_than_a_warp_keeps(sb, port):
    """4,096 a side: on a path of 9,400 nodes one sample in sixty."""
    hg = sb.HostGraph.from_pairs(path(9400)[0].astype(np.uint32), False)
    g = sb.Graph.from_host(hg)
    job = sb.Probabilistic(g, 0.2, 0.1, seed=6, slots=next(fresh_slots), **ONE_PATH)
    job.step(1)
    got = job.sampler_info()
    assert 0 < got["warp_left"] < got["warp_tried"]
    a, b = g.replay(6, 0, 200, 0.0), port_graph(port, hg.csr()).replay(6, 0, 200, 0.0)
    assert a["path_length"].max() > 8192
    for f in ("path_length", "num_paths", "vis_edges", "offsets", "nodes", "counts"):
        np.testing.assert_array_equal(a[f], getattr(b, f), err_msg=f)


def test_one_way_rows_are_not_tried(sb):
    n = 60
    off = np.arange(0, 2 * n + 1, 2).astype(np.uint64)
    adj = np.sort([[(i - 1) % n, (i + 1) % n] for i in range(n)], 1).astype(np.uint32)
    adj[7] = [8, 30]  # 6 no longer on 7's row, nor 7 on 30's
    csr = sb.CSR(n, False, off, adj.ravel(), off, adj.ravel(), np.zeros(n, np.uint32), 1, n)
    job = sb.Probabilistic(sb.Graph.upload(csr), 0.1, 0.1, seed=6, slots=next(fresh_slots))
    try:
        job.run()
    except sb.SilvanError as err:  # a walk over the missing entry
        assert err.code == sb.E_STATE
    assert job.sampler_info()["warp_tried"] == 0


def test_tried_and_untried_graphs_in_one_redrawn_round(sb, port):
    """A lattice whose samples the warps have left before, and a ring whose paths
    (a thousand nodes each) overflow the record buffers: the round is drawn again
    with larger ones, the ring's samples by warps, the lattice's by CTAs."""
    slots = next(fresh_slots)
    lattice = sb.HostGraph.from_pairs(sb.grid(384, 0.05, 0.001, 1), False)
    rings = sb.HostGraph.from_pairs(ring(4001)[0].astype(np.uint32), False)
    graphs = [sb.Graph.from_host(h) for h in (lattice, rings)]
    sb.Probabilistic(graphs[0], 0.1, 0.1, seed=1, slots=slots, **ONE_PATH).run()
    jobs = [sb.Probabilistic(g, eps, 0.1, seed=6, slots=slots, **ONE_PATH)
            for g, eps in zip(graphs, (0.1, 0.03))]
    for hg, job, eps, res in zip((lattice, rings), jobs, (0.1, 0.03), sb.run_batched(jobs)):
        csr = hg.csr()
        assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, eps, 0.1, seed=6,
                                                            **ONE_PATH))
    assert jobs[0].sampler_info()["warp_tried"] == 0
    ring_info = jobs[1].sampler_info()
    assert ring_info["warp_left"] == 0
    assert ring_info["warp_tried"] > jobs[1].result["samples_drawn"]  # drawn twice
