"""The CTA sampler's last levels (nodes marked and counted only, once a meeting
edge is known) and the places of its node states: graphs below and above the
largest that has them in shared memory for a CTA size, above it short ones
(states in the slots) and a long one (in the records), rounds of several graphs, last levels of several tiles, meeting edges
in several tiles, many hits on one node.  Against the oracle, and against the
same samples with every level on the help board, whose tiles do neither
(Sp_sampler::random_path, silvan/src/Sp_sampler.cpp:89-197)."""
import numpy as np
import pytest

from conftest import port_graph
from test_gpu_assist import NEVER, SCALARS, same_counters
from test_gpu_modes import assert_same_run

pytestmark = pytest.mark.gpu


def hubs(n, hubs_, m, seed):
    """Every node hangs on a few of `hubs_` hubs, and on m random others."""
    r = np.random.RandomState(seed)
    v = np.arange(n)
    e = [np.stack([v, r.randint(0, hubs_, n)], 1) for _ in range(2)]
    e += [np.stack([r.randint(0, n, m), r.randint(0, n, m)], 1)]
    return np.vstack(e + [[[0, n - 1]]]).astype(np.uint32)


GRAPHS = {  # name: (pairs, directed)
    "below": (hubs(32768, 60, 40000, 1), False),   # states for every CTA size
    "above": (hubs(32769, 60, 40000, 2), False),   # none for 128 threads
    "wide": (hubs(70000, 300, 200000, 3), False),  # none for 128 and 256
    "directed": (hubs(40000, 40, 300000, 4), True),
    "few": (hubs(9000, 3, 20000, 5), False),       # thousands of meeting edges
    "tail": (np.vstack([hubs(70000, 300, 200000, 6),  # a path makes it long
                        np.stack([np.arange(69999, 70039), np.arange(70000, 70040)], 1)]), False),
}


@pytest.mark.parametrize("block", [128, 256, 512, 1024])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_last_levels(sb, port, name, block):
    pairs, directed = GRAPHS[name]
    hg = sb.HostGraph.from_pairs(pairs.astype(np.uint32), directed)
    csr = hg.csr()
    g = sb.Graph.from_host(hg)
    kw = dict(seed=12, alpha=0.01, alpha_given=True)
    runs = []
    for items in (NEVER, 1):
        job = sb.Probabilistic(g, 0.05, 0.1, block=block, assist_items=items, **kw)
        runs.append((job, job.run()))
    (a, ra), (b, rb) = runs
    for f in SCALARS:
        assert ra[f] == rb[f], f
    same_counters(a, b)
    assert_same_run(a, ra, port_graph(port, csr).run(csr.diameter, 0.05, 0.1, **kw))


@pytest.mark.parametrize("names", [("few", "below"), ("few", "wide", "directed"),
                                   ("tail", "few"), ("tail",)])
def test_rounds_of_several_graphs(sb, port, names):
    kw = dict(seed=5, alpha=0.01, alpha_given=True)
    jobs, want = [], []
    for nm in names:
        pairs, directed = GRAPHS[nm]
        hg = sb.HostGraph.from_pairs(pairs.astype(np.uint32), directed)
        csr = hg.csr()
        jobs.append(sb.Probabilistic(sb.Graph.from_host(hg), 0.05, 0.1, **kw))
        want.append(port_graph(port, csr).run(csr.diameter, 0.05, 0.1, **kw))
    for job, res, o in zip(jobs, sb.run_batched(jobs), want):
        assert_same_run(job, res, o)
