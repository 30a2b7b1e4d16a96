"""Predecessors by rank far from the ends of a search: a hub of a long row between
two fans of 40 nodes and two chains, reached at levels on either side of those
whose queue bounds lie in shared memory (64) and in the slot (256).  Runs are
the oracle's (Sp_sampler::backtrack_path, silvan/src/Sp_sampler.cpp:241-265), and
finding the rank on the narrow level rather than on the hub's row keeps the few
samples through the hub from being the run's time (5 ms where it is found so,
116 ms where it is not: the bound below is between the two)."""
import numpy as np
import pytest

from test_gpu_modes import assert_same_run
from conftest import port_graph

pytestmark = pytest.mark.gpu


def hub_between_chains(chain, ways, leaves):
    def arm(first):  # a chain, then `ways` nodes between its end and the hub
        c = first + np.arange(chain)
        w = first + chain + np.arange(ways)
        z = np.zeros(ways, np.int64)
        return [np.stack([c[:-1], c[1:]], 1), np.stack([z + c[-1], w], 1), np.stack([w, z], 1)]
    two = arm(1) + arm(1 + chain + ways)
    leaf = 1 + 2 * (chain + ways) + np.arange(leaves)
    return np.concatenate(two + [np.stack([np.zeros(leaves, np.int64), leaf], 1)])


@pytest.mark.parametrize("chain,ways,leaves", [(300, 8, 200), (300, 5, 900), (120, 20, 600)])
def test_run_matches_oracle(sb, port, chain, ways, leaves):
    """A threshold of its own keeps a job's samples from the warp sampler."""
    hg = sb.HostGraph.from_pairs(hub_between_chains(chain, ways, leaves).astype(np.uint32), False)
    csr = hg.csr()
    job = sb.Probabilistic(sb.Graph.from_host(hg), 0.1, 0.1, seed=6, assist_items=1 << 30)
    res = job.run()
    assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, 0.1, 0.1, seed=6))
    assert job.sampler_info()["warp_tried"] == 0


def test_samples_through_a_far_hub_do_not_bound_the_run(sb):
    pairs = hub_between_chains(150, 40, 3000)
    g = sb.Graph.from_pairs(pairs.astype(np.uint32))
    t = [sb.Probabilistic(g, 0.02, 0.05, seed=s).run()["time_sampling_s"] for s in range(8)]
    assert min(t) < 0.05
