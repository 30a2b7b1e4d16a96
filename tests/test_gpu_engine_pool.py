"""Engines that outlive a call give way: a graph whose slots are bound by memory
leaves the small graphs after it the slots that they had, and what an idle engine
holds goes to a server or to a batch that needs it.  A few edges and the id of the
last node make a graph of millions of nodes."""
import numpy as np
import pytest

from test_gpu_modes import assert_same_run
from conftest import port_graph

pytestmark = pytest.mark.gpu

N = 9_000_000  # a slot of 400 MB


@pytest.fixture(scope="module")
def large(sb):
    i = np.arange(200)
    pairs = np.concatenate([np.stack([i, (i + 1) % 200], 1), [[0, N - 1]]])
    return sb.Graph.from_pairs(pairs.astype(np.uint32))


def estimate(sb, g, **kw):
    job = sb.Probabilistic(g, 0.3, 0.1, seed=3, **kw)
    return job, job.run()


def test_small_graphs_keep_their_slots(sb, port, small_graphs, large):
    hg, csr, _ = small_graphs["ba2k"]
    small = sb.Graph.from_host(hg)
    before = estimate(sb, small)[0].sampler_info()["slots"]
    assert 0 < estimate(sb, large)[0].sampler_info()["slots"] < before
    for _ in range(2):  # whichever engine came back last
        job, res = estimate(sb, small)
        assert job.sampler_info()["slots"] == before
        assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, 0.3, 0.1, seed=3))
        assert estimate(sb, large)[0].sampler_info()["slots"] < before


def test_a_server_after_a_batch_has_half_of_the_memory(sb, large):
    import torch
    total = torch.cuda.mem_get_info()[1]
    sb.run_batched([sb.Probabilistic(large, 0.3, 0.1, seed=s) for s in (1, 2)])
    srv = sb.Server(N)
    try:
        slots = srv.stats()["slots"]
    finally:
        srv.close()
    assert slots >= 0.9 * (total // 2) // (N * 45)  # 44.25 bytes a node and 1 MB


def test_a_bounded_batch_gets_what_idle_engines_hold(sb, large):
    """Two thirds of the memory, half of which the batch before left in the pool."""
    import torch
    total = torch.cuda.mem_get_info()[1]
    first = sb.Probabilistic(large, 0.3, 0.1, seed=1)
    sb.run_batched([first])
    want = first.result["num_samples"]
    del first
    assert torch.cuda.mem_get_info()[0] < total * 2 // 3
    job = sb.Probabilistic(large, 0.3, 0.1, seed=1)
    res, = sb.run_batched([job], total * 2 // 3)
    assert res["num_samples"] == want
    assert job.sampler_info()["slots"] >= total * 2 // 3 // (N * 45) * 0.9
