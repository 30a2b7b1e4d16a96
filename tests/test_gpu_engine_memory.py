"""Engines whose memory does not hold all the slots that the GPU can run at once:
the slots get all of it, and the warp sampler's state lies in what the CTA
sampler leaves between samples.  Results are the oracle's with room for a few
slots and a few warps as with all of them (Sp_sampler::random_path,
silvan/src/Sp_sampler.cpp:41-238)."""
import pytest

from test_gpu_modes import assert_same_run
from conftest import port_graph

pytestmark = pytest.mark.gpu

MEETS = 65536 * 16  # meeting edges of a slot


def slot_bytes(n):  # a node's record, queue, hit, touched entries and state bits
    return n * (32 + 3 * 4) + MEETS + 4 * ((n + 15) // 16)


def test_slots_get_all_the_memory(sb):
    """Half of the free memory, for graphs of four million nodes."""
    import torch

    n = 4 << 20
    free = torch.cuda.mem_get_info()[0]
    srv = sb.Server(n)
    try:
        slots = srv.stats()["slots"]
    finally:
        srv.close()
    assert slots < 1000  # bound by memory
    assert slots >= free // 2 // slot_bytes(n) * 0.98


@pytest.mark.parametrize("budget", [1, 5 << 20, 40 << 20, 300 << 20])
@pytest.mark.parametrize("extra", [{}, {"k": 6}], ids=["absolute", "topk"])
def test_bounded_batch_matches_oracle(sb, port, small_graphs, budget, extra):
    names = ["ba2k", "rmat11d", "er3k", "rmat11u"]
    eps = 0.08 if extra else 0.03
    jobs = [sb.Probabilistic(sb.Graph.from_host(small_graphs[nm][0]), eps, 0.1, seed=9, **extra)
            for nm in names]
    for nm, job, res in zip(names, jobs, sb.run_batched(jobs, budget)):
        csr = small_graphs[nm][1]
        assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, eps, 0.1, seed=9, **extra))


@pytest.mark.parametrize("slots", [1, 3, 40])
def test_few_slots_match_oracle(sb, port, small_graphs, slots):
    for nm, kw in (("rmat11d", {}), ("grid40", dict(alpha=0.0, alpha_given=True))):
        hg, csr, _ = small_graphs[nm]
        job = sb.Probabilistic(sb.Graph.from_host(hg), 0.05, 0.1, seed=4, slots=slots, **kw)
        assert_same_run(job, job.run(), port_graph(port, csr).run(csr.diameter, 0.05, 0.1, seed=4, **kw))
