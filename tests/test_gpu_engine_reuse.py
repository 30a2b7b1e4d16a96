"""Engines that outlive one call: a batch takes the pooled engine that single
jobs use (or one of its own under a memory budget), a larger graph replaces an
idle smaller engine, and the first launch of a job is sized by earlier jobs of
the same kind only.  None of it changes a result
(silvan/src/Probabilistic.cpp:812-1120)."""
import pytest

from test_gpu_modes import assert_same_run
from conftest import port_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget", [0, 1 << 30])
def test_batches_and_single_jobs_in_turn(sb, port, small_graphs, budget):
    names = ["ba2k", "rmat11d", "er3k"]
    want = {nm: port_graph(port, small_graphs[nm][1]).run(
        small_graphs[nm][1].diameter, 0.03, 0.1, seed=9) for nm in names}
    for order in (names[:1], names, names[::-1]):  # smaller and larger engines, then again
        jobs = [sb.Probabilistic(sb.Graph.from_host(small_graphs[nm][0]), 0.03, 0.1, seed=9)
                for nm in order]
        for nm, job, res in zip(order, jobs, sb.run_batched(jobs, budget)):
            assert_same_run(job, res, want[nm])
        one = sb.Probabilistic(sb.Graph.from_host(small_graphs[order[-1]][0]), 0.03, 0.1, seed=9)
        assert_same_run(one, one.run(), want[order[-1]])


def test_failed_batch_leaves_the_engine_usable(sb, port, small_graphs):
    hg, csr, _ = small_graphs["ba2k"]
    g = sb.Graph.from_host(hg)
    done = sb.Probabilistic(g, 0.05, 0.1, seed=1)
    done.run()
    with pytest.raises(sb.SilvanError):
        sb.run_batched([sb.Probabilistic(g, 0.05, 0.1, seed=2), done])
    job = sb.Probabilistic(g, 0.03, 0.1, seed=9)
    assert_same_run(job, job.run(), port_graph(port, csr).run(csr.diameter, 0.03, 0.1, seed=9))


def test_a_launch_is_sized_by_jobs_of_its_own_kind(sb, small_graphs):
    """A tight job's total says nothing about a loose one's on the same graph."""
    g = sb.Graph.from_host(small_graphs["ba2k"][0])
    for _ in range(2):
        tight = sb.Probabilistic(g, 0.004, 0.1, seed=3).run()
    for _ in range(2):
        loose = sb.Probabilistic(g, 0.05, 0.1, seed=3).run()
    used = loose["first_pass_samples"] + loose["num_samples"]
    assert tight["samples_drawn"] > 10 * used
    assert used <= loose["samples_drawn"] <= 6 * used
