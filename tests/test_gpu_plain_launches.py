"""The plain form draws eleven samples a launch and commits them at once: three
kernels a draw (the round's start, the sampler, the commit), whatever the batched
form's draws take, and the oracle's run bit for bit
(silvan/src/Probabilistic.cpp:812-1120)."""
import numpy as np
import pytest

from test_gpu_modes import assert_same_run
from conftest import port_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,eps,kw", [
    ("ba2k", 0.05, {}), ("rmat11d", 0.05, {}), ("er3k", 0.08, {"k": 6}),
    ("grid40", 0.1, {"alpha": 0.0, "alpha_given": True}),
    ("rmat11u", 0.05, {"alpha": 40.0, "alpha_given": True}),  # buckets of many entries
])
def test_three_kernels_a_draw(sb, port, small_graphs, name, eps, kw):
    hg, csr, _ = small_graphs[name]
    job = sb.Probabilistic(sb.Graph.from_host(hg), eps, 0.1, seed=7, form="plain", **kw)
    res = job.run()
    assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, eps, 0.1, seed=7, **kw))
    # a check takes a reduction, and a few kernels end each pass
    assert res["kernel_launches"] <= 3 * res["sampler_launches"] + 4 * res["checks"] + 16


@pytest.mark.parametrize("rounds", [1, 3])
def test_steps_then_run_to_the_end(sb, port, small_graphs, rounds):
    hg, csr, _ = small_graphs["ba2k"]
    job = sb.Probabilistic(sb.Graph.from_host(hg), 0.05, 0.1, seed=7, form="plain")
    while not job.step(rounds)["done"]:
        pass
    o = port_graph(port, csr).run(csr.diameter, 0.05, 0.1, seed=7)
    np.testing.assert_array_equal(job.counters()["mcrade"], o["mcrade"])
    np.testing.assert_array_equal(job.get_centrality(), o["approx"] / o["num_samples"])
