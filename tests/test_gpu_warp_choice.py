"""When the warps are tried.  A lattice whose samples they left does not rule them
out for a short graph of the same size and degree (both to a power of two), nor for
its own kind for good: after 64 launches they are tried again.  Where they leave
some of the samples, what a launch takes with and without them decides.  Each test
has an engine of its own by a slot count that no other test asks for; results do not
depend on the choice (Sp_sampler::random_path, silvan/src/Sp_sampler.cpp:41-238)."""
import numpy as np
import pytest

from test_gpu_modes import assert_same_run
from conftest import port_graph

pytestmark = pytest.mark.gpu

ONE_PATH = dict(alpha=0.0, alpha_given=True)


@pytest.fixture(scope="module")
def lattice(sb):
    return sb.Graph.from_pairs(sb.grid(384, 0.05, 0.001, 1))


def run(sb, g, eps, seed, slots, **kw):
    job = sb.Probabilistic(g, eps, 0.1, seed=seed, slots=slots, **kw)
    return job, job.run()


def test_a_lattice_leaves_the_warps_to_short_graphs_of_its_class(sb, port, lattice):
    hg = sb.HostGraph.from_pairs(sb.barabasi_albert(140000, 2, 1), False)
    csr = hg.csr()
    assert csr.n >> 17 == lattice.n >> 17 == 1
    assert len(csr.out_adj) // csr.n == 3 and 2 <= 2 * 384 * 383 * 0.95 * 2 // lattice.n < 4
    for seed in range(3):
        info = run(sb, lattice, 0.1, seed, 26, **ONE_PATH)[0].sampler_info()
    assert info["warp_tried"] == 0  # left out by now
    job, res = run(sb, sb.Graph.from_host(hg), 0.02, 7, 26)
    assert job.sampler_info()["warp_tried"] > 0
    assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, 0.02, 0.1, seed=7))


def test_left_out_graphs_are_tried_again(sb, lattice):
    tried, launches = [], []
    for seed in range(80):
        job, res = run(sb, lattice, 0.2, seed, 27, **ONE_PATH)
        tried.append(job.sampler_info()["warp_tried"] > 0)
        launches.append(res["sampler_launches"])
        if tried[1:].count(True):
            break
    assert tried[0] and tried[-1]
    assert sum(launches[1:-1]) <= 64 <= sum(launches)


def test_the_time_decides_where_some_samples_are_left(sb, port):
    """Of a 120 x 120 lattice the warps leave four samples in ten and cost a quarter
    of the sampling; of 10,000 nodes of Barabasi-Albert one in fourteen, and without
    them the sampling is half as long again."""
    hg = sb.HostGraph.from_pairs(sb.grid(120, 0.05, 0.001, 1), False)
    g, infos = sb.Graph.from_host(hg), []
    for seed in range(24):
        job, res = run(sb, g, 0.03, seed, 1183, **ONE_PATH)
        infos.append(job.sampler_info())
    assert 64 * infos[0]["warp_left"] > infos[0]["warp_tried"] > 2 * infos[0]["warp_left"]
    assert [i["warp_tried"] for i in infos[-3:]] == [0, 0, 0]
    csr = hg.csr()
    assert_same_run(job, res, port_graph(port, csr).run(csr.diameter, 0.03, 0.1, seed=23,
                                                        **ONE_PATH))
    small = sb.Graph.from_pairs(sb.barabasi_albert(10000, 5, 1))
    infos = [run(sb, small, 0.01, seed, 1183)[0].sampler_info() for seed in range(24)]
    assert all(i["warp_tried"] > 0 for i in infos[-3:])


def test_draws_ahead_where_the_ctas_take_the_time(sb):
    """Sparse directed random graphs: nearly all samples are void, and the others are
    long ones of the CTA sampler's.  The slots that are free while the slowest is
    drawn draw ahead, so that the first pass and the second take a launch each."""
    pairs = np.random.RandomState(1).randint(0, 200000, (220000, 2)).astype(np.uint32)
    g = sb.Graph.from_pairs(pairs, True)
    res = [run(sb, g, 0.005, seed, 1182)[1] for seed in range(10)]
    assert min(r["sampler_launches"] for r in res[-5:]) <= 2
