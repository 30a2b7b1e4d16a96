"""The commit of a draw where its forms meet: nodes in every sample (buckets
ordered by a whole CTA, folded 32 entries at a time), in a few (one warp), in
about 32 or 256 of a draw, entries of one, of fractions and of both mixed, in
the first pass, the top-k pass and with and without the journal of overlapped checks.  The counters are
sums in sample order and must be equal bit by bit (the reference's update loops,
silvan/src/Probabilistic.cpp:336-420)."""
import numpy as np
import pytest

from conftest import port_graph
from test_gpu_modes import assert_same_run

pytestmark = pytest.mark.gpu


def hubs(leaves, k, per, seed):
    """Each leaf hangs on `per` of k hubs (0: one to all of them, at random)."""
    r = np.random.RandomState(seed)
    e = []
    for leaf in range(k, k + leaves):
        m = per or r.randint(1, k + 1)
        e += [(leaf, h) for h in r.choice(k, m, replace=False)]
    return np.array(e, dtype=np.uint32)


def chain_of_stars(arms, leaves):
    """Centres on a path, each with its leaves: bucket sizes fall off along it."""
    e = [(i, i + 1) for i in range(arms - 1)]
    e += [(i, arms + i * leaves + j) for i in range(arms) for j in range(leaves)]
    return np.array(e, dtype=np.uint32)


GRAPHS = {
    # every x is 1, nearly every sample has the hub
    "one_hub": np.vstack([hubs(300, 1, 1, 0), [(1, 301), (301, 302)]]).astype(np.uint32),
    # x of 1/2 and 1 by a few paths
    "two_hubs": np.vstack([hubs(300, 2, 2, 1), hubs(500, 1, 1, 1)[300:]]).astype(np.uint32),
    "mixed_hubs": hubs(500, 7, 0, 2),
    "many_hubs": hubs(700, 40, 3, 3),
    "stars": chain_of_stars(12, 9),
    "path33": chain_of_stars(33, 0),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("kw", [
    dict(eps=0.02), dict(eps=0.05, k=1), dict(eps=0.03, alpha=0.0, alpha_given=True),
    dict(eps=0.03, serial_checks=True),
], ids=["eps", "topk", "one_path", "serial"])
def test_counters_match_oracle(sb, port, name, kw):
    kw = dict(kw)
    eps, serial = kw.pop("eps"), kw.pop("serial_checks", False)
    hg = sb.HostGraph.from_pairs(GRAPHS[name], False)
    csr = hg.csr()
    job = sb.Probabilistic(sb.Graph.from_host(hg), eps, 0.05, seed=31, serial_checks=serial, **kw)
    res = job.run()
    o = port_graph(port, csr).run(csr.diameter, eps, 0.05, seed=31, **kw)
    assert_same_run(job, res, o)
