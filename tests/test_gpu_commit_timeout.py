"""The bounded waits of the commit.  With no polls allowed, the CTAs that group
a draw's records by node give up at their first barrier, so the draw's buckets
are not there when the commit rounds queued behind it run: those must find no
bucket to read, the job must end with E_TIMEOUT, whichever of its draws it
happens in, and later jobs (on buffers that the failed one gave back) must
again match the oracle bit for bit (the reference commits a sample inside one
critical section, silvan/src/Probabilistic.cpp:479-544)."""
import pytest

from test_gpu_modes import assert_same_run
from conftest import port_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,extra", [("rmat11d", {}), ("ba2k", {"k": 6}),
                                        ("er3k", {"serial_checks": True})])
@pytest.mark.parametrize("rounds", [0, 1])
def test_given_up_wait_ends_the_job_alone(sb, port, small_graphs, name, extra, rounds):
    hg, csr, _ = small_graphs[name]
    g = sb.Graph.from_host(hg)
    eps = 0.08 if extra.get("k") else 0.03
    bad = sb.Probabilistic(g, eps, 0.1, seed=5, form="plain" if rounds else "batched", **extra)
    if rounds:  # the first draw of eleven samples goes well
        bad.step(rounds)
    bad.commit_polls(0)
    for _ in range(2):  # a caller that goes on all the same gets the error again
        with pytest.raises(sb.SilvanError) as err:
            while True:
                if bad.step(8)["done"]:
                    break
        assert err.value.code in (sb.E_TIMEOUT, sb.E_STATE)
    del bad
    job = sb.Probabilistic(g, eps, 0.1, seed=5, **extra)
    want = {k: v for k, v in extra.items() if k == "k"}
    assert_same_run(job, job.run(), port_graph(port, csr).run(csr.diameter, eps, 0.1, seed=5, **want))
