"""What a job holds on the device decides which requests a server runs side by
side and which large draws still fit: 20 bytes a path-map record (the sampler's
12 and 8 to group it by node) and the same per-node state whatever the commit
does with them."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TRIALS = 25


def request_bytes(csr):
    """A request's share of a server's budget: its graph, the counters and node
    buckets, the round buffers with 2^20 records, and 64 MiB to grow."""
    n, entries = csr.n, len(csr.out_adj) + (len(csr.in_adj) if csr.directed else 0)
    graph = 4 * (n + 1) * (2 if csr.directed else 1) + 4 * entries + 4 * n
    job = n * (8 + 8 + 8 * TRIALS + 4 + 1 + 4 + 4 + 4 + 4 + 8) + (csr.diameter + 1) * 8
    return graph + job + 65536 * 36 + (20 << 20) + (64 << 20)


@pytest.mark.parametrize("spare,together", [(0, 2), (-1, 1)])
def test_two_requests_fill_a_budget_of_twice_their_bytes(sb, spare, together):
    hg = sb.HostGraph.from_pairs(sb.barabasi_albert(60000, 4, 5), False)
    csr = hg.csr()
    srv = sb.Server(csr.n, budget=2 * request_bytes(csr) + spare)
    try:
        ids = [srv.submit(hg, 0.001, 0.1, seed=s) for s in (1, 2)]
        used = 0
        while any(srv.poll(i)[0] in (sb.REQ_QUEUED, sb.REQ_RUNNING) for i in ids):
            used = max(used, srv.stats()["bytes_in_use"])
            time.sleep(0.0005)
        for i in ids:
            srv.wait(i, 300)
        assert srv.stats()["max_active"] == together
        assert used == together * request_bytes(csr)
    finally:
        srv.close()


def test_a_grown_draw_holds_20_bytes_a_record(sb):
    """A ring's draws are long paths: 65,536 samples of up to 2,000 nodes.  What a
    run of them adds to the process's device memory stays below 20 bytes for each
    record of the next power of two (the buffer's size), and an allowance of a
    sixteenth for the lists of long buckets and the rounding of blocks."""
    import torch

    n = 4001
    ring = np.stack([np.arange(n), (np.arange(n) + 1) % n], 1).astype(np.uint32)
    g = sb.Graph.from_pairs(ring)
    sb.Probabilistic(g, 0.2, 0.1, alpha=0.0, alpha_given=True, seed=3).run()  # the engine is there
    before = torch.cuda.mem_get_info()[0]
    job = sb.Probabilistic(g, 0.005, 0.1, alpha=0.0, alpha_given=True, seed=3)
    res = job.run()
    held = before - torch.cuda.mem_get_info()[0]
    per_draw = min(65536, res["samples_drawn"]) * (n // 4)  # a path has n / 4 inner nodes on average
    cap = 1 << 20
    while cap < per_draw:
        cap *= 2
    assert cap >= 1 << 23
    assert held <= 20 * cap * 17 // 16 + (48 << 20), (held, cap)
