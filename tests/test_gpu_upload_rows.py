"""The checks of uploaded rows at the lengths where a row goes from a warp to its
whole CTA (512 entries), with few long rows and with one in most CTAs.  Rows that
match let the warps be tried, one entry without its counterpart rules them out, and
an entry out of order or out of range is refused, in the middle of a long row as at
its end."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BADARG = -1
fresh_slots = itertools.count(1300)


def bipartite_rows(hubs, leaves):
    """Every hub (ids 0..) wired to every leaf."""
    rows = [hubs + np.arange(leaves)] * hubs + [np.arange(hubs)] * leaves
    off = np.zeros(hubs + leaves + 1, np.uint64)
    off[1:] = np.cumsum([len(r) for r in rows])
    return off, np.concatenate(rows).astype(np.uint32)


def upload(sb, off, adj):
    n = len(off) - 1
    return sb.Graph.upload(sb.CSR(n, False, off, adj, off, adj, np.zeros(n, np.uint32), 1, 4))


def tried(sb, g):
    job = sb.Probabilistic(g, 0.2, 0.1, alpha=0.0, alpha_given=True, slots=next(fresh_slots))
    try:
        job.step(1)
    except sb.SilvanError as err:  # a walk over a missing entry
        assert err.code == sb.E_STATE
    return job.sampler_info()["warp_tried"] > 0


@pytest.mark.parametrize("hubs,leaves", [(2, 511), (2, 512), (2, 513), (3, 767), (5, 4001),
                                         (1500, 700)])
def test_long_rows_are_checked_to_the_end(sb, hubs, leaves):
    off, adj = bipartite_rows(hubs, leaves)
    assert tried(sb, upload(sb, off, adj))
    for at in (leaves // 2, leaves - 1):  # of the last hub's row
        k = int(off[hubs - 1]) + at
        one_way = np.delete(adj, k)
        o = off.copy()
        o[hubs:] -= 1
        assert not tried(sb, upload(sb, o, one_way))
        for value in (adj[k - 1], len(off) - 1):
            bad = adj.copy()
            bad[k] = value
            with pytest.raises(sb.SilvanError) as err:
                upload(sb, off, bad)
            assert err.value.code == BADARG
