"""4-cycle counter widths: endpoints whose degree, and so whose largest
count, sits at each end of the 2-, 4-, 8-, 16- and 32-bit classes, on graphs
with one hub joined to every middle vertex and endpoints joined to `degree`
consecutive middles (so a count reaches the endpoint's degree).  Whole graph,
root ranges and shards, with and without the degree-ordered copy; one graph's
endpoints fill more than one window.  Counts against the host's wedge count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C4 = "0101101001011010"


def _hub_graph(gat, middles, endpoints, seed, isolated=7):
    """endpoints: (degree, how many)."""
    rng = np.random.default_rng(seed)
    u, v = [np.zeros(middles, np.int64)], [1 + np.arange(middles)]
    at = 1 + middles
    for degree, n in endpoints:
        first = rng.integers(0, middles, n)
        u.append(np.repeat(at + np.arange(n), degree))
        v.append((1 + (first[:, None] + np.arange(degree)) % middles).ravel())
        at += n
    V = at + isolated
    u, v = np.concatenate(u), np.concatenate(v)
    perm = rng.permutation(V)  # ids as given in no order
    a, b = perm[np.concatenate([u, v])], perm[np.concatenate([v, u])]
    order = np.lexsort((b, a))
    off = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=V))])
    return gat.Graph.from_csr(off, b[order].astype(np.int32), check_symmetry=False)


@pytest.mark.parametrize("middles,endpoints", [
    (3, [(2, 5), (3, 5)]),
    (600, [(1, 900), (2, 5000), (3, 5000), (4, 5000)]),
    (600, [(15, 700), (16, 700), (255, 120), (256, 120)]),
    (600, [(2, 400), (3, 400), (4, 400), (15, 400), (16, 400), (255, 40), (256, 40), (599, 20)]),
    (70000, [(65535, 3), (65536, 3), (2, 3000)]),
    (2000, [(2, 500000), (3, 30000), (17, 3000)]),
])
def test_counter_widths(gat, oracle, middles, endpoints):
    g = _hub_graph(gat, middles, endpoints, middles)
    off, adj = g.csr()
    want = oracle.c4_rooted(off, adj, at_largest=True)
    s = gat.Schedule(C4, "exact")
    assert s.dedicated_kernel == 1
    for ordered in (True, False):
        h = gat.Graph.from_csr(off, adj, check_symmetry=False)
        h.upload(degree_order=ordered)
        ex = gat.Executor()
        assert ex.count(h, s).count == want, ordered
        assert ex.count(h, s, balg=True).count == want
        V = len(off) - 1
        cuts = [0, 1, 3, min(V, 600), min(V, 5000), V]
        assert sum(ex.count_range(h, s, a, b)[0] for a, b in zip(cuts, cuts[1:])) == want
        assert sum(ex.count_shard(h, s, i, 3)[0] for i in range(3)) == want
