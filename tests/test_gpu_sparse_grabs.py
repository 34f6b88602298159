"""Sparse graphs, whose queues are handed out several roots or units at a time,
and the forms of the search kernel with and without bitmap rows: counts of one
path against another's, whole and in shards and root ranges."""
import pytest

pytestmark = pytest.mark.gpu

K4, K5, C4 = "0111101111011110", "0111110111110111110111110", "0101101001011010"
HOUSE, CYCLE5, PATH5 = ("0100110110010110110010100", "0001100101010101010011000",
                        "0100010100010100010100010")


def _executor(gat, **fields):
    c = gat.Config.engine_default()
    for k, v in fields.items():
        setattr(c, k, v)
    return gat.Executor(c)


def _graphs(gat):
    yield gat.Graph.barabasi_albert(70001, 1, 3)     # a tree with hubs
    yield gat.Graph.barabasi_albert(150001, 2, 3)    # hubs, wide form
    yield gat.Graph.erdos_renyi(120001, 2.0, 5)      # no rows
    yield gat.Graph.erdos_renyi(9001, 14.0, 5)       # rows of every vertex
    yield gat.Graph.rmat(16, 1 << 16, seed=7)


def test_roots_taken_several_at_a_time(gat):
    dedicated, plan = gat.Executor(), _executor(gat, special_kernels=2)
    for g in _graphs(gat):
        V = g.info()[0]
        for p in (K4, K5, C4):
            s = gat.Schedule(p, "exact")
            want = plan.count(g, s).count
            assert dedicated.count(g, s).count == want, (V, p)
            assert sum(dedicated.count_shard(g, s, i, 5)[0] for i in range(5)) == want
            cuts = (0, 1, 7, V // 3, V - 1, V)
            parts = [dedicated.count_range(g, s, a, b)[0] for a, b in zip(cuts, cuts[1:])]
            assert sum(parts) == want, (V, p)


def test_kernel_forms(gat):
    """With rows, without them (by flag and by upload), and instrumented."""
    rows, plain = _executor(gat, special_kernels=2), _executor(gat, special_kernels=2, hub_bitmaps=0)
    wide = _executor(gat, special_kernels=2, threads_per_warp=8, chunk=1)
    for g in _graphs(gat):
        for p in (HOUSE, CYCLE5, PATH5, "0011001111011110"):
            for mode in ("exact", "ref"):
                s = gat.Schedule(p, mode)
                want = rows.count(g, s).count
                assert plain.count(g, s).count == want, (g.info(), p, mode)
                assert wide.count(g, s).count == want, (g.info(), p, mode)
                assert rows.count(g, s, balg=True).count == want
        s = gat.Schedule(HOUSE, "exact")
        want = rows.count(g, s).count
        g.upload(hub_min_degree=8, hub_max_bytes=1 << 30)
        assert rows.count(g, s).count == want
        g.upload(hub_max_bytes=0)
        assert rows.count(g, s).count == want
