"""The 5-cycle by path counts (cycles5.cu) against the CPU oracle, the
schedule plan (special_kernels = 2), root ranges and shards (which follow the
plan), instrumented counts and batched jobs."""
from math import comb

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C5 = "0100110100010100010110010"
RELABELLED = "0001100101010101010011000"


def _complete(gat, n):
    off = np.arange(0, n * (n - 1) + 1, n - 1)
    adj = np.concatenate([np.delete(np.arange(n), i) for i in range(n)])
    return gat.Graph.from_csr(off, adj.astype(np.int32))


def _star_ring(gat, n):
    """A hub joined to a ring of n: every root but the hub has few lower
    neighbours and the hub's row is the longest; the last ids are isolated."""
    ring = np.arange(1, n + 1)
    u = np.concatenate([np.zeros(n, int), ring])
    v = np.concatenate([ring, np.roll(ring, -1)])
    a, b = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((b, a))
    off = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n + 9))])
    return gat.Graph.from_csr(off, b[order].astype(np.int32))


@pytest.fixture(scope="module")
def executors(gat):
    cfg = gat.Config.engine_default()
    cfg.special_kernels = 2
    return gat.Executor(), gat.Executor(cfg)


@pytest.mark.parametrize("n", [3, 5, 6, 9, 33, 257])
def test_complete_graphs(gat, executors, n):
    """12 five-cycles on every five vertices."""
    g = _complete(gat, n)
    s = gat.Schedule(C5, "exact")
    for ordered in (True, False):
        g.upload(degree_order=ordered)
        assert executors[0].count(g, s).count == 12 * comb(n, 5)


@pytest.mark.parametrize("make", ["er", "ba", "rmat", "star", "er_rows_off"])
def test_against_oracle_and_plan(gat, oracle, executors, make):
    g = {"er": lambda: gat.Graph.erdos_renyi(500, 9.0, 3),
         "er_rows_off": lambda: gat.Graph.erdos_renyi(300, 14.0, 4),
         "ba": lambda: gat.Graph.barabasi_albert(701, 7, 5),
         "rmat": lambda: gat.Graph.rmat(9, 8 << 9, seed=6),
         "star": lambda: _star_ring(gat, 300)}[make]()
    if make == "er_rows_off":
        g.upload(hub_max_bytes=0)
    off, adj = g.csr()
    want = oracle.exact_count(off, adj, C5)
    b = gat.Batch()
    for p in (C5, RELABELLED):
        for variant in range(min(2, gat.Schedule.variants(p))):
            s = gat.Schedule(p, "exact", variant=variant)
            r = executors[0].count(g, s)
            assert r.count == want and r.raw_sum == want * r.divisor
            assert executors[1].count(g, s).count == want
            assert executors[0].count(g, s, balg=True).count == want
            raw = [executors[0].count_shard(g, s, i, 4) for i in range(4)]
            assert sum(x for x, _ in raw) == want * raw[0][1].divisor
            raw = [executors[0].count_range(g, s, lo, hi)
                   for lo, hi in ((0, 1), (1, 77), (77, len(off) - 1))]
            assert sum(x for x, _ in raw) == want * raw[0][1].divisor
            b.add(g, s)
            b.add_shard(g, s, 0, 1)
    b.add(g, gat.Schedule("011101110", "exact"))
    for graph in (True, False):
        b.prepare(cuda_graph=graph)
        for _ in range(2):
            b.run()
            got = b.counts()
            assert got[0] == want and got[-1] == oracle.exact_count(off, adj, "011101110")
            assert all(x in (want, want * r.divisor) for x in got[:-1])


def test_batch_of_five_cycles_alone(gat, oracle):
    graphs = [gat.Graph.barabasi_albert(200 + 31 * i, 5, i) for i in range(3)]
    b = gat.Batch()
    s = gat.Schedule(C5, "exact")
    for g in graphs:
        b.add(g, s)
    b.prepare()
    b.run()
    assert b.counts() == [oracle.exact_count(*g.csr(), C5) for g in graphs]


def test_at_the_largest_graph_that_fits(gat, executors):
    """Graphs either side of the shared-memory limit, and of the rule that
    leaves large sparse graphs to the plan, agree with the plan path."""
    s = gat.Schedule(C5, "exact")
    for n, d in ((90001, 14.0), (104001, 14.0), (39999, 5.0), (40001, 5.0)):
        g = gat.Graph.erdos_renyi(n, d, n)
        assert executors[0].count(g, s).count == executors[1].count(g, s).count
