"""The work queue of the plan interpreter: two-level plans whose lanes take
units of different rows (run_pairs), units handed to the whole tile because
their lists are far longer than their neighbours', and grabs that shrink with
the units left.  Counts against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TWO_LEVEL = ["001001110", "011101110", "0001000100011110", "0001001001011010",
             "0001001101011110", "0011001111011110", "0001100011000111110111110"]


def _hub_and_rows(gat, n, hub, seed):
    """A sparse ring with chords, one vertex joined to `hub` others, and the
    last ids isolated: short rows, one long row, empty rows."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([np.arange(n), np.arange(n), np.full(hub, n // 2)])
    v = np.concatenate([(np.arange(n) + 1) % n, (np.arange(n) + rng.integers(2, 5, n)) % n,
                        rng.choice(n, hub, replace=False)])
    keep = u != v
    e = np.unique(np.concatenate([np.stack([u, v], 1)[keep], np.stack([v, u], 1)[keep]]), axis=0)
    off = np.zeros(n + 40 + 1, np.int64)
    np.add.at(off, e[:, 0] + 1, 1)
    return gat.Graph.from_csr(np.cumsum(off), e[:, 1].astype(np.int32))


@pytest.mark.parametrize("tile,block,chunk,blocks", [(32, 256, 8, 0), (32, 64, 64, 1), (16, 128, 1, 3),
                                                     (8, 256, 64, 0), (1, 128, 16, 7)])
def test_two_level_units_of_many_rows(gat, oracle, tile, block, chunk, blocks):
    c = gat.Config.engine_default()
    c.threads_per_warp, c.threads_per_block, c.chunk, c.num_blocks = tile, block, chunk, blocks
    ex = gat.Executor(c)
    b = gat.Batch()
    want = []
    # 31, 33: fewer units than a tile and one more; 700 of 900: lists long
    # enough for the hand-over to the tile
    for n, hub in ((7, 3), (31, 5), (33, 30), (900, 700)):
        g = _hub_and_rows(gat, n, hub, n)
        off, adj = g.csr()
        for p in TWO_LEVEL:
            s = gat.Schedule(p, "exact")
            want.append(oracle.exact_count(off, adj, p))
            assert ex.count(g, s).count == want[-1], (n, p)
            parts = [ex.count_shard(g, s, i, 3) for i in range(3)]
            assert sum(r for r, _ in parts) == want[-1] * parts[0][1].divisor, (n, p)
            b.add(g, s)
    b.prepare(c)
    b.run()
    assert b.counts() == want


@pytest.mark.parametrize("tile,blocks", [(32, 0), (8, 0), (1, 0), (32, 1)])
def test_units_split_into_parts(gat, oracle, tile, blocks):
    """Plans of four levels and more on graphs with few units per tile (and,
    with one CTA, many): candidates of level 2 dealt to the parts of a unit."""
    c = gat.Config.engine_default()
    c.threads_per_warp, c.num_blocks, c.special_kernels = tile, blocks, 2
    ex = gat.Executor(c)
    cycle6_chord = "010101101000010100101010000101100010"
    for g in (gat.Graph.erdos_renyi(60, 7.0, 2), gat.Graph.barabasi_albert(90, 4, 3)):
        off, adj = g.csr()
        for p in ("0001100101010101010011000", "0111110111110111110111110", cycle6_chord):
            s = gat.Schedule(p, "exact")
            want = oracle.exact_count(off, adj, p)
            assert ex.count(g, s).count == want, p
            parts = [ex.count_shard(g, s, i, 3) for i in range(3)]
            assert sum(r for r, _ in parts) == want * parts[0][1].divisor, p
