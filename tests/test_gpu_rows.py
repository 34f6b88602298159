"""Bitmap rows below the hubs (graphs small enough for the rows to stay in
L2): counts with them, without them and with hubs alone agree with the CPU
oracle, and the number of hubs reported is the caller's threshold's alone."""
import pytest

pytestmark = pytest.mark.gpu

PATTERNS = ["011101110", "0111101111011110", "0100110110010110110010100", "0001100101010101010011000",
            "0111110111110111110111110"]


@pytest.mark.parametrize("kind,a,b", [("er", 33, 9.0), ("ba", 257, 12), ("er", 1000, 30.0),
                                      ("er", 127, 60.0), ("er", 129, 60.0)])
def test_rows_below_the_hubs(gat, oracle, golden_schedules, kind, a, b):
    g = gat.Graph.erdos_renyi(a, b, 3) if kind == "er" else gat.Graph.barabasi_albert(a, b, 3)
    off, adj = g.csr()
    cfg = gat.Config.engine_default()
    cfg.hub_bitmaps = 0
    plain, rows = gat.Executor(cfg), gat.Executor()
    cfg = gat.Config.engine_default()
    cfg.special_kernels = 2  # cliques by the plan: bounded intersections of rows
    lanes = gat.Executor(cfg)
    deg = off[1:] - off[:-1]
    for min_degree, max_bytes in ((512, 1 << 30), (int(deg.max()), 1 << 30), (512, 4096), (0, 0)):
        g.upload(hub_min_degree=min_degree, hub_max_bytes=max_bytes)
        words = (a + 31) // 32 * 4
        hubs = min(int((deg >= min_degree).sum()), max_bytes // words) if min_degree else 0
        assert g.hubs(True) == hubs and g.hubs(False) == hubs
        for p in PATTERNS:
            want = oracle.exact_count(off, adj, p)
            s = gat.Schedule(p, "exact")
            assert rows.count(g, s).count == want == plain.count(g, s).count, (p, min_degree)
            assert lanes.count(g, s).count == want, (p, min_degree)
        r = gat.Schedule("0111101111011110", "ref")
        st, want, _ = oracle.ref_engine(off, adj, golden_schedules["0111101111011110"])
        assert st == 0 and rows.count(g, r).count == want == plain.count(g, r).count
