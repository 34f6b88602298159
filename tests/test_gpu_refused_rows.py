"""Counts after an upload whose bitmap rows the device has no room for."""
import pytest

pytestmark = pytest.mark.gpu

PATTERNS = ["0111101111011110", "0101101001011010", "011101110", "0111110111110111110111110"]


def test_counts_after_a_refused_upload(gat):
    g = gat.Graph.rmat(22, 1 << 20, seed=3, device=True)
    g.upload(hub_max_bytes=0)
    ex = gat.Executor()
    schedules = [gat.Schedule(p, "exact") for p in PATTERNS]
    want = [ex.count(g, s).count for s in schedules]
    off, _ = g.csr()
    rows = int((off[1:] > off[:-1]).sum())
    assert rows * (1 << 19) > 200 << 30  # a row is 2^22 bits
    with pytest.raises(gat.GatError, match="GAT_ERR_MEMORY"):
        g.upload(hub_min_degree=1, hub_max_bytes=1 << 50)
    assert g.hubs(True) == 0
    assert [ex.count(g, s).count for s in schedules] == want
