"""Algorithmic bytes belong to the plan and the graph: the same from any launch
shape, and shards' add up to the whole's."""
import pytest

pytestmark = pytest.mark.gpu

CYCLE5, K5 = "0001100101010101010011000", "0111110111110111110111110"
CYCLE6_CHORD = "010101101000010100101010000101100010"
HOUSE = "0100110110010110110010100"


def _executor(gat, **fields):
    c = gat.Config.engine_default()
    for k, v in fields.items():
        setattr(c, k, v)
    return gat.Executor(c)


@pytest.mark.parametrize("special", [0, 2])
def test_bytes_of_any_shape(gat, special):
    g = gat.Graph.erdos_renyi(60, 7.0, 2)  # few units: those of deep plans are split
    shapes = [dict(), dict(num_blocks=1), dict(num_blocks=7, threads_per_block=64),
              dict(threads_per_warp=8), dict(threads_per_warp=1, chunk=64)]
    executors = [_executor(gat, special_kernels=special, **s) for s in shapes]
    for p in (CYCLE5, K5, CYCLE6_CHORD, HOUSE, "0001001001011010"):
        s = gat.Schedule(p, "exact")
        whole = executors[1].count(g, s, balg=True)
        for ex in executors:
            r = ex.count(g, s, balg=True)
            assert (r.count, r.balg_bytes) == (whole.count, whole.balg_bytes), p
            parts = [ex.count_shard(g, s, i, 3, balg=True) for i in range(3)]
            assert sum(x for x, _ in parts) == whole.raw_sum, p
            assert sum(r.balg_bytes for _, r in parts) == whole.balg_bytes, p
