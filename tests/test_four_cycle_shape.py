"""Which shape the 4-cycle's root kernel takes: the one that was faster on a B200
(figures beside the rule)."""
import ctypes as C

import pytest


@pytest.mark.parametrize("V,E,heavy,threads", [
    (32768, 467954, 194, 1024), (20011, 360000, 25, 512), (65536, 727718, 675, 1024),
    (131072, 1942160, 834, 1024), (131072, 999462, 828, 512), (65000, 1169910, 88, 512),
    (262144, 2986414, 1002, 512), (1 << 20, 31400304, 9000, 512)])
def test_four_cycle_root_shape(gat, V, E, heavy, threads):
    from graphautotune_b200 import _lib

    f = _lib.lib()["_ZN3gat15c4_root_threadsEill"]
    assert f(V, C.c_int64(E), C.c_int64(heavy)) == threads
