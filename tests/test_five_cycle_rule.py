"""Which graphs the 5-cycle's path counts take (c5_fits): either side of the
line as measured on a B200 (times beside the rule), the sizes as the library
sees them on the degree-ordered copy."""
import ctypes as C

import pytest


class View(C.Structure):  # DevGraphView
    _fields_ = [("V", C.c_int32), ("E", C.c_int64), ("off", C.c_void_p), ("adj", C.c_void_p),
                ("lo_off", C.c_void_p), ("lo_total", C.c_int64), ("max_degree", C.c_int32),
                ("max_lower", C.c_int32), ("hub_slot", C.c_void_p), ("bitmaps", C.c_void_p),
                ("bitmap_words", C.c_int64)]


# V, E, largest degree, longest lower list, path / plan in ms
PATHS = [
    (4000, 2040, 4, 3, .022, .042), (16000, 32320, 10, 4, .085, .089),     # sparse and small
    (16384, 8028, 152, 9, .054, .11), (20011, 360000, 785, 19, .82, 11.8),
    (24000, 120000, 15, 6, .24, .35), (32000, 192000, 18, 7, .47, .63),
    (40000, 320400, 23, 9, 1.0, 1.5), (40000, 160000, 679, 6, 1.0, 1.6),
    (64000, 1024640, 37, 16, 5.9, 15.9), (64000, 768640, 32, 12, 4.7, 7.2),
    (64000, 512000, 814, 11, 5.4, 5.9), (65536, 128451, 1351, 35, 2.5, 6.2),
    (95000, 1520000, 36, 16, 10.4, 24.9), (95000, 1710000, 1660, 19, 20., 55.),
]
PLANS = [
    (24000, 48480, 10, 4, .16, .10), (32000, 64320, 9, 4, .27, .11),
    (40000, 40400, 7, 3, .30, .074), (40000, 80400, 9, 4, .51, .10),
    (40000, 160400, 15, 6, .74, .36), (40000, 80000, 268, 4, .77, .53),
    (64000, 320640, 17, 7, 3.0, .87), (64000, 513280, 23, 9, 3.7, 2.6),
    (64000, 256000, 868, 6, 3.6, 2.3), (65536, 32768, 378, 11, .56, .40),
    (95000, 760950, 22, 9, 6.6, 4.0),
    (104001, 1456000, 40, 20, 0, 0),  # the counters do not fit
]


@pytest.mark.parametrize("paths,rows", [(True, PATHS), (False, PLANS)])
def test_the_faster_side_is_taken(gat, paths, rows):
    from graphautotune_b200 import _lib

    fits = getattr(_lib.lib(), "_ZN3gat7c5_fitsERKNS_12DevGraphViewE")
    fits.restype, fits.argtypes = C.c_bool, [C.POINTER(View)]
    for V, E, degree, lower, a, b in rows:
        assert (a < b) == paths
        g = View(V=V, E=E, lo_off=1, lo_total=E // 2, max_degree=degree, max_lower=lower)
        assert fits(C.byref(g)) == paths, (V, E)
