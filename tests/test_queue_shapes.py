"""How the queues of sparse graphs are cut, and which kernels their rows serve:
the sides that were faster on a B200 (figures beside the rules)."""
import ctypes as C
import gc

import pytest

import fake_gpu
from test_five_cycle_rule import View as _View


class View(C.Structure):  # DevGraphView
    _fields_ = [*_View._fields_, ("deep_rows", C.c_bool)]


def _clique_less(n, edges):
    return "".join("1" if (i, j) in edges or (j, i) in edges else "0"
                   for i in range(n) for j in range(n))


PRISM = _clique_less(6, {(0, 1), (1, 2), (0, 2), (3, 4), (4, 5), (3, 5), (0, 3), (1, 4), (2, 5)})
HOUSE, CYCLE5 = "0100110110010110110010100", "0001100101010101010011000"


def _plan(gat, pattern):
    from graphautotune_b200 import _lib

    s, n = gat.Schedule(pattern, "exact"), C.c_size_t()
    _lib.check(_lib.lib().gat_schedule_plan(s._h, None, 0, C.byref(n)))
    buf = C.create_string_buffer(n.value)
    _lib.check(_lib.lib().gat_schedule_plan(s._h, buf, n.value, C.byref(n)))
    return buf


# V, E, largest degree, longest lower list; patterns; whether grabs are large
@pytest.mark.parametrize("V,E,degree,lower,patterns,large", [
    (1 << 18, 1 << 20, 18, 7, (PRISM, HOUSE, CYCLE5), True),       # uniform, sparse
    (1 << 18, 1 << 21, 27, 9, (PRISM, HOUSE, CYCLE5), True),
    (1 << 20, 8 << 20, 5000, 11, (PRISM, HOUSE), True),            # many units
    (65536, 262140, 868, 6, (PRISM,), True),                       # no dense core
    (65536, 262140, 868, 6, (HOUSE, CYCLE5), False),
    (1 << 18, 500000, 3080, 40, (PRISM, HOUSE, CYCLE5), False),    # dense core
    (1024, 12000, 346, 40, (PRISM, HOUSE, CYCLE5), False),         # few units
])
def test_units_per_grab(gat, V, E, degree, lower, patterns, large):
    from graphautotune_b200 import _lib

    lib = _lib.lib()
    fill = lib["_ZN3gat14batch_fill_jobEPvPK7GatPlanRS2_RKNS_12DevGraphViewEibiii"]
    grabs = lib["_ZN3gat15batch_job_grabsEPvRK7GatPlanllii"]
    grabs.restype = C.c_int64
    tasks = lib["_ZN3gat15batch_job_tasksEPKv"]
    tasks.restype = C.c_int64
    size = lib["_ZN3gat15batch_job_bytesEv"]
    size.restype = C.c_size_t
    g = View(V=V, E=E, off=8, adj=8, lo_off=8, lo_total=E // 2, max_degree=degree,
             max_lower=lower)
    for p in patterns:
        plan = _plan(gat, p)
        job = C.create_string_buffer(size())
        fill(job, None, plan, C.byref(g), 0, C.c_bool(True), 0, 0, 0)
        per_grab = tasks(job) / grabs(job, plan, C.c_int64(E), C.c_int64(4736), 32, 8)
        assert (per_grab >= 4) if large else (per_grab <= 2), (p, per_grab)


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.Fake(fake_gpu.build(tmp_path_factory.mktemp("fake")))


def test_rows_that_deep_plans_leave_alone(gat, fake, monkeypatch):
    """Graphs without long rows whose bitmap rows hold few of the entries."""
    from graphautotune_b200 import _lib

    for name, (res, args) in _lib._SIGS.items():
        fn = getattr(fake.lib, name)
        fn.restype, fn.argtypes = res, args
    gc.collect()
    monkeypatch.setattr(_lib, "_lib", fake.lib)
    ex = gat.Executor()
    for g, deep in ((gat.Graph.erdos_renyi(5000, 2.0, 1), 0), (gat.Graph.erdos_renyi(40000, 16.0, 1), 0),
                    (gat.Graph.erdos_renyi(2000, 12.0, 1), 1), (gat.Graph.barabasi_albert(30000, 2, 1), 1)):
        for mode in ("exact", "ref"):
            ex.count(g, gat.Schedule(HOUSE, mode))
            assert fake["deep_rows"] == deep, (g.info(), mode)
    del ex, g
    gc.collect()
