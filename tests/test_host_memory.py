"""The library's handling of device memory, on a CUDA runtime in host memory
(fake_gpu): what a call leaves behind when an allocation is refused."""
import gc

import numpy as np
import pytest

import fake_gpu

K4, C4 = "0111101111011110", "0101101001011010"
C5 = "0001100101010101010011000"
HOUSE = "0100110110010110110010100"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return fake_gpu.Fake(fake_gpu.build(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def on_fake(gat, fake, monkeypatch):
    """The package's classes on the fake runtime."""
    from graphautotune_b200 import _lib

    for name, (res, args) in _lib._SIGS.items():
        fn = getattr(fake.lib, name)
        fn.restype, fn.argtypes = res, args
    gc.collect()
    monkeypatch.setattr(_lib, "_lib", fake.lib)
    for name in fake_gpu.SLOTS:
        if name != "live":
            fake[name] = fake_gpu.NEVER if name in ("refuse", "throw") else 0
    yield fake
    gc.collect()  # handles go where they came from


def test_bitmaps_that_do_not_fit(gat, on_fake):
    """The upload that cannot get its bitmaps says so and leaves no part of
    them; counts that follow, single and batched, run without bitmaps."""
    g = gat.Graph.barabasi_albert(2000, 4, 1)
    g.upload()  # 64 KB of neighbours, 8 KB a table of vertices
    ex = gat.Executor()
    for p in (K4, C4, HOUSE, C5):  # (the executor keeps the scratch of these)
        ex.count(g, gat.Schedule(p, "exact"))
    assert on_fake["c5_bitmaps"] == 1
    g.upload(hub_min_degree=0)
    live = on_fake["live"]
    on_fake["refuse"] = 100_000
    for degree_order in (True, False):
        with pytest.raises(gat.GatError, match="GAT_ERR_MEMORY"):
            g.upload(degree_order=degree_order)
        if degree_order:
            assert on_fake["live"] == live
        for p in (C5, K4, C4, HOUSE):
            ex.count(g, gat.Schedule(p, "exact"))
        assert on_fake["c5_bitmaps"] == 0
    # the copy with the given ids makes its bitmaps when a count asks for them
    g.upload(hub_min_degree=0)
    with pytest.raises(gat.GatError, match="GAT_ERR_MEMORY"):
        g.upload()
    ref = gat.Schedule(HOUSE, "ref")
    with pytest.raises(gat.GatError, match="GAT_ERR_MEMORY"):
        ex.count(g, ref)
    ex.count(g, ref)
    on_fake["refuse"] = fake_gpu.NEVER  # (a batch has scratch of its own)
    b = gat.Batch()
    for p in (C5, HOUSE):
        b.add(g, gat.Schedule(p, "exact"))
    b.prepare(cuda_graph=False)
    b.run()
    assert on_fake["c5_bitmaps"] == 0
    g.upload()
    ex.count(g, gat.Schedule(C5, "exact"))
    assert on_fake["c5_bitmaps"] == 1
    assert on_fake["misuse"] == 0


def _counted(gat, g, cfg):
    """One count and one batch of the 5-cycle under a configuration."""
    s = gat.Schedule(C5, "exact")
    gat.Executor(cfg).count(g, s)
    yield "count"
    b = gat.Batch()
    b.add(g, s)
    b.prepare(cfg, cuda_graph=False)
    b.run()
    yield "batch"


def test_five_cycles_take_num_blocks(gat, on_fake):
    g = gat.Graph.barabasi_albert(500, 4, 1)
    cfg = gat.Config.engine_default()
    for blocks, grid in ((7, 7), (0, 200), (10_000, 200)):  # 100 SMs of two CTAs
        cfg.num_blocks = blocks
        for how in _counted(gat, g, cfg):
            assert on_fake["c5_grid"] == grid, how


def test_five_cycles_without_bitmaps(gat, on_fake):
    """hub_bitmaps = 0: never, where the graph has them."""
    g = gat.Graph.barabasi_albert(500, 4, 1)
    cfg = gat.Config.engine_default()
    for flag in (1, 0):
        cfg.hub_bitmaps = flag
        for how in _counted(gat, g, cfg):
            assert on_fake["c5_bitmaps"] == flag, how


UPLOADS = [dict(hub_min_degree=0), dict(degree_order=False), dict(hub_min_degree=20), dict()]


def test_batches_keep_their_arrays(gat, on_fake):
    """A prepared batch counts on the arrays it was prepared with, whatever
    its graphs' later uploads let go of; nothing stays behind the batch."""
    gat.Graph.barabasi_albert(500, 4, 1).upload()
    gc.collect()
    none = on_fake["live"]  # (what the pool itself holds)
    g = gat.Graph.barabasi_albert(500, 4, 1)
    g.upload()
    live = on_fake["live"]
    b = gat.Batch()
    for p, mode in ((C5, "exact"), (HOUSE, "exact"), (HOUSE, "ref")):
        b.add(g, gat.Schedule(p, mode))
    b.prepare(cuda_graph=False)
    for again in UPLOADS:
        g.upload(**again)
        b.run()
        assert on_fake["misuse"] == 0, again
    del b
    gc.collect()
    g.upload()
    assert on_fake["live"] == live
    del g
    gc.collect()
    assert on_fake["live"] == none


@pytest.mark.parametrize("pattern,mode", [(C5, "exact"), (K4, "exact"), (C4, "exact"),
                                          (HOUSE, "exact"), (HOUSE, "ref")])
def test_counts_keep_their_arrays(gat, on_fake, pattern, mode):
    """A graph uploaded again by another thread while a count runs."""
    g = gat.Graph.barabasi_albert(500, 4, 1)
    ex, s = gat.Executor(), gat.Schedule(pattern, mode)
    try:
        for again in UPLOADS:
            g.upload()
            ex.count(g, s)  # (the given-id copy's bitmaps are made on first use)
            on_fake.during(lambda: g.upload(**again))
            ex.count(g, s)
            on_fake.during(None)
            assert on_fake["misuse"] == 0, again
    finally:
        on_fake.during(None)


def test_host_memory_runs_out_before_the_copies(gat, on_fake):
    """A graph from host arrays whose host copy cannot be allocated: no copy
    from the caller's arrays is on its way when the call ends."""
    import ctypes as C

    off, adj = gat.Graph.barabasi_albert(500, 4, 1).csr()
    call = on_fake.lib.fake_from_csr_device
    call.argtypes = [C.c_int32, C.c_int64, C.c_void_p, C.c_void_p]
    args = (500, len(adj), off.ctypes.data, adj.ctypes.data)
    on_fake["throw"] = off.nbytes
    live, on_fake["pending"] = on_fake["live"], 0
    try:
        assert call(*args) == -1
    finally:
        on_fake["throw"] = fake_gpu.NEVER
    assert on_fake["pending"] == 0 and on_fake["live"] == live


def test_uploads_after_a_device_reset(gat, on_fake):
    """cudaDeviceReset takes the library's pool with it, with handles alive or
    not; the addresses are given out again."""
    s = gat.Schedule(HOUSE, "exact")
    old = [(gat.Executor(), gat.Graph.barabasi_albert(500, 4, 1)) for _ in range(2)]
    old[0][0].count(old[0][1], s)
    del old[0]
    for _ in range(2):
        on_fake.lib.fake_reset()
        ex, g = gat.Executor(), gat.Graph.barabasi_albert(500, 4, 1)
        ex.count(g, s)
        g.upload(hub_min_degree=0)
        ex.count(g, s)
        assert on_fake["misuse"] == 0
        del ex, g
        gc.collect()
    del old
    gc.collect()
    assert on_fake["misuse"] == 0
