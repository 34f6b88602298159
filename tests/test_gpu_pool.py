"""The library's device memory pool: graphs uploaded, counted and freed by
several threads on their own streams, and the kept pages given back when the
last handle goes."""
import threading

import pytest

pytestmark = pytest.mark.gpu

K4 = "0111101111011110"


def test_threads_upload_count_and_free(gat, oracle):
    import torch

    graphs = [gat.Graph.barabasi_albert(300 + 57 * i, 6, i) for i in range(4)]
    arrays = [g.csr() for g in graphs]
    want = [oracle.exact_count(o, a, K4) for o, a in arrays]
    bad = []

    def work(i):
        try:
            st = torch.cuda.Stream()
            ex = gat.Executor()
            s = gat.Schedule(K4, "exact")
            for _ in range(12):
                g = gat.Graph.from_csr(*arrays[i], check_symmetry=False, device=True,
                                       stream=st.cuda_stream)
                g.upload(stream=st.cuda_stream)
                whole = ex.count(g, s, stream=st.cuda_stream).count
                parts = sum(ex.count_shard(g, s, k, 3, stream=st.cuda_stream)[0] for k in range(3))
                if (whole, parts) != (want[i], want[i]):
                    bad.append((i, whole, parts, want[i]))
                del g
        except Exception as e:  # a thread's failure is the test's
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_last_handle_gives_the_pages_back():
    """In a process of its own: no other handle may be alive."""
    import subprocess
    import sys
    from pathlib import Path

    code = """
import torch, gc, graphautotune_b200 as g
g.Graph.rmat(10, 1 << 13, seed=1, device=True).upload()
gc.collect(); torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
ex = g.Executor()
gr = g.Graph.rmat(18, 1 << 21, seed=1, device=True); gr.upload()
del gr; gc.collect()
held = torch.cuda.mem_get_info()[0]
del ex; gc.collect()
after = torch.cuda.mem_get_info()[0]
assert held < before - (32 << 20), (before, held)
assert held > before - (2 << 30) - (64 << 20), (before, held)
assert after > before - (32 << 20), (before, after)
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parents[1],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
