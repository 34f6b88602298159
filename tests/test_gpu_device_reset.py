"""A process that resets its device goes on with new handles."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import ctypes, gc, graphautotune_b200 as g
K4 = "0111101111011110"
rt = ctypes.CDLL("libcudart.so.12", mode=ctypes.RTLD_GLOBAL)  # the one libgat is linked with

def counts():
    gr = g.Graph.barabasi_albert(400, 6, 1)
    ex = g.Executor()
    out = [ex.count(gr, g.Schedule(p, "exact")).count for p in (K4, "0100110110010110110010100")]
    gr.upload(hub_min_degree=8)
    return out + [ex.count(gr, g.Schedule(K4, "exact")).count]

want = counts()
for _ in range(2):
    gc.collect()  # the handles go before their context does
    assert rt.cudaDeviceReset() == 0
    assert counts() == want
print("same", want)
"""


def test_counts_after_a_reset():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=Path(__file__).resolve().parents[1],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
