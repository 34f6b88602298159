"""Builds the library's host code against a CUDA runtime that lives in host
memory (fake_gpu.cpp)."""
import ctypes as C
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent
ROOT = HERE.parents[1]
CSRC = ROOT / "graphautotune_b200" / "csrc"
SOURCES = [HERE / "fake_gpu.cpp", *(CSRC / f"{n}.cpp" for n in
                                    ("schedule", "plan", "graph", "devmem", "capi"))]
SLOTS = ("refuse", "throw", "misuse", "live", "pending", "c5_launches", "c5_grid", "c5_bitmaps",
         "searches", "cliques", "deep_rows")
NEVER = 2 ** 63 - 1


def build(folder: Path) -> Path:
    from graphautotune_b200.build import nvcc

    cuda = Path(nvcc()).resolve().parents[1] / "include"
    objs = []
    for s in SOURCES:
        objs.append(folder / (s.stem + ".o"))
        procs = [*(procs if len(objs) > 1 else []), subprocess.Popen(
            ["g++", "-O1", "-std=c++17", "-fPIC", "-fopenmp", "-I", str(cuda), "-I", str(CSRC),
             "-I", str(ROOT / "include"), "-c", str(s), "-o", str(objs[-1])])]
    assert not any([p.wait() for p in procs])
    out = folder / "libgat_fake.so"
    subprocess.run(["g++", "-shared", "-fopenmp", "-Wl,-Bsymbolic", "-o", str(out), *map(str, objs)],
                   check=True)
    return out


class Fake:
    """The library on the fake runtime; `state` counts and injects."""

    def __init__(self, path: Path):
        self.lib = C.CDLL(str(path))
        self._state = (C.c_int64 * len(SLOTS)).in_dll(self.lib, "fake_state")

    def during(self, call) -> None:
        """call() runs while each counting kernel does (None: nothing)."""
        self._during = C.CFUNCTYPE(None)(call) if call else None
        C.c_void_p.in_dll(self.lib, "fake_during").value = (
            C.cast(self._during, C.c_void_p).value if call else None)

    def __getitem__(self, name: str) -> int:
        return self._state[SLOTS.index(name)]

    def __setitem__(self, name: str, value: int) -> None:
        self._state[SLOTS.index(name)] = value
