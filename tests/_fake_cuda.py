"""The library's host code on a CUDA runtime without a device (fake_cudart.cpp): its own objects,
linked with that runtime, in the place of libionsolver.so while a test runs."""
from __future__ import annotations

import ctypes as C
import re
import shutil
import subprocess
from pathlib import Path

import pytest

from ionsolver_gb300 import _native as N
from ionsolver_gb300 import build as B

SOURCE = Path(__file__).resolve().parent / "fake_cudart.cpp"


class Fake:
    def __init__(self, lib: C.CDLL):
        self.lib = lib
        lib.fake_fail.argtypes = [C.c_char_p, C.c_int]
        lib.fake_memory.argtypes = [C.c_size_t]
        lib.fake_used.restype = C.c_size_t
        lib.fake_launch.restype = C.c_char_p

    def fail(self, call: str, times: int = 1) -> None:
        """The next ``times`` calls of a runtime function (or launches of a kernel) fail."""
        self.lib.fake_fail(call.encode(), times)

    def launches(self) -> list[dict]:
        out = []
        g, b, s, d = C.c_uint(), C.c_uint(), C.c_size_t(), C.c_int()
        for i in range(self.lib.fake_launches()):
            name = self.lib.fake_launch(i, C.byref(g), C.byref(b), C.byref(s), C.byref(d)).decode()
            out.append(dict(name=re.sub(r"^.*?\d(?=k_)", "", name), grid=g.value, block=b.value, smem=s.value, device=d.value))
        return out

    def kernel(self, prefix: str) -> dict:
        """The last launch of a kernel."""
        return [x for x in self.launches() if x["name"].startswith(prefix)][-1]


@pytest.fixture
def fake(tmp_path, monkeypatch):
    """A fresh copy of the library on the fake runtime (its static state included)."""
    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    B.build()
    objects = sorted(str(p) for p in B.OUT.glob("*.o"))
    include = Path(B.nvcc()).resolve().parent.parent / "include"
    out = tmp_path / "libionsolver_fake.so"
    # only these names leave the library: the static variables of inline functions would be one in
    # the whole process, and this copy's runtime is not the others'
    names = tmp_path / "names.map"
    names.write_text("{ global: ion_*; fake_*; local: *; };\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", f"-I{include}", str(SOURCE), *objects, "-Wl,-Bsymbolic",
                    f"-Wl,--version-script={names}", "-o", str(out)], check=True)
    lib = C.CDLL(str(out))
    for name, (res, args) in N._SIGS.items():
        f = getattr(lib, name)
        f.restype, f.argtypes = res, args
    monkeypatch.setattr(N, "_lib", lib)
    return Fake(lib)
