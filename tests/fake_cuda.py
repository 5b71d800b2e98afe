"""The library's host code over a stand-in for the CUDA runtime (cpp/fake_cudart.cpp):
which kernels a call launches, without a GPU.  Addresses passed to it are only
looked at for their alignment.  Run in a process of its own per case, since the
library keeps what it learned of a device."""
from __future__ import annotations

import ctypes
import json
import re
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
PKG = ROOT / "efficient-dpp_gb300"
CLUSTER, COOPERATIVE, PROGRAMMATIC = 1, 2, 4
IN, OUT, IN1, OUT1, LOC, WS = (k << 40 for k in range(1, 7))  # 16-byte-aligned addresses
BIG = 1 << 42  # bytes of any workspace
KERNELS = {k for f in (PKG / "csrc").glob("*.cu*") for k in re.findall(r"\b\w+_kernel\b", f.read_text())}


def build(folder: Path) -> Path:
    import shutil
    nvcc = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve()
    lib = folder / "lib" / "libedpp_fake.so"  # no tuning table beside it
    lib.parent.mkdir(parents=True, exist_ok=True)
    objs = [str(o) for o in sorted((PKG / "_build").glob("*.o"))]
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-Wl,-Bsymbolic", "-o", str(lib),
                    f"-I{nvcc.parent.parent / 'include'}", str(ROOT / "tests/cpp/fake_cudart.cpp"),
                    *objs, "-ldl", "-pthread"], check=True)
    return lib


class Fake:
    def __init__(self, path):
        sys.path.insert(0, str(PKG))
        import edpp
        self.lib = ctypes.CDLL(str(path))
        for name, (res, args) in edpp.SIGNATURES.items():
            f = getattr(self.lib, name)
            f.restype, f.argtypes = res, args
        self.lib.fake_log.restype = ctypes.c_char_p

    def launches(self, call, refuse=0, blocks_per_sm=2):
        """(status, [(kernel, blocks, kind, its mangled template arguments)]) of call(lib)."""
        self.lib.fake_reset(refuse, blocks_per_sm)
        status = call(self.lib)
        out = []
        for line in self.lib.fake_log().decode().splitlines():
            name, blocks, kind = line.split()
            kernel, = (k for k in KERNELS if f"{len(k)}{k}" in name)  # of the mangled name
            out.append([kernel, int(blocks), int(kind), name.split(kernel, 1)[1]])
        return status, out


def run(path, source: str):
    """Runs `source` (which sets `result`, JSON values) with `fake` in a new process."""
    code = ("import json, sys\nsys.path.insert(0, sys.argv[1])\nfrom fake_cuda import *\n"
            "fake = Fake(sys.argv[2])\n" + source + "\nprint(json.dumps(result))\n")
    r = subprocess.run([sys.executable, "-c", code, str(Path(__file__).parent), str(path)],
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    return json.loads(r.stdout.splitlines()[-1])
