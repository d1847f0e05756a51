"""libhx's host code on the CPU: its objects linked with tests/cpp/host_cudart.cpp in
place of the CUDA runtime, and a script run against that library in a process of its own
(a write past a buffer ends the process)."""
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PRELUDE = """
import ctypes, sys
sys.path.insert(0, {root!r})
import hashinator_gb300 as hx
lib = hx.lib({lib!r})
lib.fake_find.restype = ctypes.c_void_p
lib.fake_find.argtypes = [ctypes.c_size_t]
lib.fake_fail_pool_from.argtypes = [ctypes.c_size_t]
lib.fake_pool_held.restype = ctypes.c_uint64
lib.fake_capacity.argtypes = [ctypes.c_uint64]
KEYS = 1 << 20  # an address: nothing reads it here
"""


def host_library(tmp_path) -> Path:
    from hashinator_gb300 import build
    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    build.build_lib()
    out = tmp_path / "libhx_host.so"
    include = Path(nvcc).resolve().parents[1] / "include"
    cxx = shutil.which("g++") or shutil.which("c++")
    objs = [str(build.BUILD / (Path(s).stem + ".o")) for s in build.CUDA_SOURCES]
    subprocess.run([cxx, "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", f"-I{include}",
                    str(ROOT / "tests" / "cpp" / "host_cudart.cpp"), *objs, "-o", str(out), "-ldl"], check=True)
    return out


def run_on_host(tmp_path, script: str) -> None:
    lib = host_library(tmp_path)
    r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=str(ROOT), lib=str(lib)) + script],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, f"exit {r.returncode}\n{r.stdout[-2000:]}{r.stderr[-3000:]}"
