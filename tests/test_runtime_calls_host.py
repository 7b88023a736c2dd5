"""What the host code asks of the CUDA runtime, without a device.

The library's own objects are linked with ``fake_cudart.cpp``, a runtime that launches nothing and
refuses the launches it is told to, and a child process (so that the two runtimes never meet)
drives them through the C ABI with host memory in the place of device memory.
"""

import json
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

from conftest import ROOT

PKG = ROOT / "spacetime-topology-optimization_b200"

CHILD = r"""
import ctypes, json, sys
import numpy as np
lib = ctypes.CDLL(sys.argv[1])
case = json.loads(sys.argv[2])
P, I, L, D = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_double
for f in ("stt_hier_workspace_bytes", "stt_solve_workspace_bytes", "stt_vcycle_workspace_bytes"):
    getattr(lib, f).restype = L
for f in ("stt_mma_workspace_bytes", "fake_largest_smem", "fake_lowest_ceiling"):
    getattr(lib, f).restype = ctypes.c_size_t
lib.stt_last_error.restype = ctypes.c_char_p
keep = []

def mem(n, dtype=np.float64):
    a = np.zeros(n * np.dtype(dtype).itemsize + 256, np.uint8)
    keep.append(a)
    return P(a.ctypes.data + -a.ctypes.data % 256)

def arr(a):
    a = np.ascontiguousarray(a, np.float64)
    keep.append(a)
    return P(a.ctypes.data)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not cxx or not Path(nvcc).exists():
        pytest.skip("needs g++ and the CUDA toolkit")
    sys.path.insert(0, str(PKG))
    try:
        import build_ext
    finally:
        sys.path.pop(0)
    build_ext.build()
    objs = [build_ext.BUILD / (s.stem + ".o") for s in sorted(build_ext.CSRC.glob("*.cu"))]
    out = tmp_path_factory.mktemp("fake") / "libfake.so"
    subprocess.run([cxx, "-shared", "-fPIC", "-O1", "-Wl,-Bsymbolic", "-I", str(Path(nvcc).resolve().parents[1] / "include"),
                    str(ROOT / "tests" / "fake_cudart.cpp"), *map(str, objs), "-lpthread", "-o", str(out)], check=True)

    def run(body, **case):
        res = subprocess.run([sys.executable, "-c", CHILD + body, str(out), json.dumps(case)], cwd=ROOT,
                             capture_output=True, text=True, timeout=300)
        assert res.returncode == 0, res.stderr[-2000:]
        return json.loads(res.stdout.splitlines()[-1])

    return run


MMA = r"""
n = 600

def subsolv(m):
    ws = lib.stt_mma_workspace_bytes(m, L(n))
    v = [mem(n) for _ in range(6)]
    PQ = [mem(m * n) for _ in range(2)]
    one, out = arr(np.ones(m)), [mem(m + 1) for _ in range(6)]
    return lib.stt_mma_subsolv(I(m), L(n), D(1e-1), *v, *PQ, L(n), D(1.0), one, one, arr(np.full(m, 1000.0)), one,
                               mem(n), mem(n), mem(n), *out, None, None, mem(ws, np.uint8), ctypes.c_size_t(ws), None)
"""


@pytest.mark.parametrize("first,then", [(8, 6), (6, 8), (24, 21), (47, 33), (64, 49)])
def test_an_mma_call_leaves_room_for_larger_ones_of_its_kernel(fake, first, then):
    """Numbers of constraints that share a kernel need different amounts of shared memory.  The
    ceiling belongs to the kernel, so no call may set it to its own size: another thread's call, in
    the middle of its Newton steps, would have its launches refused."""
    got = fake(MMA + r"""
rcs = [subsolv(m) for m in (case["first"], case["then"])]
print(json.dumps(dict(rcs=rcs, launches=lib.fake_launches(b"mma_assemble_kernel"),
                      largest=lib.fake_largest_smem(b"mma_assemble_kernel"),
                      lowest=lib.fake_lowest_ceiling(b"mma_assemble_kernel"))))
""", first=first, then=then)
    assert got["launches"] > 0 and 5 not in got["rcs"], got  # 5: a CUDA call failed
    assert got["lowest"] >= got["largest"], got
