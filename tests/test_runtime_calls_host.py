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


@pytest.mark.parametrize("most", [4, 1, 0])
def test_a_device_with_smaller_clusters_takes_those(fake, most):
    """(A partition of a GPU may have fewer SMs together than a cluster of eight needs.)"""
    got = fake(r"""
lib.fake_most(I(case["most"]))
try:
""" + "".join("    " + line + "\n" for line in CYCLE.splitlines()) + r"""
except AssertionError:
    print(json.dumps("none"))
else:
    print(json.dumps([vcycle(), pcg(), lib.fake_cluster(b"tree_factor_kernel"), lib.fake_cluster(b"tree_solve_kernel")]))
""", d=2, nelx=40, nely=20, mce=200, prec=1, rows=2, most=most)
    assert got == ("none" if most == 0 else [0, 0, most, most]), got


@pytest.mark.parametrize("d,nelx,nely,blocks", [(1, 600, 1, 38), (2, 1, 600, 76), (2, 300, 2, 61), (2, 100, 7, 51),
                                                (2, 80, 8, 81), (2, 45, 15, 46), (1, 63, 1, 64)])
def test_short_lines_of_a_long_coarsest_grid_share_blocks(fake, d, nelx, nely, blocks):
    """The elimination's steps follow from the number of blocks: more than 64 lines go up to 32 unknowns a
    block."""
    got = fake(CYCLE + r"""
print(json.dumps(dict(blocks=lib.fake_blocks(b"tree_assemble_kernel"), rc=vcycle(),
                      solves=lib.fake_launches(b"tree_solve_kernel"))))
""", d=d, nelx=nelx, nely=nely, mce=700, prec=0, rows=1)
    assert got == dict(blocks=blocks, rc=0, solves=1), got


@pytest.mark.parametrize("nelx,nely,rows,kernel", [
    (32, 16, 128, "tree_factor_kernel"), (500, 13, 64, "tree_factor_kernel"),
    (500, 13, 65, "band_factor_tiled_kernelILi2E"), (3000, 3, 1, "band_factor_tiled_kernelILi2E"),
    (700, 20, 1, "band_factor_tiled_kernelILi4E"), (40, 38, 1, "band_factor_kernel")])
def test_long_and_wide_coarsest_grids_take_their_factorisation(fake, nelx, nely, rows, kernel):
    got = fake(CYCLE + r"""
print(json.dumps([lib.fake_launches(case["kernel"].encode()), vcycle()]))
""", d=2, nelx=nelx, nely=nely, mce=nelx * nely, prec=0, rows=rows, kernel=kernel)
    assert got == [1, 0], got


@pytest.mark.parametrize("mce,kernel,early", [(1520, "coarse_solve_kernel", 0), (700, "tree_solve_kernel", 1)])
def test_the_chain_of_a_banded_coarse_solve_is_not_launched_early(fake, mce, kernel, early):
    got = fake(CYCLE + r"""
print(json.dumps([vcycle(), lib.fake_early(case["kernel"].encode()), lib.fake_early(b"restrict")]))
""", d=2, nelx=80, nely=76, mce=mce, prec=0, rows=2, kernel=kernel)
    assert got == [0, early, 1], got


MMA = r"""
n = case.get("n", 600)

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


@pytest.mark.parametrize("nelx,nely,rows,small", [(180, 60, 1, 1), (180, 60, 12, 1), (180, 60, 13, 0), (256, 128, 4, 1),
                                                  (540, 270, 1, 0), (2048, 1024, 1, 0)])
def test_small_filter_launches_take_small_tiles(fake, nelx, nely, rows, small):
    """Fewer 32 x 32 tiles than SMs: tiles of 32 x 8, one row a thread."""
    got = fake(r"""
nx, ny, rows = case["nelx"], case["nely"], case["rows"]
x, a, b = (mem(rows * nx * ny) for _ in range(3))
rcs = [lib.stt_cone_filter(I(nx), I(ny), I(rows), D(4.0), x, L(nx * ny), a, b, L(nx * ny), D(8.0), D(0.5), None),
       lib.stt_cone_filter_adjoint(I(nx), I(ny), I(rows), D(4.0), x, L(nx * ny), a, L(nx * ny), D(8.0), D(0.5), b,
                                   L(nx * ny), None)]
print(json.dumps(rcs + [lib.fake_launches(b"cone_filter_kernelILi%dELi3ELi%dELi%dE" % (adj, *tile))
                        for adj in (0, 1) for tile in ((1, 8), (2, 16))]))
""", nelx=nelx, nely=nely, rows=rows)
    assert got == [0, 0] + 2 * [small, 1 - small], got


@pytest.mark.parametrize("d,nelx,nely,rows,split", [(1, 24, 24, 1, 0), (1, 1023, 1023, 1, 0), (1, 1023, 1023, 2, 1),
                                                    (2, 24, 24, 1, 1)])
def test_small_one_dof_applies_take_one_loop(fake, d, nelx, nely, rows, split):
    got = fake(r"""
from oracle import sttopt_oracle as O

d, nx, ny, rows = (case[k] for k in ("d", "nelx", "nely", "rows"))
n = d * (nx + 1) * (ny + 1)
rc = lib.stt_q4_apply(I(0), I(d), I(nx), I(ny), I(rows), mem(8), L(n), mem(8), L(n), mem(8), L(nx * ny), None, L(0), None,
                      I(0), arr(O.plane_stress_KE(0.3) if d == 2 else O.diffusion_KE()), None)
print(json.dumps([rc] + [lib.fake_launches(b"q4_apply_modal_kernelILi%dEdLi0ELb%dE" % (d, k)) for k in (0, 1)]))
""", d=d, nelx=nelx, nely=nely, rows=rows)
    assert got == [0, 1 - split, split], got


CYCLE = r"""
from oracle import sttopt_oracle as O

d, nelx, nely, mce, prec, rows = (case[k] for k in ("d", "nelx", "nely", "mce", "prec", "rows"))
KE = arr(O.plane_stress_KE(0.3) if d == 2 else O.diffusion_KE())
wb = lib.stt_hier_workspace_bytes(I(d), I(nelx), I(nely), I(rows), I(mce), I(prec))
h = P()
rho = mem(rows * nelx * nely)
assert lib.stt_hier_create(ctypes.byref(h), mem(wb, np.uint8), L(wb), I(d), I(nelx), I(nely), I(rows), rho,
                           L(nelx * nely), None, L(0), None, KE, I(mce), I(prec), None) == 0, lib.stt_last_error()
nd = d * (nelx + 1) * (nely + 1)
nd += nd % 2
r, z = mem(rows * nd), mem(rows * nd)
ws = lib.stt_solve_workspace_bytes(h, I(rows), I(1))
w = mem(ws, np.uint8)

def vcycle():
    return lib.stt_vcycle(h, I(rows), r, L(nd), z, L(nd), D(0.6), I(2), I(1), w, L(ws), None)

def pcg():
    rel, conv, n = mem(rows), mem(rows, np.int32), mem(1, np.int32)
    return lib.stt_pcg_mg(h, I(rows), r, L(nd), z, L(nd), I(0), D(1e-8), I(5), D(0.6), I(2), I(1), I(0), I(0), I(0),
                          rel, conv, n, w, L(ws), None)
"""


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("d,nelx,nely,mce,kernel", [
    (2, 40, 20, 200, "tree_solve_kernel"), (1, 40, 20, 200, "tree_solve_kernel"), (2, 16, 8, 700, "tree_solve_kernel"),
    (2, 72, 70, 1300, "coarse_solve_kernel")])
def test_a_refused_coarse_solve_fails_the_call(fake, d, nelx, nely, mce, kernel, prec):
    """A coarse solve that does not run leaves the level's vector as it was: the V-cycle and the
    PCG must say so, whatever the launches after it did, and a later call must not."""
    got = fake(CYCLE + r"""
kernel = case["kernel"].encode()
before = [vcycle(), pcg(), lib.fake_launches(kernel)]
lib.fake_refuse(kernel)
refused = [vcycle(), pcg()]
message = lib.stt_last_error().decode()
lib.fake_refuse(b"")
print(json.dumps(dict(before=before, refused=refused, message=message, after=[vcycle(), pcg()])))
""", d=d, nelx=nelx, nely=nely, mce=mce, prec=prec, rows=2, kernel=kernel)
    assert got["before"][:2] == [0, 0] and got["before"][2] > 0, got
    assert got["refused"] == [5, 5] and "refused by the test" in got["message"], got  # STT_ERR_CUDA
    assert got["after"] == [0, 0], got


@pytest.mark.parametrize("rows", [1, 15, 16, 30, 31, 60, 120])
@pytest.mark.parametrize("d,nelx,nely", [(2, 32, 16), (2, 26, 26), (1, 32, 16)])
def test_the_coarse_solve_runs_all_rows_at_once_where_it_can(fake, d, nelx, nely, rows):
    """The runtime here holds 120 CTAs of any cluster size.  A row takes as many as leave room for
    all rows (twice as many rows as clusters would run one half after the other)."""
    got = fake(CYCLE + r"""
lib.fake_forget()
rc = vcycle()
print(json.dumps(dict(rc=rc, solve=lib.fake_cluster(b"tree_solve_kernel"))))
""", d=d, nelx=nelx, nely=nely, mce=700, prec=0, rows=rows)
    assert got["rc"] == 0 and got["solve"] in (1, 2, 4, 8), got
    assert rows * got["solve"] <= 120, got
    assert rows > 15 or got["solve"] == 8, got


@pytest.mark.parametrize("m", [22, 23, 24, 46, 47, 48])
def test_the_advance_pass_leaves_room_for_two_blocks_an_sm(fake, m):
    """With more blocks than SMs: 228 KB an SM, less 1 KB a block for the system and 0.5 KB of
    static memory."""
    got = fake(MMA + r"""
rc = subsolv(case["m"])
print(json.dumps(dict(rc=rc, smem=lib.fake_largest_smem(b"ELb1EE"), launches=lib.fake_launches(b"ELb1EE"))))
""", m=m, n=148 * 256 + 1)
    assert got["rc"] == 0 and got["launches"] > 0
    assert 2 * (got["smem"] + 1536) <= 228 << 10, got
