"""A row map written by the kernel just before a V-cycle.

On a hierarchy of one level the V-cycle is the coarse solve alone, which is launched while the
kernel before it still runs and fetches its factor early; which factor, the row map says.  The
map's new rows are written behind some milliseconds of other work on the same stream, so a map
read early gives the rows it held before (also rows of the hierarchy).  Every result equals, bit
for bit, the same solve with the map at rest.
"""

import ctypes

import numpy as np
import pytest
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelx,nely,mce", [(7, 5, 700), (31, 15, 700), (48, 32, 200)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_row_map_written_just_before(pkg, nelx, nely, mce, precision):
    from sttopt_b200 import _lib, torch_mg

    lib, dev, H = _lib.lib(), torch.device("cuda"), 4
    rng = np.random.default_rng(nelx)
    n = 2 * (nelx + 1) * (nely + 1)
    mask = np.ones((nely + 1, nelx + 1, 2), bool)
    mask[-1] = False
    t = lambda a: torch.tensor(a, device=dev)
    levels = torch_mg.build_hierarchy(t(rng.uniform(0.1, 1.0, (H, nelx * nely))), t(O.element_dof_map(nelx, nely)),
                                      t(O.plane_stress_KE(0.3)), t(mask.reshape(-1)), nelx, nely,
                                      max_coarse_elements=mce, precision=precision)
    h = levels[0]._hier
    r = t(rng.standard_normal(n) * mask.reshape(-1)).repeat(3, 1).contiguous()
    rows = torch.zeros(3, dtype=torch.int32, device=dev)
    view = ctypes.c_void_p()
    _lib.check(lib.stt_hier_select(h.handle, _lib.ptr(rows), ctypes.byref(view)))
    ws = _lib.workspace(lib.stt_vcycle_workspace_bytes(view, 3, 1), dev)

    def cycle():
        z = torch.empty_like(r)
        _lib.check(lib.stt_vcycle(view, 3, _lib.ptr(r), n, _lib.ptr(z), n, 0.6, 2, 1, _lib.ptr(ws), ws.numel(),
                                  _lib.stream()))
        return z

    maps = [torch.tensor(rng.permutation(H)[:3].astype(np.int32), device=dev) for _ in range(12)]
    want = []
    for m in maps:
        rows.copy_(m)
        torch.cuda.synchronize()
        want.append(cycle())
    torch.cuda.synchronize()
    busy = torch.rand(2048, 2048, device=dev)
    got = []
    for m in maps:
        busy = (busy @ busy).clamp_(0, 1)
        torch.add(m, 0, out=rows)
        got.append(cycle())
    torch.cuda.synchronize()
    _lib.check(lib.stt_hier_destroy(view))
    for a, b in zip(got, want):
        assert torch.equal(a, b)
