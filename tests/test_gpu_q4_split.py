"""The one-dof operator with and without its loop free of range tests.

Launches of few nodes take the tested loop alone, a batch of many rows the other in bands whose loads
all lie inside the grid; both round an output alike, so a row of the batch equals, bit for bit,
the row alone.  The grids put the last band's end and its look-ahead on either side of the rule
and strips on, before and after the grid's edge, with every option.
"""

import numpy as np
import pytest
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("nelx,nely", [(59, 64), (60, 67), (61, 68), (29, 69), (30, 70), (90, 99), (91, 101), (121, 133)])
def test_rows_do_not_depend_on_the_loop(pkg, nelx, nely, dtype):
    from sttopt_b200 import _lib

    lib = _lib.lib()
    n = (nelx + 1) * (nely + 1)
    rows = (4 << 20) // n + 1
    g = torch.Generator(device="cuda")
    g.manual_seed(nelx)
    rand = lambda *s: torch.rand(*s, dtype=dtype, device="cuda", generator=g)
    U, rho, RD = rand(rows, n) - 0.5, rand(rows, nelx * nely), rand(rows, n)
    FX = (rand(n) < 0.1).to(torch.uint8)
    KE = _lib.dbl_array(O.diffusion_KE().ravel())
    code = _lib.STT_FP64 if dtype == torch.float64 else _lib.STT_FP32

    def apply(u, r, rd, fl):
        out = torch.full_like(u, float("nan"))
        _lib.check(lib.stt_q4_apply(code, 1, nelx, nely, u.shape[0], _lib.ptr(u), n, _lib.ptr(out), n, _lib.ptr(r),
                                    nelx * nely, _lib.ptr(rd), n if rd is not None else 0, _lib.ptr(FX) if fl else None,
                                    fl, KE, _lib.stream()))
        return out

    for fl in (0, _lib.STT_PROJECT_OUT, _lib.STT_PROJECT_IN | _lib.STT_PROJECT_OUT):
        for rd in (None, RD):
            batch = apply(U, rho, rd, fl)
            for s in (0, 1, rows - 1):
                one = apply(U[s:s + 1].clone(), rho[s:s + 1].clone(), None if rd is None else rd[s:s + 1].clone(), fl)
                assert torch.equal(one[0], batch[s]), (fl, s)
