"""The marching operator at the edges of its bands and strips.

A block marches a band of 32 node rows over strips of 30 node columns; bands whose loads all
lie inside the grid take a loop without range tests, the others the tested one.  The grids
put the last band's end and its look-ahead on either side of that rule (64 to 134 rows of
nodes, the smallest with two bands up to four), with strips that end on, before and after
the grid's edge, for one and two dofs a node, both precisions and every option (input and
output projection, reaction term), against the oracle's FP64 product.

Tolerance: an output adds at most 4 elements' 8 products, and the modal form takes fewer than
64 roundings on the way to it, none on a magnitude above S = 4 max(rho) max_i sum_j |KE_ij|
max|u| (the reaction term adds max|rdiag| max|u|), so 64 u S with u the unit roundoff.
"""

import numpy as np
import pytest
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(58, 63), (59, 64), (60, 67), (61, 68), (29, 69), (30, 70), (31, 71), (89, 95), (90, 99), (91, 101),
         (119, 102), (8, 103), (121, 133)]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("d", [1, 2])
@pytest.mark.parametrize("nelx,nely", GRIDS)
def test_apply_at_band_and_strip_edges(pkg, nelx, nely, d, dtype):
    from sttopt_b200 import _lib

    lib = _lib.lib()
    rng = np.random.default_rng(nelx * 1000 + nely * 2 + d)
    rows, nn = 2, (nelx + 1) * (nely + 1)
    n = nn * d
    KE = O.plane_stress_KE(0.3) if d == 2 else O.diffusion_KE()
    edof = O.element_dof_map(nelx, nely, d)
    # inputs that FP32 holds exactly, so that the oracle sees the same ones
    f32 = lambda a: a.astype(np.float32).astype(np.float64)
    rho = f32(rng.uniform(1e-3, 1.0, (rows, nelx * nely)))
    u = f32(rng.standard_normal((rows, n)))
    rdiag = f32(rng.uniform(0.0, 0.5, (rows, n)))
    free = rng.uniform(size=n) > 0.1
    flags = np.zeros(nn, np.uint8)
    for k in range(d):
        flags |= ((~free.reshape(nn, d)[:, k]).astype(np.uint8) << k).astype(np.uint8)
    dev = torch.device("cuda")
    t = lambda a: torch.tensor(a, dtype=dtype, device=dev)
    U, R, RD, FX = t(u), t(rho), t(rdiag), torch.tensor(flags, device=dev)
    code = _lib.STT_FP64 if dtype == torch.float64 else _lib.STT_FP32
    S = 4.0 * rho.max() * np.abs(KE).sum(1).max() * np.abs(u).max() + rdiag.max() * np.abs(u).max()
    tol = 64.0 * (2.0 ** -53 if dtype == torch.float64 else 2.0 ** -24) * S
    for fl in (0, _lib.STT_PROJECT_OUT, _lib.STT_PROJECT_IN | _lib.STT_PROJECT_OUT):
        for react in (False, True):
            out = torch.full_like(U, float("nan"))
            _lib.check(lib.stt_q4_apply(code, d, nelx, nely, rows, _lib.ptr(U), n, _lib.ptr(out), n, _lib.ptr(R),
                                        nelx * nely, _lib.ptr(RD) if react else None, n if react else 0,
                                        _lib.ptr(FX) if fl else None, fl, _lib.dbl_array(KE.ravel()),
                                        _lib.stream()))
            got = out.cpu().numpy().astype(np.float64)
            v = u * free if fl & _lib.STT_PROJECT_IN else u
            want = O.matvec(v, rho, edof, KE, n)
            if react:
                want = want + rdiag * v
            if fl & _lib.STT_PROJECT_OUT:
                want = want * free
            assert np.abs(got - want).max() <= tol, (fl, react)
