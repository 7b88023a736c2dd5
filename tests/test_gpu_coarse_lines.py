"""Several short grid lines a block, wide lines, and long coarsest grids, in the coarse solve.

Coarsest grids of more than 64 lines take up to 32 unknowns a block, so a block may hold whole lines
and the last one fewer; the grids here put the lines on either side of that number and of a
whole number of blocks, with one line a block where two do not fit, in both line directions, take
lines of 58 to 64 unknowns (64 a block, of which none is staged in shared memory), and go on to grids
whose vectors fill a row's shared memory or no longer fit it (the banded factorisation with blocks of
32 and of 64, which more than 64 rows of the former take too).  A one-level hierarchy's V-cycle is the
solve alone: ``z = A^{-1} r``, against scipy's sparse factorisation.

Tolerance: with dofs held every four nodes the matrices' condition numbers stay under 1e3 (measured on
the CPU), so two backward-stable FP64 solves agree to 1e-12 or so; FP32 rounding of the right-hand
side and the result (2^-24 each, amplified by at most the square root of the condition number in these
norms) to 2e-6.
"""

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(28, 28, 2), (31, 31, 2), (40, 30, 2), (30, 44, 2), (80, 31, 2), (62, 1, 2), (63, 1, 2), (64, 1, 2),
         (65, 2, 1), (70, 7, 2), (71, 8, 2), (95, 1, 1), (3, 150, 2), (300, 2, 2), (600, 1, 1), (700, 1, 2),
         (1200, 3, 1), (500, 13, 2), (250, 30, 2), (2047, 3, 2), (3000, 3, 2), (700, 20, 2)]
CASES = [(*g, 3) for g in GRIDS] + [(400, 13, 2, 64), (400, 13, 2, 65), (200, 27, 2, 65)]


def _problem(nelx, nely, d, rows):
    rng = np.random.default_rng(nelx * 10 + nely + d)
    nn = (nelx + 1) * (nely + 1)
    rho = rng.uniform(0.1, 1.0, (rows, nelx * nely))
    mask = np.ones((nely + 1, nelx + 1, d), bool)
    mask[::4, ::4] = False
    mask[-1, -1, -1] = False
    return rho, mask.reshape(-1), rng.standard_normal((rows, nn * d)) * mask.reshape(-1)


def _matrix(rho, mask, nelx, nely, d):
    KE = O.plane_stress_KE(0.3) if d == 2 else O.diffusion_KE()
    edof = O.element_dof_map(nelx, nely, d)
    n = mask.size
    i, j = np.repeat(edof, edof.shape[1], axis=1).reshape(-1), np.tile(edof, edof.shape[1]).reshape(-1)
    K = sp.coo_matrix(((rho[:, None] * KE.reshape(1, -1)).reshape(-1), (i, j)), shape=(n, n)).tocsc()
    free = np.flatnonzero(mask)
    return K[free][:, free], free


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nelx,nely,d,rows", CASES)
def test_short_lines_and_long_grids(pkg, nelx, nely, d, rows, precision):
    from sttopt_b200 import torch_mg

    dev = torch.device("cuda")
    rho, mask, r = _problem(nelx, nely, d, rows)
    KE = O.plane_stress_KE(0.3) if d == 2 else O.diffusion_KE()
    levels = torch_mg.build_hierarchy(torch.tensor(rho, device=dev),
                                      torch.tensor(O.element_dof_map(nelx, nely, d), device=dev),
                                      torch.tensor(KE, device=dev), torch.tensor(mask, device=dev), nelx, nely,
                                      max_coarse_elements=nelx * nely, precision=precision)
    assert len(levels) == 1
    z = torch_mg.VCycle(levels)(torch.tensor(r, device=dev)).cpu().numpy()
    tol = 1e-11 if precision == "fp64" else 1e-5
    for s in sorted({0, 1, rows // 2, rows - 1}):
        K, free = _matrix(rho[s], mask, nelx, nely, d)
        want = np.zeros(mask.size)
        want[free] = spl.spsolve(K, r[s][free])
        assert np.linalg.norm(z[s] - want) <= tol * np.linalg.norm(want), (s, np.linalg.norm(z[s] - want) / np.linalg.norm(want))
        assert not z[s][~mask].any()
