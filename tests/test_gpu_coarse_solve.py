"""The coarsest level's direct solve by odd-even elimination of the grid lines.

A hierarchy whose level 0 is already the coarsest makes the V-cycle that solve alone:
``z = A^{-1} r`` with the projected operator.  It is compared with a dense FP64 solve of the
same matrix on the CPU, for line blocks of every padded width (8 to 64 unknowns, with and
without padding), both line directions, one line up to many (the odd-even order's last
strides with and without a right neighbour), one and two dofs a node, and wide or very long
grids, which take the banded factorisation.

Tolerance: with densities in [0.1, 1] and the left edge and the top row held the matrices'
condition numbers stay under 1e5 (measured on the CPU), so two backward-stable FP64 solves
agree to a few 1e-11; FP32 rounding of the right-hand side and the result (2^-24 each,
amplified by at most the square root of the condition number in these norms) to ~2e-5.
"""

import numpy as np
import pytest
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(2, 1), (1, 2), (3, 3), (7, 3), (5, 17), (16, 8), (17, 9), (40, 11), (13, 31), (26, 19), (33, 23), (25, 26),
         (40, 27), (64, 3), (27, 31), (36, 34), (600, 2), (700, 2)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("d", [1, 2])
@pytest.mark.parametrize("nelx,nely", GRIDS)
def test_coarsest_level_alone_is_an_exact_solve(pkg, nelx, nely, d, precision):
    from sttopt_b200 import torch_mg

    rng = np.random.default_rng(nelx * 100 + nely + d)
    rows, nn = 2, (nelx + 1) * (nely + 1)
    rho = rng.uniform(0.1, 1.0, (rows, nelx * nely))
    KE = O.plane_stress_KE(0.3) if d == 2 else O.diffusion_KE()
    edof = O.element_dof_map(nelx, nely, d)
    mask = np.ones((nely + 1, nelx + 1, d), bool)
    mask[:, 0] = False  # the left edge and the top row held, and one more dof
    mask[0] = False
    mask[nely // 2, -1, -1] = False
    mask = mask.reshape(-1)
    r = rng.standard_normal((rows, nn * d)) * mask
    dev = torch.device("cuda")
    levels = torch_mg.build_hierarchy(torch.tensor(rho, device=dev), torch.tensor(edof, device=dev),
                                      torch.tensor(KE, device=dev), torch.tensor(mask, device=dev), nelx, nely,
                                      max_coarse_elements=nelx * nely, precision=precision)
    assert len(levels) == 1
    z = torch_mg.VCycle(levels)(torch.tensor(r, device=dev)).cpu().numpy()
    tol = 1e-10 if precision == "fp64" else 2e-5
    for s in range(rows):
        K = np.zeros((nn * d, nn * d))
        np.add.at(K, (edof[:, :, None], edof[:, None, :]), rho[s][:, None, None] * KE)
        free = np.flatnonzero(mask)
        want = np.zeros(nn * d)
        want[free] = np.linalg.solve(K[np.ix_(free, free)], r[s][free])
        assert np.linalg.norm(z[s] - want) <= tol * np.linalg.norm(want), (s, nelx, nely)
        assert not z[s][~mask].any()
