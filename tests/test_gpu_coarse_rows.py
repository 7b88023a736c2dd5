"""The coarse solve and factorisation at every cluster size.

How many CTAs a row takes depends on how many rows there are and how many clusters the device
holds; the blocks' elimination order and sums do not.  So a row of a batch equals, bit for bit, the
same row alone (eight CTAs): with a factor for each row and with one factor shared, for narrow
and wide line blocks (64 unknowns, none of which is staged in shared memory, included), few and
many lines, and numbers of rows on either side of the points where the cluster size changes.
"""

import numpy as np
import pytest
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu


def _levels(rho, nelx, nely, d):
    from sttopt_b200 import torch_mg

    dev = torch.device("cuda")
    mask = np.ones((nely + 1, nelx + 1, d), bool)
    mask[-1] = False
    KE = O.plane_stress_KE(0.3) if d == 2 else O.diffusion_KE()
    levels = torch_mg.build_hierarchy(rho, torch.tensor(O.element_dof_map(nelx, nely, d), device=dev),
                                      torch.tensor(KE, device=dev), torch.tensor(mask.reshape(-1), device=dev), nelx,
                                      nely, max_coarse_elements=nelx * nely, precision="fp64")
    assert len(levels) == 1
    return torch_mg.VCycle(levels)


@pytest.mark.parametrize("rows", [15, 16, 34, 75, 160])
@pytest.mark.parametrize("nelx,nely,d", [(32, 16, 2), (26, 26, 2), (31, 30, 2), (24, 12, 2), (32, 16, 1), (3, 2, 2),
                                         (60, 3, 1)])
def test_rows_do_not_depend_on_the_cluster_size(pkg, nelx, nely, d, rows):
    rng = np.random.default_rng(nelx + rows)
    n = d * (nelx + 1) * (nely + 1)
    rho = torch.tensor(rng.uniform(0.1, 1.0, (rows, nelx * nely)), device="cuda")
    r = torch.tensor(rng.standard_normal((rows, n)), device="cuda")
    z = _levels(rho, nelx, nely, d)(r)
    shared = _levels(rho[0], nelx, nely, d)
    zs = shared(r)
    assert torch.isfinite(z).all()
    for s in sorted({0, 1, rows // 2, rows - 1}):
        assert torch.equal(_levels(rho[s], nelx, nely, d)(r[s]).reshape(-1), z[s]), s
        assert torch.equal(shared(r[s]).reshape(-1), zs[s]), s
