"""Level 0's FP32 smoothing passes with two columns a lane, at every band height.

A warp marches a band of 4 to 64 rows, the longest that gives each SM its warps, so batches of many
rows reach the longer ones, whose ring of asynchronous copies wraps many times.  The grids end at a band, a row
past it and inside one, with 2 x 2 coarsenings (transfers joined) and others.  As at four rows, the
same hierarchy with a reaction of zeros takes the one-column passes, and both V-cycles are compared with the
FP64 hierarchy's.

Tolerance: both FP32 cycles round the same sums (in another order), so their distances from the
FP64 cycle are of one size: at most four times the other's, plus 16 units of the FP32 roundoff.
"""

import numpy as np
import pytest
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu

CASES = [(122, 126, 300), (122, 126, 150), (122, 126, 80), (122, 126, 40), (118, 128, 300), (118, 128, 160),
         (116, 64, 320), (116, 62, 640), (60, 192, 450), (60, 190, 200), (117, 63, 400), (81, 60, 600)]


def _band(cols, nelx, nely, rows):
    strips, nny, band = -(-(nelx + 1) // cols), nely + 1, 64
    while band > 4 and strips * -(-nny // band) * rows < 148 * (12 if band > 8 else 8):
        band //= 2
    return band


def test_the_cases_reach_every_band():
    for cols in (58, 60):
        assert {_band(cols, *c) for c in CASES} == {8, 16, 32, 64}


@pytest.mark.parametrize("nelx,nely,rows", CASES)
def test_two_column_passes_in_long_bands(pkg, nelx, nely, rows):
    from sttopt_b200 import torch_mg

    rng = np.random.default_rng(nelx * 1000 + nely + rows)
    nn = (nelx + 1) * (nely + 1)
    mask = rng.uniform(size=(nely + 1, nelx + 1, 2)) > 0.01
    mask[:, 0] = False
    dev = torch.device("cuda")
    mask = torch.tensor(mask.reshape(-1), device=dev)
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    rho = 0.1 + 0.9 * torch.rand(rows, nelx * nely, dtype=torch.float64, device=dev, generator=g)
    r = torch.randn(rows, nn * 2, dtype=torch.float64, device=dev, generator=g) * mask
    edof = torch.tensor(O.element_dof_map(nelx, nely, 2), device=dev)
    KE = torch.tensor(O.plane_stress_KE(0.3), device=dev)

    def cycle(precision, reaction=None):
        levels = torch_mg.build_hierarchy(rho, edof, KE, mask, nelx, nely, reaction=reaction,
                                          max_coarse_elements=nelx * nely // 8, precision=precision)
        assert len(levels) > 1
        return torch_mg.VCycle(levels)(r)

    exact = cycle("fp64")
    one, two = cycle("mixed", torch.zeros_like(rho)), cycle("mixed")
    assert not two[:, ~mask].any()
    size = exact.norm(dim=1)
    e1, e2 = (one - exact).norm(dim=1) / size, (two - exact).norm(dim=1) / size
    bad = e2 > 4.0 * e1 + 16 * 2.0 ** -24
    assert not bad.any(), (bad.nonzero().flatten()[:8].tolist(), float(e1.max()), float(e2.max()))
