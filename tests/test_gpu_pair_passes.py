"""Level 0's FP32 smoothing passes with two columns a lane, at the edges of strips and bands.

The plane-stress mixed hierarchy without a reaction takes them; the same hierarchy with a
reaction of zeros is the same operator through the one-column passes and separate transfers.
Both V-cycles are compared with the FP64 hierarchy's on the same right-hand side.  The grids put
strips of 58 and 60 columns and bands of 4 to 64 rows on either side of the grid's edges, with
2 x 2 coarsenings (transfers joined) and others, and dofs fixed at random inside the grid.

Tolerance: both FP32 cycles round the same sums (in another order), so their distances from
the FP64 cycle are of one size: at most four times the other's, plus 16 units of the FP32
roundoff.  A wrong row, weight or mask shows at 1e-3.
"""

import numpy as np
import pytest
import torch

from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(56, 24), (58, 32), (60, 34), (62, 66), (114, 36), (116, 62), (118, 64), (120, 68), (122, 126),
         (300, 62), (54, 27), (81, 60), (60, 45), (117, 63)]


@pytest.mark.parametrize("rows", [1, 5])
@pytest.mark.parametrize("nelx,nely", GRIDS)
def test_two_column_passes(pkg, nelx, nely, rows):
    from sttopt_b200 import torch_mg

    rng = np.random.default_rng(nelx * 1000 + nely + rows)
    nn = (nelx + 1) * (nely + 1)
    rho = rng.uniform(0.1, 1.0, (rows, nelx * nely))
    mask = rng.uniform(size=(nely + 1, nelx + 1, 2)) > 0.01
    mask[:, 0] = False
    mask = mask.reshape(-1)
    r = rng.standard_normal((rows, nn * 2)) * mask
    dev = torch.device("cuda")
    t = lambda a: torch.tensor(a, device=dev)
    edof = t(O.element_dof_map(nelx, nely, 2))

    def cycle(precision, reaction=None):
        levels = torch_mg.build_hierarchy(t(rho), edof, t(O.plane_stress_KE(0.3)), t(mask), nelx, nely,
                                          reaction=reaction, max_coarse_elements=nelx * nely // 8, precision=precision)
        assert len(levels) > 1
        return torch_mg.VCycle(levels)(t(r)).cpu().numpy()

    exact = cycle("fp64")
    zero = t(np.zeros((rows, nelx * nely)))
    one, two = cycle("mixed", zero), cycle("mixed")
    assert not two[:, ~mask].any()
    for s in range(rows):
        size = np.linalg.norm(exact[s])
        e1, e2 = np.linalg.norm(one[s] - exact[s]) / size, np.linalg.norm(two[s] - exact[s]) / size
        assert e2 <= 4.0 * e1 + 16 * 2.0 ** -24, (s, e1, e2)
