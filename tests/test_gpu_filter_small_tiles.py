"""The cone filter's two tile shapes on the same rows.

A batch of rows that fills the GPU takes 32 x 32 tiles and two rows a thread, a row alone 32 x 8 tiles and
one; an output's taps are added in the same order in both, and so is Hs near the border.  So a row of
the batch equals, bit for bit, the row alone: at every radius, on grids whose edges fall on either side
of both tiles' edges and on grids narrower than the stencil, filter and projection, and the adjoint.
"""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rmin", [1.0, 2.0, 2.6, 4.0, 5.0, 6.0, 6.5, 8.0])
@pytest.mark.parametrize("nelx,nely", [(5, 3), (32, 8), (33, 9), (31, 33), (64, 32), (65, 63), (180, 60)])
def test_rows_do_not_depend_on_the_tile(pkg, nelx, nely, rmin):
    from sttopt_b200 import filters

    g = torch.Generator(device="cuda")
    g.manual_seed(nelx + nely)
    rows = 160
    x = torch.rand(rows, nely, nelx, dtype=torch.float64, device="cuda", generator=g)
    w = torch.randn(rows, nely, nelx, dtype=torch.float64, device="cuda", generator=g)
    H, _ = filters.density_filter(nelx, nely, rmin)

    def both(x, w):
        x = x.clone().requires_grad_(True)
        xp, xt = filters.filter_and_project(x, H, 8.0, 0.5)
        (gx,) = torch.autograd.grad(xp, [x], w)
        y = x.detach().clone().requires_grad_(True)
        f = filters.apply_density_filter(y, H)
        (gy,) = torch.autograd.grad(f, [y], w)
        return xp.detach(), xt.detach(), gx, f.detach(), gy

    batch = both(x, w)
    for s in (0, 1, rows - 1):
        for a, b in zip(batch, both(x[s], w[s])):
            assert torch.equal(a[s], b.reshape(a[s].shape)), s
