"""The cone filter's kernels at the edges of their tiles: every stencil radius (each its own
kernel), grids one element short of, equal to and past a tile of 32 x 32 (two rows a
thread) or several, smaller than the stencil, one batch row and many; forward with the
projection, and the adjoint.

Against the oracle's explicit matrix at 1e-13 relative: both sides are FP64 sums of at most
225 positive products and one quotient (225 * 2^-53 = 2.5e-14), tanh to an ulp."""

import numpy as np
import pytest
import torch

from conftest import rel_err
from oracle import sttopt_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rmin", [0.7, 1.5, 2.5, 4.0, 4.2, 5.9, 6.5, 8.0])
@pytest.mark.parametrize("nelx,nely,rows", [(31, 31, 3), (32, 32, 150), (33, 33, 2), (65, 31, 5), (5, 3, 2),
                                            (64, 33, 1), (95, 130, 4)])
def test_filter_tiles(pkg, nelx, nely, rows, rmin):
    from sttopt_b200 import filters

    rng = np.random.default_rng(int(10 * rmin) + nelx)
    x = rng.uniform(0, 1, (rows, nely, nelx))
    g = rng.standard_normal((rows, nely, nelx))
    Hm, Hs = O.density_filter(nelx, nely, rmin)
    Hs = np.asarray(Hs).ravel()
    H, _ = filters.density_filter(nelx, nely, rmin)
    X = torch.tensor(x, device="cuda").requires_grad_(True)
    xp, xt = filters.filter_and_project(X, H, 8.0, 0.5)
    (gx,) = torch.autograd.grad(xp, [X], torch.tensor(g, device="cuda"))
    want = (Hm @ x.reshape(rows, -1).T).T / Hs
    den = 2 * np.tanh(4.0)
    t = np.tanh(8.0 * (want - 0.5))
    assert rel_err(xt.cpu().numpy().reshape(rows, -1), want) < 1e-13
    assert rel_err(xp.detach().cpu().numpy().reshape(rows, -1), (np.tanh(4.0) + t) / den) < 1e-13
    back = (Hm @ (g.reshape(rows, -1) * 8.0 * (1 - t * t) / den / Hs).T).T
    assert rel_err(gx.cpu().numpy().reshape(rows, -1), back) < 1e-13 * 10  # signed sums: cancellation
