"""mmasub's gradient rows by sign, in every row chunk and block tail.

The passes sum a row's positive and negative parts, so the rows cover gradients that are all
positive, all negative, mixed and zero (with and without a sign bit), at numbers of
constraints on either side of the row chunks and of variables on either side of a warp and a
block, against the oracle's mmasub.

Bound: 1e-9 of each output's largest magnitude, what the same outputs are held to elsewhere
(the passes round in another order along the same Newton path).
"""

import numpy as np
import pytest
import torch

from oracle import mma_oracle as M

pytestmark = pytest.mark.gpu
TOL = 1e-9


def _case(m, n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.2, 0.8, n)
    g = rng.standard_normal((m, n)) / n
    kinds = rng.integers(0, 5, m)
    kinds[0] = 1
    for i, k in enumerate(kinds):
        if k == 0:
            g[i] = np.abs(g[i])
        elif k == 1:
            g[i] = -np.abs(g[i])
        elif k == 2:
            g[i] = np.where(rng.uniform(size=n) < 0.5, 0.0, -0.0)
        elif k == 3:
            g[i, :: 3] = 0.0
    df0 = rng.standard_normal(n) / n
    zero, one = np.zeros(m), np.ones(m)
    fval = rng.uniform(-0.3, 0.1, m)
    return (m, n, 1, x, np.zeros(n), np.ones(n), x.copy(), x.copy(), 0.0, df0, fval, g, np.zeros(n), np.ones(n), 1.0,
            zero, 1e3 * one, one)


@pytest.mark.parametrize("m,n", [(1, 31), (4, 33), (8, 255), (9, 257), (12, 512), (13, 300), (16, 1000), (17, 1025),
                                 (20, 777), (21, 640), (25, 513), (33, 700), (49, 900)])
def test_gradient_rows_by_sign(pkg, m, n):
    from sttopt_b200 import mma

    args = _case(m, n, 100 * m + n)
    want = M.mmasub(*args)
    t = [torch.as_tensor(v).cuda() if isinstance(v, np.ndarray) else v for v in args]
    got = mma.mmasub(*t)
    for k, (gv, wv) in enumerate(zip(got, want)):
        gv = gv.detach().cpu().numpy() if torch.is_tensor(gv) else np.asarray(gv)
        wv = np.asarray(wv)
        scale = max(float(np.abs(wv).max()), 1e-300)
        assert float(np.abs(gv - wv).max()) <= TOL * scale, (k, float(np.abs(gv - wv).max()) / scale)
