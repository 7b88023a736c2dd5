"""The assemble and advance passes' tile at the edges of its 8 x 8 products.

Its rows are the constraints and one or two more, padded with zeros; of 23, 24, 47 and 48 constraints
and more blocks than the 148 SMs the advance pass stores no padding, and a product's rows past the last
repeat it and are not read.  The numbers of constraints put the last product's first, second and last
row there, through both entry points: ``mmasub`` (rows rebuilt from the gradients) and ``subsolv`` (P
and Q given), against the oracle's.

Bound: 1e-9 of each output's largest magnitude, what the same outputs are held to elsewhere.
"""

import numpy as np
import pytest
import torch

from oracle import mma_oracle as M

pytestmark = pytest.mark.gpu
TOL = 1e-9


def _check(got, want):
    for k, (g, w) in enumerate(zip(got, want)):
        g = g.detach().cpu().numpy() if torch.is_tensor(g) else np.asarray(g)
        w = np.asarray(w)
        scale = max(float(np.abs(w).max()), 1e-300)
        assert float(np.abs(g.reshape(-1) - w.reshape(-1)).max()) <= TOL * scale, k


@pytest.mark.parametrize("m,n", [(5, 300), (6, 300), (7, 520), (14, 300), (15, 700), (22, 300), (23, 600), (24, 513),
                                 (31, 500), (39, 600), (46, 600), (47, 700), (48, 513), (55, 600), (62, 600),
                                 (63, 700), (64, 900), (23, 148 * 256), (23, 148 * 256 + 1), (24, 38200),
                                 (47, 38200), (48, 148 * 256 + 1)])
def test_tile_rows(pkg, m, n):
    from sttopt_b200 import mma

    rng = np.random.default_rng(1000 * m + n)
    x = rng.uniform(0.2, 0.8, n)
    zero, one = np.zeros(m), np.ones(m)
    args = (m, n, 1, x, np.zeros(n), np.ones(n), x.copy(), x.copy(), 0.0, rng.standard_normal(n) / n,
            rng.uniform(-0.3, 0.1, m), rng.standard_normal((m, n)) / n, np.zeros(n), np.ones(n), 1.0, zero, 1e3 * one,
            one)
    t = lambda v: torch.as_tensor(v).cuda() if isinstance(v, np.ndarray) else v
    _check(mma.mmasub(*map(t, args)), M.mmasub(*args))
    low, upp = x - 0.5, x + 0.5
    alfa, beta = np.maximum(0.0, x - 0.2), np.minimum(1.0, x + 0.2)
    P, Q = rng.uniform(0, 1, (m, n)) / n, rng.uniform(0, 1, (m, n)) / n
    b = (P / (upp - x) + Q / (x - low)).sum(1) + rng.uniform(-0.1, 0.3, m)
    args = (m, n, 1e-7, low, upp, alfa, beta, rng.uniform(0.01, 1, n) / n, rng.uniform(0.01, 1, n) / n, P, Q, 1.0, zero,
            b, 1e3 * one, one)
    _check(mma.subsolv(*map(t, args)), M.subsolv(*args))
