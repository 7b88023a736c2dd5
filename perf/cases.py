"""The work this framework is used for, as measurable cases over its public entry points.

Every case is one call (or one call and its backward pass) that a topology-optimisation
program makes again and again, on fresh densities of the kind it meets: smoothed noise in
[1e-3, 1], stages cut from a time field that rises from the build plate.

==============  ======================================================================
``path``        what one pass is
==============  ======================================================================
``apply``       the projected operator ``torch_fem.operator`` on a stack of vectors (what a
                caller's own Krylov loop pays per iteration)
``whole``       ``compliance.whole_compliance`` and its gradient: one load case, hierarchy
                build, FP64 MG-PCG, element sensitivities
``loads``       ``torch_solve.femsolve`` with an FP32 V-cycle for several load cases of one
                density, and the gradient of a functional that is not the compliance, so
                the adjoint iterates
``loop``        one iteration of the production loop: the virtual-heat time field, the whole
                structure and every self-weight stage with the smooth stage mask as one
                batched solve, and two Jacobian rows (structure, time) in density and
                diffusivity
``spacetime``   ``spacetime.objective_and_gradient``: heat time field, hard-threshold stages
``uneven``      ``spacetime.objective_and_gradient_many`` on problems of several grid sizes
``mma``         ``mma.unit_box_step``: the optimiser's update after each evaluation
``filter``      ``filters.filter_and_project`` forward and backward
==============  ======================================================================
"""

import math
import random
import types

import numpy as np
import torch

from __graft_entry__ import load_package

load_package()
from sttopt_b200 import (compliance, fem, filters, gravity, load_cases, mma, sensitivity, spacetime,  # noqa: E402
                         torch_fem, torch_mg, torch_solve, virtual_heat)

EMIN, EMAX, PENAL, NU = 1e-9, 1.0, 3.0, 0.3
F64 = torch.float64


def listed():
    return [
        # a batched FP32 apply at the benchmark's grid and stage count: pure bandwidth
        dict(name="apply_f32_2048x1024_16rows", path="apply", nelx=2048, nely=1024, rows=16, dtype="float32", dofs=2),
        # the smallest solve in use (a half MBB beam): launches, synchronisations, one coarse factorisation
        dict(name="whole_mbb_120x40", path="whole", nelx=120, nely=40, support="mbb"),
        # one large FP64 load case
        dict(name="whole_cantilever_1024x512", path="whole", nelx=1024, nely=512, support="cantilever"),
        # load cases on a grid that coarsens by 2 and by 3
        dict(name="loads_540x270_4rows", path="loads", nelx=540, nely=270, rows=4),
        # the production loop at the size it is run at day to day
        dict(name="loop_180x60_8stages", path="loop", nelx=180, nely=60, stages=8, beta_t=20.0, time_map="one_minus"),
        # the space-time objective: a small design study, the gradient-check size in FP64, the benchmark
        dict(name="spacetime_256x128_8stages", path="spacetime", nelx=256, nely=128, stages=8, precision="mixed"),
        dict(name="spacetime_f64_512x256_16stages", path="spacetime", nelx=512, nely=256, stages=16,
             precision="fp64"),
        dict(name="spacetime_2048x1024_16stages", path="spacetime", nelx=2048, nely=1024, stages=16,
             precision="mixed"),
        # many problems of uneven sizes and stage counts at once
        dict(name="uneven_9problems", path="uneven", problems=9, top=768),
        # the update of the 180x60 loop (density and diffusivity, one constraint a stage and one more), and of
        # the benchmark's grid
        dict(name="mma_21600vars_9rows", path="mma", vars=21600, rows=9),
        dict(name="mma_4194304vars_17rows", path="mma", vars=4194304, rows=17),
        # the design variable's filter and projection at the benchmark's grid
        dict(name="filter_2048x1024", path="filter", nelx=2048, nely=1024, rmin=4.0, beta=8.0),
    ]


def draw(rng: random.Random):
    path = rng.choice(["apply", "whole", "loads", "loop", "spacetime", "spacetime", "uneven", "mma", "filter"])
    if path == "apply":
        nelx, nely = rng.randint(24, 2048), rng.randint(24, 1024)
        rows = rng.randint(1, 16)
        return dict(path=path, nelx=nelx, nely=nely, rows=rows, dtype=rng.choice(["float32", "float64"]),
                    dofs=rng.choice([1, 2, 2]))
    if path == "whole":
        nelx, nely = _grid(rng, 3_000, 500_000)
        return dict(path=path, nelx=nelx, nely=nely, support=rng.choice(["mbb", "cantilever"]))
    if path == "loads":
        nelx, nely = _grid(rng, 10_000, 400_000)
        return dict(path=path, nelx=nelx, nely=nely, rows=rng.randint(1, 6))
    if path == "loop":
        nelx, nely = _grid(rng, 2_700, 180_000)
        return dict(path=path, nelx=nelx, nely=nely, stages=rng.randint(3, 12), beta_t=rng.uniform(10.0, 40.0),
                    time_map=rng.choice(["one_minus", "one_minus", "neg_log"]))
    if path == "spacetime":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        nelx, nely = _grid(rng, 8_000, 1_000_000 if precision == "mixed" else 250_000)
        return dict(path=path, nelx=nelx, nely=nely, stages=rng.randint(4, 16), precision=precision)
    if path == "uneven":
        return dict(path=path, problems=rng.randint(3, 9), top=rng.choice([256, 512, 768]))
    if path == "mma":
        n = 2 * int(round(math.exp(rng.uniform(math.log(2_700), math.log(2_000_000)))))
        return dict(path=path, vars=n, rows=rng.randint(2, 20))
    nelx, nely = rng.randint(90, 2048), rng.randint(30, 1024)
    return dict(path="filter", nelx=nelx, nely=nely, rmin=round(rng.uniform(1.5, 6.0), 2),
                beta=rng.choice([1.0, 4.0, 8.0, 32.0]))


def _grid(rng, lo, hi):
    """A grid that coarsens by 2s and 3s to a few hundred elements, its element count spread
    over the logarithm of [lo, hi], at most four times as wide as high."""
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    best = None
    for _ in range(200):
        nely = rng.randint(7, 19)
        nelx = rng.randint(nely, min(4 * nely, 700 // nely))
        while nelx * nely < target / 4:
            nelx *= rng.choice([2, 2, 3])
            nely *= rng.choice([2, 2, 3])
        if rng.random() < 0.5:
            nelx, nely = 2 * nelx, 2 * nely
        if nely <= nelx <= 4 * nely and lo <= nelx * nely <= hi:
            off = abs(math.log(nelx * nely / target))
            if best is None or off < best[0]:
                best = (off, nelx, nely)
    return (best[1], best[2]) if best else (240, 80)


# ---- inputs -------------------------------------------------------------------------


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _cone(rmin):
    r = int(math.ceil(rmin)) - 1
    k = torch.zeros(2 * r + 1, 2 * r + 1, dtype=F64, device="cuda")
    for j in range(-r, r + 1):
        for i in range(-r, r + 1):
            k[j + r, i + r] = max(0.0, rmin - math.hypot(i, j))
    return k[None, None]


def _cone_filter(x, rmin):
    k = _cone(rmin)
    r = k.shape[-1] // 2
    num = torch.nn.functional.conv2d(x[None, None], k, padding=r)
    den = torch.nn.functional.conv2d(torch.ones_like(x)[None, None], k, padding=r)
    return (num / den)[0, 0]


def _smoothed(nelx, nely, g, rmin=4.0):
    """Seeded noise through the cone filter, mapped to [1e-3, 1]."""
    x = _cone_filter(torch.randn(nely, nelx, dtype=F64, device="cuda", generator=g), rmin)
    x = (x - x.min()) / (x.max() - x.min())
    return 1e-3 + (1 - 1e-3) * x


def _body(x, rows, g):
    """Rows of nodal forces: each element's share of a smooth random field times its density."""
    nely, nelx = x.shape
    f = torch.stack([_cone_filter(torch.randn(nely, nelx, dtype=F64, device="cuda", generator=g), 6.0) * x
                     for _ in range(2 * rows)]).reshape(rows, 2, nely, nelx).permute(0, 2, 3, 1)
    return _spread(f.repeat(1, 1, 1, 4) / 4, nelx, nely, 2)


def _uniform(shape, g, lo=-1.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, dtype=F64, device="cuda", generator=g)


def _support(case):
    """Load vector and free dofs: a half MBB beam, or the left edge clamped and a unit load
    at the middle of the right edge."""
    nelx, nely = case["nelx"], case["nely"]
    if case.get("support") == "mbb":
        return load_cases.load_case(load_cases.LoadCase.MBB, nelx, nely, 0.0, 0.0, 1.0)
    return load_cases.mid_right_cantilever(nelx, nely)


def _grid_state(case, dofs=2):
    nelx, nely = case["nelx"], case["nely"]
    KE = torch.as_tensor(fem.plane_stress_KE(NU) if dofs == 2 else fem.diffusion_KE(), dtype=F64, device="cuda")
    edof = torch_mg.element_dof_map_tensor(nelx, nely, torch.device("cuda", torch.cuda.current_device()), dofs)
    return KE, edof, dofs * (nelx + 1) * (nely + 1)


def _uneven_shapes(case):
    sizes = [s for s in ((256, 128), (512, 256), (768, 384)) if s[0] <= case["top"]]
    return [(*sizes[k % len(sizes)], 4 + (5 * k) % 13) for k in range(case["problems"])]


def prepare(case, seed):
    g = _gen(seed)
    s = dict(case=case, path=case["path"])
    path = case["path"]
    if path == "apply":
        nelx, nely, d, rows = case["nelx"], case["nely"], case["dofs"], case["rows"]
        dtype = getattr(torch, case["dtype"])
        KE, edof, ndof = _grid_state(case, d)
        x = _smoothed(nelx, nely, g)
        up = torch.linspace(1, 0, nely, dtype=F64, device="cuda")[:, None]  # built from the plate upwards
        rho = torch.stack([EMIN + (x * (up <= (r + 1) / rows)) ** PENAL for r in range(rows)]).reshape(rows, -1)
        mask = torch.ones((nely + 1, (nelx + 1) * d), dtype=torch.bool, device="cuda")
        mask[-1] = False
        s.update(U=torch.randn(rows, ndof, dtype=F64, device="cuda", generator=g).to(dtype), rho=rho.to(dtype),
                 edof=edof, KE=KE, ndof=ndof, mask=mask.reshape(-1))
    elif path in ("whole", "loads"):
        KE, edof, ndof = _grid_state(case)
        F, free = _support(case)
        free = torch.as_tensor(free, device="cuda")
        x = _smoothed(case["nelx"], case["nely"], g)
        s.update(KE=KE, edof=edof, ndof=ndof, free=free, x=x)
        if path == "whole":
            s.update(F=torch.as_tensor(F, device="cuda"))
        else:  # body forces on the material, and displacement functionals weighted by it
            mask = torch_fem.free_mask(ndof, free, device="cuda")
            s.update(mask=mask, rho=(EMIN + x ** PENAL * (EMAX - EMIN)).reshape(-1),
                     F=_body(x, case["rows"], g) * mask, G=_body(x, case["rows"], g) * mask)
    elif path == "loop":
        nelx, nely = case["nelx"], case["nely"]
        KE, edof, ndof = _grid_state(case)
        _, free = load_cases.build_plate_clamp(nelx, nely)
        F = torch.zeros(nely + 1, nelx + 1, 2, dtype=F64, device="cuda")
        F[0, -1, 1] = -1.0
        s.update(KE=KE, edof=edof, ndof=ndof, free=torch.as_tensor(free, device="cuda"), F=F.reshape(-1),
                 x=_smoothed(nelx, nely, g), mu=_uniform((nely, nelx), g, 0.4, 0.6), w=_uniform((nely, nelx), g),
                 mesh=virtual_heat.ScalarMesh.build(nelx, nely, "bottom_edge", "cuda", F64),
                 C=gravity.gravity_load_matrix(nelx, nely), weights=_uniform(case["stages"], g, 0.5, 1.5),
                 times=[(k + 1) / case["stages"] for k in range(case["stages"])],
                 cfg=types.SimpleNamespace(chi_contrast=1000.0, drain_beta=25.0, time_map=case["time_map"],
                                           heat_cg_rtol=1e-8))
    elif path == "spacetime":
        nelx, nely = case["nelx"], case["nely"]
        s.update(x=_smoothed(nelx, nely, g), w=_uniform((nely, nelx), g),
                 problem=spacetime.SpaceTimeProblem(nelx, nely, torch.device("cuda", torch.cuda.current_device())))
    elif path == "uneven":
        dev = torch.device("cuda", torch.cuda.current_device())
        shapes = _uneven_shapes(case)
        s.update(xs=[_smoothed(a, b, g) for a, b, _ in shapes], ws=[_uniform((b, a), g) for a, b, _ in shapes],
                 stages=[n for _, _, n in shapes],
                 problems={(a, b): spacetime.SpaceTimeProblem(a, b, dev) for a, b, _ in shapes})
    elif path == "mma":
        n, m = case["vars"], case["rows"]
        x = _uniform(n, g, 0.05, 0.95)
        step = torch.randn(2, n, dtype=F64, device="cuda", generator=g) * 0.02
        x1 = (x + step[0]).clamp(0, 1)
        x2 = (x1 + step[1]).clamp(0, 1)
        normal = lambda *shape: torch.randn(*shape, dtype=F64, device="cuda", generator=g)  # noqa: E731
        s.update(x=x, history=mma.History(x1, x2, x - 0.2, x + 0.2), move=_uniform(n, g, 0.02, 0.1),
                 df0dx=normal(n) * (4.0 / n), fval=normal(m) * 0.1, dfdx=normal(m, n) * (4.0 / n))
    else:
        nelx, nely = case["nelx"], case["nely"]
        H, _ = filters.density_filter(nelx, nely, case["rmin"])
        s.update(H=H, x=_smoothed(nelx, nely, g, 2.0), g=_uniform((nely, nelx), g))
    return s


# ---- one pass -----------------------------------------------------------------------


def run(s):
    case, path = s["case"], s["path"]
    if path == "apply":
        return torch_fem.operator(s["U"], s["rho"], s["edof"], s["KE"], s["ndof"], s["mask"])
    if path == "whole":
        x = s["x"].detach().requires_grad_(True)
        c, U = compliance.whole_compliance(x, s["KE"], s["edof"], EMIN, EMAX, PENAL, s["free"], s["F"], s["ndof"])
        (gx,) = torch.autograd.grad(c, [x])
        return dict(c=c.detach(), U=U.detach(), gx=gx)
    if path == "loads":
        rho, F = s["rho"].detach().requires_grad_(True), s["F"].detach().requires_grad_(True)
        U = torch_solve.femsolve(rho, F, s["edof"], s["KE"], s["mask"], case["nelx"], case["nely"],
                                 precision="mixed")
        g_rho, g_F = torch.autograd.grad(U, [rho, F], s["G"])
        return dict(U=U.detach(), g_rho=g_rho, g_F=g_F)
    if path == "loop":
        x, mu = s["x"].detach().requires_grad_(True), s["mu"].detach().requires_grad_(True)
        sol = virtual_heat.heat_time_field(s["cfg"], s["mesh"], x, mu, conduction_penal=3.0)
        c, stages, U = compliance.batched_whole_and_gravity_compliance(
            x, sol.tPhys, s["KE"], s["edof"], EMIN, EMAX, PENAL, s["free"], s["F"], s["ndof"], s["C"],
            case["beta_t"], s["times"])
        stages = torch.stack(stages)
        out = torch.stack([c + (s["weights"] * stages).sum(), (s["w"] * sol.tPhys).sum()])
        gx, gmu = sensitivity.jacobian_rows(out, [x, mu])
        return dict(c=c.detach(), stages=stages.detach(), U=U.detach(), t=sol.tPhys.detach(), gx=gx, gmu=gmu)
    if path == "spacetime":
        return _few(spacetime.objective_and_gradient(s["x"], s["w"], n_stage=case["stages"],
                                                     precision=case["precision"], problem=s["problem"]))
    if path == "uneven":
        return [_few(o) for o in spacetime.objective_and_gradient_many(s["xs"], s["ws"], s["stages"],
                                                                       problems=s["problems"])]
    if path == "mma":
        n = case["vars"]
        x, lam, h = mma.unit_box_step(s["history"], 2, s["x"], s["move"], 0.0, s["df0dx"], s["fval"], s["dfdx"],
                                      a0=1.0, c=1000.0, raa0=1e-5 / n)
        return dict(x=x, lam=lam, low=h.low, upp=h.upp)
    x = s["x"].detach().requires_grad_(True)
    xPhys, xTilde = filters.filter_and_project(x, s["H"], case["beta"], 0.5)
    (gx,) = torch.autograd.grad(xPhys, [x], s["g"])
    return dict(xPhys=xPhys.detach(), xTilde=xTilde, gx=gx)


def _few(o):
    return {k: o[k] for k in ("objective", "c_s", "tPhys", "gradient")}


# ---- what a pass cannot do without ---------------------------------------------------


def work(case):
    path = case["path"]
    if path == "mma":  # the m x n gradient and 7 n-vectors in, 3 out; one Newton matrix
        n, m = case["vars"], case["rows"]
        return dict(bytes=8.0 * n * (m + 10), flops=1.0 * n * m * (m + 20))
    if path == "uneven":
        shapes = _uneven_shapes(case)
        each = [work(dict(path="spacetime", nelx=a, nely=b, stages=n)) for a, b, n in shapes]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    nel, nnode = case["nelx"] * case["nely"], (case["nelx"] + 1) * (case["nely"] + 1)
    if path == "filter":
        taps = math.pi * case["rmin"] ** 2
        return dict(bytes=8.0 * nel * 5, flops=4.0 * nel * taps)
    if path == "apply":
        es, d, rows = (4 if case["dtype"] == "float32" else 8), case["dofs"], case["rows"]
        return dict(bytes=float(es * rows * (2 * d * nnode + nel)), flops=rows * nel * 32.0 * d * d)
    if path == "whole":  # density and load in, displacement and gradient out
        return dict(bytes=8.0 * (2 * nel + 4 * nnode), flops=nel * 1000.0)
    if path == "loads":
        rows = case["rows"]
        return dict(bytes=8.0 * (2 * nel + rows * 8 * nnode), flops=rows * nel * 1000.0)
    if path == "loop":  # densities, diffusivity and weights in; rows of U, t and two rows of two gradients out
        rows = case["stages"] + 1
        return dict(bytes=8.0 * (8 * nel + rows * 2 * nnode), flops=rows * nel * 1000.0)
    return dict(bytes=8.0 * 4 * nel, flops=case["stages"] * nel * 1000.0)  # x, w in; tPhys, gradient out


# ---- the same in plain torch, 64 bits --------------------------------------------------


def _ke(dofs):
    """The bilinear element's matrix (plane stress at nu, or diffusion) by 2 x 2 Gauss
    quadrature, local order bottom-left, bottom-right, top-right, top-left."""
    a = 0.5 / math.sqrt(3.0)
    K = np.zeros((4 * dofs, 4 * dofs))
    C = np.array([[1, NU, 0], [NU, 1, 0], [0, 0, (1 - NU) / 2]]) / (1 - NU * NU)
    for x in (0.5 - a, 0.5 + a):
        for y in (0.5 - a, 0.5 + a):
            dN = np.array([[y - 1, 1 - y, y, -y], [x - 1, -x, x, 1 - x]])
            if dofs == 1:
                K += dN.T @ dN / 4
            else:
                B = np.zeros((3, 8))
                B[0, 0::2], B[1, 1::2] = dN
                B[2, 0::2], B[2, 1::2] = dN[1], dN[0]
                K += B.T @ C @ B / 4
    K = np.round((K + K.T) / 2 * 24 * (1 - NU * NU), 9) / (24 * (1 - NU * NU))
    return torch.as_tensor((K + K.T) / 2, dtype=F64, device="cuda")


def _corners(U, nelx, nely, d):
    """(rows, nely, nelx, 4 d) element dofs of nodal rows."""
    g = U.reshape(-1, nely + 1, nelx + 1, d)
    return torch.cat([g[:, 1:, :-1], g[:, 1:, 1:], g[:, :-1, 1:], g[:, :-1, :-1]], dim=-1)


def _spread(fe, nelx, nely, d):
    """The transpose of ``_corners``."""
    out = fe.new_zeros(fe.shape[0], nely + 1, nelx + 1, d)
    out[:, 1:, :-1] += fe[..., :d]
    out[:, 1:, 1:] += fe[..., d:2 * d]
    out[:, :-1, 1:] += fe[..., 2 * d:3 * d]
    out[:, :-1, :-1] += fe[..., 3 * d:]
    return out.reshape(fe.shape[0], -1)


class _Direct:
    """Block Cholesky of ``K(rho) + diag`` column by column of the grid (fixed dofs held)."""

    def __init__(self, rho, free, nelx, nely, d, rdiag=None):
        self.nelx, self.nely, self.d, self.nb = nelx, nely, d, d * (nely + 1)
        self.rho = rho.reshape(-1, nely, nelx)
        self.KE = _ke(d)
        self.free = free.reshape(nely + 1, nelx + 1, d).permute(1, 0, 2).reshape(nelx + 1, self.nb).to(F64)
        self.rdiag = None if rdiag is None else \
            rdiag.reshape(-1, nely + 1, nelx + 1, d).permute(0, 2, 1, 3).reshape(-1, nelx + 1, self.nb)
        r = torch.arange(nely, device="cuda")[:, None]
        i = torch.arange(d, device="cuda")[None, :]
        self.idx = torch.cat([d * (r + 1) + i, d * r + i], dim=1)  # bottom, top node of an element side
        self.left = torch.cat([torch.arange(d), torch.arange(3 * d, 4 * d)]).cuda()
        self.right = torch.cat([torch.arange(d, 2 * d), torch.arange(2 * d, 3 * d)]).cuda()
        self.L = []
        S = self.diagonal(0)
        for j in range(nelx + 1):
            self.L.append(torch.linalg.cholesky(S))
            if j < nelx:
                W = torch.linalg.solve_triangular(self.L[j], self.couple(j), upper=False)
                S = self.diagonal(j + 1) - W.mT @ W

    def block(self, j, a, b):
        """Element column j's block between node sides a and b."""
        ke = self.KE[a][:, b]
        v = (self.rho[:, :, j, None, None] * ke).reshape(self.rho.shape[0], -1)
        flat = (self.idx[:, :, None] * self.nb + self.idx[:, None, :]).reshape(-1)
        return v.new_zeros(v.shape[0], self.nb * self.nb).index_add_(1, flat, v).reshape(-1, self.nb, self.nb)

    def diagonal(self, j):
        D = 0
        if j < self.nelx:
            D = D + self.block(j, self.left, self.left)
        if j > 0:
            D = D + self.block(j - 1, self.right, self.right)
        if self.rdiag is not None:
            D = D + torch.diag_embed(self.rdiag[:, j])
        f = self.free[j]
        return D * f[:, None] * f[None, :] + torch.diag(1 - f)

    def couple(self, j):
        return self.block(j, self.left, self.right) * self.free[j][:, None] * self.free[j + 1][None, :]

    def solve(self, F):
        n = self.nelx
        g = F.reshape(-1, self.nely + 1, n + 1, self.d).permute(2, 0, 1, 3).reshape(n + 1, -1, self.nb, 1)
        g = g * self.free[:, None, :, None]
        rows = g.shape[1]
        g = [v for v in g]
        pick = (lambda L: L.expand(rows, -1, -1)) if self.rho.shape[0] == 1 else (lambda L: L)
        for j in range(n):
            g[j + 1] = g[j + 1] - self.couple(j).mT @ torch.cholesky_solve(g[j], pick(self.L[j]))
        x = [None] * (n + 1)
        for j in range(n, -1, -1):
            b = g[j] if j == n else g[j] - self.couple(j) @ x[j + 1]
            x[j] = torch.cholesky_solve(b, pick(self.L[j])) * self.free[j][:, None]
        return torch.stack(x)[..., 0].reshape(n + 1, rows, self.nely + 1, self.d).permute(1, 2, 0, 3).reshape(rows, -1)


class _Solve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, rho, F, free, nelx, nely, d, rdiag):
        A = _Direct(rho, free, nelx, nely, d, rdiag)
        U = A.solve(F)
        ctx.A, ctx.shape = A, rho.shape
        ctx.save_for_backward(U)
        return U

    @staticmethod
    def backward(ctx, gU):
        A, (U,) = ctx.A, ctx.saved_tensors
        lam = A.solve(gU)
        le, ue = _corners(lam, A.nelx, A.nely, A.d), _corners(U, A.nelx, A.nely, A.d)
        grho = -((le @ A.KE) * ue).sum(-1).reshape(U.shape[0], -1)
        if A.rho.shape[0] == 1:
            grho = grho.sum(0)
        return (grho.reshape(ctx.shape), lam) + (None,) * 5


def _energy(U, rho, nelx, nely):
    ue = _corners(U, nelx, nely, 2)
    return (rho.reshape(-1, nely, nelx) * ((ue @ _ke(2)) * ue).sum(-1)).sum((1, 2))


def _free(ndof, free):
    m = torch.zeros(ndof, dtype=torch.bool, device="cuda")
    m[free] = True
    return m


def _heat(x, mu, nelx, nely, time_map="one_minus"):
    """The virtual-heat time field (element values), the plate at the bottom."""
    nel = nelx * nely
    chi = ((x.flatten() ** 3).clamp(min=1e-6) * 1000.0 ** (mu.flatten() - 0.5))[None]
    alpha = 25.0 / nel
    plate = torch.zeros(nely + 1, nelx + 1, dtype=F64, device="cuda")
    plate[-1] = 1.0
    rdiag = _spread(torch.full((1, nely, nelx, 4), alpha / 4, dtype=F64, device="cuda"), nelx, nely, 1)
    lift = plate.reshape(1, -1)
    fe = chi.reshape(1, nely, nelx, 1) * (_corners(lift, nelx, nely, 1) @ _ke(1))
    F = -(_spread(fe, nelx, nely, 1) + rdiag * lift)
    T = _Solve.apply(chi, F, lift == 0, nelx, nely, 1, rdiag) + lift
    part = x >= x.max() / 2
    if time_map == "one_minus":
        t = 1 - T
    else:
        floor = 1e-3 * _corners(T, nelx, nely, 1).mean(-1)[0][part].min().detach()
        t = -torch.log(T.clamp(min=0) + floor)
    te = _corners(t, nelx, nely, 1).mean(-1)[0]
    return te / te[part].max().detach()


def _self_weight(xt, nelx, nely):
    fe = xt.reshape(-1, nely, nelx, 1).expand(-1, -1, -1, 4) / (4 * nelx * nely)
    f = -_spread(fe, nelx, nely, 1)
    return torch.stack([torch.zeros_like(f), f], dim=-1).reshape(f.shape[0], -1)


def _clamped_plate(nelx, nely):
    m = torch.ones(nely + 1, nelx + 1, 2, dtype=torch.bool, device="cuda")
    m[-1] = False
    return m.reshape(-1)


def _simp(x):
    return EMIN + x ** PENAL * (EMAX - EMIN)


def _spacetime_exact(x, w, stages):
    nely, nelx = x.shape
    x = x.detach().requires_grad_(True)
    t = _heat(x, torch.full_like(x, 0.5), nelx, nely)
    ts = t.detach().flatten()
    member = torch.stack([(ts <= (k + 1) / stages).to(F64) for k in range(stages)])
    xt = x.flatten() * member
    rho, F = _simp(xt), _self_weight(xt, nelx, nely)
    free = _clamped_plate(nelx, nely)
    c = _energy(_Solve.apply(rho, F, free, nelx, nely, 2, None), rho, nelx, nely)
    J = c.sum() + (w * t).sum()
    (gx,) = torch.autograd.grad(J, [x])
    return dict(objective=J.detach(), c_s=c.detach(), tPhys=t.detach(), gradient=gx)


def _mma_exact(s, n, m):
    """Svanberg's update and the primal-dual barrier solve of its subproblem."""
    x0, h, move = s["x"], s["history"], s["move"]
    osc = (x0 - h.xold1) * (h.xold1 - h.xold2)
    fac = torch.where(osc > 0, 1.2 * torch.ones_like(osc), torch.where(osc < 0, 0.7 * torch.ones_like(osc), 1.0))
    low = torch.minimum(torch.maximum(x0 - fac * (h.xold1 - h.low), x0 - 20.0 * move), x0 - 0.02 * move)
    upp = torch.maximum(torch.minimum(x0 + fac * (h.upp - h.xold1), x0 + 20.0 * move), x0 + 0.02 * move)
    alfa = torch.maximum(low + 0.1 * (x0 - low), x0 - move).clamp(min=0)
    beta = torch.minimum(upp - 0.1 * (upp - x0), x0 + move).clamp(max=1)
    raa = 1e-5 / n
    u0, l0 = upp - x0, x0 - low

    def split(gr):
        p, q = gr.clamp(min=0), (-gr).clamp(min=0)
        e = 0.001 * (p + q) + raa
        return (p + e) * u0 * u0, (q + e) * l0 * l0

    (p0, q0), (P, Q) = split(s["df0dx"]), split(s["dfdx"])
    b = P @ (1 / u0) + Q @ (1 / l0) - s["fval"]
    one = torch.ones(m, dtype=F64, device="cuda")
    a, c, d, a0 = 0 * one, 1000.0 * one, 0 * one, 1.0
    x = (alfa + beta) / 2
    scalar = torch.ones((), dtype=F64, device="cuda")
    pt = [x, one, scalar, one, (1 / (x - alfa)).clamp(min=1), (1 / (beta - x)).clamp(min=1), torch.maximum(one, c / 2),
          scalar, one]

    def kkt(pt, eps):
        x, y, z, lam, xsi, eta, mu, zet, sl = pt
        u, v = upp - x, x - low
        return torch.cat([(p0 + lam @ P) / u ** 2 - (q0 + lam @ Q) / v ** 2 - xsi + eta, c + d * y - mu - lam,
                          (a0 - zet - a @ lam)[None], P @ (1 / u) + Q @ (1 / v) - a * z - y + sl - b,
                          xsi * (x - alfa) - eps, eta * (beta - x) - eps, mu * y - eps, (zet * z - eps)[None],
                          lam * sl - eps])

    eps = 1.0
    while eps > 1e-7:
        r = kkt(pt, eps)
        for _ in range(200):
            if float(r.abs().max()) <= 0.9 * eps:
                break
            x, y, z, lam, xsi, eta, mu, zet, sl = pt
            u, v, xa, bx = upp - x, x - low, x - alfa, beta - x
            pl, ql = p0 + lam @ P, q0 + lam @ Q
            G = P / u ** 2 - Q / v ** 2
            delx = pl / u ** 2 - ql / v ** 2 - eps / xa + eps / bx
            dely, delz = c + d * y - lam - eps / y, a0 - a @ lam - eps / z
            dell = P @ (1 / u) + Q @ (1 / v) - a * z - y - b + eps / lam
            Dx = 2 * (pl / u ** 3 + ql / v ** 3) + xsi / xa + eta / bx
            Dy = d + mu / y
            A = torch.zeros(m + 1, m + 1, dtype=F64, device="cuda")
            A[:m, :m] = torch.diag(sl / lam + 1 / Dy) + (G / Dx) @ G.T
            A[:m, m] = A[m, :m] = a
            A[m, m] = -zet / z
            sol = torch.linalg.solve(A, torch.cat([dell + dely / Dy - G @ (delx / Dx), delz[None]]))
            dlam, dz = sol[:m], sol[m]
            dx = -(delx + dlam @ G) / Dx
            dy = (dlam - dely) / Dy
            step = [dx, dy, dz, dlam, -xsi + (eps - xsi * dx) / xa, -eta + (eps + eta * dx) / bx,
                    -mu + (eps - mu * dy) / y, -zet + (eps - zet * dz) / z, -sl + (eps - sl * dlam) / lam]
            lim = max([1.0, float((-1.01 * dx / xa).max()), float((1.01 * dx / bx).max())]
                      + [float((-1.01 * dv / v_).max()) for dv, v_ in zip(step[1:], pt[1:])])
            norm = float(torch.linalg.norm(r))
            for k in range(50):
                new = [v_ + dv / (lim * 2.0 ** k) for v_, dv in zip(pt, step)]
                r = kkt(new, eps)
                if not float(torch.linalg.norm(r)) > norm:
                    break
            pt = new
        eps *= 0.1
    return dict(x=pt[0], lam=pt[3], low=low, upp=upp)


def exact(case, seed):
    path = case["path"]
    s = prepare(case, seed)
    if path == "mma":
        return _mma_exact(s, case["vars"], case["rows"])
    if path == "filter":
        x = s["x"].detach().requires_grad_(True)
        xt = _cone_filter(x, case["rmin"])
        b = case["beta"]
        xp = (math.tanh(b / 2) + torch.tanh(b * (xt - 0.5))) / (2 * math.tanh(b / 2))
        (gx,) = torch.autograd.grad(xp, [x], s["g"])
        return dict(xPhys=xp.detach(), xTilde=xt.detach(), gx=gx)
    if path == "apply":
        nelx, nely, d = case["nelx"], case["nely"], case["dofs"]
        out = []
        for u, rho in zip(s["U"].to(F64), s["rho"].to(F64)):
            fe = rho.reshape(1, nely, nelx, 1) * (_corners(u * s["mask"], nelx, nely, d) @ _ke(d))
            out.append(_spread(fe, nelx, nely, d)[0] * s["mask"])
        return torch.stack(out)
    if path == "uneven":
        if sum(_cost(a, b, n) for a, b, n in _uneven_shapes(case)) > 1.5e12:
            return None
        return [_spacetime_exact(x, w, n) for x, w, n in zip(s["xs"], s["ws"], s["stages"])]
    nelx, nely = case["nelx"], case["nely"]
    if _cost(nelx, nely, case.get("stages", 0) + 1) > 1.5e12:
        return None
    if path == "spacetime":
        return _spacetime_exact(s["x"], s["w"], case["stages"])
    if path == "whole":
        x = s["x"].detach().requires_grad_(True)
        rho = _simp(x.flatten())[None]
        U = _Solve.apply(rho, s["F"], _free(s["ndof"], s["free"]), nelx, nely, 2, None)
        c = _energy(U, rho, nelx, nely)[0]
        (gx,) = torch.autograd.grad(c, [x])
        return dict(c=c.detach(), U=U[0].detach(), gx=gx)
    if path == "loads":
        rho, F = s["rho"].detach().requires_grad_(True), s["F"].detach().requires_grad_(True)
        U = _Solve.apply(rho, F, s["mask"], nelx, nely, 2, None)
        g_rho, g_F = torch.autograd.grad(U, [rho, F], s["G"])
        return dict(U=U.detach(), g_rho=g_rho, g_F=g_F)
    x, mu = s["x"].detach().requires_grad_(True), s["mu"].detach().requires_grad_(True)
    t = _heat(x, mu, nelx, nely, case["time_map"])
    bt = case["beta_t"]
    masks = [(1 - (math.tanh(bt * ti) + torch.tanh(bt * (t - ti))) / (math.tanh(bt * ti) + math.tanh(bt * (1 - ti))))
             .clamp(min=0).flatten() for ti in s["times"]]
    xt = x.flatten() * torch.stack(masks)
    rho = _simp(torch.cat([x.reshape(1, -1), xt]))
    F = torch.cat([s["F"][None], _self_weight(xt, nelx, nely)])
    U = _Solve.apply(rho, F, _clamped_plate(nelx, nely), nelx, nely, 2, None)
    c = _energy(U, rho, nelx, nely)
    out = torch.stack([c[0] + (s["weights"] * c[1:]).sum(), (s["w"] * t).sum()])
    rows = [torch.autograd.grad(o, [x, mu], retain_graph=True, allow_unused=True) for o in out]
    gx, gmu = (torch.stack([torch.zeros_like(x).flatten() if r[k] is None else r[k].flatten() for r in rows])
               for k in (0, 1))
    return dict(c=c[0].detach(), stages=c[1:].detach(), U=U.detach(), t=t.detach(), gx=gx, gmu=gmu)


def _cost(nelx, nely, rows):
    """Multiply-adds of the block factorisations, a rough measure of their time."""
    return rows * (nelx + 1) * (2.0 * (nely + 1)) ** 3
