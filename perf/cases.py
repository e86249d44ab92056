"""The work that users of geoflow_b200 have it do, as measurable cases.

A case is a dict of plain values.  `listed()` holds the fixed ones, `draw(rng)`
gives more of the same ranges, `prepare` makes what a program has in hand before
the call (grid, problem, operator, fields), `run` is one pass through the public
entry points, `exact` the same outputs from plain torch in 64 bits.

Kinds, and what each stands for:

  apply     GHelmholtz.opVec_prod: the operator of every implicit solve and
            diffusion term, on affine, per-node ("regular") and deformed
            geometry, with constant and per-node coefficients.
  gather    GGFX.doOp, the direct-stiffness gather-scatter between elements.
  step      GBurgers.step on a box: advection (prescribed velocity), Burgers and
            heat, with the RK schemes the stepper has, with or without a filter.
  sphere    GBurgers.step, tracer advection on the icosahedral sphere.
  solve     GCG.solve of (M + K) x = b with Jacobi or multigrid preconditioning.
  gradient  GBurgers.adjoint_gradient, the backward direction.
  ensemble  Ensemble.solve, many small independent solves at once.

Fields are sums of a few Fourier modes plus noise per unique node, so they are
continuous across elements, as the state of a spectral-element run is.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

import geoflow_b200 as G
from geoflow_b200 import _abi as A

SCHEMES = {"rk1": A.GF_RK1, "rk2": A.GF_RK2, "rk3": A.GF_RK3, "rk4": A.GF_RK4,
           "ssp22": A.GF_SSP22, "ssp33": A.GF_SSP33, "ssp34": A.GF_SSP34}
EQNS = {"advect": A.GF_EQN_ADVECT, "burgers": A.GF_EQN_BURGERS, "heat": A.GF_EQN_HEAT}
OPS = {"smooth": G.GGFX.Smooth, "max": G.GGFX.Max, "min": G.GGFX.Min}


def listed():
    return [
        # the FP32 operator inside mixed-precision solves, at the size of the
        # Helmholtz benchmark
        {"name": "apply_affine_f32", "kind": "apply", "dtype": "f32", "p": 7, "ne": "32x32x32",
         "geom": "affine", "coef": "scalar"},
        # variable viscosity and reaction on the reference's per-node geometry,
        # ragged element counts
        {"name": "apply_nodal_f64", "kind": "apply", "dtype": "f64", "p": 6, "ne": "17x22x19",
         "geom": "regular", "coef": "node"},
        # curved elements (terrain-like), an ordinary size
        {"name": "apply_deformed_f64", "kind": "apply", "dtype": "f64", "p": 7, "ne": "16x15x14",
         "geom": "deformed", "coef": "scalar"},
        # continuity of an FP32 field, between two operators of a time step
        {"name": "gather_f32", "kind": "gather", "dtype": "f32", "p": 5, "ne": "37x35x33",
         "op": "smooth", "periodic": True},
        # the 2-d advection run of the CPU-sized configuration: launch bound
        {"name": "step_advect2d_f64", "kind": "step", "dtype": "f64", "p": 4, "ne": "16x16",
         "eqn": "advect", "scheme": "rk4", "steps": 10, "filter": False},
        # 3-d Burgers turbulence in FP32 with the SSP scheme of the RK benchmark
        {"name": "step_burgers3d_f32", "kind": "step", "dtype": "f32", "p": 5, "ne": "40x40x40",
         "eqn": "burgers", "scheme": "ssp33", "steps": 2, "filter": False},
        # the same equation in FP64 with RK4 and a stabilising filter, odd order
        # and ragged element counts
        {"name": "step_burgers3d_f64", "kind": "step", "dtype": "f64", "p": 6, "ne": "21x24x19",
         "eqn": "burgers", "scheme": "rk4", "steps": 1, "filter": True},
        # one tracer on the sphere
        {"name": "sphere_f32", "kind": "sphere", "dtype": "f32", "p": 6, "level": 4,
         "scheme": "rk4", "steps": 4, "nu": 0.0},
        # a small 2-d solve: iterations of a few microseconds each
        {"name": "solve_jacobi2d", "kind": "solve", "p": 5, "ne": "32x32", "precond": "jacobi"},
        # the headline solve
        {"name": "solve_multigrid3d", "kind": "solve", "p": 7, "ne": "32x32x32",
         "precond": "multigrid"},
        # gradient of a final-time misfit (data assimilation), order of the
        # adjoint configuration
        {"name": "gradient_f64", "kind": "gradient", "p": 6, "ne": "12x12x12", "scheme": "rk4",
         "steps": 6, "every": 3},
        # uneven 2-d solves advanced together, sizes and orders of the ensemble
        # configuration
        {"name": "ensemble_solve", "kind": "ensemble",
         "members": "8:7,8:4,48:5,48:4,64:5,16:3,32:4,64:7,32:7,8:3,24:8,16:8"},
    ]


def draw(rng):
    """One more case of the listed ranges: 2-d and 3-d, orders 2..9 (the solves
    and the ensemble within the orders their set-up takes), element counts that
    spread the node count over its logarithm, odd counts as likely as even."""

    def grid(dim, p, lo, hi):
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        side = (n / (p + 1) ** dim) ** (1.0 / dim)
        ne = [max(2, int(round(side * rng.uniform(0.8, 1.25)))) for _ in range(dim)]
        while math.prod(ne) * (p + 1) ** dim > hi and max(ne) > 2:
            ne[ne.index(max(ne))] -= 1
        return "x".join(str(k) for k in ne)

    kind = rng.choice(["apply", "apply", "gather", "step", "step", "step", "sphere", "solve",
                       "gradient", "ensemble"])
    dtype = rng.choice(["f32", "f64"])
    if kind == "apply":
        dim, p = rng.choice([2, 3, 3]), rng.randint(2, 9)
        geom = rng.choice(["affine", "regular", "deformed"])
        return {"kind": kind, "dtype": dtype, "p": p, "geom": geom,
                "ne": grid(dim, p, 2e4, 1.6e7 if geom == "affine" else 3e6),
                "coef": rng.choice(["scalar", "node"])}
    if kind == "gather":
        dim, p = rng.choice([2, 3, 3]), rng.randint(2, 9)
        return {"kind": kind, "dtype": dtype, "p": p, "ne": grid(dim, p, 2e4, 1.4e7),
                "op": rng.choice(sorted(OPS)), "periodic": rng.random() < 0.5}
    if kind == "step":
        dim, p = rng.choice([2, 3, 3]), rng.randint(3, 8)
        return {"kind": kind, "dtype": dtype, "p": p, "ne": grid(dim, p, 5e3, 1.2e7 if dim == 3 else 1e6),
                "eqn": rng.choice(["advect", "burgers", "burgers", "heat"]),
                "scheme": rng.choice(["rk2", "rk3", "rk4", "rk4", "ssp22", "ssp33", "ssp34"]),
                "steps": rng.randint(1, 3), "filter": rng.random() < 0.3}
    if kind == "sphere":
        return {"kind": kind, "dtype": dtype, "p": rng.randint(3, 8), "level": rng.randint(2, 4),
                "scheme": rng.choice(["rk3", "rk4", "rk4"]), "steps": rng.randint(1, 6),
                "nu": rng.choice([0.0, 0.0, 1e-4])}
    if kind == "solve":
        if rng.random() < 0.5:
            p = rng.randint(3, 8)
            return {"kind": kind, "p": p, "ne": grid(2, p, 2e3, 1.2e5), "precond": "jacobi"}
        p, s = rng.choice([3, 4, 5, 7]), rng.choice([6, 8, 12, 16, 24])
        return {"kind": kind, "p": p, "ne": f"{s}x{s}x{s}", "precond": "multigrid"}
    if kind == "gradient":
        p, steps = rng.randint(3, 7), rng.randint(2, 6)
        return {"kind": kind, "p": p, "ne": grid(3, p, 2e4, 6e5),
                "scheme": rng.choice(["rk4", "ssp33"]), "steps": steps,
                "every": rng.randint(1, steps)}
    members = ",".join(f"{rng.choice([8, 16, 24, 32, 48, 64])}:{rng.randint(3, 8)}"
                       for _ in range(rng.randint(6, 16)))
    return {"kind": kind, "members": members}


# ---------------------------------------------------------------------------
# the grids, in plain torch
# ---------------------------------------------------------------------------
def _ne(case):
    return [int(v) for v in case["ne"].split("x")]


def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.float64


def _gll(p):
    """GLL nodes, weights and the derivative matrix D[l, j] = phi_j'(xi_l)."""
    Pp = np.polynomial.legendre.Legendre.basis(p)
    xi = np.concatenate([[-1.0], np.sort(np.real(Pp.deriv().roots())), [1.0]]) if p > 1 \
        else np.array([-1.0, 1.0])
    for _ in range(3):  # Newton on (1 - x^2) P_p'(x), whose derivative is -p (p + 1) P_p
        inner = xi[1:-1]
        xi[1:-1] = inner + (1 - inner**2) * Pp.deriv()(inner) / (p * (p + 1) * Pp(inner))
    xi = 0.5 * (xi - xi[::-1])
    L = Pp(xi)
    W = 2.0 / (p * (p + 1) * L**2)
    n = p + 1
    D = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            if i != j:
                D[i, j] = L[i] / (L[j] * (xi[i] - xi[j]))
    D[0, 0], D[-1, -1] = -p * (p + 1) / 4.0, p * (p + 1) / 4.0
    return xi, W, D


def _lagrange(xa, xb):
    """Matrix interpolating values at nodes xa to nodes xb."""
    M = np.ones((len(xb), len(xa)))
    for j in range(len(xa)):
        for k in range(len(xa)):
            if k != j:
                M[:, j] *= (xb - xa[k]) / (xa[j] - xa[k])
    return M


class _Box:
    """A box of elements: node coordinates, lattice numbering and the
    spectral-element operators as torch matrix products in 64 bits.  Fields are
    [element, (k,) j, i], x fastest, elements in lexicographic order."""

    def __init__(self, ne, p, length, periodic):
        self.ne, self.p, self.n, self.dim = ne, p, p + 1, len(ne)
        self.length, self.per = length, periodic
        dev = torch.device("cuda")
        xi, W, D = _gll(p)
        self.D = torch.from_numpy(D).to(dev)
        self.W = torch.from_numpy(W).to(dev)
        dim, n = self.dim, self.n
        nel = math.prod(ne)
        e = torch.arange(nel, device=dev)
        ec = []
        for d in range(dim):
            ec.append(e % ne[d])
            e = e // ne[d]
        self.h = [length / v for v in ne]
        xid = torch.from_numpy(xi).to(dev)
        idx = torch.zeros([nel] + [1] * dim, dtype=torch.int64, device=dev)
        self.x, stride = [], 1
        for d in range(dim):
            shape = [1] * (dim + 1)
            shape[dim - d] = n
            c = ec[d].view([nel] + [1] * dim)
            loc = torch.arange(n, device=dev).view(shape)
            self.x.append(((c + 0.5 * (xid.view(shape) + 1.0)) * self.h[d]))
            M = ne[d] * p + (0 if periodic else 1)
            idx = idx + ((c * p + loc) % M if periodic else c * p + loc) * stride
            stride *= M
        self.nL = stride
        self.idx = idx.expand([nel] + [n] * dim).reshape(-1)
        self.shape = [nel] + [n] * dim
        self.N = nel * n**dim
        w = self.W
        self.W3 = w[:, None, None] * w[:, None] * w if dim == 3 else w[:, None] * w
        self.X = [2.0 / v for v in self.h]  # dxi/dx
        self.J = math.prod(v / 2.0 for v in self.h)
        self.mult = torch.zeros(self.nL, dtype=torch.float64, device=dev).index_add_(
            0, self.idx, torch.ones(self.N, dtype=torch.float64, device=dev))
        self.dev = dev

    def field(self, gen, modes, amp, noise, kmax=3):
        """Fourier modes plus noise per unique node, continuous and periodic in
        the box; 64-bit, flat."""
        u = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
        for _ in range(modes):
            k = [int(torch.randint(-kmax, kmax + 1, (1,), generator=gen)) for _ in range(self.dim)]
            a = float(torch.randn(1, generator=gen))
            ph = float(torch.rand(1, generator=gen)) * 2 * math.pi
            arg = sum(2 * math.pi * k[d] / self.length * self.x[d] for d in range(self.dim))
            u += a * torch.cos(arg + ph)
        u = u.reshape(-1)
        if noise:
            g = torch.Generator(device=self.dev)
            g.manual_seed(int(torch.randint(1 << 30, (1,), generator=gen)))
            u += noise * torch.randn(self.nL, dtype=torch.float64, device=self.dev, generator=g)[self.idx]
        u = self.dss(u, mean=True)  # the same bits in every copy
        return u * (amp / u.abs().max())

    def grad(self, u):
        """Reference derivatives D_d u of [*, (k,) j, i] values."""
        g = [u @ self.D.T, self.D @ u]
        if self.dim == 3:
            g.append(torch.einsum("kl,elji->ekji", self.D, u))
        return g

    def div_t(self, g):
        """sum_d D_d^T g_d."""
        o = g[0] @ self.D + self.D.T @ g[1]
        if self.dim == 3:
            o = o + torch.einsum("lk,elji->ekji", self.D, g[2])
        return o

    def dss(self, u, mean=False):
        s = torch.zeros(self.nL, dtype=u.dtype, device=u.device).index_add(0, self.idx, u.reshape(-1))
        if mean:
            s = s / self.mult
        return s[self.idx].reshape(u.shape)


def _metric(box, amp=0.03):
    """A smooth deformation x_k = X_k + amp L sin(2 pi X_{k+1} / L) of the box:
    planes dXi_i/dx_k (i * dim + k) and the Jacobian, 64-bit on the host."""
    dim, L = box.dim, box.length
    shape = box.shape
    F = torch.zeros(shape + [dim, dim], dtype=torch.float64, device=box.dev)  # dx_k/dX_l
    for k in range(dim):
        F[..., k, k] = 1.0
        nx = (k + 1) % dim
        F[..., k, nx] += amp * 2 * math.pi * torch.cos(2 * math.pi * box.x[nx] / L)
    inv = torch.linalg.inv(F)  # dX_i/dx_k
    planes = [(inv[..., i, k] * box.X[i]).reshape(-1) for i in range(dim) for k in range(dim)]
    jac = (torch.linalg.det(F) * box.J).reshape(-1)
    return torch.cat(planes + [jac]).cpu().numpy()


def _gen(seed):
    g = torch.Generator()
    g.manual_seed(seed)
    return g


def _problem(ctx, ne, p, length, periodic, geom="affine", node_geom=None):
    dim = len(ne)
    grid = G.GridBox(dim, ne, p, length=[length] * dim, periodic=[int(periodic)] * dim)
    return G.Problem(ctx, grid, dirichlet_mask=not periodic, structured=geom != "deformed",
                     geometry=geom, node_geom=node_geom)


# ---------------------------------------------------------------------------
# inputs: the same tensors for prepare and exact
# ---------------------------------------------------------------------------
def _inputs(case, seed):
    kind, gen = case["kind"], _gen(seed)
    dt = _dtype(case)
    if kind == "apply":
        box = _Box(_ne(case), case["p"], 1.0, False)
        i = {"box": box, "u": box.field(gen, 4, 1.0, 0.2).to(dt), "p": 0.7, "q": 1.3}
        if case["coef"] == "node":
            i["p"] = (1.0 + 0.5 * box.field(gen, 3, 1.0, 0.0)).to(dt)
            i["q"] = (1.0 + 0.5 * box.field(gen, 3, 1.0, 0.0)).to(dt)
        return i
    if kind == "gather":
        box = _Box(_ne(case), case["p"], 1.0, case["periodic"])
        g = torch.Generator(device=box.dev)
        g.manual_seed(seed)
        # what an operator leaves: one value per copy
        u = torch.randn(box.N, dtype=torch.float64, device=box.dev, generator=g)
        return {"box": box, "u": u.to(dt)}
    if kind in ("step", "gradient"):
        length = 2 * math.pi
        box = _Box(_ne(case), case["p"], length, True)
        eqn = case.get("eqn", "burgers")
        ns = box.dim if eqn == "burgers" else 1
        u = [box.field(gen, 6, 1.0 if kind == "step" else 0.5, 1e-3).to(dt) for _ in range(ns)]
        c = None
        if eqn == "advect":
            c = [(0.5 + 0.5 * box.field(gen, 2, 1.0, 0.0, 2)).to(dt) for _ in range(box.dim)]
        xi = _gll(case["p"])[0]
        # a resolved flow (grid Reynolds number 2 at unit speed) that decays, and
        # a step inside the advective and the diffusive limit: the state stays
        # bounded however often the pass is repeated
        hmin, nu = min(box.h) * 0.5 * (xi[1] - xi[0]), 0.5 * max(box.h) / case["p"]
        i = {"box": box, "u": u, "c": c, "eqn": eqn, "nu": nu,
             "dt": min(0.1 * hmin, 0.05 * hmin**2 / (nu * box.dim))}
        if kind == "gradient":
            i["obs"] = [a + box.field(gen, 4, 0.1, 0.0) for a in u]
        return i
    if kind == "solve":
        return _solve_inputs(_ne(case), case["p"], gen)
    raise ValueError(kind)


def _solve_inputs(ne, p, gen):
    """b = M f, f a sum of sine modes with zero boundary values."""
    box = _Box(ne, p, 1.0, False)
    f = torch.zeros(box.shape, dtype=torch.float64, device=box.dev)
    for _ in range(8 if box.dim == 3 else 4):
        k = torch.randint(1, 9, (box.dim,), generator=gen)
        t = float(torch.randn(1, generator=gen))
        for d in range(box.dim):
            t = t * torch.sin(math.pi * int(k[d]) * box.x[d])
        f += t
    return {"box": box, "b": (f * (box.W3 * box.J)).reshape(-1)}


def _sphere(case, seed):
    """The icosahedral grid, a cosine bell at a seeded centre and the
    solid-body wind; dt at CFL 0.05 (without diffusion the scheme amplifies
    the shortest waves slowly, and the state is stepped many times)."""
    grid = G.IcosGrid(case["level"], case["p"], ctx=_context())
    gen = _gen(seed)
    lat, lon = ((float(torch.rand(1, generator=gen)) - 0.5) * 2.0 for _ in range(2))
    u = G.workloads.icos_cosine_bell(grid.xyz, lat, math.pi + lon)
    c = G.workloads.icos_solid_body_wind(grid.xyz, alpha=0.3)
    cmax = float(np.max(np.sqrt(sum(a * a for a in c))))
    dt, dev = _dtype(case), torch.device("cuda")
    return {"grid": grid, "u": torch.from_numpy(u).to(dev, dt),
            "c": [torch.from_numpy(a).to(dev, dt) for a in c], "dt": 0.05 * grid.minnodedist / cmax}


def _members(case):
    return [tuple(int(v) for v in m.split(":")) for m in case["members"].split(",")]


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def _context():
    return G.Context(torch.cuda.current_device())


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    if kind == "sphere":
        i = _sphere(case, seed)
        prob = i["grid"].problem(ctx)
        eq = G.GBurgers(prob, A.GF_EQN_ADVECT, case["nu"], SCHEMES[case["scheme"]])
        return {"kind": kind, "steps": case["steps"], "eq": eq, "u": [i["u"]], "c": i["c"], "dt": i["dt"]}
    if kind == "ensemble":
        gen, probs, bs = _gen(seed), [], []
        for ne, p in _members(case):
            probs.append(_problem(ctx, [ne, ne], p, 1.0, False))
            bs.append(_solve_inputs([ne, ne], p, gen)["b"])
        tr = G.CGTraits(maxit=20000, normtype=A.GF_NORM_EUC, tol=1e-10, relative=1,
                        precond=A.GF_PRECOND_JACOBI, precision=A.GF_CG_FP64)
        return {"kind": kind, "ens": G.Ensemble(ctx, probs), "tr": tr, "b": bs,
                "x": [torch.zeros_like(b) for b in bs]}
    i = _inputs(case, seed)
    box = i["box"]
    geom = case.get("geom", "affine")
    prob = _problem(ctx, box.ne, box.p, box.length, box.per, geom,
                    _metric(box) if geom == "deformed" else None)
    state = {"kind": kind, "prob": prob}
    if kind == "apply":
        H = G.GHelmholtz(prob)
        H.set_Lap_scalar(i["p"])
        H.set_mass_scalar(i["q"])
        state.update(H=H, u=i["u"], out=torch.empty_like(i["u"]))
    elif kind == "gather":
        state.update(ggfx=G.GGFX(prob), u=i["u"], op=OPS[case["op"]])
    elif kind == "step":
        state.update(eq=G.GBurgers(prob, EQNS[i["eqn"]], i["nu"], SCHEMES[case["scheme"]]), u=i["u"],
                     c=i["c"], dt=i["dt"], steps=case["steps"],
                     filters=[G.GProjectionFilter(prob, 1, 0.05)] if case["filter"] else None)
    elif kind == "solve":
        pre = A.GF_PRECOND_JACOBI if case["precond"] == "jacobi" else A.GF_PRECOND_PMG
        tr = G.CGTraits(maxit=20000, normtype=A.GF_NORM_EUC, tol=1e-10, relative=1, precond=pre,
                        poly_degree=1)
        H = G.GHelmholtz(prob)
        H.set_Lap_scalar(1.0)
        H.set_mass_scalar(1.0)
        state.update(cg=G.GCG(tr, prob), H=H, b=i["b"], xb=torch.zeros_like(i["b"]),
                     x=torch.zeros_like(i["b"]))
    else:
        state.update(eq=G.GBurgers(prob, A.GF_EQN_BURGERS, i["nu"], SCHEMES[case["scheme"]]), u=i["u"],
                     obs=i["obs"], dt=i["dt"], steps=case["steps"], every=case["every"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "apply":
        state["H"].opVec_prod(state["u"], None, state["out"])
        return {"out": state["out"]}
    if kind == "gather":
        state["ggfx"].doOp(state["u"], state["op"])
        return {"u": state["u"]}
    if kind in ("step", "sphere"):
        state["eq"].step(state["u"], state["c"], dt=state["dt"], nsteps=state["steps"],
                         filters=state.get("filters"))
        return {"u": state["u"]}
    if kind == "solve":
        state["x"].zero_()
        state["cg"].solve(state["H"], state["b"], state["xb"], state["x"])
        return {"x": state["x"]}
    if kind == "ensemble":
        for x in state["x"]:
            x.zero_()
        state["ens"].solve(state["b"], state["x"], state["tr"])
        return {"x": state["x"]}
    J, grad = state["eq"].adjoint_gradient(state["u"], None, state["obs"], state["dt"],
                                           state["steps"], state["every"])
    return {"J": J, "grad": grad}


# ---------------------------------------------------------------------------
# the work and the tolerance
# ---------------------------------------------------------------------------
def work(case):
    """Bytes of each input read once and each output written once (per RK stage
    for the steppers, per iteration for the solves, with the iteration counts
    that the present convergence needs), and the flops of the contractions."""
    kind, s = case["kind"], 4 if case.get("dtype") == "f32" else 8
    if kind == "ensemble":
        its, total, fl = 60, 0, 0
        for ne, p in _members(case):
            N = ne * ne * (p + 1) ** 2
            total += its * N * 8 * 4
            fl += its * N * (8 * (p + 1) + 16)
        return {"bytes": total, "flops": fl}
    if kind == "sphere":
        rows = 20 * (2 ** case["level"]) ** 2 * 3  # quadrilaterals after bisection, about
        N, n = rows * (case["p"] + 1) ** 2, case["p"] + 1
        st = case["steps"] * int(case["scheme"][2:])
        planes = 2 + (2 if case["nu"] == 0.0 else 14)
        return {"bytes": st * N * s * planes, "flops": st * N * (4 * n + 10)}
    ne, p = _ne(case), case["p"]
    dim, n = len(ne), p + 1
    N = math.prod(ne) * n**dim
    if kind == "apply":
        planes = 2 + {"affine": 0, "regular": dim + 1, "deformed": dim * (dim + 1) // 2 + 1}[case["geom"]]
        planes += 2 if case["coef"] == "node" else 0
        return {"bytes": N * s * planes, "flops": N * (2 * dim * n if case["geom"] == "affine" else 4 * dim * n)}
    if kind == "gather":
        return {"bytes": 2 * N * s, "flops": N}
    if kind == "solve":
        NL = math.prod(v * p + 1 for v in ne)
        its = 11 if case["precond"] == "multigrid" else 8 * int(max(ne) * p ** 0.5 / 8 + 4)
        if case["precond"] == "multigrid":  # FP64 step and a V-cycle of FP32 applies and passes
            return {"bytes": its * (NL * (10 * 8 + 30 * 4)), "flops": its * 6 * N * 2 * dim * n}
        return {"bytes": its * NL * 8 * 8, "flops": its * N * 2 * dim * n}
    stages = {"rk1": 1, "rk2": 2, "rk3": 3, "rk4": 4, "ssp22": 2, "ssp33": 3, "ssp34": 4}
    st = case["steps"] * stages[case["scheme"]]
    if kind == "gradient":
        st *= 4  # forward, recomputation, and a reverse stage of twice a forward one
    eqn = case.get("eqn", "burgers")
    ns = dim if eqn == "burgers" else 1
    planes = 2 * ns + 1 + (dim if eqn == "advect" else 0)
    return {"bytes": st * N * s * planes, "flops": st * ns * N * 4 * dim * n}


def tolerance(case):
    """About four times the error against `exact` over the listed and some drawn
    cases.  The gather-scatter folds in a fixed order, so it has none."""
    kind, f32 = case["kind"], case.get("dtype") == "f32"
    if kind == "gather":
        return "exact"
    if kind == "apply":  # weak Laplacian of a noisy field: 2e-7..4e-7 and 1e-15..4e-15
        return {"rel": 1.5e-6} if f32 else {"rel": 1.5e-14}
    if kind in ("step", "sphere"):  # increments of O(dt) added to the state: 1e-7, 2e-16
        return {"rel": 5e-7} if f32 else {"rel": 2e-15}
    if kind == "gradient":  # 1e-15
        return {"rel": 5e-15}
    # stopped at a relative residual of 1e-10 (1e-12..8e-12 from the solution); an
    # iteration more or less moves the result by several times its error
    return {"rel": 1e-10}


# ---------------------------------------------------------------------------
# the same outputs in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _butcher(order):
    alpha = {1: [0], 2: [0, 1], 3: [0, 1 / 3, 2 / 3], 4: [0, 0.5, 0.5, 1.0]}[order]
    c = {1: [1], 2: [0.5, 0.5], 3: [0.25, 0, 0.75], 4: [1 / 6, 1 / 3, 1 / 3, 1 / 6]}[order]
    return alpha, c  # each stage uses the slope before it, beta[m][m-1] = alpha[m]


def _stepper(scheme, rhs, smooth):
    """One step u -> u of the stepper: Butcher schemes smooth each slope and the
    last stage's input and result, SSP schemes smooth each substep."""
    many = lambda f, *a: [f(*v) for v in zip(*a)]

    def rk(u, h):
        order = int(scheme[2:])
        alpha, c = _butcher(order)
        out, K = list(u), None
        for m in range(order):
            um = u if K is None else many(lambda a, b: a + alpha[m] * h * b, u, K)
            if m == order - 1:
                um = many(smooth, um)
            K = many(smooth, rhs(um))
            out = many(lambda a, b: a + c[m] * h * b, out, K)
        return many(smooth, out)

    def euler(u, h):
        return many(lambda a, b: a + h * b, u, rhs(u))

    def comb(a, x, b, y):
        return many(lambda v, w: smooth(a * v + b * w), x, y)

    def ssp(u, h):
        if scheme == "ssp22":
            x = many(smooth, euler(u, h))
            return comb(0.5, euler(x, h), 0.5, u)
        if scheme == "ssp33":
            x = many(smooth, euler(u, h))
            x = comb(0.25, euler(x, h), 0.75, u)
            return comb(2 / 3, euler(x, h), 1 / 3, u)
        x = comb(0.5, euler(u, h), 0.5, u)
        x = comb(0.5, euler(x, h), 0.5, x)
        x = many(lambda v, w, z: smooth(v / 6 + w / 6 + 2 * z / 3), euler(x, h), x, u)
        return comb(0.5, euler(x, h), 0.5, x)

    return rk if scheme.startswith("rk") else ssp


def _box_rhs(box, eqn, nu, c):
    mass = box.W3 * box.J
    m1 = mass.expand(box.shape)
    imass = 1.0 / box.dss(m1, mean=True)
    cs = None if c is None else [a.double().reshape(box.shape) for a in c]

    def rhs(u):
        vel = u if eqn == "burgers" else cs
        out = []
        for a in u:
            g = box.grad(a)
            r = -nu * box.div_t([mass * box.X[d] ** 2 * g[d] for d in range(box.dim)])
            if eqn != "heat":
                r = r - mass * sum(vel[d] * box.X[d] * g[d] for d in range(box.dim))
            out.append(imass * r)
        return out

    return rhs


def _solve_exact(box, b):
    """(K + M) x = Q^T b with zero boundary values by fast diagonalisation of
    the 1-d assembled operators."""
    D, W = box.D.cpu().numpy(), box.W.cpu().numpy()
    K1 = D.T @ np.diag(W) @ D
    n, p, dim = box.n, box.p, box.dim
    V, lam, shape = [], [], []
    for d in range(dim):
        M = box.ne[d] * p + 1
        K, m = np.zeros((M, M)), np.zeros(M)
        for e in range(box.ne[d]):
            s = slice(e * p, e * p + n)
            K[s, s] += K1 * box.X[d]
            m[s] += W / box.X[d]
        m = m[1:-1]
        w, v = np.linalg.eigh(K[1:-1, 1:-1] / np.sqrt(np.outer(m, m)))
        V.append(torch.from_numpy(v / np.sqrt(m)[:, None]).to(box.dev))  # V^T M V = I
        lam.append(torch.from_numpy(w).to(box.dev))
        shape.append(M)
    L = torch.zeros(box.nL, dtype=torch.float64, device=box.dev).index_add_(0, box.idx, b)
    L = L.reshape(shape[::-1])
    inner = L[tuple(slice(1, -1) for _ in range(dim))]
    if dim == 2:
        t = V[1].T @ inner @ V[0]
        t = t / (1.0 + lam[1][:, None] + lam[0])
        x = V[1] @ t @ V[0].T
    else:
        t = torch.einsum("zk,zyx->kyx", V[2], V[1].T @ (inner @ V[0]))
        t = t / (1.0 + lam[2][:, None, None] + lam[1][:, None] + lam[0])
        x = torch.einsum("kz,zyx->kyx", V[2], V[1] @ (t @ V[0].T))
    out = torch.zeros_like(L)
    out[tuple(slice(1, -1) for _ in range(dim))] = x
    return out.reshape(-1)[box.idx]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        gen, out = _gen(seed), []
        for ne, p in _members(case):
            i = _solve_inputs([ne, ne], p, gen)
            out.append(_solve_exact(i["box"], i["b"]))
        return {"x": out}
    if kind == "sphere":
        return _sphere_exact(case, seed)
    i = _inputs(case, seed)
    box = i["box"]
    if kind == "apply":
        u = i["u"].double().reshape(box.shape)
        pv, qv = (v.double().reshape(box.shape) if torch.is_tensor(v) else v for v in (i["p"], i["q"]))
        g = box.grad(u)
        if case["geom"] == "deformed":
            m = torch.from_numpy(_metric(box)).to(box.dev).reshape([box.dim**2 + 1] + box.shape)
            mass, dim = box.W3 * m[-1], box.dim
            f = [sum(m[a * dim + k] * g[a] for a in range(dim)) for k in range(dim)]  # du/dx_k
            g = [pv * mass * sum(m[a * dim + k] * f[k] for k in range(dim)) for a in range(dim)]
        else:
            mass = box.W3 * box.J
            g = [pv * mass * box.X[d] ** 2 * g[d] for d in range(box.dim)]
        return {"out": (box.div_t(g) + qv * mass * u).reshape(-1)}
    if kind == "gather":
        u = i["u"].double()
        if case["op"] == "smooth":
            return {"u": box.dss(u, mean=True)}
        L = torch.zeros(box.nL, dtype=torch.float64, device=box.dev)
        L.scatter_reduce_(0, box.idx, u, "amax" if case["op"] == "max" else "amin",
                          include_self=False)
        return {"u": L[box.idx]}
    if kind == "step":
        step = _stepper(case["scheme"], _box_rhs(box, i["eqn"], i["nu"], i["c"]),
                        lambda v: box.dss(v, mean=True))
        u = [a.double().reshape(box.shape) for a in i["u"]]
        for _ in range(case["steps"]):
            u = step(u, i["dt"])
            if case["filter"]:
                xi, lo = _gll(box.p)[0], _gll(box.p - 1)[0]
                F = 0.05 * _lagrange(lo, xi) @ _lagrange(xi, lo) + 0.95 * np.eye(box.n)
                F = torch.from_numpy(F).to(box.dev)
                u = [F @ (a @ F.T) for a in u]
                if box.dim == 3:
                    u = [torch.einsum("kl,elji->ekji", F, a) for a in u]
        return {"u": [a.reshape(-1) for a in u]}
    if kind == "solve":
        return {"x": _solve_exact(box, i["b"])}
    step = _stepper(case["scheme"], _box_rhs(box, "burgers", i["nu"], None),
                    lambda v: box.dss(v, mean=True))
    u0 = [a.reshape(box.shape).clone().requires_grad_() for a in i["u"]]
    u = u0
    for _ in range(case["steps"]):
        u = torch.utils.checkpoint.checkpoint(lambda *a: tuple(step(list(a), i["dt"])), *u,
                                              use_reentrant=False)
    mass = box.W3 * box.J
    J = 0.5 * sum((mass * (a - o.reshape(box.shape)) ** 2).sum() for a, o in zip(u, i["obs"]))
    grads = torch.autograd.grad(J, u0)
    return {"J": float(J.detach()), "grad": [a.reshape(-1) for a in grads]}


def _sphere_exact(case, seed):
    i = _sphere(case, seed)
    grid, dev = i["grid"], torch.device("cuda")
    n, nel = grid.n, grid.nelems
    xi, W, D = _gll(grid.p)
    D, W = torch.from_numpy(D).to(dev), torch.from_numpy(W).to(dev)
    m = torch.from_numpy(grid.node_geom).to(dev).reshape(7, nel, n, n)
    idx = torch.from_numpy(grid.node_class).to(dev).long()
    mult = torch.zeros(grid.nclass, dtype=torch.float64, device=dev).index_add_(
        0, idx, torch.ones(grid.ndof(), dtype=torch.float64, device=dev))

    def smooth(v):
        s = torch.zeros(grid.nclass, dtype=torch.float64, device=dev).index_add_(0, idx, v.reshape(-1))
        return (s / mult)[idx].reshape(v.shape)

    mass = W[:, None] * W * m[6]
    imass = 1.0 / smooth(mass)
    c = [a.double().reshape(nel, n, n) for a in i["c"]]

    def rhs(u):
        g = [u[0] @ D.T, D @ u[0]]
        du = [m[k] * g[0] + m[3 + k] * g[1] for k in range(3)]
        r = -mass * sum(c[k] * du[k] for k in range(3))
        if case["nu"]:
            f = [mass * sum(m[3 * a + k] * du[k] for k in range(3)) for a in range(2)]
            r = r - case["nu"] * (f[0] @ D + D.T @ f[1])
        return [imass * r]

    step = _stepper(case["scheme"], rhs, smooth)
    u = [i["u"].double().reshape(nel, n, n)]
    for _ in range(case["steps"]):
        u = step(u, i["dt"])
    return {"u": [u[0].reshape(-1)]}
