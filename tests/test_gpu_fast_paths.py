"""Kernels that a rule on geometry, dimension or size selects, each against the
general path that the same grid takes in another description:

* affine 3-d right-hand side and its VJP (even-odd D and K1) against the
  per-node geometry kernels;
* 2-d boxes whose RK steps or CG iterations run inside one cluster against
  the same grid without its box description (separate kernels, CSR members):
  the steps bit for bit, the solves to the stop tolerance;
* the line-by-line Helmholtz applies (diagonal and full metric) against dense
  FP64 contractions in numpy.

Tolerances: FP64 sums of at most 3 * 12 terms differ by rounding order, a few
hundred eps of the largest term (1e-12); FP32 likewise (2e-5).  Solves stop at a
relative residual of 1e-11, which leaves them within 1e-8 of each other."""
import numpy as np
import pytest

from geoflow_b200 import _abi as A

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11]


def cuda(a, dt):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(device="cuda", dtype=dt)


def rel(a, b):
    import torch
    a, b = a.double(), b.double()
    return float((a - b).abs().max() / b.abs().max())


def bits_equal(a, b):
    import torch
    i = torch.int64 if a.dtype == torch.float64 else torch.int32
    return torch.equal(a.view(i), b.view(i))


@pytest.mark.parametrize("p", ORDERS)
@pytest.mark.parametrize("eqn", [A.GF_EQN_ADVECT, A.GF_EQN_BURGERS, A.GF_EQN_HEAT])
def test_affine_rhs_equals_nodal(ctx, p, eqn):
    import torch
    from geoflow_b200 import GBurgers, GridBox, Problem
    g = GridBox(3, [3, 2, 2], p, length=[1.0, 0.7, 1.9], periodic=[1, 0, 1])
    pa, pn = Problem(ctx, g, dirichlet_mask=False), Problem(ctx, g, dirichlet_mask=False,
                                                            geometry="regular")
    rng = np.random.default_rng(p)
    ns = 3 if eqn == A.GF_EQN_BURGERS else 1
    u0 = [rng.standard_normal(g.ndof()) for _ in range(ns)]
    c0 = [rng.standard_normal(g.ndof()) for _ in range(3)] if eqn == A.GF_EQN_ADVECT else None
    for dt, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        u = [cuda(a, dt) for a in u0]
        c = [cuda(a, dt) for a in c0] if c0 else None
        out = []
        for prob in (pa, pn):
            o = prob.zeros(dt, ncomp=ns)
            GBurgers(prob, eqn, 0.03).dudt(u, c, o)
            out.append(o)
        for a, b in zip(*out):
            assert rel(a, b) < tol, (dt, rel(a, b))
    # the VJP (FP64)
    u, lam = [cuda(a, torch.float64) for a in u0], [cuda(rng.standard_normal(g.ndof()), torch.float64)
                                                   for _ in range(ns)]
    c = [cuda(a, torch.float64) for a in c0] if c0 else None
    out = []
    for prob in (pa, pn):
        o = prob.zeros(ncomp=ns)
        GBurgers(prob, eqn, 0.03).dudt_vjp(u, c, lam, o)
        out.append(o)
    for a, b in zip(*out):
        assert rel(a, b) < 1e-12, rel(a, b)


def test_rhs_with_an_asymmetric_derivative_matrix(ctx):
    """A caller's D that is not centro-antisymmetric keeps the general kernels."""
    import torch
    from geoflow_b200 import GBurgers, GridBox, Problem
    g = GridBox(3, [2, 2, 2], 4)
    g.D = g.D * (1.0 + 0.1 * np.random.default_rng(0).standard_normal(g.D.size))
    u = [cuda(np.random.default_rng(k).standard_normal(g.ndof()), torch.float64) for k in range(3)]
    out = []
    for geom in ("affine", "regular"):
        prob = Problem(ctx, g, geometry=geom)
        o = prob.zeros(ncomp=3)
        GBurgers(prob, A.GF_EQN_BURGERS, 0.1).dudt(u, None, o)
        out.append(o)
    for a, b in zip(*out):
        assert rel(a, b) < 1e-12


@pytest.mark.parametrize("ne,p,per", [([1, 3], 1, [0, 1]), ([16, 16], 4, [1, 1]), ([5, 3], 11, [0, 0]),
                                      ([17, 9], 6, [1, 0]), ([2, 40], 2, [0, 1]), ([3, 2], 9, [1, 1])])
@pytest.mark.parametrize("scheme", [A.GF_RK2, A.GF_RK3, A.GF_RK4, A.GF_SSP22, A.GF_SSP33, A.GF_SSP34])
def test_cluster_steps_equal_separate_kernels(ctx, ne, p, per, scheme):
    import torch
    from geoflow_b200 import GBurgers, GridBox, Problem
    g = GridBox(2, ne, p, periodic=per)
    rng = np.random.default_rng(p + scheme)
    for geom in ("affine", "regular"):
        probs = [Problem(ctx, g, structured=s, geometry=geom) for s in (True, False)]
        for eqn, ns in ((A.GF_EQN_ADVECT, 1), (A.GF_EQN_BURGERS, 2), (A.GF_EQN_HEAT, 1)):
            u0 = [0.3 * rng.standard_normal(g.ndof()) for _ in range(ns)]
            c0 = [rng.standard_normal(g.ndof()) for _ in range(2)]
            for dt in (torch.float64, torch.float32):
                c = [cuda(a, dt) for a in c0] if eqn == A.GF_EQN_ADVECT else None
                us = []
                for prob in probs:
                    u = [cuda(a, dt) for a in u0]
                    GBurgers(prob, eqn, 1e-2, scheme=scheme).step(u, c, dt=1e-4, nsteps=3)
                    us.append(u)
                for a, b in zip(*us):
                    assert bits_equal(a, b), (geom, eqn, dt)


@pytest.mark.parametrize("ne,p,per", [([2, 3], 1, [0, 0]), ([8, 8], 3, [0, 0]), ([32, 32], 5, [0, 0]),
                                      ([5, 7], 11, [1, 0]), ([1, 4], 6, [1, 0]), ([40, 3], 2, [0, 1]),
                                      ([9, 6], 8, [0, 0])])
@pytest.mark.parametrize("norm", [A.GF_NORM_INF, A.GF_NORM_EUC, A.GF_NORM_L2, A.GF_NORM_L1])
def test_cluster_cg_equals_separate_kernels(ctx, ne, p, per, norm):
    import torch
    from geoflow_b200 import CGTraits, GCG, GHelmholtz, GridBox, Problem
    g = GridBox(2, ne, p, length=[1.0, 1.7], periodic=per)
    rng = np.random.default_rng(p)
    first = g.members[g.class_ptr[:-1]][g.node_class]
    b = cuda(rng.standard_normal(g.ndof()), torch.float64)
    x0 = rng.standard_normal(g.ndof())[first]
    lift = np.where(g.mask == 0.0, rng.standard_normal(g.ndof())[first], 0.0)
    for pre in (A.GF_PRECOND_NONE, A.GF_PRECOND_JACOBI):
        for xb in (None, lift):
            res = []
            for s in (True, False):
                prob = Problem(ctx, g, structured=s)
                H = GHelmholtz(prob)
                H.set_Lap_scalar(0.3)
                H.set_mass_scalar(2.0)
                tr = CGTraits(maxit=4000, normtype=norm, tol=1e-11, relative=1, precond=pre)
                cg = GCG(tr, prob)
                x = cuda(x0, torch.float64)
                rc = cg.solve(H, b, *([] if xb is None else [cuda(xb, torch.float64)]), x)
                res.append((rc, cg.iter_, x, np.array(cg.get_residuals())))
            (ra, ia, xa, ha), (rb, ib, xbb, hb) = res
            assert ra == rb == 0
            assert abs(ia - ib) <= max(2, ib // 20)
            assert rel(xa, xbb) < 1e-8
            assert abs(ha[0] - hb[0]) <= 1e-9 * hb[0]


def asymmetric_grid(ne, p, **kw):
    """A box whose derivative matrix is not centro-antisymmetric."""
    from geoflow_b200 import GridBox
    g = GridBox(len(ne), ne, p, **kw)
    g.D = g.D * (1.0 + 0.1 * np.random.default_rng(p).standard_normal(g.D.size))
    return g


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("p", [1, 2, 5, 7, 8])
def test_applies_with_an_asymmetric_derivative_matrix(ctx, dim, p):
    """The affine apply, by FMA and (p = 7) by tensor cores, against the per-node
    kernel of the same grid; then a solve with each preconditioner."""
    import torch
    from geoflow_b200 import CGTraits, GCG, GHelmholtz, Problem
    g = asymmetric_grid([3, 2, 2][:dim], p, length=[1.0, 0.7, 1.3][:dim])
    u = np.random.default_rng(p).standard_normal(g.ndof())
    probs = [Problem(ctx, g, geometry=geom) for geom in ("affine", "regular")]
    Hs = [GHelmholtz(prob) for prob in probs]
    for H in Hs:
        H.set_Lap_scalar(0.6)
        H.set_mass_scalar(1.7)
    lib = A.load()
    for dt, mode, tol in ((torch.float64, A.GF_FP32_APPLY_FMA, 1e-12),
                          (torch.float32, A.GF_FP32_APPLY_FMA, 2e-5),
                          (torch.float32, A.GF_FP32_APPLY_TF32, 2e-5)):
        prev = lib.gf_set_fp32_apply(mode)
        try:
            out = []
            for prob, H in zip(probs, Hs):
                o = prob.zeros(dt)
                H.opVec_prod(cuda(u, dt), None, o)
                out.append(o)
        finally:
            lib.gf_set_fp32_apply(prev)
        assert rel(*out) < tol, (dt, mode, rel(*out))
    b = cuda(np.random.default_rng(p + 1).standard_normal(g.ndof()), torch.float64)
    kinds = [(1, A.GF_PRECOND_JACOBI, A.GF_CG_FP64), (0, A.GF_PRECOND_JACOBI, A.GF_CG_FP64)]
    if dim == 3 and p >= 5:  # enough unknowns for a batch of FP32 iterations
        kinds += [(0, A.GF_PRECOND_JACOBI, A.GF_CG_MIXED), (0, A.GF_PRECOND_PMG, A.GF_CG_FP64)]
    xs = []
    for i, pre, prec in kinds:
        x = probs[i].zeros()
        tr = CGTraits(maxit=8000, normtype=A.GF_NORM_EUC, tol=1e-11, relative=1, precond=pre,
                      precision=prec)
        assert GCG(tr, probs[i]).solve(Hs[i], b, probs[i].zeros(), x) == 0, (pre, prec)
        xs.append(x)
    for x in xs[1:]:
        assert rel(x, xs[0]) < 1e-8


@pytest.mark.parametrize("ne,p", [([2, 3], 2), ([6, 5], 4), ([4, 4], 7)])
def test_solves_with_an_asymmetric_derivative_matrix(ctx, ne, p):
    """The 2-d FP64 solves, alone and in an ensemble, solve with the operator of
    opVec_prod: as the same grid without its box description, and the assembled
    residual by opVec_prod vanishes."""
    import torch
    from geoflow_b200 import CGTraits, Ensemble, GCG, GGFX, GHelmholtz, Problem
    g = asymmetric_grid(ne, p)
    probs = [Problem(ctx, g, structured=s) for s in (True, False)]
    b = cuda(np.random.default_rng(p).standard_normal(g.ndof()), torch.float64)
    tr = CGTraits(maxit=4000, normtype=A.GF_NORM_EUC, tol=1e-11, relative=1,
                  precond=A.GF_PRECOND_JACOBI, precision=A.GF_CG_FP64)
    xs = []
    for prob in probs:
        H = GHelmholtz(prob)
        H.set_Lap_scalar(0.3)
        H.set_mass_scalar(2.0)
        x = prob.zeros()
        assert GCG(tr, prob).solve(H, b, prob.zeros(), x) == 0
        xs.append(x)
    xe = probs[0].zeros()
    rc, _, _, st = Ensemble(ctx, probs[:1]).solve([b], [xe], tr, p=0.3, q=2.0)
    assert rc == 0 and list(st) == [0]
    assert rel(xs[0], xs[1]) < 1e-8
    assert rel(xe, xs[1]) < 1e-8
    H = GHelmholtz(probs[1])
    H.set_Lap_scalar(0.3)
    H.set_mass_scalar(2.0)
    for x in (xs[0], xe):
        ax = probs[1].zeros()
        H.opVec_prod(x, None, ax)
        r = (b - ax) * cuda(g.mask, torch.float64)
        s = b.clone()
        for v in (r, s):
            GGFX(probs[1]).doOp(v, GGFX.Sum)
        assert float((r * cuda(g.mask, torch.float64)).abs().max()) < 1e-9 * float(s.abs().max())


def stretched(g):
    """Elements of unequal size: columns and rows of growing width."""
    eg = g.elem_geom.reshape(g.nelems, 3)
    e = np.arange(g.nelems)
    sx, sy = 1.0 + 0.5 * np.sin(e % g.ne[0]), 1.0 + 0.3 * np.cos(e // g.ne[0])
    eg[:, 0] /= sx
    eg[:, 1] /= sy
    eg[:, 2] *= sx * sy
    return g


# more than 2048 points per CTA (16 CTAs), where the vectors are in global memory; rows
# that do not divide by the CTAs, CTAs without a row; unequal elements; either side
# of the size limit of the cluster
@pytest.mark.parametrize("ne,p,per,unequal", [([44, 44], 5, [0, 0], 0), ([50, 35], 6, [1, 0], 1),
                                              ([3, 700], 4, [0, 1], 0), ([600, 8], 2, [1, 0], 1),
                                              ([12, 9], 7, [0, 0], 1), ([9, 6], 3, [1, 1], 1),
                                              ([56, 56], 5, [0, 0], 0), ([57, 57], 5, [0, 0], 0),
                                              ([160, 16], 5, [0, 0], 0)])
def test_cluster_cg_large_and_unequal(ctx, ne, p, per, unequal):
    import torch
    from geoflow_b200 import CGTraits, GCG, GHelmholtz, GridBox, Problem
    g = GridBox(2, ne, p, periodic=per)
    if unequal:
        g = stretched(g)
    rng = np.random.default_rng(p)
    first = g.members[g.class_ptr[:-1]][g.node_class]
    b = cuda(rng.standard_normal(g.ndof()), torch.float64)
    x0 = rng.standard_normal(g.ndof())[first]
    for norm in (A.GF_NORM_EUC, A.GF_NORM_L2):
        res = []
        for s in (True, False):
            prob = Problem(ctx, g, structured=s)
            H = GHelmholtz(prob)
            H.set_Lap_scalar(0.02)
            H.set_mass_scalar(2.0)
            cg = GCG(CGTraits(maxit=8000, normtype=norm, tol=1e-11, relative=1,
                              precond=A.GF_PRECOND_JACOBI), prob)
            x = cuda(x0, torch.float64)
            assert cg.solve(H, b, prob.zeros(), x) == 0
            res.append((cg.iter_, x, np.array(cg.get_residuals())))
        (ia, xa, ha), (ib, xb, hb) = res
        assert abs(ia - ib) <= max(2, ib // 20)
        assert rel(xa, xb) < 1e-8
        assert abs(ha[0] - hb[0]) <= 1e-9 * hb[0]


# FP64 ensembles: clusters with members of about 50 k and 200 k points; grid-wide with
# one member that is too large for the shared memory of a cluster, and with one that
# the others would wait for; unequal elements and a ragged box on either path
@pytest.mark.parametrize("boxes", [[([37, 38], 6), ([8, 5], 3), ([64, 64], 7), ([64, 63], 7)],
                                   [([64, 65], 9), ([9, 14], 8), ([20, 3], 4)],
                                   [([60, 61], 8), ([7, 5], 6)],
                                   [([6, 7], 5)]])
def test_ensemble_fp64_paths_equal_single_solves(ctx, boxes):
    import torch
    from geoflow_b200 import CGTraits, Ensemble, GCG, GHelmholtz, GridBox, Problem
    tr = CGTraits(maxit=8000, normtype=A.GF_NORM_EUC, tol=1e-11, relative=1,
                  precond=A.GF_PRECOND_JACOBI, precision=A.GF_CG_FP64)
    grids = [GridBox(2, ne, p) for ne, p in boxes]
    if len(grids) > 1:
        grids[1] = stretched(grids[1])
    rng = np.random.default_rng(len(boxes))
    bs = [cuda(rng.standard_normal(g.ndof()), torch.float64) for g in grids]
    probs = [Problem(ctx, g) for g in grids]
    xs = [p.zeros() for p in probs]
    rc, it, nrm, st = Ensemble(ctx, probs).solve(bs, xs, tr, p=0.02, q=2.0)
    assert rc == 0 and list(st) == [0] * len(boxes)
    for g, b, x, k in zip(grids, bs, xs, it):
        prob = Problem(ctx, g, structured=False)
        H = GHelmholtz(prob)
        H.set_Lap_scalar(0.02)
        H.set_mass_scalar(2.0)
        cg = GCG(tr, prob)
        ref = prob.zeros()
        assert cg.solve(H, b, prob.zeros(), ref) == 0
        assert abs(int(k) - cg.iter_) <= max(2, cg.iter_ // 20)
        assert rel(x, ref) < 1e-8


def test_cluster_cg_outcomes(ctx):
    """maxit, an exact start and a non-finite right-hand side."""
    import torch
    from geoflow_b200 import CGTraits, GCG, GFError, GHelmholtz, GridBox, Problem
    g = GridBox(2, [6, 6], 5)
    prob = Problem(ctx, g)
    H = GHelmholtz(prob)
    H.set_mass_scalar(1.0)
    b = cuda(np.random.default_rng(0).standard_normal(g.ndof()), torch.float64)
    for maxit in (0, 1, 7):
        cg = GCG(CGTraits(maxit=maxit, tol=1e-12, relative=1, precond=1), prob)
        assert cg.solve(H, b, prob.zeros(), prob.zeros()) == 1 and cg.iter_ == maxit
    zero = prob.zeros()
    cg = GCG(CGTraits(maxit=50, tol=1e-12, relative=1, precond=1), prob)
    assert cg.solve(H, zero, prob.zeros(), prob.zeros()) == 0 and cg.iter_ == 0
    b[50] = float("nan")  # an interior node of element 1
    with pytest.raises(GFError):
        cg.solve(H, b, prob.zeros(), prob.zeros())


@pytest.mark.parametrize("p", ORDERS)
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("geom", ["regular", "deformed", "affine"])
def test_line_applies(ctx, p, dim, geom):
    import torch
    from geoflow_b200 import GHelmholtz, GridBox, Problem
    ne = [3, 2, 2][:dim]
    g = GridBox(dim, ne, p)
    N, n = g.ndof(), p + 1
    rng = np.random.default_rng(10 * p + dim)
    shape = [g.nelems] + [n] * dim
    D, W = g.D.reshape(n, n).T, g.W  # D[l, m]
    w = W
    for _ in range(dim - 1):
        w = np.multiply.outer(W, w)
    if geom == "deformed":
        X = rng.standard_normal((dim, dim, N)) * 0.3 + 2.0 * np.eye(dim)[:, :, None]
        J = 0.1 + rng.random(N)
        prob = Problem(ctx, g, structured=False, geometry="deformed",
                       node_geom=np.concatenate([X.reshape(-1), J]))
    else:
        prob = Problem(ctx, g, geometry=geom)
        eg = g.elem_geom.reshape(g.nelems, dim + 1)
        X = np.zeros((dim, dim, N))
        for d in range(dim):
            X[d, d] = np.repeat(eg[:, d], n**dim)
        J = np.repeat(eg[:, dim], n**dim)
    u, pv, qv = rng.standard_normal(N), 1.0 + rng.random(N), 1.0 + rng.random(N)
    mass = w[None] * J.reshape(shape)

    def along(M, f, d):  # contraction along reference direction d (0 = x, the last axis)
        return np.moveaxis(np.tensordot(M, f, axes=(1, dim - d)), 0, dim - d)

    U = u.reshape(shape)
    du = [along(D, U, d) for d in range(dim)]
    phys = [sum(X[i, k].reshape(shape) * du[i] for i in range(dim)) for k in range(dim)]
    for vec in (False, True):
        P, Q = (pv.reshape(shape), qv.reshape(shape)) if vec else (0.6, 1.7)
        ref = Q * mass * U
        for i in range(dim):
            flux = P * mass * sum(X[i, k].reshape(shape) * phys[k] for k in range(dim))
            ref = ref + along(D.T, flux, i)
        ref = cuda(ref.reshape(-1), torch.float64)
        for dt, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
            H = GHelmholtz(prob)
            H.set_Lap_scalar(cuda(pv, dt) if vec else 0.6)
            H.set_mass_scalar(cuda(qv, dt) if vec else 1.7)
            out = prob.zeros(dt)
            H.opVec_prod(cuda(u, dt), None, out)
            assert rel(out, ref) < tol, (vec, dt, rel(out, ref))


@pytest.mark.parametrize("scheme", [A.GF_RK1, A.GF_RK2, A.GF_RK3, A.GF_RK4])
def test_reverse_passes_box_equal_csr(ctx, scheme):
    """The fused reverse class passes on a box against the CSR member lists."""
    import torch
    from geoflow_b200 import GBurgers, GridBox, Problem
    g = GridBox(3, [3, 2, 4], 3, periodic=[1, 0, 1])
    rng = np.random.default_rng(scheme)
    u0 = [0.3 * rng.standard_normal(g.ndof()) for _ in range(3)]
    obs = [0.3 * rng.standard_normal(g.ndof()) for _ in range(3)]
    out = []
    for s in (True, False):
        prob = Problem(ctx, g, dirichlet_mask=False, structured=s)
        B = GBurgers(prob, GBurgers.BURGERS, 1e-2, scheme=scheme)
        out.append(B.adjoint_gradient([cuda(a, torch.float64) for a in u0], None,
                                      [cuda(a, torch.float64) for a in obs], 1e-3, 5, 2))
    (ja, ga), (jb, gb) = out
    assert abs(ja - jb) <= 1e-13 * abs(jb)
    for a, b in zip(ga, gb):
        assert rel(a, b) < 1e-13


@pytest.mark.parametrize("ne,p,per", [([33, 31, 33], 2, [0, 1, 0]), ([14, 11, 10], 6, [1, 0, 0]),
                                      ([7, 8, 9], 9, [1, 1, 0]), ([9, 10, 8], 9, [0, 1, 0]),
                                      ([40, 41, 43], 1, [1, 0, 0]), ([75, 77], 7, [0, 0]),
                                      ([262, 260], 2, [1, 0])])
def test_lattice_runs_equal_csr(ctx, ne, p, per):
    """Lattices of more than 2^18 points are walked in runs (smaller ones, point by
    point): gathers and RK steps bit for bit as the member lists have them."""
    import torch
    from geoflow_b200 import GBurgers, GGFX, GridBox, Problem
    g = GridBox(len(ne), ne, p, periodic=per)
    rng = np.random.default_rng(p)
    probs = [Problem(ctx, g, dirichlet_mask=False, structured=s) for s in (True, False)]
    v = rng.standard_normal(g.ndof())
    u0 = [0.3 * rng.standard_normal(g.ndof()) for _ in ne]
    for dt in (torch.float64, torch.float32):
        for op in (A.GF_DSS_SUM, A.GF_DSS_SMOOTH, A.GF_DSS_MAX, A.GF_DSS_MIN):
            a, b = cuda(v, dt), cuda(v, dt)
            assert GGFX(probs[0]).doOp(a, op) and GGFX(probs[1]).doOp(b, op)
            assert bits_equal(a, b), (dt, op)
        for scheme in (A.GF_RK2, A.GF_RK4, A.GF_SSP33):
            us = []
            for prob in probs:
                u = [cuda(a, dt) for a in u0]
                GBurgers(prob, A.GF_EQN_BURGERS, 1e-2, scheme=scheme).step(u, None, dt=1e-4, nsteps=1)
                us.append(u)
            for a, b in zip(*us):
                assert bits_equal(a, b), (dt, scheme)


@pytest.mark.parametrize("ne,p", [([33, 31, 33], 2), ([11, 10, 9], 7)])
def test_multigrid_runs(ctx, ne, p):
    """Multigrid on more than 2^18 points against the Jacobi solve of the same grid
    without its box description."""
    import torch
    from geoflow_b200 import CGTraits, GCG, GHelmholtz, GridBox, Problem
    g = GridBox(3, ne, p)
    b = cuda(np.random.default_rng(p).standard_normal(g.ndof()), torch.float64)
    xs = []
    for s, pre in ((True, A.GF_PRECOND_PMG), (False, A.GF_PRECOND_JACOBI)):
        prob = Problem(ctx, g, structured=s)
        H = GHelmholtz(prob)
        H.set_mass_scalar(20.0)
        x = prob.zeros()
        cg = GCG(CGTraits(maxit=4000, tol=1e-11, relative=1, precond=pre), prob)
        assert cg.solve(H, b, x) == 0
        xs.append(x)
    assert rel(*xs) < 1e-8


def test_ssp_steps_allocate_what_they_use(ctx):
    """Work vectors of an SSP advance: one slope and the results of the substeps but
    the last, per component; none for step_b's running sum."""
    import torch
    from geoflow_b200 import GBurgers, GridBox, Problem

    def advance(ne):
        g = GridBox(3, [ne] * 3, 5)
        prob = Problem(ctx, g, dirichlet_mask=False)
        u = prob.zeros(ncomp=3)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        GBurgers(prob, A.GF_EQN_BURGERS, 1e-2, scheme=A.GF_SSP33).step(u, None, dt=1e-4)
        torch.cuda.synchronize()
        return (free - torch.cuda.mem_get_info()[0]) / (8 * g.ndof())

    advance(2)  # loads the kernels
    assert advance(24) < 3 * (1 + 2) + 1  # in vectors of 24 MB
