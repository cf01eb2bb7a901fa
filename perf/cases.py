"""The work that users of this framework have it do, as measurable cases.

A strength-reduction or limit-load run is a sequence of Newton iterations, and every one of
them calls the same few public entry points on the same mesh handle: the residual at a trial
displacement, the residual with its tangent and the regularised stiffness, the
A-orthogonalisation of the deflation basis, and the preconditioned solves.  Each of these is
a kind of case here; three more are a whole Newton solve, one Newton iteration of the seepage
problem, and the host-buffer return mapping that the MEX functions call.

    residual   CONSTITUTIVE.build_F_all: F at a reduction factor and a displacement (line
               searches and the lambda + eps difference call nothing else)
    tangent    CONSTITUTIVE.build_F_and_DS_all and build_K_r_QQ_vals: what a Newton iteration
               starts with
    basis      DFGMRES.A_orthogonalize of a k-column deflation basis against the new K_r
    linear     the linear part of a Newton iteration: preconditioner update for the new K_r,
               A-orthogonalisation, and the pair of deflated FGMRES solves, to the relative
               tolerance 1e-1 of the slope scripts, with the FP64 or the mixed (FP32)
               V-cycle
    newton     newton_ind_SSR from an accepted continuation step to the next omega
    seepage    one Newton iteration of newton_flow: system, preconditioner update,
               A-orthogonalisation and solve of the non-symmetric pressure tangent (1e-6)
    host       sg_constitutive3d on host arrays: stress, tangent and branch per point

Meshes are the slope scripts': the 2D profile with spacing h, and the 3D profile extruded by
``depth`` metres at ``n_h`` cells per metre, homogeneous or with the four material layers.
A program sets its mesh handle up once and runs on it for hours, so the handles are kept
between states (a few at a time); everything else is made from the seed: strength and
stiffness of each layer, displacement, reduction factor, regularisation, basis vectors.
"""
import collections
import math

import numpy as np
import torch

from slope_stability_octave_b200 import _lib, fem, newton, problems, seepage, workloads
from slope_stability_octave_b200.constitutive import CONSTITUTIVE
from slope_stability_octave_b200.device import DeviceMesh, dot, hptr
from slope_stability_octave_b200.linear_solvers import set_linear_solver

F64 = torch.float64
PROFILE = (15, 10, 15, 10, 10)     # x1 x2 x3 y1 y2 of the slope scripts


def listed():
    return [
        # the line search of the 2D benchmark slope (h = 0.5): the smallest call, all latency
        dict(name="residual_2d_h05", kind="residual", dim=2, h=0.5, layered=False),
        # start of a Newton iteration on the reference's stored 2D run (h = 1/4)
        dict(name="tangent_2d_h025", kind="tangent", dim=2, h=0.25, layered=False),
        # the same in 3D on a mesh with odd counts everywhere (a script with its own depth and
        # spacing)
        dict(name="tangent_3d_ragged", kind="tangent", dim=3, n_h=0.93, depth=12.7, layered=True),
        # a whole Newton solve of the omega-constrained step, small 3D slope
        dict(name="newton_3d_z5", kind="newton", dim=3, n_h=1.0, depth=5.0, layered=False),
        # a seepage Newton iteration, pressure on the nodes of a 10 m slope
        dict(name="seepage_3d_z10", kind="seepage", dim=3, n_h=1.0, depth=10.0, k=4),
        # the 40 m slope: line search, basis in the middle of a continuation step, solves
        dict(name="residual_3d_z40", kind="residual", dim=3, n_h=1.0, depth=40.0, layered=False),
        dict(name="basis_3d_z40_k21", kind="basis", dim=3, n_h=1.0, depth=40.0, layered=False, k=21),
        dict(name="linear_3d_z40", kind="linear", dim=3, n_h=1.0, depth=40.0, layered=False, k=9, mixed=False),
        # the layered slope at h = 0.6 m (2.9M unknowns, 8M points): the largest systems
        dict(name="tangent_3d_layered", kind="tangent", dim=3, n_h=5 / 3, depth=40.0, layered=True),
        dict(name="basis_3d_layered_k38", kind="basis", dim=3, n_h=5 / 3, depth=40.0, layered=True, k=38),
        dict(name="linear_3d_layered_mixed", kind="linear", dim=3, n_h=5 / 3, depth=40.0, layered=True, k=15,
             mixed=True),
        # return mapping of host arrays, the five branches 20 % each (a MEX call on a mid-size mesh)
        dict(name="host_return_map", kind="host", n=150_001),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["residual", "residual", "tangent", "tangent", "basis", "linear", "linear", "newton", "seepage",
                       "host"])
    if kind == "host":
        return dict(kind=kind, n=int(_log_uniform(rng, 1e3, 3e5)))
    case = dict(kind=kind, dim=3 if kind in ("newton", "seepage") or rng.random() < 0.7 else 2)
    # nodes of the 3D mesh: about 5500 depth n_h^3; solves and bases up to the 40 m slope,
    # whole Newton solves and seepage up to about 60,000 nodes
    if case["dim"] == 2:
        case["h"] = round(_log_uniform(rng, 0.2, 1.0), 3)
    else:
        most = dict(residual=1.0e6, tangent=1.0e6, basis=2.2e5, linear=2.2e5, newton=4e4, seepage=6e4)[kind]
        nodes = _log_uniform(rng, 4e3, most)
        n_h = rng.uniform(0.6, min(5 / 3, (nodes / 5500) ** (1 / 3)) if nodes > 5500 * 0.7 ** 3 else 0.7)
        case["n_h"] = round(max(n_h, (nodes / 5500 / 40) ** (1 / 3)), 3)
        case["depth"] = round(min(40.0, max(1.0, nodes / 5500 / case["n_h"] ** 3)), 1)
    if kind != "seepage":
        case["layered"] = rng.random() < 0.5 and case["dim"] == 3
    if kind == "basis":
        case["k"] = int(_log_uniform(rng, 2, 80))
    if kind == "linear":
        case["k"] = rng.randint(0, 24)
        case["mixed"] = rng.random() < 0.5
    if kind == "seepage":
        case["k"] = rng.randint(0, 8)
    return case


# ------------------------------------------------------------------ meshes (kept, a few at a time)

_kept = collections.OrderedDict()


def _problem(case):
    key = (case["dim"], case.get("h"), case.get("n_h"), case.get("depth"), case.get("layered", False))
    if key in _kept:
        _kept.move_to_end(key)
        return _kept[key]
    while len(_kept) >= 5:
        _kept.popitem(last=False)
    if case["dim"] == 2:
        P = problems.slope_2d(case["h"])
    else:
        make = problems.slope_3d_layered if case.get("layered") else problems.slope_3d
        P = make(case["n_h"], PROFILE + (case["depth"],))
    P.dmesh = DeviceMesh(P.mesh, P.dphi, P.weight, P.n_q)
    P.xyz = torch.from_numpy(np.ascontiguousarray(P.mesh.coord)).cuda()
    _kept[key] = P
    return P


# ------------------------------------------------------------------ seeded inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * seed + 17)


def _modes(P, g, count, waves, dim=None):
    """``count`` smooth fields on the nodes (rows, node-major): each a sum of three products
    of cosines with up to ``waves`` half waves along each axis in a random direction."""
    dim = P.mesh.dim if dim is None else dim
    X = P.xyz
    lo, hi = X.min(1).values[:, None], X.max(1).values[:, None]
    Xn = (X - lo) / (hi - lo) * math.pi
    out = torch.zeros((count, X.shape[1], dim), dtype=F64, device="cuda")
    for row in out:
        for _ in range(3):
            m = torch.randint(0, waves + 1, (X.shape[0], 1), generator=g, device="cuda")
            shift = torch.rand((X.shape[0], 1), generator=g, device="cuda", dtype=F64) * math.pi
            way = torch.randn(dim, generator=g, device="cuda", dtype=F64)
            row += torch.cos(m * Xn + shift).prod(0)[:, None] * way
    return out.reshape(count, -1)


def _displacement(P, g):
    """One-dimensional settlement under gravity with smooth lateral and vertical movements
    that bring part of the slope to yield."""
    y = P.xyz[1]
    settle = -20.0 / 54000.0 * (20.0 * y - 0.5 * y * y)
    U = _modes(P, g, 1, 5)[0] * 1.5e-3
    U = U.view(-1, P.mesh.dim)
    U[:, 1] += settle
    return (U.reshape(-1) * P.dmesh.mask).contiguous()


def _constitutive(P, seed):
    """CONSTITUTIVE with each layer's cohesion, friction angle and stiffness moved by the seed."""
    rng = np.random.default_rng(seed)
    m = P.mat
    kinds, layer = np.unique(m["c0"].reshape(P.mesh.n_e, P.n_q)[:, 0], return_inverse=True)
    per = lambda lo, hi: np.repeat(rng.uniform(lo, hi, kinds.size)[layer], P.n_q)
    stiff = per(0.85, 1.15)
    return CONSTITUTIVE(P.dmesh, m["c0"] * per(0.8, 1.25), m["phi"] * per(0.92, 1.08), m["psi"], "B",
                        m["shear"] * stiff, m["bulk"] * stiff, m["lame"] * stiff)


def _scalars(seed):
    rng = np.random.default_rng([seed, 5])
    return float(rng.uniform(0.9, 1.3)), float(10 ** rng.uniform(-2.0, -1.0))     # lambda, r


def prepare(case, seed):
    kind = case["kind"]
    if kind == "host":
        d = workloads.constitutive_points(case["n"], seed=seed)
        n = case["n"]
        d = {k: np.ascontiguousarray(d[k]) for k in ("E", "c_bar", "sin_phi", "shear", "bulk", "lame")}
        return dict(d, kind=kind, n=n, S=np.zeros((n, 6)), DS=np.zeros((n, 36)), branch=np.zeros(n, np.uint8))
    P = _problem(case)
    g = _generator(seed)
    lam, r = _scalars(seed)
    if kind == "seepage":
        return _prepare_seepage(P, case, g)
    cons = _constitutive(P, seed)
    s = dict(kind=kind, P=P, lam=lam, r=r, U=_displacement(P, g))
    if kind == "residual":
        return dict(s, cons=cons)
    cons.init_K_r_pattern()
    if kind == "tangent":
        return dict(s, cons=cons)
    solver = set_linear_solver("DFGMRES_B200_MIXED" if case.get("mixed") else "DFGMRES_B200", 1e-1, 100, 1e-3, 0,
                               P.dmesh, P.mesh.coord)
    f = torch.from_numpy(np.ascontiguousarray(P.f.T)).cuda().reshape(-1)
    if kind == "newton":
        # the last accepted step of a continuation: equilibrium at lambda = 0.9
        U1, flag, _, _ = newton.newton(torch.zeros_like(f), 1e-4, 100, 10, 1e-4, None, P.dmesh.mask, f, _reduced(cons, 0.9),
                                       solver)
        assert flag == 0
        solver.expand_deflation_basis(U1)
        return dict(kind=kind, P=P, cons=cons, solver=solver, U=U1, f=f, lam=0.9, omega=1.08 * dot(f * P.dmesh.mask, U1))
    if case["k"]:
        solver.basis = solver._rows(case["k"])
        solver.basis.copy_(_modes(P, g, case["k"], 7) * P.dmesh.mask)
    F = cons.build_F_and_DS_all(lam, s["U"])
    K = cons.build_K_r_QQ_vals(r)
    if kind == "basis":
        return dict(kind=kind, P=P, solver=solver, K=K)
    # the hierarchy stands since the first iteration of the run, on the elastic matrix
    solver.setup_preconditioner(cons.elastic_K_QQ())
    torch.cuda.synchronize()
    mask = P.dmesh.mask
    return dict(kind=kind, P=P, solver=solver, K=K, b1=f * mask, b2=(f - F) * mask, mixed=case["mixed"])


def _reduced(cons, lam):
    cons.reduction(lam)
    return cons


def _prepare_seepage(P, case, g):
    """The homogeneous seepage slope: phreatic boundary, conductivity of each element
    lognormal about the script's, pressure about the boundary's with part of it in the
    penalty band."""
    Q_w, pw_D = problems.homo_slope_seepage_bc(P.mesh.coord)
    cond = torch.exp(0.5 * torch.randn(P.mesh.n_e, generator=g, device="cuda", dtype=F64))
    S = seepage.SeepageSystem(P.dmesh, P.hat, cond.repeat_interleave(P.n_q).cpu().numpy(), Q_w)
    solver = seepage.seepage_solver(P.dmesh, Q_w)
    pD = torch.from_numpy(pw_D).cuda()
    pw = pD + S.mask * (40.0 * _modes(P, g, 1, 4, dim=1)[0] + 20.0)
    solver.setup_preconditioner(S.system(pD, 1)[0])
    if case["k"]:
        solver.basis = solver._rows(case["k"])
        solver.basis.copy_(_modes(P, g, case["k"], 5, dim=1) * S.mask)
    K, F = S.new_values(), S.new_node_vector()
    torch.cuda.synchronize()
    return dict(kind="seepage", P=P, S=S, solver=solver, pw=pw, K=K, F=F, cond=cond)


# ------------------------------------------------------------------ one pass

def run(s):
    kind = s["kind"]
    if kind == "residual":
        return s["cons"].build_F_all(s["lam"], s["U"])
    if kind == "tangent":
        c = s["cons"]
        F = c.build_F_and_DS_all(s["lam"], s["U"])
        K = c.build_K_r_QQ_vals(s["r"])
        return dict(F=F, S=c.S, DS=c.DS, K=K, branch=c.branch)
    if kind == "host":
        _lib.call("sg_constitutive3d", *[hptr(s[k]) for k in ("E", "c_bar", "sin_phi", "shear", "bulk", "lame")],
                  s["n"], hptr(s["S"]), hptr(s["DS"]), hptr(s["branch"]))
        return dict(S=s["S"], DS=s["DS"], branch=s["branch"])
    solver = s["solver"].copy()        # every continuation attempt works on a copy of the solver
    if kind == "basis":
        solver.A_orthogonalize(s["K"])
        return dict(W=solver.basis, AW=solver.AW)
    if kind == "linear":
        K = s["K"]
        solver.setup_preconditioner(K)
        solver.A_orthogonalize(K)
        (x1, _), (x2, _) = solver.solve_pair(K, s["b1"], s["b2"])
        if s["mixed"]:     # an FP32 V-cycle's directions to 1e-1: single precision is all they hold
            return dict(x1=x1.float(), x2=x2.float())
        return dict(x1=x1, x2=x2)
    if kind == "seepage":
        S = s["S"]
        K, F = S.system(s["pw"], 2, K=s["K"], F=s["F"])
        solver.setup_preconditioner(K)
        solver.A_orthogonalize(K)
        dp, _ = solver.solve(K, F)
        return dict(K=K, F=F, dp=dp)
    U, lam, _, _, _ = newton.newton_ind_SSR(s["U"], s["omega"], s["lam"], 100, 10, 1e-4, 1e-4, None, s["P"].dmesh.mask,
                                            s["f"], s["cons"], solver)
    return dict(U=U, lam=lam)


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "host":
        return dict(bytes=case["n"] * (80 + 48 + 288 + 1), flops=case["n"] * 900)
    P = _problem(case)
    m = P.dmesh
    dim, n_int, nodes, blocks = m.dim, m.n_int, m.n_n, m.n_blocks
    n, bb = dim * nodes, dim * dim
    ns, rows = (6, 6) if dim == 3 else (3, 4)
    # per point: gradients, weight, c0 phi psi shear lame; mesh: element nodes; U in, F out
    point = 8 * (dim * m.n_p + 1 + 5)
    elements = m.n_e * m.n_p * 4 + 16 * n
    strain_force = n_int * m.n_p * dim * 2 * dim * 2
    if kind == "residual":
        return dict(bytes=n_int * point + elements, flops=strain_force + n_int * 250)
    if kind == "tangent":
        nl = dim * m.n_p
        return dict(bytes=n_int * (point + 8 * (rows + ns * ns) + 1) + elements + 2 * 8 * bb * blocks,
                    flops=strain_force + n_int * (900 + nl * ns * dim * 2 + nl * (nl + 1) // 2 * dim * 2))
    matrix = blocks * (8 * bb + 4) + 4 * nodes
    if kind == "basis":
        k = case["k"]
        return dict(bytes=matrix + 3 * 8 * n * k, flops=k * (2 * bb * blocks + 2 * n * k + 2 * n * (k + 1)))
    if kind == "linear":
        # every product with the matrix that two solves of one iteration each need (residual,
        # six in the V-cycle, Arnoldi), on a matrix that is read from memory each time
        k = case["k"]
        cycle = (6 * blocks * (4 * bb if case["mixed"] else 8 * bb)) + 2 * matrix
        return dict(bytes=matrix + 2 * cycle + 3 * 8 * n * k + 4 * 8 * n, flops=(16 + k) * 2 * bb * blocks)
    if kind == "seepage":
        scalar = blocks * 12 + 4 * nodes
        return dict(bytes=n_int * 8 * (dim * m.n_p + 1 + 1 + dim) + m.n_e * (m.n_p * 4 + 8) + 10 * scalar,
                    flops=n_int * m.n_p * m.n_p * 2 * (dim + 1) + 20 * blocks)
    return dict(bytes=4 * (2 * n_int * (point + 8 * ns * ns) + 10 * matrix), flops=4 * 20 * 2 * bb * blocks)


# ------------------------------------------------------------------ the same in 64 bits of plain torch

def _principal_law(lamb, c, sp, G, la):
    """Mohr-Coulomb return in principal strains lamb (n, 3), e1 >= e2 >= e3: principal stresses
    f, their derivative J (n, 3, 3) and the pairs whose stresses are merged."""
    e1, e2, e3 = lamb.T
    tr = e1 + e2 + e3
    one = torch.ones_like(lamb)
    eye = torch.eye(3, dtype=F64, device=lamb.device)
    nrm = torch.stack([2 * G * (1 + sp), 0 * G, -2 * G * (1 - sp)], 1) + (2 * la * sp)[:, None]
    f_tr = (nrm * lamb).sum(1) - c

    def average(a, b):       # stiffness averaged over a merged pair
        M = torch.zeros((3, 3), dtype=F64, device=lamb.device)
        M[a, a] = M[a, b] = M[b, a] = M[b, b] = 0.5
        M[3 - a - b, 3 - a - b] = 1.0
        return M

    def face(M):
        C = la[:, None, None] + 2 * G[:, None, None] * M
        nf = nrm @ M
        flow = torch.stack([2 * G * (1 + sp), 0 * G, -2 * G * (1 - sp)], 1) @ M + (2 * la * sp)[:, None]
        m = torch.stack([1 + sp, 0 * sp, -(1 - sp)], 1) @ M
        den = (flow * m).sum(1)
        dl = ((nf * lamb).sum(1) - c) / den
        f = (C @ lamb[..., None])[..., 0] - dl[:, None] * flow
        J = C - flow[:, :, None] * nf[:, None, :] / den[:, None, None]
        return f, J, dl

    M0, ML, MR = eye, average(0, 1), average(1, 2)
    fe = la[:, None] * tr[:, None] + 2 * G[:, None] * lamb
    Je = la[:, None, None] + 2 * G[:, None, None] * eye
    fs, Js, dls = face(M0)
    fl, Jl, dll = face(ML)
    fr, Jr, dlr = face(MR)
    gsl, gsr = (e1 - e2) / (1 + sp), (e2 - e3) / (1 - sp)
    gla, gra = (e1 + e2 - 2 * e3) / (3 - sp), (2 * e1 - e2 - e3) / (3 + sp)
    elastic = f_tr <= 0
    smooth = ~elastic & (dls <= gsl) & (dls <= gsr)
    left = ~elastic & ~smooth & (gsl < gsr) & (dll >= gsl) & (dll <= gla)
    right = ~elastic & ~smooth & ~left & (gsl > gsr) & (dlr >= gsr) & (dlr <= gra)
    f = (c / (2 * sp))[:, None] * one
    J = torch.zeros_like(Je)
    branch = torch.full_like(e1, 4)
    for number, (on, fb, Jb) in enumerate(((elastic, fe, Je), (smooth, fs, Js), (left, fl, Jl), (right, fr, Jr))):
        f = torch.where(on[:, None], fb, f)
        J = torch.where(on[:, None, None], Jb, J)
        branch = torch.where(on, torch.full_like(e1, number), branch)
    return f, J, branch


def _return_map(E, c, sp, G, la, tangent):
    """Stress (n, 6) and tangent (n, 6, 6) of engineering strains (n, 6), from the spectral
    decomposition of the strain tensor."""
    place = ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))
    T = torch.zeros((E.shape[0], 3, 3), dtype=F64, device=E.device)
    for a, (i, j) in enumerate(place):
        T[:, i, j] = T[:, j, i] = E[:, a] * (1.0 if i == j else 0.5)
    val, vec = torch.linalg.eigh(T.cpu())
    lamb, N = val.flip(1).to(E.device), vec.flip(2).to(E.device)
    f, J, branch = _principal_law(lamb, c, sp, G, la)
    S = torch.einsum("nik,nk,njk->nij", N, f, N)
    S = torch.stack([S[:, i, j] for i, j in place], 1)
    if not tangent:
        return S, None
    gap = lamb[:, :, None] - lamb[:, None, :]
    quotient = (f[:, :, None] - f[:, None, :]) / torch.where(gap.abs() > 0, gap, torch.ones_like(gap))
    quotient = torch.where((branch == 0)[:, None, None], 2 * G[:, None, None].expand_as(gap), quotient)
    quotient.diagonal(dim1=1, dim2=2).zero_()
    D = torch.empty((E.shape[0], 6, 6), dtype=F64, device=E.device)
    for b, (i, j) in enumerate(place):
        H = torch.zeros((3, 3), dtype=F64, device=E.device)
        H[i, j] = H[j, i] = 1.0 if i == j else 0.5
        Hp = torch.einsum("nik,ij,njl->nkl", N, H, N)
        dS = quotient * Hp
        dS.diagonal(dim1=1, dim2=2).add_(torch.einsum("nkl,nl->nk", J, Hp.diagonal(dim1=1, dim2=2)))
        dS = torch.einsum("nik,nkl,njl->nij", N, dS, N)
        for a, (p, q) in enumerate(place):
            D[:, a, b] = dS[:, p, q]
    return S, D


def _davis_b(c0, phi, psi, lam):
    c1, f1, s1 = c0 / lam, torch.atan(torch.tan(phi) / lam), torch.atan(torch.tan(psi) / lam)
    beta = torch.cos(f1) * torch.cos(s1) / (1 - torch.sin(f1) * torch.sin(s1))
    fl = torch.atan(beta * torch.tan(f1))
    return 2 * beta * c1 * torch.cos(fl), torch.sin(fl)


def _strain_matrix(dphi, n_e, n_q):
    """B (n_e, n_q, n_strain, dim n_p) of the elements from their gradients."""
    d = [torch.as_tensor(x, device="cuda").reshape(n_e, n_q, -1) for x in dphi]
    dim, n_p = len(d), d[0].shape[2]
    B = torch.zeros((n_e, n_q, 6 if dim == 3 else 3, n_p, dim), dtype=F64, device="cuda")
    for a in range(dim):
        B[:, :, a, :, a] = d[a]
    for row, (i, j) in zip(range(dim, B.shape[2]), ((0, 1), (1, 2), (0, 2)) if dim == 3 else ((0, 1),)):
        B[:, :, row, :, i] = d[j]
        B[:, :, row, :, j] = d[i]
    return B.reshape(n_e, n_q, -1, n_p * dim)


def _exact_elements(s, tangent):
    P, c = s["P"], s["cons"]
    mesh, dim, n_q = P.mesh, P.mesh.dim, P.n_q
    n_e, n = mesh.n_e, dim * mesh.n_n
    cb, sp = _davis_b(c.c0, c.phi, c.psi, s["lam"])
    elem = torch.as_tensor(mesh.elem.T.astype(np.int64), device="cuda")                  # n_e x n_p
    dofs = (elem[:, :, None] * dim + torch.arange(dim, device="cuda")).reshape(n_e, -1)
    w = torch.as_tensor(P.weight, device="cuda").reshape(n_e, n_q)
    ns, rows = (6, 6) if dim == 3 else (3, 4)
    nl = dofs.shape[1]
    F = torch.zeros(n, dtype=F64, device="cuda")
    S_all = torch.empty((n_e, n_q, rows), dtype=F64, device="cuda")
    D_all = torch.empty((n_e, n_q, ns, ns), dtype=F64, device="cuda") if tangent else None
    if tangent:
        a, b = torch.broadcast_tensors(elem[:, :, None], elem[:, None, :])
        pairs, slot = torch.unique((a * mesh.n_n + b).reshape(-1), return_inverse=True)
        slot = slot.reshape(n_e, -1)
        nb = pairs.numel()
        Kt = torch.zeros((nb, dim * dim), dtype=F64, device="cuda")
        Kel = torch.zeros_like(Kt)
    for e0 in range(0, n_e, 4000):
        e1 = min(n_e, e0 + 4000)
        g = slice(e0 * n_q, e1 * n_q)
        B = _strain_matrix([d[g] for d in P.dphi], e1 - e0, n_q)
        E = torch.einsum("eqsl,el->eqs", B, s["U"][dofs[e0:e1]]).reshape(-1, ns)
        E6 = E
        if dim == 2:       # plane strain
            E6 = torch.zeros((E.shape[0], 6), dtype=F64, device="cuda")
            E6[:, 0], E6[:, 1], E6[:, 3] = E.T
        S, D = _return_map(E6, cb[g], sp[g], c.shear[g], c.lame[g], tangent)
        if dim == 2:
            S = S[:, [0, 1, 3, 2]]
            D = D[:, [0, 1, 3]][:, :, [0, 1, 3]] if tangent else None
        S_all[e0:e1] = S.reshape(-1, n_q, rows)
        Fe = torch.einsum("eq,eqsl,eqs->el", w[e0:e1], B, S_all[e0:e1, :, :ns])
        F.index_add_(0, dofs[e0:e1].reshape(-1), Fe.reshape(-1))
        if tangent:
            D_all[e0:e1] = D.reshape(-1, n_q, ns, ns)
            # elastic: 2 G dev + K vol with iota = (1 1 1 0 0 0); in 2D the scripts' iota is (1 1 1)
            iota = torch.zeros(ns, dtype=F64, device="cuda")
            iota[:3] = 1.0
            vol = iota[:, None] * iota
            dev = torch.diag(torch.tensor([1.0] * dim + [0.5] * (ns - dim), dtype=F64, device="cuda")) - vol / 3
            Del = (2 * c.shear[g][:, None, None] * dev + c.bulk[g][:, None, None] * vol).reshape(-1, n_q, ns, ns)
            for out, DD in ((Kt, D_all[e0:e1]), (Kel, Del)):
                Ke = torch.einsum("eq,eqsl,eqst,eqtm->elm", w[e0:e1], B, 0.5 * (DD + DD.transpose(2, 3)), B)
                Ke = Ke.reshape(-1, nl // dim, dim, nl // dim, dim).transpose(2, 3).reshape(-1, dim * dim)
                out.index_add_(0, slot[e0:e1].reshape(-1), Ke)
    if not tangent:
        return F
    mask = torch.as_tensor(mesh.Q.T.copy(), device="cuda")
    row, col = pairs // mesh.n_n, pairs % mesh.n_n
    free = mask[row][:, :, None] & mask[col][:, None, :]
    unit = (row == col)[:, None, None] & torch.eye(dim, dtype=torch.bool, device="cuda")
    K = (s["r"] * Kel + (1 - s["r"]) * Kt).reshape(-1, dim, dim)
    K = torch.where(free, K, unit.to(F64)).reshape(-1)
    return dict(F=F, S=S_all.reshape(-1), DS=D_all.transpose(2, 3).reshape(-1), K=K, branch=None)


def _exact_basis(s):
    """A_orthogonalize.m: columns last to first, one pass against the kept ones."""
    P, W, K = s["P"], s["solver"].basis, s["K"]
    dim, nn = P.mesh.dim, P.mesh.n_n
    elem = torch.as_tensor(P.mesh.elem.T.astype(np.int64), device="cuda")
    pairs = torch.cat([torch.unique((elem[:, i] * nn)[:, None] + elem) for i in range(elem.shape[1])])
    pairs = torch.unique(pairs)
    row, col = pairs // nn, pairs % nn
    Kb = K.view(-1, dim, dim)

    def times(v):
        y = torch.zeros((nn, dim), dtype=F64, device="cuda")
        return y.index_add_(0, row, torch.einsum("pab,pb->pa", Kb, v.view(nn, dim)[col])).reshape(-1)

    kept, images, signs = [], [], []
    for v in W.flip(0):
        Av = times(v)
        u, Au = v.clone(), Av.clone()
        for w, Aw, sign in zip(kept, images, signs):
            h = sign * torch.dot(Av, w)
            u -= h * w
            Au -= h * Aw
        norm = torch.dot(u, Av)
        if abs(norm) > s["solver"].tolerance_deflation_basis:
            kept.append(u / norm.abs().sqrt())
            images.append(Au / norm.abs().sqrt())
            signs.append(torch.sign(norm))
    return dict(W=torch.stack(kept[::-1]), AW=torch.stack(images[::-1]))


def _exact_seepage(s):
    P, S = s["P"], s["S"]
    mesh, n_q, n_e = P.mesh, P.n_q, P.mesh.n_e
    nn = mesh.n_n
    elem = torch.as_tensor(mesh.elem.T.astype(np.int64), device="cuda")
    D = torch.stack([torch.as_tensor(x, device="cuda").reshape(n_e, n_q, -1) for x in P.dphi], 3)   # e q i d
    hat = torch.as_tensor(np.ascontiguousarray(P.hat.T), device="cuda")                             # q i
    w = torch.as_tensor(P.weight, device="cuda").reshape(n_e, n_q)
    wc = w * s["cond"][:, None]
    p = s["pw"][elem]
    y = torch.as_tensor(mesh.coord[1].copy(), device="cuda")[elem]
    X = torch.as_tensor(mesh.coord.copy(), device="cuda")[:, elem[:, :4]]                            # d e v
    edge = lambda a, b: X[:, :, a] - X[:, :, b]
    lengths = [edge(a, b).square().sum(0).sqrt() for a, b in ((0, 1), (0, 2), (1, 2), (0, 3), (1, 3))]
    odd = (edge(2, 3)[:2].square().sum(0) + edge(1, 3)[2].square()).sqrt()      # the scripts' L34
    eps = (seepage.GRHO * torch.stack(lengths + [odd]).min(0).values / 2)[:, None]
    pint = torch.einsum("qi,ei->eq", hat, p)
    band = (pint > 0) & (pint < eps)
    perm = torch.where(band, pint / eps, (pint >= eps).to(F64))
    der = torch.where(band, 1 / eps, torch.zeros_like(pint))
    gy = torch.einsum("eqid,ei->eqd", D, y)
    flux = torch.einsum("eqid,ei->eqd", D, p) + seepage.GRHO * perm[:, :, None] * gy
    F = torch.zeros(nn, dtype=F64, device="cuda")
    F.index_add_(0, elem.reshape(-1), -torch.einsum("eq,eqid,eqd->ei", wc, D, flux).reshape(-1))
    Ke = torch.einsum("eq,eqid,eqjd->eij", wc, D, D)
    Ke += torch.einsum("eq,eqid,eqd,qj->eij", wc * der * seepage.GRHO, D, gy, hat)
    a, b = torch.broadcast_tensors(elem[:, :, None], elem[:, None, :])
    pairs, slot = torch.unique((a * nn + b).reshape(-1), return_inverse=True)
    K = torch.zeros(pairs.numel(), dtype=F64, device="cuda").index_add_(0, slot, Ke.reshape(-1))
    free = torch.as_tensor(S.Q_w, device="cuda")
    row, col = pairs // nn, pairs % nn
    K = torch.where(free[row] & free[col], K, (row == col).to(F64))
    return dict(K=K, F=F * free, dp=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("linear", "newton"):
        return None            # what a solver returns at its tolerance depends on its preconditioner
    if kind == "host":
        s = prepare(case, seed)
        t = {k: torch.as_tensor(s[k], device="cuda") for k in ("E", "c_bar", "sin_phi", "shear", "lame")}
        S, D = _return_map(t["E"], t["c_bar"], t["sin_phi"], t["shear"], t["lame"], True)
        return dict(S=S, DS=D.transpose(1, 2).reshape(-1, 36), branch=None)
    n_int = _problem(case).dmesh.n_int
    if kind == "seepage":
        return _exact_seepage(prepare(case, seed)) if n_int < 600_000 else None
    if kind == "basis":
        return _exact_basis(prepare(case, seed)) if n_int < 2_500_000 else None
    if n_int > (1_800_000 if kind == "residual" else 500_000):
        return None            # over 20 seconds
    return _exact_elements(prepare(case, seed), kind == "tangent")
