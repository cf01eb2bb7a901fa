"""Pieces of the AMG that run in one launch each: the coarsest level's inverse over sizes around
its 32-wide tiles and around the largest size of the one-launch steps, and the Chebyshev steps
fused with their residual for each parity of the degree (the steps alternate between two arrays).

A cycle is compared with the restated one on the exported hierarchy, 1e-10 of its norm (the bound
of the cycle test at the default options) and 1e-4 in mixed precision; a dense inverse with a direct
solve, n roundings amplified by the matrix's condition number."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from oracle.amg_ref import Hierarchy
from slope_stability_octave_b200 import problems
from slope_stability_octave_b200.linear_solvers import AMG
from test_gpu_amg import elastic_problem, export

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def elastic(cuda_device):
    return elastic_problem()


@pytest.mark.parametrize("degree", [1, 2, 3, 4])
@pytest.mark.parametrize("coarse_size", [100, 1200])
def test_cycle_of_each_degree(elastic, cuda_device, degree, coarse_size):
    P, K = elastic
    amg = AMG(P.dmesh, cheb_degree=degree, coarse_size=coarse_size)
    amg.update(K)
    lev = export(amg, len(amg.info()["levels"]))
    H = Hierarchy.from_levels([A for A, _, _ in lev], [p for _, p, _ in lev[:-1]], [b for _, _, b in lev],
                              cheb_degree=degree)
    r = np.random.default_rng(degree).normal(size=P.dmesh.n_dof) * P.mesh.Q.T.ravel()
    want = H.vcycle(r)
    rd = torch.from_numpy(r).to(cuda_device)
    z = torch.empty_like(rd)
    amg.apply(rd, z)
    assert np.linalg.norm(z.cpu().numpy() - want) <= 1e-10 * np.linalg.norm(want)
    assert torch.equal(rd.cpu(), torch.from_numpy(r))
    amg.apply(rd, rd)                                     # in place: the same cycle
    assert torch.equal(rd, z)
    mixed = AMG(P.dmesh, cheb_degree=degree, coarse_size=coarse_size, mixed=True)
    mixed.update(K)
    rd = torch.from_numpy(r).to(cuda_device)
    mixed.apply(rd, z)
    assert np.linalg.norm(z.cpu().numpy() - want) <= 1e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("h,steps", [(4, True), (2, True), (1.5, False)])
def test_inverse_of_one_level(cuda_device, h, steps):
    """A hierarchy of one level is its dense inverse: 314, 1402 and 2630 unknowns, none a
    multiple of the tile, the last beyond the one-launch steps."""
    P = problems.slope_2d(h).to_device()
    P.cons.init_K_r_pattern()
    P.cons.reduction(1.0)
    P.cons.build_F_and_DS_reduced(torch.zeros(P.dmesh.n_dof, dtype=torch.float64, device=cuda_device))
    K = P.cons.build_K_r_QQ_vals(1e-2)
    amg = AMG(P.dmesh, coarse_size=12000)
    amg.update(K)
    n = P.dmesh.n_dof
    assert len(amg.info()["levels"]) == 1 and n % 32 and (n <= 2048) == steps
    A = export(amg, 1)[0][0]
    r = torch.from_numpy(np.random.default_rng(1).normal(size=n)).to(cuda_device)
    z = torch.empty_like(r)
    amg.apply(r, z)
    want = np.linalg.solve(A.toarray(), r.cpu().numpy())
    tol = n * np.finfo(float).eps * np.linalg.cond(A.toarray())
    assert np.linalg.norm(z.cpu().numpy() - want) <= tol * np.linalg.norm(want)


def star_mesh(n):
    """Tetrahedra from the centre of a ball to the triangles of n points on its surface (P2): the
    centre's row couples every node."""
    from scipy.spatial import ConvexHull
    k = np.arange(n)
    z = 1.0 - (2.0 * k + 1.0) / n
    phi = k * np.pi * (3.0 - np.sqrt(5.0))
    s = np.sqrt(1.0 - z * z)
    pts = np.stack([s * np.cos(phi), s * np.sin(phi), z], 1)
    xyz = list(np.vstack([[0.0, 0.0, 0.0], pts]))
    ref = problems.slope_3d(1, dims=(15, 10, 15, 10, 10, 2)).mesh      # order of the mid-edge nodes
    X = ref.coord[:, ref.elem[:, 0]]
    pairs = [min(((a, b) for a in range(4) for b in range(a)), key=lambda e: np.linalg.norm(
        0.5 * (X[:, e[0]] + X[:, e[1]]) - X[:, q])) for q in range(4, 10)]
    mid, elem = {}, []
    for t in ConvexHull(pts).simplices + 1:
        v = [0, *t]
        if np.linalg.det(np.array([xyz[t[0]], xyz[t[1]], xyz[t[2]]])) * \
                np.linalg.det(X[:, 1:4].T - X[:, 0]) < 0:
            v[2], v[3] = v[3], v[2]
        for a, b in pairs:
            e = (min(v[a], v[b]), max(v[a], v[b]))
            if e not in mid:
                mid[e] = len(xyz)
                xyz.append(0.5 * (xyz[e[0]] + xyz[e[1]]))
            v.append(mid[e])
        elem.append(v)
    return np.array(xyz).T, np.array(elem, np.int64).T


@pytest.mark.parametrize("n", [20, 62, 130])
def test_products_of_long_rows(cuda_device, n):
    """A P and P'(A P) of a slope with a separate ball whose centre couples all its nodes: rows
    within the shared arrays of the A P product, rows that shrink its runs, and rows beyond them,
    and a coarse block that sums most of the ball's pairs."""
    slope = problems.slope_3d(1, dims=(15, 10, 15, 10, 10, 5)).mesh
    coord, elem = star_mesh(n)
    Q = np.ones((3, coord.shape[1]), bool)
    Q[:, coord[2] < -0.7] = False
    n_s = slope.coord.shape[1]
    P = problems.slope_3d_from_mesh(np.hstack([slope.coord, coord]), np.hstack([slope.elem, elem + n_s]),
                                    np.hstack([slope.Q, Q])).to_device()
    P.cons.init_K_r_pattern()
    P.cons.reduction(1.0)
    P.cons.build_F_and_DS_reduced(torch.zeros(P.dmesh.n_dof, dtype=torch.float64, device=cuda_device))
    K = P.cons.build_K_r_QQ_vals(1e-2)
    amg = AMG(P.dmesh, max_levels=2)
    amg.update(K)
    assert len(amg.info()["levels"]) == 2
    (A, Pr, _), (Ac, _, _) = export(amg, 2)
    AP = A @ Pr
    assert AP.tobsr((3, 6)).indices.size >= 32768
    want = (Pr.T @ AP).tocsr()
    dead = np.asarray(abs(want).max(axis=1).todense()).ravel() == 0.0
    want = want + sp.diags(dead.astype(float))
    assert abs(Ac - want).max() <= 1e-12 * abs(want).max()
    mixed = AMG(P.dmesh, max_levels=2, mixed=True)
    mixed.update(K)
    for a in (amg, mixed):                 # the later updates of the mixed form are in FP32
        a.update(K)
    r = torch.from_numpy(np.random.default_rng(n).normal(size=P.dmesh.n_dof) * P.mesh.Q.T.ravel()).to(cuda_device)
    z, z32 = torch.empty_like(r), torch.empty_like(r)
    amg.apply(r, z)
    mixed.apply(r, z32)
    assert (z - z32).norm() <= 1e-4 * z.norm()
