"""Pieces of the AMG that run in one launch each: the coarsest level's inverse over sizes around
its 32-wide tiles and around the largest size of the one-launch steps, and the Chebyshev steps
fused with their residual for each parity of the degree (the steps alternate between two arrays).

A cycle is compared with the restated one on the exported hierarchy, 1e-10 of its norm (the bound
of the cycle test at the default options) and 1e-4 in mixed precision; a dense inverse with a direct
solve, n roundings amplified by the matrix's condition number."""
import numpy as np
import pytest
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
