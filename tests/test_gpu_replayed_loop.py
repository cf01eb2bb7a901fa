"""The replayed DFGMRES loop against the host-driven one where its kernels branch: no basis, a basis
with A W, a basis without it (A z is formed, as for the seepage tangent, which is not symmetric),
few iterations and more than 32 and than 64 (the rotations are staged 32 at a time, the triangle up
to 64), and a graph captured for one form and used by the other.

Iterates agree within 1e-12 and residual histories within 1e-10 relative (+1e-12): the bounds of
the existing comparison of the two loops."""
import ctypes as C

import numpy as np
import pytest
import torch

from slope_stability_octave_b200 import _lib, problems
from slope_stability_octave_b200.device import cur_stream, ptr
from slope_stability_octave_b200.linear_solvers import AMG, DFGMRES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system(cuda_device):
    P = problems.slope_3d(1, dims=(15, 10, 15, 10, 10, 2)).to_device()
    P.cons.init_K_r_pattern()
    P.cons.reduction(1.0)
    P.cons.build_F_and_DS_reduced(torch.zeros(P.dmesh.n_dof, dtype=torch.float64, device=cuda_device))
    return P, P.cons.build_K_r_QQ_vals(1e-2).clone()


def solve(ws, P, K, amg, W, AW, k, b, maxit):
    x = torch.empty_like(b)
    it, rel = C.c_int32(), C.c_double()
    hist = np.zeros(maxit + 1)
    _lib.call("sg_dfgmres_solve", ws, P.dmesh.bsr, ptr(K), amg.handle if amg else None, ptr(W) if k else None,
              ptr(AW) if AW is not None else None, k, ptr(b), ptr(x), 1e-10, maxit, C.byref(it), C.byref(rel),
              hist.ctypes.data_as(C.c_void_p), cur_stream())
    return x, it.value, hist[: it.value + 1]


@pytest.mark.parametrize("maxit,with_amg", [(3, True), (60, True), (33, False), (70, False)])
def test_forms_of_the_projection(system, cuda_device, maxit, with_amg):
    P, K = system
    amg = AMG(P.dmesh) if with_amg else None
    if amg:
        amg.update(K)
    sol = DFGMRES(P.dmesh, 1e-10, maxit, 1e-3, amg=amg)
    g = torch.Generator(device="cuda").manual_seed(maxit)
    sol.basis = torch.randn((5, P.dmesh.n_dof), dtype=torch.float64, device=cuda_device, generator=g) * P.dmesh.mask
    sol.A_orthogonalize(K)
    W = sol.basis
    k = W.shape[0]
    AW = torch.empty_like(W)
    for i in range(k):
        P.dmesh.spmv(K, W[i], AW[i])
    b = P.f_device() * P.dmesh.mask
    # the forms one after the other on one workspace, the first one again at the end
    forms = [(0, None), (k, AW), (k, None), (0, None), (k, None), (k, AW)]
    out = {}
    for graph in (1, 0):
        _lib.call("sg_krylov_set_graph", sol._ws.handle, graph)
        out[graph] = [solve(sol._ws.handle, P, K, amg, W, aw, kk, b, maxit) for kk, aw in forms]
    for (xg, ig, hg), (xh, ih, hh) in zip(out[1], out[0]):
        assert ig == ih and ig > 0
        assert (xg - xh).abs().max() <= 1e-12 * xh.abs().max()
        assert np.all(np.abs(hg - hh) <= 1e-12 + 1e-10 * hh)
