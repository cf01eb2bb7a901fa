"""The one-pass Gram matrix and the in-place products of the A-orthogonalisation at the edges of
their eight-column tiles (up to 48 columns, where the results replace the input columns), with and
without a dropped column, and one column past them, against the column-blocked Gram-Schmidt.
Tolerance 1e-9 of the largest entry, as between the two paths elsewhere: both sum in FP64 in
different orders, amplified by the conditioning of the random basis (about 1e3)."""
import numpy as np
import pytest
import torch

from slope_stability_octave_b200 import _lib
from slope_stability_octave_b200.linear_solvers import DFGMRES
from test_gpu_krylov import elastic_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,drop", [(3, False), (4, False), (8, False), (9, True), (16, True), (24, False), (25, True),
                                    (32, False), (41, True), (48, True), (49, False)])
def test_tile_edges(cuda_device, k, drop):
    P, K, KQ, q = elastic_system()
    n = P.dmesh.n_dof
    W = np.zeros((k, n))
    W[:, q] = np.random.default_rng(60 + k).normal(size=(k, q.size))
    if drop:
        W[k // 2] = 0.25 * W[0] - W[k - 1]
    out = {}
    for mode in (1, 0):
        sol = DFGMRES(P.dmesh, 1e-8, 40, 1e-3)
        _lib.call("sg_krylov_set_aorth", sol._ws.handle, mode)
        sol.basis = torch.from_numpy(W).to(cuda_device)
        sol.A_orthogonalize(K)
        torch.cuda.synchronize()
        out[mode] = (sol.basis.clone(), sol.AW.clone())
    for got, ref in zip(out[1], out[0]):
        assert got.shape == ref.shape and got.shape[0] == k - int(drop)
        assert ((got - ref).abs().max() / ref.abs().max()).item() <= 1e-9
