"""The products A S of the A-orthogonalisation, from four columns on, carry the rounding error of a
lane's sum over its blocks on meshes of up to 750,000 unknowns.

One row of the matrix gets multiples v of the identity, 2^53 and -2^53 first and last among every
fourth block and ones between them: a plain FP64 sum of such a run loses every one, a sum that
carries its error none, and what the four runs add up to is a small whole number.  (A run's first
and last two blocks are added in pairs first; the partners of the large entries are zero.)  Each
column has a unit of its own elsewhere, so that the basis is A-orthonormal as it stands and the
returned A W is A S itself: equality is exact."""
import numpy as np
import pytest
import torch

from slope_stability_octave_b200.linear_solvers import DFGMRES
from test_gpu_krylov import elastic_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [4, 8, 9, 16, 17, 21])
def test_row_sums_carry_their_error(cuda_device, k):
    P, _, _, _ = elastic_system()
    mesh, nn = P.mesh, P.mesh.n_n
    elem = mesh.elem.T.astype(np.int64)
    pairs = np.unique((elem[:, :, None] * nn + elem[:, None, :]).ravel())     # blocks by row, then column
    row, col = pairs // nn, pairs % nn
    start = np.searchsorted(row, np.arange(nn + 1))
    node = int(np.argmax(np.diff(start)))
    p0, p1 = start[node], start[node + 1]
    near = set(col[p0:p1])
    run = np.arange(p0, p1, 4)                                                # the first lane group's blocks
    run = run[: 2 * (run.size // 2)]                                          # whole pairs
    assert run.size >= 8
    v = np.ones(p1 - p0)
    v[run - p0] = np.where(np.arange(run.size) % (run.size - 1) == 0, 0.0, 1.0)
    v[run[[1, -2]] - p0] = 0.0
    v[run[0] - p0], v[run[-1] - p0] = 2.0 ** 53, -(2.0 ** 53)
    K = np.zeros((pairs.size, 9))
    K[p0:p1, [0, 4, 8]] = v[:, None]
    S = np.zeros((k, nn, 3))
    scale = 2.0 ** (np.arange(k) % 5)
    if node in col[run[[0, -1]]]:                                             # the row's own block is not one of the two
        pytest.skip("the row starts or ends with its own block")
    others = np.array([j for j in sorted(near) if j != node])
    S[:, others, 0] = scale[:, None]
    far = [j for j in range(nn) if j not in near][: 1 + 2 * k : 2][:k]
    for i, j in enumerate(far):
        S[i, j, 1] = 1.0
        K[np.searchsorted(pairs, j * nn + j), 4] = 1.0                        # that unit's own diagonal entry
    sol = DFGMRES(P.dmesh, 1e-8, 40, 1e-3)
    sol.basis = torch.from_numpy(S.reshape(k, -1)).to(cuda_device)
    Kd = torch.from_numpy(K.ravel()).to(cuda_device)
    assert Kd.numel() == P.dmesh.n_blocks * 9
    sol.A_orthogonalize(Kd)
    assert sol.k == k
    expect = np.zeros_like(S)
    expect[:, node, 0] = scale * np.count_nonzero((v == 1.0) & (col[p0:p1] != node))     # the large two cancel
    for i, j in enumerate(far):
        expect[i, j, 1] = 1.0
    assert np.array_equal(sol.AW.cpu().numpy().reshape(S.shape), expect)
