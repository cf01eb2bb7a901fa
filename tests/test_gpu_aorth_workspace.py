"""The A-orthogonalisation works in the memory its workspace was made with: the first call on a
new workspace allocates nothing on the device for bases of up to 64 columns (the workspace's
column capacity), whichever of its products the number of columns takes."""
import numpy as np
import pytest
import torch

from slope_stability_octave_b200 import _lib
from slope_stability_octave_b200.linear_solvers import DFGMRES
from test_gpu_krylov import elastic_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3, 4, 16, 25, 48, 49, 64])
def test_first_call_allocates_nothing(cuda_device, k):
    P, K, KQ, q = elastic_system()
    W = np.zeros((k, P.dmesh.n_dof))
    W[:, q] = np.random.default_rng(70 + k).normal(size=(k, q.size))
    sol = DFGMRES(P.dmesh, 1e-8, 40, 1e-3)
    sol.basis = torch.from_numpy(W).to(cuda_device)
    count = _lib.lib().sg_device_alloc_count
    before = count(0)
    sol.A_orthogonalize(K)
    assert count(0) == before
    assert sol.k == k
