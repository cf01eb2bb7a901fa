"""sg_residual_dev, the stress-only residual at a strength that is already reduced, called itself (the
Python layer goes through sg_element_response_dev): against the chain of separate kernels at the
same strength, with and without branch ids, on a factored and on an unfactored mesh.  F within
1e-11 of its largest entry and branch ids equal, as for the response; its inputs stay as they
were.  In 2D and beyond sixteen points it is refused."""
import numpy as np
import pytest
import torch

from slope_stability_octave_b200 import _lib, fem
from slope_stability_octave_b200.constitutive import CONSTITUTIVE
from slope_stability_octave_b200.device import DeviceMesh
from test_gpu_response import problem

pytestmark = pytest.mark.gpu


def setup(dim, cells, nq, numbering):
    mesh, dphi, w = problem(dim, cells, nq, numbering)
    mat = fem.materials(np.zeros(mesh.n_e, int), nq, [[6, 45, 0, 40000, 0.3, 20, 20]])
    dm = DeviceMesh(mesh, dphi, w, nq)
    cons = CONSTITUTIVE(dm, mat["c0"], mat["phi"], mat["psi"], "B", mat["shear"], mat["bulk"], mat["lame"])
    U = np.random.default_rng(5).normal(size=(dim, mesh.n_n)) * 3e-3 * mesh.Q
    return dm, cons, torch.from_numpy(np.ascontiguousarray(U.T).ravel()).cuda()


@pytest.mark.parametrize("cells,nq,numbering", [(1, 11, "reference"), (3, 11, "reference"), (2, 11, "swapped"),
                                                (2, 16, "reference"), (1, 1, "swapped")])
def test_against_the_separate_kernels(cuda_device, cells, nq, numbering):
    dm, cons, U = setup(3, cells, nq, numbering)
    cons.reduction(1.4)
    cons.constitutive_problem_stress(U)
    ref, branch = cons.build_F().clone(), cons.branch.clone()
    c_bar, sin_phi = cons.c_bar.clone(), cons.sin_phi.clone()
    for got_branch in (torch.full_like(branch, 99), None):
        F = torch.full_like(ref, float("nan"))
        dm.residual(U, cons.c_bar, cons.sin_phi, cons.shear, cons.lame, got_branch, F)
        assert (F - ref).abs().max() <= 1e-11 * ref.abs().max()
        assert got_branch is None or torch.equal(got_branch, branch)
    assert torch.equal(cons.c_bar, c_bar) and torch.equal(cons.sin_phi, sin_phi)


@pytest.mark.parametrize("dim,nq", [(2, 7), (3, 17)])
def test_refused(cuda_device, dim, nq):
    dm, cons, U = setup(dim, 1, nq, "reference")
    with pytest.raises(_lib.SlopeGPUError):
        dm.residual(U, cons.c_bar, cons.sin_phi, cons.shear, cons.lame, None, torch.empty_like(U))
