"""Which meshes the factored element kernels take: every P2 tetrahedral mesh in the reference's
local numbering, whatever its rule, layers or origin (the generators' and the reference's HDF5
meshes), and no other."""
import os

import numpy as np
import pytest

from slope_stability_octave_b200 import fem, problems
from slope_stability_octave_b200.device import DeviceMesh
from test_gpu_response import problem

pytestmark = pytest.mark.gpu
GOLDEN_MESH = os.path.join(os.path.dirname(__file__), "golden", "mesh_ssr3d_stored_runs.npz")


@pytest.mark.parametrize("dim,nq,numbering,factored", [
    (3, 11, "reference", True), (3, 1, "reference", True), (3, 16, "reference", True), (3, 11, "swapped", False),
    (3, 4, "swapped", False), (2, 7, "reference", False)])
def test_numberings_and_rules(cuda_device, dim, nq, numbering, factored):
    mesh, dphi, w = problem(dim, 2, nq, numbering)
    assert DeviceMesh(mesh, dphi, w, nq).factored == factored


@pytest.mark.parametrize("case", ["slope", "layered", "box", "homo", "hetero"])
def test_meshes_in_use(cuda_device, case):
    if case == "box":
        mesh = fem.mesh_p2_box(3, 4, 2)
        xi, wf = fem.quadrature_p2_tet()
        hat, a, b, c = fem.local_basis_p2_tet(xi)
        *d, w = fem.geometry_3d(mesh, a, b, c, wf)
        assert DeviceMesh(mesh, tuple(d), w, 11).factored
        return
    if case in ("homo", "hetero"):
        g = np.load(GOLDEN_MESH)
        P = problems.slope_3d_from_mesh(g[f"{case}_coord"], g[f"{case}_elem"], g[f"{case}_Q"])
    else:
        make = problems.slope_3d_layered if case == "layered" else problems.slope_3d
        P = make(0.93, (15, 10, 15, 10, 10, 3.1))
    assert DeviceMesh(P.mesh, P.dphi, P.weight, P.n_q).factored
