"""GPU parity of the fused element response (reduction, strain, return mapping, internal force
in one kernel) against the oracle, at the places where its tiles and dispatch turn: element
counts that do not fill a CTA's pass, rules of 1 to 16 points, meshes whose gradients factor
into barycentric directions and meshes whose local numbering keeps them from it, the three
Davis types, with and without the tangent.

Tolerances, from the rounding of each quantity: the strain sums thirty products whose terms are
some 10 times their sum (1e-14), stress and force inherit it with the force's cancellation over
the elements of a node: 1e-11 of the largest entry, as for the chain of separate kernels.  The
tangent is compared at the kernel's own strain; it divides by differences of principal strains,
of which random strains have a few at 1e-4 of their size: 1e-10 of the largest entry."""
import numpy as np
import pytest
import torch

from oracle import native
from oracle.octave_ref import OctavePattern
from slope_stability_octave_b200 import fem
from slope_stability_octave_b200.constitutive import CONSTITUTIVE
from slope_stability_octave_b200.device import DeviceMesh

pytestmark = pytest.mark.gpu


def problem(dim, cells, nq, numbering):
    if dim == 3:
        mesh = fem.mesh_p2_3d(1, 2, 1, 2, 1, 1, cells)
        xi, wf = fem.quadrature_p2_tet()
    else:
        mesh = fem.mesh_p2_2d(1.0, 2, 1, 2, 1, cells)
        xi, wf = fem.quadrature_p2_tri()
    pick = np.arange(nq) % xi.shape[1]          # the rule cut short, or with points repeated
    xi, wf = np.ascontiguousarray(xi[:, pick]), np.ascontiguousarray(np.abs(wf[pick]))
    if dim == 3:
        hat, a, b, c = fem.local_basis_p2_tet(xi)
        *d, w = fem.geometry_3d(mesh, a, b, c, wf)
    else:
        hat, a, b = fem.local_basis_p2_tri(xi)
        *d, w = fem.geometry_2d(mesh, a, b, wf)
    if numbering == "swapped":                   # local nodes 4 and 5 change places
        order = np.arange(mesh.elem.shape[0])
        order[[4, 5]] = order[[5, 4]]
        mesh = fem.Mesh(mesh.coord, np.ascontiguousarray(mesh.elem[order]), mesh.Q)
        d = [np.ascontiguousarray(x[:, order]) for x in d]
    return mesh, tuple(d), w


@pytest.mark.parametrize("dim,cells,nq,numbering,davis", [
    (3, 1, 11, "reference", "B"), (3, 3, 11, "reference", "A"), (3, 2, 11, "swapped", "B"), (3, 1, 1, "reference", "C"),
    (3, 2, 7, "reference", "B"), (3, 2, 14, "reference", "A"), (3, 1, 16, "swapped", "C"), (2, 1, 7, "reference", "B"),
    (2, 2, 1, "reference", "A"), (2, 3, 16, "swapped", "C")])
def test_response_matches_oracle(cuda_device, dim, cells, nq, numbering, davis):
    mesh, dphi, w = problem(dim, cells, nq, numbering)
    rng = np.random.default_rng(100 * dim + 10 * cells + nq)
    mat = fem.materials(rng.integers(0, 2, mesh.n_e), nq, [[6, 30, 5, 40000, 0.3, 20, 20], [12, 40, 0, 20000, 0.25, 19, 19]])
    dm = DeviceMesh(mesh, dphi, w, nq)
    assert dm.fused_response
    cons = CONSTITUTIVE(dm, mat["c0"], mat["phi"], mat["psi"], davis, mat["shear"], mat["bulk"], mat["lame"])
    U = rng.normal(size=(dim, mesh.n_n)) * 2e-3 * mesh.Q
    Ud = torch.from_numpy(np.ascontiguousarray(U.T).ravel()).to(cuda_device)
    pat = OctavePattern(dim, mesh.elem, mesh.n_n, dphi, w, mesh.Q, mat["shear"], mat["bulk"])
    cb, sp = native.reduction(mat["c0"], mat["phi"], mat["psi"], 1.3, davis)
    S, _, br = native.constitutive(dim, pat.strain(U), cb, sp, mat["shear"], mat["bulk"], mat["lame"], want_ds=False)
    F_ref = pat.force(S).T.ravel()
    for F in (cons.build_F_all(1.3, Ud), cons.build_F_reduced(Ud), cons.build_F_and_DS_all(1.3, Ud),
              cons.build_F_and_DS_reduced(Ud)):
        assert np.abs(F.cpu().numpy() - F_ref).max() <= 1e-11 * np.abs(F_ref).max()
        assert np.mean(cons.branch.cpu().numpy() == br) > 0.999
    for got, ref in ((cons.c_bar, cb), (cons.sin_phi, sp), (cons.S, S)):
        assert np.abs(got.cpu().numpy().ravel() - np.ravel(ref)).max() <= 1e-11 * np.abs(ref).max()
    E = cons.E.cpu().numpy().reshape(mesh.n_e * nq, -1)
    assert np.abs(E - pat.strain(U)).max() <= 1e-12 * np.abs(E).max()
    _, DS, br = native.constitutive(dim, E, cons.c_bar.cpu().numpy(), cons.sin_phi.cpu().numpy(), mat["shear"],
                                    mat["bulk"], mat["lame"])
    same = cons.branch.cpu().numpy() == br
    D = cons.DS.cpu().numpy().reshape(DS.shape)
    assert np.abs(D - DS)[same].max() <= 1e-10 * np.abs(DS).max()


def test_response_nan_and_infinite_displacement(cuda_device):
    """What is not finite stays visible: no point with such a strain is taken for elastic."""
    mesh, dphi, w = problem(3, 1, 11, "reference")
    mat = fem.materials(np.zeros(mesh.n_e, int), 11, [[6, 30, 0, 40000, 0.3, 20, 20]])
    dm = DeviceMesh(mesh, dphi, w, 11)
    cons = CONSTITUTIVE(dm, mat["c0"], mat["phi"], mat["psi"], "B", mat["shear"], mat["bulk"], mat["lame"])
    for bad in (float("nan"), float("inf")):
        U = torch.zeros(dm.n_dof, dtype=torch.float64, device=cuda_device)
        U[3 * int(mesh.elem[0, 0])] = bad
        cons.build_F_all(1.0, U)
        touched = cons.branch.view(mesh.n_e, 11)[0]
        assert (touched != 0).any()


@pytest.mark.parametrize("cells,nq,numbering", [(1, 11, "reference"), (3, 11, "reference"), (2, 11, "swapped"),
                                                (1, 1, "reference"), (2, 14, "reference")])
def test_assembly_over_rules_and_numberings(cuda_device, cells, nq, numbering):
    """K_t of tangents with all 36 entries free (sym(D) counts) against the element sums in
    plain FP64, where the moments of the rule carry the blocks (11 points, factored gradients) and
    where the direct sum does; a block adds up to some 24 x nq terms of alternating sign,
    1e-12 of the largest entry as in the other assembly tests."""
    mesh, dphi, w = problem(3, cells, nq, numbering)
    dm = DeviceMesh(mesh, dphi, w, nq)
    n_e, n_n = mesh.n_e, mesh.n_n
    g = torch.Generator(device="cuda").manual_seed(cells * 100 + nq)
    DS = torch.randn((n_e * nq, 6, 6), dtype=torch.float64, device="cuda", generator=g) * 1e4
    K = dm.new_block_values()
    dm.assemble(DS, K)
    d = [torch.from_numpy(x).cuda().view(n_e, nq, 10) for x in dphi]
    B = torch.zeros((n_e, nq, 6, 10, 3), dtype=torch.float64, device="cuda")
    for c in range(3):
        B[:, :, c, :, c] = d[c]
    for row, (i, j) in ((3, (0, 1)), (4, (1, 2)), (5, (0, 2))):
        B[:, :, row, :, i], B[:, :, row, :, j] = d[j], d[i]
    B = B.reshape(n_e, nq, 6, 30)
    D = 0.5 * (DS + DS.transpose(1, 2)).view(n_e, nq, 6, 6)
    Ke = torch.einsum("eq,eqsl,eqst,eqtm->elm", torch.from_numpy(w).cuda().view(n_e, nq), B, D, B)
    elem = torch.from_numpy(mesh.elem.T.astype(np.int64)).cuda()
    a, b = torch.broadcast_tensors(elem[:, :, None], elem[:, None, :])
    _, slot = torch.unique((a * n_n + b).reshape(-1), return_inverse=True)
    ref = torch.zeros((dm.n_blocks, 9), dtype=torch.float64, device="cuda")
    ref.index_add_(0, slot, Ke.view(n_e, 10, 3, 10, 3).transpose(2, 3).reshape(-1, 9))
    assert (K.view(-1, 9) - ref).abs().max() <= 1e-12 * ref.abs().max()
