"""The element blocks of P2 tetrahedra through each of their kernels: the factored kernel with 16-byte
and with 8-byte copies of DS, and, for a mesh in another local numbering, the bulk-staged kernel
(DS on a 16-byte boundary) and the plain-load kernel (DS 8 bytes off it).  The two of a mesh
perform the same operations: bitwise the same K_t, over a ragged last batch of eight elements, and no
bounded wait of the bulk copies gives up."""
import ctypes as C

import numpy as np
import pytest
import torch

from slope_stability_octave_b200 import _lib, fem
from slope_stability_octave_b200.device import DeviceMesh
from test_gpu_mesh_ops import build_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("numbering", ["reference", "swapped"])
def test_aligned_and_offset_tangents_agree(cuda_device, numbering):
    mesh, dphi, w, nq, _ = build_case("slope3d")
    if numbering == "swapped":                   # local nodes 4 and 5 change places
        order = [0, 1, 2, 3, 5, 4, 6, 7, 8, 9]
        mesh = fem.Mesh(mesh.coord, np.ascontiguousarray(mesh.elem[order]), mesh.Q)
        dphi = tuple(np.ascontiguousarray(x[:, order]) for x in dphi)
    assert mesh.n_e % 8 != 0
    dm = DeviceMesh(mesh, dphi, w, nq)
    assert dm.factored == (numbering == "reference")
    g = torch.Generator(device="cuda").manual_seed(17)
    DS = torch.randn(dm.n_int * 36, dtype=torch.float64, device="cuda", generator=g)
    off = torch.empty(DS.numel() + 1, dtype=torch.float64, device="cuda")[1:]
    off.copy_(DS)
    assert DS.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 8
    st = C.c_int32(-1)
    assert _lib.lib().sg_device_status(1, C.byref(st)) == 0        # cleared
    K = dm.new_block_values()
    K_off = torch.full_like(K, float("nan"))
    dm.assemble(DS, K)
    dm.assemble(off, K_off)
    torch.cuda.synchronize()
    assert torch.equal(K, K_off)
    assert _lib.lib().sg_device_status(0, C.byref(st)) == 0 and st.value == 0
