"""The Davis reduction at reduction factors far below one, where tan(phi) / lambda exceeds the square
root of the largest double: the limits of its formulas for psi = 0, t = tan(phi),
    A       sin -> 1,          c -> 2 c0 / t
    B, C    sin -> 1/sqrt(2),  c -> sqrt(2) c0 / t
A dozen roundings: 1e-14 relative."""
import numpy as np
import pytest
import torch

from slope_stability_octave_b200 import _lib
from slope_stability_octave_b200.device import cur_stream, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("davis", ["A", "B", "C"])
@pytest.mark.parametrize("lam", [1e-100, 1e-150, 1e-160, 1e-250, 1e-305])
def test_limits_of_the_reduction(cuda_device, davis, lam):
    phi = torch.tensor([0.1, 0.5, 1.2], dtype=torch.float64, device=cuda_device)
    c0 = torch.tensor([6.0, 15.0, 1.0], dtype=torch.float64, device=cuda_device)
    psi, c, s = torch.zeros_like(phi), torch.empty_like(phi), torch.empty_like(phi)
    _lib.call("sg_reduction_dev", ptr(c0), ptr(phi), ptr(psi), lam, davis.encode(), 3, ptr(c), ptr(s), cur_stream())
    sine, factor = (1.0, 2.0) if davis == "A" else (np.sqrt(0.5), np.sqrt(2.0))
    assert (s.cpu().numpy() == pytest.approx(sine, rel=1e-14))
    assert (c.cpu().numpy() == pytest.approx(factor * (c0 / torch.tan(phi)).cpu().numpy(), rel=1e-14))
