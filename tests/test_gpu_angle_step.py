"""The FBP's last factor, the mean wrapped angular step, applied in place."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 4097])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("angles", ["one", "two", "wraps", "backwards", "many"])
def test_angle_step_scale(cuda, n, offset, angles):
    """Lengths around the four-element loads, a buffer that does not start on one, scans that pass 2 pi or run
    backwards, and the zero of a single view.  Tolerance 1e-6: the same float32 steps, summed in another order."""
    from xrecon_b200 import _native
    from xrecon_b200.projector import mean_angle_step
    ang = {"one": torch.tensor([0.3]), "two": torch.tensor([0.1, 0.4]),
           "wraps": torch.remainder(torch.arange(50) * 0.37 + 6.0, 2 * math.pi),
           "backwards": 1.0 - torch.arange(50) * 0.02, "many": torch.arange(3000) * (2 * math.pi / 3000)}[angles].to(cuda)
    x = torch.rand(n + offset, generator=torch.Generator().manual_seed(n)).to(cuda)
    want = x.clone()
    want[offset:] = x[offset:] * (0.5 * mean_angle_step(ang))
    got = _native.angle_step_scale_(x[offset:], ang, 0.5)
    assert got.data_ptr() == x[offset:].data_ptr()
    assert torch.allclose(x, want, rtol=1e-6, atol=0.0)
