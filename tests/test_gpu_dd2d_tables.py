"""The 2D gathers through tables (single images; up to four images of the pixel
gathers) where tables can go wrong and the column walks of larger batches do
not."""
import math

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SCAN = {"parallel": 0, "flat": 1, "arc": 2}
IMAGE_IN = ("A", "BT", "BWT")
OPS = ("A", "BT", "BWT", "AT", "B", "BW")


def _opts(scan, W, H, Nu, du, sod=500.0, sdd=1000.0, shift=(0.4, -0.3, 0.2)):
    e = du if scan == "parallel" else du * sod / sdd if scan == "flat" else 2 * math.atan(du / (2 * sdd))
    return np.array([W, H, Nu, 1.0, 1.0, e, sod, sdd, shift[0], shift[1], shift[2] * e, SCAN[scan]], np.float32)


def _run(op, x, opts, ang, cuda):
    from xrecon_b200 import _native
    from xrecon_b200.backend import HostGeometry
    return _native.apply(2, op, torch.from_numpy(x).to(cuda), HostGeometry(2, opts.tolist()).struct,
                         torch.from_numpy(ang).to(cuda))


@pytest.mark.parametrize("V", [1, 4])
@pytest.mark.parametrize("scan,W,Nu,du", [("parallel", 256, 700, 0.4), ("flat", 256, 700, 0.8), ("arc", 256, 256, 2.0),
                                          ("arc", 256, 700, 0.8), ("arc", 400, 1500, 0.55), ("arc", 24, 600, 0.2)])
def test_every_edge_finds_its_column(cuda, scan, W, Nu, du, V):
    """Few views, so that a pixel edge assigned to the wrong column, or a chained boundary not clipped to its pixel,
    is not averaged away.  Bound: a handful of float32 roundings (4e-7), or half as much again as the walk's error
    where the detector's float32 angles leave more."""
    opts = _opts(scan, W, W - 7, Nu, du)
    if W == 24:
        opts[3:5] = 4.0 * opts[5] * 500.0  # four columns of 2e-4 rad a pixel
    rng = np.random.default_rng(V)
    ang = (np.arange(V) * (2 * np.pi / V) + 0.313).astype(np.float32)
    sino = rng.random((8, 1, V, Nu)).astype(np.float32)
    for op in ("AT", "B", "BW"):
        want = O.dd2d(op, sino, opts, ang)
        walked = rel_l2(_run(op, sino, opts, ang, cuda).cpu().numpy(), want)
        tabled = [rel_l2(_run(op, sino[i:i + 1], opts, ang, cuda).cpu().numpy(), want[i:i + 1]) for i in range(3)]
        assert max(tabled) < max(4e-7, 1.5 * walked), (op, tabled, walked)
