"""The 2D gathers' launch shapes against the FP64 oracle: batch sizes on both
sides of every interleaving width and of the row tables' limit, images that do
not fill their tiles, detectors of a few cells, columns wider and narrower than
a pixel; rows holding non-finite values; and a scratch too small for the tables.

Tolerance: 1e-5 relative L2, the bound of every operator against the oracle."""
import ctypes
import math

import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SCAN = {"parallel": 0, "flat": 1, "arc": 2}


def _opts(scan, W, H, Nu, du):
    du_eff = du if scan == "parallel" else du * 0.5 if scan == "flat" else 2 * math.atan(du / 2000.0)
    return np.array([W, H, Nu, 1.0, 1.1, du_eff, 500.0, 1000.0, 0.4, -0.3, 0.2 * du_eff, SCAN[scan]], np.float32)


def _run(op, x, opts, ang, cuda):
    from xrecon_b200 import _native
    from xrecon_b200.backend import HostGeometry
    return _native.apply(2, op, torch.from_numpy(x).to(cuda), HostGeometry(2, opts.tolist()).struct,
                         torch.from_numpy(ang).to(cuda))


CASES = [(1, 33, 17, 41, 1.6, 9), (2, 16, 16, 16, 3.0, 16), (3, 5, 61, 1, 160.0, 7), (4, 70, 35, 3, 60.0, 33),
         (5, 31, 32, 65, 1.0, 8), (9, 17, 9, 256, 0.15, 12), (1, 1, 1, 2, 2.0, 1), (1, 130, 129, 300, 1.0, 140)]


@pytest.mark.parametrize("scan", ["parallel", "flat", "arc"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "b%d_%dx%d_nu%d" % c[:4])
def test_2d_launch_shapes_match_the_oracle(cuda, scan, case):
    B, W, H, Nu, du, V = case
    opts = _opts(scan, W, H, Nu, du)
    rng = np.random.default_rng(B + W)
    ang = (np.arange(V) * (2 * np.pi / V) + 0.013).astype(np.float32)
    img = rng.random((B, 1, H, W)).astype(np.float32)
    sino = rng.random((B, 1, V, Nu)).astype(np.float32)
    for op in ("A", "AT", "B", "BW", "BT", "BWT"):
        # The arc transposes follow float32 boundary angles (a quantum of 4.8e-7 rad) without averaging them: on
        # columns of 1.5e-4 rad that is no longer within 1e-5 of the oracle's own order of roundings, on any path.
        if scan == "arc" and op in ("BT", "BWT") and opts[5] < 5e-4:
            continue
        x = img if op in ("A", "BT", "BWT") else sino
        assert rel_l2(_run(op, x, opts, ang, cuda).cpu().numpy(), O.dd2d(op, x, opts, ang)) < 1e-5, op


@pytest.mark.parametrize("scan", ["parallel", "flat", "arc"])
def test_non_finite_rows_reach_only_their_pixels(cuda, scan):
    opts = _opts(scan, 40, 24, 50, 2.0)
    ang = (np.arange(11) * 0.57).astype(np.float32)
    sino = np.random.default_rng(2).random((8, 1, 11, 50)).astype(np.float32)
    sino[:, 0, 3, 20], sino[:, 0, 7, 49], sino[:, 0, 9, 0] = np.nan, np.inf, -np.inf
    for op in ("AT", "B", "BW"):
        walked = _run(op, sino, opts, ang, cuda)     # eight images: columns walked
        tabled = _run(op, sino[:1], opts, ang, cuda)  # one image: row tables
        assert torch.equal(torch.isfinite(walked[:1]), torch.isfinite(tabled)), op
        ok = torch.isfinite(tabled)
        assert 0 < int(ok.sum()) < tabled.numel()
        assert rel_l2(tabled[ok].cpu().numpy(), walked[:1][ok].cpu().numpy()) < 1e-5, op


def test_scratch_without_room_for_the_tables(cuda):
    from xrecon_b200 import _native
    L = _native.lib()
    geom = _native.Geom2d(W=64, H=48, Nu=160, type=1, dx=1.0, dy=1.0, du=1.1, sod=500.0, sdd=900.0,
                          shift_x=0.0, shift_y=0.0, shift_u=0.0)
    V = 4000
    ang = torch.linspace(0, 2 * math.pi, V + 1)[:-1].to(cuda)
    sino = torch.rand(1, 1, V, 160, generator=torch.Generator().manual_seed(3)).to(cuda)
    assert L.xr_dd2d_workspace_size(_native.OPS["B"], ctypes.byref(geom), 1, V) > 32 << 20
    want = _native.apply(2, "B", sino, geom, ang)
    out = torch.empty_like(want)
    rc = L.xr_dd2d_noalloc(_native.OPS["B"], ctypes.byref(geom), sino.data_ptr(), 0, out.data_ptr(), 0,
                           ang.data_ptr(), 1, V, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, L.xr_last_error().decode()
    assert rel_l2(out.cpu().numpy(), want.cpu().numpy()) < 1e-5
