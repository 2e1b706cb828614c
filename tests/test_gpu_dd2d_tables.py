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


OUTLIERS = [1e20, float(np.finfo(np.float32).min), np.inf, np.nan]


def _untouched(op, x, at, opts, ang):
    """Oracle of x without the element `at` of every image, and the outputs that this element does not reach."""
    alone, rest = np.zeros_like(x), x.copy()
    alone[(slice(None), 0) + at] = 1.0
    rest[(slice(None), 0) + at] = 0.0
    return O.dd2d(op, rest, opts, ang), O.dd2d(op, alone, opts, ang) == 0


@pytest.mark.parametrize("B", [1, 4, 8])
@pytest.mark.parametrize("scan", ["parallel", "flat", "arc"])
@pytest.mark.parametrize("value", OUTLIERS)
def test_an_outlier_reaches_only_what_it_touches(cuda, scan, value, B):
    """One very large, infinite or NaN pixel or cell: outputs that do not overlap it are those of the rest (1e-5
    relative L2, the bound of every operator), and those that do carry it."""
    opts = _opts(scan, 40, 31, 60, 1.6)
    rng = np.random.default_rng(3)
    ang = (np.arange(9) * 0.71 + 0.05).astype(np.float32)
    img = rng.random((B, 1, 31, 40)).astype(np.float32)
    sino = rng.random((B, 1, 9, 60)).astype(np.float32)
    for op in OPS:
        x, at = (img, (11, 9)) if op in IMAGE_IN else (sino, (4, 22))
        want, free = _untouched(op, x, at, opts, ang)
        x = x.copy()
        x[(slice(None), 0) + at] = value
        got = _run(op, x, opts, ang, cuda).cpu().numpy()
        assert 0 < free.sum() < free.size
        assert rel_l2(got[free], want[free]) < 1e-5, op
        hit = np.abs(got[~free])
        assert (hit > 1e12).any() if np.isfinite(value) else not np.isfinite(hit).all(), op


@pytest.mark.parametrize("value", OUTLIERS)
def test_an_outlier_in_a_ragged_batch(cuda, value):
    """The same for the projections of a ragged batch; its filter spreads the value over every column of a view, so
    of the reconstructions only the other instance's is compared."""
    from xrecon_b200 import geometry as G
    from xrecon_b200.projector import Projector2d
    from xrecon_b200.ragged import RaggedFBP2d
    P = [Projector2d(G.Volume2d((n, n - 3), 1.0), G.FanBeam2d(G.Detector2d(m, 2.2), 500.0, 1000.0, "arc")).to(cuda)
         for n, m in ((40, 60), (33, 47))]
    ang = [torch.arange(V) * (2 * math.pi / V) + 0.05 for V in (9, 14)]
    rng = np.random.default_rng(4)
    img = [rng.random((1, 1, n - 3, n)).astype(np.float32) for n in (40, 33)]
    plan = RaggedFBP2d(P, ang)
    clean = [r.clone() for r in plan([torch.from_numpy(x).to(cuda) for x in img])[1]]
    opts = P[0].options.cpu().numpy()
    want, free = _untouched("A", img[0], (11, 9), opts, ang[0].numpy())
    img[0][0, 0, 11, 9] = value
    sino, recon = plan([torch.from_numpy(x).to(cuda) for x in img])
    got = sino[0].cpu().numpy()
    assert 0 < free.sum() < free.size
    assert rel_l2(got[free], want[free]) < 1e-5
    assert torch.equal(recon[1], clean[1])


@pytest.mark.parametrize("value", [1e20, np.inf])
def test_an_outlier_in_a_ragged_row(cuda, value):
    """Row tables of a ragged batch: with a filter of one tap the filtered row is the row itself, and a view that
    holds the value is walked."""
    from xrecon_b200 import geometry as G
    from xrecon_b200.projector import Projector2d
    from xrecon_b200.ragged import RaggedFBP2d
    P = Projector2d(G.Volume2d((40, 37), 1.0), G.FanBeam2d(G.Detector2d(60, 2.2), 500.0, 1000.0, "arc")).to(cuda)
    with torch.no_grad():
        taps = torch.zeros_like(P.filter).reshape(-1)
        taps[taps.numel() // 2] = 1.0
        P.filter.copy_(taps.reshape(P.filter.shape))
    ang = torch.arange(9) * 0.71 + 0.05
    plan = RaggedFBP2d([P], [ang], graph=False)
    img = torch.rand(37, 40, generator=torch.Generator().manual_seed(5)).to(cuda)
    plan([img])
    sino = plan.sino.clone().view(1, 1, 9, 60)
    opts, w = P.options.cpu().numpy(), P.weight.detach().cpu().numpy().reshape(-1)
    weighted = sino.cpu().numpy() * w
    want, free = _untouched("BW", weighted, (4, 22), opts, ang.numpy())
    plan.sino.view(9, 60)[4, 22] = value
    plan.launch(project=False)
    got = plan.reconstructions()[0].cpu().numpy()
    d = ang.diff().double()
    scale = float(((d + math.pi) % (2 * math.pi) - math.pi).abs().mean()) / 2
    assert 0 < free.sum() < free.size
    if np.isfinite(value):  # an infinity times the filter's zeros is NaN in every column of its view
        assert rel_l2(got[free], want[free] * scale) < 1e-5
    else:
        assert not np.isfinite(got[~free]).any()


# (W, H, view angle): lines behind the source's plane along the axis, on either axis, and a view with none
ELONGATED = [(40, 200, math.pi / 4 - 0.05), (200, 40, 3 * math.pi / 4 - 0.05), (200, 40, math.pi / 4 - 0.02)]


@pytest.mark.parametrize("scan", ["flat", "arc"])
@pytest.mark.parametrize("W,H,beta", ELONGATED)
def test_lines_behind_the_source_plane(cuda, scan, W, H, beta):
    """Elongated images close to the source: the columns reach the lines in front of the source's plane as the oracle
    has them (1e-5, the bound of every operator), whatever lies behind it.  On the arc detector the oracle's chained
    operators stop at the first column past 90 degrees; there the single image is held to the batch's walk."""
    sod, sdd, n = 110.0, 220.0, 200
    du = 4.4 if scan == "flat" else 2 * sdd * math.tan(2.7 / n / 2)
    opts = _opts(scan, W, H, n, du, sod, sdd, (0.0, 0.0, 0.0))
    ang = np.array([beta], np.float32)
    rng = np.random.default_rng(W)
    img, sino = rng.random((8, 1, H, W)).astype(np.float32), rng.random((8, 1, 1, n)).astype(np.float32)
    for op in OPS:
        x = img if op in IMAGE_IN else sino
        walked, single = _run(op, x, opts, ang, cuda).cpu().numpy(), _run(op, x[:1], opts, ang, cuda).cpu().numpy()
        assert np.count_nonzero(single) > 0
        assert rel_l2(single, walked[:1]) < 1e-5, op
        if scan == "flat" or op in ("A", "AT"):
            want = O.dd2d(op, x, opts, ang)
            assert rel_l2(walked, want) < 1e-5 and rel_l2(single, want[:1]) < 1e-5, op


def test_lines_behind_the_source_plane_in_a_ragged_batch(cuda):
    from xrecon_b200 import geometry as G
    from xrecon_b200.projector import Projector2d
    from xrecon_b200.ragged import RaggedFBP2d
    P = Projector2d(G.Volume2d((40, 200), 1.0), G.FanBeam2d(G.Detector2d(200, 4.4), 110.0, 220.0, "flat")).to(cuda)
    ang = torch.tensor([math.pi / 4 - 0.05, 3 * math.pi / 4 + 0.05])
    img = torch.rand(1, 1, 200, 40, generator=torch.Generator().manual_seed(6))
    sino, recon = RaggedFBP2d([P], [ang])([img.to(cuda)])
    assert rel_l2(sino[0].cpu().numpy(), O.dd2d("A", img.numpy(), P.options.cpu().numpy(), ang.numpy())) < 1e-5
    assert rel_l2(recon[0].cpu().numpy(), P.filtered_backprojection(sino[0], ang.to(cuda)).cpu().numpy()) < 1e-5


@pytest.mark.parametrize("du,n,x", [(2e-7, 600, 0.0), (5e-8, 600, 0.0), (3e-7, 2200000, 150.0)])
@pytest.mark.parametrize("B", [1, 8])
def test_columns_finer_than_the_guess(cuda, du, n, x, B):
    """Arc columns of less than the column guess's error in radians (2e-6 towards x = 150 mm), at view angles that
    float32 resolves: every column is found, whichever way the batch is gathered (1e-5, the bound of every
    operator).  Towards x = 150 mm only A^T: the angles' float32 unit there is a tenth of a column, and the chained
    operators' own roundings are 1.6e-4 whatever finds the column."""
    sod = 500.0
    opts = _opts("arc", 24, 20, n, du * 1000.0, sod, 1000.0, (x, 0.0, 0.0))
    opts[3:5] = 0.7 * 600 * du * sod / 24
    ang = np.array([0.01, -0.008], np.float32)
    sino = np.random.default_rng(7).random((B, 1, 2, n), dtype=np.float32)
    sino[0, 0, 1, n // 2] = np.inf if B == 1 else 1.0  # one image: a walked row among tabled ones
    for op in ("AT", "B", "BW") if x == 0.0 else ("AT",):
        want = O.dd2d(op, sino, opts, ang)
        ok = np.isfinite(want)
        got = _run(op, sino, opts, ang, cuda).cpu().numpy()
        assert rel_l2(got[ok], want[ok]) < 1e-5, op


def test_ragged_tables_are_capped(cuda):
    """An image whose line tables alone are past the cap of a batch's tables (1 GiB) is walked, beside one that has
    tables; both agree with the single-scan calls (two FP32 orders of summation: 1e-5)."""
    from xrecon_b200 import geometry as G
    from xrecon_b200.projector import Projector2d
    from xrecon_b200.ragged import RaggedFBP2d
    P = [Projector2d(G.Volume2d((n, n - 3), 300.0 / n), G.FanBeam2d(G.Detector2d(90, 8.0), 500.0, 1000.0, "arc")).to(cuda)
         for n in (8200, 64)]
    ang = [torch.arange(V) * (2 * math.pi / V) + 0.05 for V in (2, 9)]
    plan = RaggedFBP2d(P, ang, autotune=False, graph=False)
    assert plan.workspace.numel() < 1 << 30
    gen = torch.Generator(device=cuda).manual_seed(9)
    img = [torch.rand(1, 1, n - 3, n, generator=gen, device=cuda) for n in (8200, 64)]
    sino, recon = plan(img)
    for i in range(2):
        want = P[i].projection(img[i], ang[i].to(cuda))
        assert float((sino[i] - want).norm() / want.norm()) < 1e-5
        want = P[i].filtered_backprojection(sino[i], ang[i].to(cuda))
        assert float((recon[i] - want).norm() / want.norm()) < 1e-5


@pytest.mark.parametrize("op,B", [("A", 1), ("BT", 1), ("B", 1), ("AT", 3), ("A", 8), ("BW", 8)])
def test_without_memory_for_the_tables(cuda, monkeypatch, op, B):
    """Where the device has no room for the tables or the interleaved batch, the call goes without: the same to
    float32 rounding (1e-5 relative L2, two orders of summation)."""
    import ctypes

    from xrecon_b200 import _native
    from xrecon_b200.backend import HostGeometry
    opts = _opts("flat", 130, 121, 200, 1.8)
    geom = HostGeometry(2, opts.tolist()).struct
    ang = (np.arange(50) * 0.13).astype(np.float32)
    shape = (B, 1, 121, 130) if op in IMAGE_IN else (B, 1, 50, 200)
    x = np.random.default_rng(10).random(shape).astype(np.float32)
    want = _run(op, x, opts, ang, cuda)
    least = _native.lib().xr_dd2d_workspace_min(_native.OPS[op], ctypes.byref(geom), B, 50)
    room = _native._workspace

    def short(nbytes, device):
        if nbytes > least:
            raise torch.cuda.OutOfMemoryError("no room")
        return room(nbytes, device)
    monkeypatch.setattr(_native, "_workspace", short)
    got = _run(op, x, opts, ang, cuda)
    assert float((got - want).norm() / want.norm()) < 1e-5


def test_line_tables_take_the_place_of_the_transpose(cuda):
    """Host only: scratch of one large image's projection, view tables and line tables but no transpose."""
    import ctypes

    from xrecon_b200 import _native
    from xrecon_b200.backend import HostGeometry
    geom = HostGeometry(2, _opts("flat", 4096, 4096, 64, 90.0, 3000.0, 6000.0).tolist()).struct
    lines = 2 * 4096 * 4098 * 16
    size = _native.lib().xr_dd2d_workspace_size(_native.OPS["A"], ctypes.byref(geom), 1, 1)
    assert size < lines + (1 << 20)
