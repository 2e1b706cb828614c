"""The staged projection's launch shapes (rows per thread, warps per CTA, pixels
per pass) against the FP64 oracle: detector heights on both sides of every
shape, columns of under one and over two pixels, and a few lines with rows of
more than a voxel, which leave the fine walk.

Tolerance: 1e-5 relative L2, the bound of every operator against the oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nv", [1, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 160])
@pytest.mark.parametrize("du,dv", [(1.3, 1.0), (4.4, 1.0), (1.3, 1.52)])
def test_projection_launch_shapes_match_the_oracle(cuda, Nv, du, dv):
    from xrecon_b200 import _native
    from xrecon_b200 import geometry as G
    from xrecon_b200.backend import HostGeometry
    D = max(4, int(Nv * 0.45))
    geo = G.ConeBeam3d(G.Detector3d((45, Nv), (du, dv), (0.3, 0.2)), 200.0, 400.0, "flat")
    opts = np.array(G.pack_options3d(G.Volume3d((26, 23, D), 1.0, (0.4, -0.2, 0.3)), geo), np.float32)
    geom = HostGeometry(3, opts.tolist()).struct
    plan = _native.cell_plan(geom)
    assert plan["ok"] and plan["fine"]
    ang = np.array([0.03, 0.7, np.pi / 4, 2.2, 3.9, 5.6], np.float32)
    img = np.random.default_rng(Nv).random((1, 2, D, 23, 26)).astype(np.float32)
    for op in ("A", "BT", "BWT"):
        got = _native.apply(3, op, torch.from_numpy(img).to(cuda), geom, torch.from_numpy(ang).to(cuda))
        assert rel_l2(got.cpu().numpy(), O.dd3d(op, img, opts, ang)) < 1e-5, op


@pytest.mark.parametrize("scan,W,D,Nu,Nv,du,dv,dz", [("parallel", 64, 40, 96, 50, 1.7, 1.7, 1.0),
                                                     ("parallel", 64, 40, 200, 50, 0.8, 1.2, 1.0),
                                                     ("flat", 48, 60, 64, 96, 2.0, 1.1, 0.7),
                                                     ("flat", 64, 40, 96, 50, 1.7, 1.7, 1.0)])
def test_rows_of_a_thread_keep_their_precision(cuda, scan, W, D, Nu, Nv, du, dv, dz):
    """Longer runs of rows a thread must not cost precision: with eight rows a thread the projection was within
    2.6e-7 of the oracle on these scans; a quarter to spare."""
    from xrecon_b200 import _native
    from xrecon_b200 import geometry as G
    from xrecon_b200.backend import HostGeometry
    det = G.Detector3d((Nu, Nv), (du, dv), (0.3, 0.2))
    geo = G.ParallelBeam3d(det) if scan == "parallel" else G.ConeBeam3d(det, 200.0, 400.0, scan)
    opts = np.array(G.pack_options3d(G.Volume3d((W, W - 3, D), (1.0, 1.0, dz), (0.4, -0.2, 0.3)), geo), np.float32)
    ang = (np.arange(5) * (2 * np.pi / 5) + 0.21).astype(np.float32)
    img = np.random.default_rng(3).random((1, 1, D, W - 3, W)).astype(np.float32)
    got = _native.apply(3, "A", torch.from_numpy(img).to(cuda), HostGeometry(3, opts.tolist()).struct,
                        torch.from_numpy(ang).to(cuda))
    assert rel_l2(got.cpu().numpy(), O.dd3d("A", img, opts, ang)) < 3.2e-7


@pytest.mark.parametrize("Nv,V", [(24, 640), (64, 640), (128, 256), (160, 256)])
@pytest.mark.parametrize("du,dv", [(1.3, 1.0), (4.4, 1.0), (1.3, 3.0)])
def test_projection_shapes_of_large_grids_match_the_oracle(cuda, Nv, V, du, dv):
    """As above with the views repeated until the grid takes the shapes of large scans (16 and 32 rows a thread; rows
    of a voxel and a half, for which that is 16), and every repeat the same bits."""
    from xrecon_b200 import _native
    from xrecon_b200 import geometry as G
    from xrecon_b200.backend import HostGeometry
    D = max(4, int(Nv * 0.45 * dv))
    geo = G.ConeBeam3d(G.Detector3d((45, Nv), (du, dv), (0.3, 0.2)), 200.0, 400.0, "flat")
    opts = np.array(G.pack_options3d(G.Volume3d((26, 23, D), 1.0, (0.4, -0.2, 0.3)), geo), np.float32)
    geom = HostGeometry(3, opts.tolist()).struct
    assert _native.cell_launch_plan(geom, 1, V)["rows_per_thread"] == (16 if dv > 1.0 or Nv == 24 else 32)
    ang = np.array([0.03, 0.7, np.pi / 4, 2.2, 3.9, 5.6, 4.4, 1.2], np.float32)
    img = np.random.default_rng(Nv).random((1, 1, D, 23, 26)).astype(np.float32)
    for op in ("A", "BT", "BWT"):
        got = _native.apply(3, op, torch.from_numpy(img).to(cuda), geom, torch.from_numpy(np.tile(ang, V // 8)).to(cuda))
        first = got[:, :, :8]
        assert rel_l2(first.cpu().numpy(), O.dd3d(op, img, opts, ang)) < 1e-5, op
        assert torch.equal(got.reshape(1, 1, V // 8, 8, Nv, 45), first[:, :, None].expand(1, 1, V // 8, 8, Nv, 45)), op
