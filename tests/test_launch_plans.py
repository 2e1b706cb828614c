"""Host-only plan queries: what the 3D kernels are launched with, and that the GPU
tests of launch shapes and view splits reach every one of them."""
import numpy as np
import pytest

from conftest import load_golden
from xrecon_b200 import _native
from xrecon_b200 import geometry as G
from xrecon_b200.backend import HostGeometry


def _struct(opts):
    return HostGeometry(3, np.asarray(opts).tolist()).struct


def _shape_case(Nv, du, dv):
    """The geometry of test_gpu_cell_shapes.py."""
    D = max(4, int(Nv * 0.45))
    geo = G.ConeBeam3d(G.Detector3d((45, Nv), (du, dv), (0.3, 0.2)), 200.0, 400.0, "flat")
    return _struct(np.array(G.pack_options3d(G.Volume3d((26, 23, D), 1.0, (0.4, -0.2, 0.3)), geo), np.float32))


# many views; rows a thread, warps: the least warps x (rows + 9) over the detector's CTAs of at most 128 rows
@pytest.mark.parametrize("Nv,rows,warps", [(1, 8, 1), (8, 8, 1), (9, 8, 2), (16, 8, 2), (17, 16, 2), (32, 16, 2),
                                           (33, 16, 3), (64, 32, 2), (65, 32, 3), (128, 32, 4), (129, 32, 3),
                                           (160, 32, 3)])
@pytest.mark.parametrize("du,dv,pixels", [(1.3, 1.0, 2), (4.4, 1.0, 3), (1.3, 1.52, 2)])
def test_projection_launch_shape(Nv, rows, warps, du, dv, pixels):
    plan = _native.cell_launch_plan(_shape_case(Nv, du, dv), 4, 2000)
    assert plan == dict(rows_per_thread=rows, warps=warps, pixels=pixels)


# few views: a grid under 148 x 16 warps takes the fewest rows that eight warps hold; then the least of rounds x (rows + 9)
@pytest.mark.parametrize("Nv,V,rows,warps", [(24, 6, 8, 3), (64, 6, 8, 8), (65, 6, 16, 5), (128, 6, 16, 8), (160, 6, 16, 5),
                                             (64, 640, 32, 2), (128, 256, 32, 4), (160, 256, 32, 3)])
def test_projection_launch_shape_of_small_grids(Nv, V, rows, warps):
    plan = _native.cell_launch_plan(_shape_case(Nv, 1.3, 1.0), 1, V)
    assert plan == dict(rows_per_thread=rows, warps=warps, pixels=2)
    assert _native.cell_launch_plan(_shape_case(Nv, 1.3, 1.0), 4, 2000)["rows_per_thread"] in (16, 32)  # and back


def test_projection_keeps_the_default_shape_for_coarse_rows():
    geo = G.ConeBeam3d(G.Detector3d((45, 160), (1.3, 4.0)), 200.0, 400.0, "flat")
    g = _struct(np.array(G.pack_options3d(G.Volume3d((26, 23, 70), 1.0), geo), np.float32))
    assert not _native.cell_plan(g)["fine"]
    assert _native.cell_launch_plan(g, 1, 2000) == dict(rows_per_thread=16, warps=5, pixels=2)
    short = _struct(np.array(G.pack_options3d(G.Volume3d((26, 23, 9), 1.0), G.ConeBeam3d(
        G.Detector3d((45, 20), (1.3, 4.0)), 200.0, 400.0, "flat")), np.float32))
    assert not _native.cell_plan(short)["fine"]
    assert _native.cell_launch_plan(short, 1, 20)["rows_per_thread"] == 8
    assert _native.cell_launch_plan(short, 1, 2000)["rows_per_thread"] == 16


@pytest.mark.parametrize("scan", ["flat", "arc", "parallel"])
@pytest.mark.parametrize("Nu", [1, 33, 64, 95])
@pytest.mark.parametrize("V,split", [(17, 1), (33, 2), (70, 4), (129, 8)])
def test_backprojection_split(scan, Nu, V, split):
    """The geometries of test_gpu_pfx_split.py: few tiles, so views are split as far as 16 a CTA allow; odd counts too."""
    from test_gpu_pfx_split import _opts
    plan = _native.pfx_launch_plan(_struct(_opts(scan, Nu)), 2, V)
    assert plan == dict(staged=True, split=split)


def test_backprojection_split_depends_on_the_grid():
    big = _native.geom3d_from_values(load_golden("options")["c5_3d_flat"])
    assert _native.pfx_launch_plan(big, 1, 1440) == dict(staged=True, split=1)
    small = _struct(np.array(G.pack_options3d(
        G.Volume3d((256, 256, 64), 1.0), G.ConeBeam3d(G.Detector3d((384, 96), 1.5), 500.0, 1000.0, "flat")), np.float32))
    assert _native.pfx_launch_plan(small, 1, 720)["split"] > 1

