"""The staged backprojection with its views split over a cluster and with odd
column counts: against the FP64 oracle (1e-5 relative L2, the bound of every
operator) and, bit for bit, against the unstaged gather; a wait that runs out in a
cluster's CTAs is reported and leaves the next call correct."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from oracle import oracle as O
from test_gpu_pfx_stage import HOOK_PFX_NOSTAGE, HOOK_PFX_UNFIT, HOOK_TMA_STALL, _run, native  # noqa: F401

pytestmark = pytest.mark.gpu


def _opts(scan, Nu):
    from xrecon_b200 import geometry as G
    det = G.Detector3d((Nu, 21), (90.0 / Nu, 1.9), (0.3, -0.2))
    geo = G.ParallelBeam3d(det) if scan == "parallel" else G.ConeBeam3d(det, 300.0, 600.0, scan)
    return np.array(G.pack_options3d(G.Volume3d((34, 31, 19), 1.0, (0.2, 0.4, -0.3)), geo), np.float32)


@pytest.mark.parametrize("scan", ["flat", "arc", "parallel"])
@pytest.mark.parametrize("Nu", [1, 33, 64, 95])
@pytest.mark.parametrize("V", [17, 33, 70, 129])
def test_split_views_and_odd_columns(cuda, native, scan, Nu, V):  # noqa: F811
    opts = _opts(scan, Nu)
    ang = (np.arange(V) * (2 * np.pi / V) + 0.011).astype(np.float32)
    sino = np.random.default_rng(V).random((2, 1, V, 21, Nu)).astype(np.float32)
    for op in ("B", "BW", "AT"):
        staged = _run(native, op, sino, opts, ang, cuda, 0)
        assert rel_l2(staged, O.dd3d(op, sino, opts, ang)) < 1e-5, op
        assert np.array_equal(staged, _run(native, op, sino, opts, ang, cuda, HOOK_PFX_NOSTAGE)), op
        assert rel_l2(_run(native, op, sino, opts, ang, cuda, HOOK_PFX_UNFIT), staged) < 1e-6, op


def test_wait_that_runs_out_in_a_cluster(cuda, native):  # noqa: F811
    opts = _opts("flat", 64)
    ang = (np.arange(129) * (2 * np.pi / 129)).astype(np.float32)
    sino = np.random.default_rng(1).random((1, 1, 129, 21, 64)).astype(np.float32)
    _run(native, "B", sino, opts, ang, cuda, 0)
    assert native.device_error(clear=True) == 0
    native.set_wait_limits(256, 0)
    _run(native, "B", sino, opts, ang, cuda, HOOK_TMA_STALL)
    assert native.device_error(clear=True) & 1
    native.set_wait_limits(0, 0)
    assert rel_l2(_run(native, "B", sino, opts, ang, cuda, 0), O.dd3d("B", sino, opts, ang)) < 1e-5
    assert native.device_error(clear=True) == 0
