"""The 2-D pair on both sides of the lines between its kernels -- footprints of a few bins or many,
few views or many, small images or large -- and candidate counts at the edges of a step of 192.
Bit-identical to the reference restatement on flat detectors."""
import numpy as np
import pytest

from ctsim_b200 import circular_betas
from ctsim_b200.geometry import FanGeometry

pytestmark = pytest.mark.gpu


def _geom(nx, ny, d, nu, du, betas):
    return FanGeometry((nx, ny), (d, d), (0.25, -0.5), nu, du, 0.75, 1000.0, 500.0, 1500.0, betas)


def _image(g, seed=1):
    return np.random.default_rng(seed).random(g.image_shape, dtype=np.float32)


# bins per pixel at the axis: narrow, near the lines (footprints on both sides of four bins), very wide
@pytest.mark.parametrize("ratio", [1.0, 2.4, 2.6, 3.0, 3.1, 3.3, 4.0, 17.0])
@pytest.mark.parametrize("size", [(33, 20), (7, 64)])
def test_projection_across_footprint_widths(ratio, size):
    import torch
    from ctsim_b200.fan import FanPlan
    from oracle.bindings import oracle_fbct
    nx, ny = size
    g = _geom(nx, ny, 1.0, int(max(size) * ratio * 1.6) + 5, 1.5 / ratio, circular_betas(11) + 0.02)
    x = _image(g)
    plan = FanPlan(g)
    for m in ("dd", "tf"):
        got = plan.project(torch.from_numpy(x).cuda(), m).cpu().numpy()
        assert np.array_equal(got, oracle_fbct(f"proj,{m}", g, x)), m


@pytest.mark.parametrize("size", [(191, 1), (16, 12), (193, 1), (24, 16), (55, 7)])
def test_projection_at_a_steps_edges(size):
    """191, 192, 193, 384 and 385 candidates, all in one block of 64 bins."""
    import torch
    from ctsim_b200.fan import FanPlan
    from oracle.bindings import oracle_fbct
    nx, ny = size
    g = _geom(nx, ny, 1.0, 64, max(size) * 1.5 / 60, np.array([0.0, 0.3, -0.4, np.pi - 0.2, 1.4]))
    x = _image(g)
    plan = FanPlan(g)
    for m in ("dd", "tf"):
        got = plan.project(torch.from_numpy(x).cuda(), m).cpu().numpy()
        assert np.array_equal(got, oracle_fbct(f"proj,{m}", g, x)), m


@pytest.mark.parametrize("size,views", [((20, 9), (1, 7, 8, 33)), ((200, 163), (7, 8, 15, 16)), ((200, 164), (8, 15, 16)),
                                        ((512, 512), (15, 16, 31, 32)), ((1030, 1020), (32, 40))])
def test_backprojection_across_views_and_sizes(size, views):
    import torch
    from ctsim_b200.fan import FanPlan
    from oracle.bindings import oracle_fbct
    nx, ny = size
    for v in views:
        g = _geom(nx, ny, 100.0 / nx, 70, 2.5, circular_betas(v) + 0.02)
        y = np.random.default_rng(v).random(g.sino_shape, dtype=np.float32)
        plan = FanPlan(g)
        for m in ("dd", "tf"):
            got = plan.backproject(torch.from_numpy(y).cuda(), m, scale=2.0).cpu().numpy()
            assert np.array_equal(got, np.float32(2.0) * oracle_fbct(f"back,{m}", g, y)), (v, m)
