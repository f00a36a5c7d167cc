"""The 2-D pair's steps: candidate counts around a step of 256, detectors around a block of 64
bins, footprints wider than the products kept per candidate, view counts around a step of 32,
odd image widths.  Bit-identical to the reference restatement on flat detectors."""
import numpy as np
import pytest

from ctsim_b200 import circular_betas
from ctsim_b200.geometry import FanGeometry

pytestmark = pytest.mark.gpu

# (nx, ny, pixel, nu, du, views)
CASES = [(3, 2, 1.0, 5, 1.2, 1), (16, 16, 1.0, 64, 1.2, 31), (17, 15, 1.0, 65, 1.2, 32), (40, 33, 0.8, 130, 0.9, 33),
         (65, 20, 2.0, 100, 0.4, 65), (9, 70, 3.0, 63, 0.5, 40)]


@pytest.mark.parametrize("case", CASES)
def test_fan_pair_matches_oracle_bit_for_bit(case):
    import torch
    from ctsim_b200.fan import FanPlan
    from oracle.bindings import oracle_fbct
    nx, ny, d, nu, du, views = case
    g = FanGeometry((nx, ny), (d, d), (0.25, -0.5), nu, du, 0.75, 1000.0, 500.0, 1500.0, circular_betas(views) + 0.01)
    rng = np.random.default_rng(nx)
    x, y = rng.random(g.image_shape, dtype=np.float32), rng.random(g.sino_shape, dtype=np.float32)
    plan = FanPlan(g)
    for m in ("dd", "tf"):
        got = plan.project(torch.from_numpy(x).cuda(), m).cpu().numpy()
        assert np.array_equal(got, oracle_fbct(f"proj,{m}", g, x)), m
        got = plan.backproject(torch.from_numpy(y).cuda(), m).cpu().numpy()
        assert np.array_equal(got, oracle_fbct(f"back,{m}", g, y)), m
