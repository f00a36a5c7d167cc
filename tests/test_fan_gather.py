"""The 2-D forward projector's bins that gather their pixels themselves (views whose rays run
along the rows) on curved and flat detectors, with a source close enough to the image that a
pixel's shadow may reach past 90 degrees of fan angle.  Curved detectors agree to the parity
tolerance (the tangent and arc tangent are not the reference's bit for bit), flat ones exactly."""
import numpy as np
import pytest

from ctsim_b200.geometry import FanGeometry

pytestmark = pytest.mark.gpu
REL_L2 = 1e-5

BETAS = np.pi / 2 + np.array([-0.02, 0.0, 0.013, np.pi - 0.03, np.pi + 0.005])

# (nx, ny, pixel, nu, du, offset_u, SAD, SDD, flat)
CASES = {
    "near_curved": (8, 8, 1.0, 24, 0.7, 0.0, 7.2, 10.0, 0),
    "near_curved_wide": (12, 9, 1.0, 60, 0.5, 0.25, 9.2, 10.0, 0),
    "near_flat": (8, 8, 1.0, 40, 0.7, 0.0, 7.2, 10.0, 1),
    "curved": (40, 33, 1.0, 70, 1.2, 0.75, 1000.0, 1500.0, 0),
    "curved_coarse": (64, 20, 0.5, 9, 9.0, 0.0, 300.0, 500.0, 0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_gathered_bins_match_oracle(name):
    import torch
    from ctsim_b200.fan import FanPlan
    from oracle.bindings import oracle_fbct
    nx, ny, d, nu, du, off, sad, sdd, flat = CASES[name]
    g = FanGeometry((nx, ny), (d, d), (0.0, 0.0), nu, du, off, sad, sdd - sad, sdd, BETAS, flat)
    x = np.random.default_rng(nu).random(g.image_shape, dtype=np.float32)
    plan = FanPlan(g)
    for m in ("dd", "tf"):
        got = plan.project(torch.from_numpy(x).cuda(), m).cpu().numpy()
        want = oracle_fbct(f"proj,{m}", g, x)
        if flat:
            assert np.array_equal(got, want), m
        # a bin that misses a pixel is off by far more than the rounding of its own sum
        assert np.abs(got.astype(np.float64) - want).max() <= REL_L2 * np.abs(want).max(), m
