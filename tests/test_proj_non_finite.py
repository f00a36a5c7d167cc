"""Infinite and NaN voxels in the forward projector that starts plans (staged voxel columns):
they reach the detector bins that they reach in the oracle, and every other bin keeps the bits
it has with those voxels finite.  Row pairs, column parts and candidate groups as in the shapes
test; the offsets keep voxel and bin edges apart, so that no bin is touched by rounding alone."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu

# (nz, nv, dz, dv, nu, du)
CASES = {"two_taps": (50, 90, 2.0, 2.0, 41, 0.9), "three_taps": (40, 64, 1.0, 1.6, 41, 0.9),
         "four_taps": (96, 40, 0.5, 1.9, 41, 0.9), "tall": (230, 385, 1.0, 1.6, 30, 1.6), "wide": (20, 30, 1.0, 1.3, 90, 0.4)}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("name", sorted(CASES))
def test_non_finite_voxels_stay_where_they_are(name, bad, dtype):
    import torch
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    nz, nv, dz, dv, nu, du = CASES[name]
    mask = np.ones((11, 12), bool)
    mask[2, 3] = False
    g = CTGeometry((12, 11, nz), (1.0, 1.0, dz), (0.23, 0.11, 0.07), (nu, nv), (du, dv), (0.31, 0.17), 1000.0, 500.0,
                   1500.0, circular_betas(5) + 0.013, map=mask)
    x = np.random.default_rng(11).random(g.image_shape, dtype=np.float32) + 0.5
    spots = [(nz // 2, 5, 6), (0, 8, 2), (nz - 1, 1, 10), (nz // 3, 2, 3)]  # the last is off the map
    y = x.copy()
    for s in spots:
        y[s] = bad
    dt = getattr(torch, dtype)
    plan = Plan(g)
    assert plan.tuning["proj_layout"] == 3
    for m in ("dd", "tf"):
        want = oracle_cbct(f"proj,{m}", g, y)
        for groups in (1, 2, 4):
            plan.set_tuning(proj_groups=groups, proj_rows=32, proj_layout=3)
            clean = plan.project(torch.from_numpy(x).cuda().to(dt), m, out_dtype=torch.float32).cpu().numpy()
            got = plan.project(torch.from_numpy(y).cuda().to(dt), m, out_dtype=torch.float32).cpu().numpy()
            plan.check()
            fin = np.isfinite(want)
            assert not fin.all() and fin.any()
            assert np.array_equal(np.isfinite(got), fin), (m, groups)
            assert np.array_equal(got[fin], clean[fin]), (m, groups)
