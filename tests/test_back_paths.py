"""The matched backprojection's voxel and row paths: one or two voxels per register, passes
cut by the last slice, extents of up to two, three and more rows, detectors that clip the
shadow at either end, row counts that fit no vector load, and 16-bit sinograms.  Every result
is within the FP32 parity tolerance (relative L2 1e-5) of the oracle, and a non-finite
detector pixel reaches exactly the voxels it reaches there."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu
REL_L2 = 1e-5


def _rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b))


def _geom(nz, nv, dz, dv, nu=30, flat=1, offset_v=0.0):
    return CTGeometry((11, 6, nz), (1.0, 1.0, dz), (0.25, 0, 0), (nu, nv), (1.3, dv), (0.5, offset_v), 1000.0, 500.0,
                      1500.0, circular_betas(35), flatPanel=flat)


CASES = {
    "one_slice": (1, 2, 1.0, 1.6), "pass_of_31": (31, 40, 1.0, 1.6), "pass_of_33": (33, 7, 1.0, 1.6),
    "pass_of_77": (77, 130, 1.0, 1.6), "clipped": (130, 60, 1.0, 1.6), "clipped_rows3": (100, 90, 1.0, 1.1),
    "second_pass": (300, 384, 1.0, 1.7), "rows3": (64, 132, 1.0, 0.9), "wide_rows": (40, 200, 2.0, 0.8),
    "unit_height": (50, 96, 1.0, 1.5),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("nu", [30, 7])
def test_paths_match_oracle(name, nu):
    import torch
    from ctsim_b200._lib import CtsimError
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = _geom(*CASES[name], nu=nu)
    y = np.random.default_rng(5).random(g.sino_shape, dtype=np.float32)
    yd = torch.from_numpy(y).cuda()
    yb = yd.to(torch.bfloat16)
    plan = Plan(g)
    for m in ("dd", "tf"):
        want, want_b = oracle_cbct(f"back,{m}", g, y), oracle_cbct(f"back,{m}", g, yb.float().cpu().numpy())
        for mz in (1, 2, 4, 8):
            try:
                plan.set_tuning(back_mz=mz, back_mz_tf=mz)
            except CtsimError:
                continue
            assert _rel(plan.backproject(yd, m).cpu().numpy(), want) <= REL_L2, (m, mz)
            assert _rel(plan.backproject(yb, m, out_dtype=torch.float32).cpu().numpy(), want_b) <= REL_L2, (m, mz)
        plan.check()


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("name", ["pass_of_77", "clipped", "rows3", "clipped_rows3"])
def test_non_finite_pixels_stay_where_they_are(name, bad):
    import torch
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = _geom(*CASES[name])
    y = np.random.default_rng(6).random(g.sino_shape, dtype=np.float32)
    y[3, 12, g.nv // 2] = bad
    y[20, 15, 0] = bad
    plan = Plan(g)
    got = plan.backproject(torch.from_numpy(y).cuda(), "dd").cpu().numpy()
    assert np.array_equal(np.isfinite(got), np.isfinite(oracle_cbct("back,dd", g, y)))
