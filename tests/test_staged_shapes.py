"""The staged forward projector's launch shapes: row pairs per warp (detectors of up to 64,
128, 256, 384 rows and taller, in one or several blocks along the rows), voxels per row
extent (two, three, more), candidate groups and slots per stage, and shadows that lie off the
detector's middle.  Every result is within the FP32 parity tolerance (relative L2 1e-5) of the
oracle; slots and launch order change no bit."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu
REL_L2 = 1e-5


def _rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b))


def _geom(nz, nv, dz, dv, couch=0.0, offset_v=0.0, flat=1, n=12, nu=41):
    return CTGeometry((n, n - 1, nz), (1.0, 1.0, dz), (0.25, 0, 0), (nu, nv), (0.9, dv), (0.5, offset_v), 1000.0, 500.0,
                      1500.0, circular_betas(5), couchZ=np.full(5, couch, np.float32), flatPanel=flat)


# (nz, nv, dz, dv): a row is dv / (1.5 dz) voxels long at the axis
CASES = {
    "two_rows": (3, 2, 1.0, 1.6), "64_rows": (40, 64, 1.0, 1.6), "65_rows": (44, 65, 1.0, 1.6),
    "128_rows": (60, 128, 1.0, 1.2), "129_rows": (130, 129, 1.0, 1.6), "257_rows": (150, 257, 1.0, 0.9),
    "384_rows": (200, 384, 1.0, 0.9), "385_rows": (230, 385, 1.0, 1.6), "800_rows": (90, 800, 1.0, 0.5),
    "two_taps": (50, 90, 2.0, 2.0), "four_taps": (96, 40, 0.5, 1.9), "nine_taps": (120, 20, 0.2, 2.4),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_row_shapes_and_extents_match_oracle(name):
    import torch
    from ctsim_b200._lib import CtsimError
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = _geom(*CASES[name])
    x = np.random.default_rng(7).random(g.image_shape, dtype=np.float32)
    xd = torch.from_numpy(x).cuda()
    plan = Plan(g)
    for m in ("dd", "tf"):
        want = oracle_cbct(f"proj,{m}", g, x)
        for groups in (1, 2, 4, 8):
            same = None
            for slots in (1, 5, 16, 32):
                try:
                    plan.set_tuning(proj_groups=groups, proj_rows=32, proj_layout=3, proj_slots=slots)
                except CtsimError:  # tall detectors: more groups than the unstaged kernel's shared memory holds
                    assert groups > 1 and g.nv > 384
                    continue
                got = plan.project(xd, m).cpu().numpy()
                plan.check()
                assert _rel(got, want) <= REL_L2, (m, groups, slots)
                assert same is None or np.array_equal(got, same), (m, groups, slots)
                same = got


@pytest.mark.parametrize("couch,offset_v,flat", [(30.0, 0.0, 1), (-25.0, 6.5, 1), (0.0, -40.0, 1), (12.0, 9.0, 0)])
def test_shadows_off_the_middle_match_oracle(couch, offset_v, flat):
    import torch
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = _geom(40, 100, 1.0, 1.1, couch, offset_v, flat)
    x = np.random.default_rng(8).random(g.image_shape, dtype=np.float32)
    plan = Plan(g)
    for m in ("dd", "tf"):
        got = plan.project(torch.from_numpy(x).cuda(), m).cpu().numpy()
        plan.check()
        assert _rel(got, oracle_cbct(f"proj,{m}", g, x)) <= REL_L2, m


def test_wide_footprints_and_map():
    """Footprints of up to ten detector columns (several column parts) and map-off columns."""
    import torch
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    rng = np.random.default_rng(9)
    g = CTGeometry((10, 12, 6), (2.0, 2.0, 1.0), (0, 0, 0), (83, 12), (0.4, 1.6), (0, 0), 1000.0, 500.0, 1500.0,
                   circular_betas(7), map=rng.random((12, 10)) > 0.3)
    x = rng.random(g.image_shape, dtype=np.float32)
    plan = Plan(g)
    for m in ("dd", "tf"):
        got = plan.project(torch.from_numpy(x).cuda(), m).cpu().numpy()
        assert _rel(got, oracle_cbct(f"proj,{m}", g, x)) <= REL_L2, m


@pytest.mark.parametrize("nz,nv,dz,dv,layout", [(60, 41, 1.0, 1.6, 3), (96, 40, 0.5, 1.9, 3), (256, 70, 0.5, 3.0, 3),
                                               (257, 70, 0.5, 3.0, 2), (120, 20, 0.2, 3.2, 2), (301, 128, 1.0, 3.0, 2)])
def test_default_route_at_its_lines(nz, nv, dz, dv, layout):
    """The default projector on both sides of the lines between staged columns and paired sums
    (voxels per row, slices) is within the parity tolerance of the oracle."""
    import torch
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = _geom(nz, nv, dz, dv)
    plan = Plan(g)
    assert plan.tuning["proj_layout"] == layout
    x = np.random.default_rng(nz).random(g.image_shape, dtype=np.float32)
    for m in ("dd", "tf"):
        got = plan.project(torch.from_numpy(x).cuda(), m).cpu().numpy()
        plan.check()
        assert _rel(got, oracle_cbct(f"proj,{m}", g, x)) <= REL_L2, m
