"""Launch shapes that are set, restored, tuned and reused: what one method's tuning leaves to the
others, detectors too tall for some shapes, plans of the same sizes and other spacings."""
import time

import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu


def _geom(nz=30, nv=160, dz=1.0, dv=0.5, n=14, views=7, nu=36):
    return CTGeometry((n, n - 2, nz), (1.0, 1.0, dz), (0.3, 0, 0), (nu, nv), (1.6, dv), (0, 0), 1000.0, 500.0, 1500.0,
                      circular_betas(views))


def _image(g):
    import torch
    return torch.from_numpy(np.random.default_rng(3).random(g.image_shape, dtype=np.float32)).cuda()


def test_tuning_one_method_leaves_the_forward_projectors_as_they_were():
    import torch
    from ctsim_b200.projector import Plan
    g = _geom()
    x = _image(g)
    fresh, tuned = Plan(g), Plan(g)
    assert fresh.tuning["proj_layout"] == 3
    tuned.autotune("back,dd", 3)
    tuned.autotune("back,hpd", 3)
    for layout in (2, 1, 3):
        fresh.set_tuning(proj_layout=layout)
        tuned.set_tuning(proj_layout=layout)
        assert {k: fresh.tuning[k] for k in ("proj_groups", "proj_rows", "proj_slots")} == {
            k: tuned.tuning[k] for k in ("proj_groups", "proj_rows", "proj_slots")}
        assert torch.equal(fresh.project(x, "dd"), tuned.project(x, "dd")), layout


def test_set_tuning_takes_back_what_get_tuning_gave():
    import torch
    from ctsim_b200.projector import Plan
    g = _geom()
    x = _image(g)
    plan = Plan(g)
    for layout, groups in ((3, 4), (2, 8), (1, 1)):
        plan.set_tuning(proj_layout=layout, proj_groups=groups, proj_rows=32)
        want, saved = plan.project(x, "dd"), plan.tuning
        other = Plan(g)
        other.set_tuning(**saved)
        assert other.tuning == saved
        assert torch.equal(other.project(x, "dd"), want), layout


@pytest.mark.parametrize("nv,dv", [(768, 0.5), (1100, 0.4), (768, 4.0)])
def test_autotune_and_groups_on_tall_detectors(nv, dv):
    """Detectors of which the unstaged projector's shared memory does not hold eight groups."""
    import torch
    from ctsim_b200._lib import CtsimError
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = _geom(nz=90, nv=nv, dv=dv)
    x = _image(g)
    want = {m: oracle_cbct(f"proj,{m}", g, x.cpu().numpy()) for m in ("dd", "tf")}
    plan = Plan(g)
    assert plan.tuning["proj_layout"] == 3
    for groups in (1, 2, 4, 8):
        plan.set_tuning(proj_groups=groups, proj_rows=32, proj_layout=3)
        for m in ("dd", "tf"):
            got = plan.project(x, m).cpu().numpy()
            assert np.linalg.norm(got - want[m]) <= 1e-5 * np.linalg.norm(want[m]), (groups, m)
    with pytest.raises(CtsimError):
        plan.set_tuning(proj_groups=8, proj_rows=32, proj_layout=1)
    with pytest.raises(CtsimError):
        plan.set_tuning(proj_groups=3, proj_layout=3)
    for m in ("dd", "tf"):
        t = plan.autotune(f"proj,{m}", 2)
        assert t["proj_layout"] in (1, 2, 3)
        got = plan.project(x, m).cpu().numpy()
        assert np.linalg.norm(got - want[m]) <= 1e-5 * np.linalg.norm(want[m]), m


def test_choices_are_kept_by_spacings_too():
    """A choice is reused for the same geometry, measured anew for plans of the same sizes whose
    rows or voxels are longer.  Reuse takes microseconds, measuring two dozen shapes of 60 views
    takes tens of milliseconds."""
    import torch
    from ctsim_b200 import _lib
    from ctsim_b200.projector import Plan

    def seconds(plan, method):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        plan.autotune(method, 60)
        return time.perf_counter() - t0

    _lib.check(_lib.load().ctsim_autotune_clear())
    plans = [Plan(_geom(nz=64, nv=90, dv=dv, dz=dz, n=64, views=60, nu=90))
             for dv, dz in ((1.6, 1.0), (1.6, 1.0), (6.0, 1.0), (20.0, 1.0), (1.6, 4.0))]
    for method in ("proj,dd", "back,dd"):
        first, again, long_rows, longer, tall = [seconds(p, method) for p in plans]
        assert again < 0.1 * first, method
        if method == "proj,dd":
            assert long_rows > 10 * again and longer > 10 * again
        else:
            assert tall > 10 * again
