"""The forward projector over staged prefix columns and the choice between it, staged voxel
columns and paired sums: volumes past the pairs' size with rows of more than three voxels, rows
of any length, columns too tall for three stages of voxels; one plan and a batch.  Within the
FP32 parity tolerance (relative L2 1e-5) of the oracle; images of mean zero keep the prefix sums,
whose rounding a row's difference inherits, of the order of a row's own value."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu
REL_L2 = 1e-5


def _rel(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b))


def _geom(n, nz, dz, nv, dv, nu, views=2, d=0.5):
    return CTGeometry((n, n - 1, nz), (d, d, dz), (0.25, 0, 0), (nu, nv), (1.5 * d, dv), (0.5, 0.25), 1000.0, 500.0,
                      1500.0, circular_betas(views) + 0.3)


def _image(g, seed):
    return np.random.default_rng(seed).random(g.image_shape, dtype=np.float32) - np.float32(0.5)


# (n, nz, dz, nv, dv, nu): past 160 MB of pairs, rows of 3.2, 4 and 12 voxels
CASES = {"rows_of_3": (400, 140, 0.5, 50, 2.4, 90), "rows_of_4_129": (406, 129, 0.5, 36, 3.0, 70),
         "rows_of_12": (512, 90, 0.5, 12, 9.0, 60)}


@pytest.mark.parametrize("name", sorted(CASES))
def test_staged_sums_match_oracle(name):
    import torch
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = _geom(*CASES[name])
    x = _image(g, 3)
    xd = torch.from_numpy(x).cuda()
    plan = Plan(g)
    assert plan.tuning["proj_layout"] == 3
    assert plan.tuning["proj_slots"] == 8
    want = oracle_cbct("proj,dd", g, x)
    got = plan.project(xd, "dd").cpu().numpy()
    plan.check()
    assert _rel(got, want) <= REL_L2
    plan.set_tuning(proj_slots=3)  # slots change no bit
    assert np.array_equal(plan.project(xd, "dd").cpu().numpy(), got)
    assert _rel(plan.project(xd, "tf").cpu().numpy(), oracle_cbct("proj,tf", g, x)) <= REL_L2


def test_tall_columns_are_staged_as_sums():
    """Columns of which three stages of voxels do not fit, two of sums do: A runs, and is linear
    in the image to a factor of two, bit for bit."""
    import torch
    from ctsim_b200.projector import Plan
    g = _geom(97, 2300, 0.5, 500, 1.4, 60)
    plan = Plan(g)
    assert plan.tuning["proj_layout"] == 3
    x = torch.from_numpy(_image(g, 3)).cuda()
    got = plan.project(x, "dd")
    plan.check()
    assert torch.equal(plan.project(2 * x, "dd"), 2 * got)


def test_batch_of_every_form():
    """Plans of voxel columns, prefix columns and paired sums in one batched call."""
    import torch
    from ctsim_b200.projector import Plan, batch_project
    geoms = [_geom(*CASES["rows_of_12"]), _geom(24, 40, 1.0, 40, 1.6, 50), _geom(30, 50, 0.5, 10, 9.0, 50)]
    plans = [Plan(g) for g in geoms]
    assert [p.tuning["proj_layout"] for p in plans] == [3, 3, 2]
    xs = [torch.from_numpy(_image(g, i)).cuda() for i, g in enumerate(geoms)]
    for m in ("dd", "tf"):
        outs = [torch.empty(g.sino_shape, device="cuda") for g in geoms]
        batch_project(m, [(p, x, o, 0, 1, 2) for p, x, o in zip(plans, xs, outs)])
        for p, x, o in zip(plans, xs, outs):
            p.check()
            assert torch.equal(o, p.project(x, m)), m


def test_slots_of_two_buffers_stay_accepted():
    """Slots that two stages hold are accepted (as many as fit are used) and change no bit."""
    import torch
    from ctsim_b200._lib import CtsimError
    from ctsim_b200.projector import Plan
    g = _geom(20, 512, 0.5, 300, 1.2, 40)
    x = torch.from_numpy(_image(g, 5)).cuda()
    plan = Plan(g)
    want = plan.project(x, "dd")
    plan.set_tuning(proj_layout=3, proj_slots=32)
    assert plan.tuning["proj_slots"] == 32
    assert torch.equal(plan.project(x, "dd"), want)
    with pytest.raises(CtsimError, match="fewer slots"):
        plan.set_tuning(proj_layout=3, proj_slots=64)


def test_long_rows_cost_no_padding():
    """A thin slice under rows of a hundred millimetres: scratch of the size of its sums."""
    from ctsim_b200.projector import Plan
    n = 256
    plan = Plan(_geom(n, 1, 0.5, 2, 100.0, 60))
    assert plan.device_bytes < 32 * n * n
