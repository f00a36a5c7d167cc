"""Batched forward projections of plans that differ in slices, in-plane size, views and rows: one
launch over staged voxel columns of several strides.  Bit-identical to each plan's own A."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu


def _geom(n, nz, nv, dv=1.6, views=9, flat=1):
    return CTGeometry((n, n - 3, nz), (1.0, 1.0, 1.0), (0.25, 0, 0), (2 * n + 5, nv), (1.1, dv), (0.5, 0.25), 1000.0, 500.0,
                      1500.0, circular_betas(views), flatPanel=flat)


# each list one class of row pairs: ascending, descending and mixed strides, many small plans
LISTS = {
    "ascending": [(12, 1, 10), (13, 7, 20), (20, 33, 30), (31, 90, 64)],
    "descending": [(40, 300, 128), (12, 200, 100), (33, 60, 120), (10, 2, 66)],
    "four_pairs": [(12, 500, 256), (25, 100, 200), (14, 230, 130)],
    "two_warps": [(12, 600, 700), (18, 250, 500)],
    "many": [(8 + i % 5, 1 + 3 * i, 20 + i % 40) for i in range(70)],
}


@pytest.mark.parametrize("name", sorted(LISTS))
@pytest.mark.parametrize("groups", [1, 4])
def test_uneven_batches_equal_each_plans_own_projection(name, groups):
    import torch
    from ctsim_b200.projector import Plan, batch_project
    geoms = [_geom(*c, views=1 + i % 9, flat=1 - i % 2) for i, c in enumerate(LISTS[name])]
    plans = [Plan(g) for g in geoms]
    for p in plans:
        assert p.tuning["proj_layout"] == 3
        p.set_tuning(proj_groups=groups)
    rng = np.random.default_rng(4)
    xs = [torch.from_numpy(rng.random(g.image_shape, dtype=np.float32)).cuda() for g in geoms]
    for m in ("dd", "tf"):
        want = [p.project(x, m) for p, x in zip(plans, xs)]
        outs = [torch.full(g.sino_shape, float("nan"), device="cuda") for g in geoms]
        batch_project(m, [(p, x, o, 0, 1, g.noViews) for p, x, o, g in zip(plans, xs, outs, geoms)])
        for i, p in enumerate(plans):
            p.check()
            assert torch.equal(outs[i], want[i]), (m, i)
