"""The voxel-driven backprojection's passes: one or two voxels per register, one to eight
32-slice blocks per pass, the last pass cut to the blocks that remain.  Every slice count
around a block or pass edge gives the reference's image, bit for bit on a flat panel."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [1, 31, 32, 33, 64, 65, 96, 129, 193, 257])
def test_slice_counts_at_pass_edges_are_bit_identical(nz):
    import torch
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    # rows off both detector ends (pd drops them, hpd clamps them), columns off one side, 33
    # views (a second 32-view chunk of one view)
    g = CTGeometry((9, 5, nz), (1.0, 1.0, 0.7), (0.25, 0, 0.5), (14, max(2, nz // 2)), (1.6, 1.3), (2.0, 0.25), 1000.0,
                   500.0, 1500.0, circular_betas(33), couchZ=np.linspace(-3, 3, 33).astype(np.float32))
    y = np.random.default_rng(nz).random(g.sino_shape, dtype=np.float32)
    plan = Plan(g)
    for m in ("pd", "hpd", "var"):
        want = oracle_cbct(f"back,{m}", g, y)
        for mz in (1, 2, 4, 8):
            plan.set_tuning(pd_mz=mz)
            got = plan.backproject(torch.from_numpy(y).cuda(), m).cpu().numpy()
            assert np.array_equal(got, want), (m, mz, float(np.abs(got - want).max()))
