"""The matched backprojection of voxels over more than two detector rows (thick slices, fine
rows), which sums its rows in a loop: whole passes, passes cut by the last slice, every z-pass
depth.  Within the parity tolerance (relative L2 1e-5) of the oracle; the pass depth changes no
bit."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu
REL_L2 = 1e-5


# (nz, rows per voxel at the axis)
@pytest.mark.parametrize("nz", [1, 33, 64, 160, 256, 300])
@pytest.mark.parametrize("rows", [2.05, 2.5, 5.0, 8.5])
def test_tall_voxels_match_oracle_at_every_depth(nz, rows):
    import torch
    from ctsim_b200._lib import CtsimError
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    nv = max(2, int(nz * rows * 0.9))  # clipped at both ends
    g = CTGeometry((9, 7, nz), (1.0, 1.0, 1.0), (0.25, 0, 0), (24, nv), (1.3, 1.5 / rows), (0.5, 0.25), 1000.0, 500.0,
                   1500.0, circular_betas(5))
    y = np.random.default_rng(nz).random(g.sino_shape, dtype=np.float32)
    yd = torch.from_numpy(y).cuda()
    plan = Plan(g)
    for m in ("dd", "tf"):
        first = plan.backproject(yd, m)
        plan.check()
        want = oracle_cbct(f"back,{m}", g, y)
        assert np.linalg.norm(first.cpu().numpy().astype(np.float64) - want) <= REL_L2 * np.linalg.norm(want), m
        for mz in (1, 2, 4, 8):
            try:
                plan.set_tuning(back_mz=mz, back_mz_tf=mz)
            except CtsimError:
                continue
            assert torch.equal(plan.backproject(yd, m), first), (m, mz)
