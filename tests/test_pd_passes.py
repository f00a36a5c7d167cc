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


@pytest.mark.parametrize("views,stride,begin", [(64, 1, 0), (65, 1, 0), (97, 1, 0), (70, 2, 1)])
def test_view_chunks_continue_the_sums_in_order(views, stride, begin):
    """A sinogram of more than two 32-view chunks of 5.2 MB views (and one of exactly two, which
    is one launch) gives the reference's image bit for bit, also over every second view."""
    import torch
    from dataclasses import replace
    from ctsim_b200.projector import Plan
    from oracle.bindings import oracle_cbct
    g = CTGeometry((9, 5, 6), (1.0, 1.0, 0.7), (0.25, 0, 0.5), (20, 65536), (1.6, 0.0005), (0.5, 0.25), 1000.0, 500.0,
                   1500.0, circular_betas(views * stride + begin),
                   couchZ=np.linspace(-3, 3, views * stride + begin).astype(np.float32))
    sel = slice(begin, None, stride)
    part = replace(g, betas=np.ascontiguousarray(g.betas[sel]), couchZ=np.ascontiguousarray(g.couchZ[sel]))
    y = np.random.default_rng(views).random(part.sino_shape, dtype=np.float32)
    plan = Plan(g)
    d = torch.from_numpy(y).cuda()
    for m in ("pd", "hpd", "var"):
        want = oracle_cbct(f"back,{m}", part, y)
        got = plan.backproject(d, m, view_begin=begin, view_stride=stride, view_count=views).cpu().numpy()
        assert np.array_equal(got, want), (m, float(np.abs(got - want).max()))
