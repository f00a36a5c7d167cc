"""The matched backprojection on detectors of more rows than 16 bits count (32768) and of more
than the loop-free row paths take (8192), through the entry point that has no bound of its own
on them (plans stop at 6080): shadows high up the detector, inside it and cut by its last row.
Within the FP32 parity tolerance (relative L2 1e-5) of the oracle, whose row weights the kernel
forms with the same float operations."""
import ctypes

import numpy as np
import pytest

from ctsim_b200 import CTGeometry, _lib, circular_betas

REL_L2 = 1e-5

# (nz, nv, row that the volume's middle projects to, dv)
CASES = [(50, 8192, 8150.0, 1.6), (50, 8193, 8150.0, 1.6), (20, 9000, 8999.0, 1.1), (300, 33000, 32770.0, 1.6),
         (50, 40000, 35000.25, 1.1), (200, 40000, 39999.0, 1.6), (31, 40001, 39990.0, 0.6)]


def _geom(nz, nv, row, dv):
    return CTGeometry((9, 8, nz), (1.0, 1.0, 1.0), (0.25, 0, 0), (7, nv), (1.6, dv), (0.5, (nv - 1) / 2 - row), 1000.0,
                      500.0, 1500.0, circular_betas(3))


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_backprojection_high_up_the_detector(case):
    import torch
    from oracle.bindings import oracle_cbct
    g = _geom(*case)
    y = np.random.default_rng(2).random(g.sino_shape, dtype=np.float32)
    want = oracle_cbct("back,dd", g, y)
    assert np.linalg.norm(want) > 0
    gs = _lib.CtsimGeom(*g.scalars()[:18], g.noViews, int(g.flatPanel))
    betas, couch, mp = (np.ascontiguousarray(a) for a in (g.betas, g.couchZ, g.map))
    yd = torch.from_numpy(y).cuda()
    out = torch.empty(g.image_shape, device="cuda")
    _lib.check(_lib.load().ctsim_back_dd_noalloc(ctypes.byref(gs), betas.ctypes.data, couch.ctypes.data, mp.ctypes.data,
                                                 yd.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream),
               "ctsim_back_dd_noalloc")
    torch.cuda.synchronize()
    got = out.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= REL_L2
