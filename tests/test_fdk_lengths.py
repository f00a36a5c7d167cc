"""The row filter's transform lengths (64 to 4096: every mix of radix-8 and radix-4 passes), odd
row counts and both detectors, against the oracle's float64 filter (relative L2 1e-5)."""
import numpy as np
import pytest

from ctsim_b200 import CTGeometry, circular_betas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,nv", [(5, 9), (33, 1 + 8), (64, 7), (100, 16), (200, 3), (300, 8), (513, 5), (1025, 17)])
@pytest.mark.parametrize("flat", [1, 0])
def test_filter_lengths_match_oracle(nu, nv, flat):
    import torch
    from ctsim_b200.fdk import FDK
    from oracle import fdk_oracle
    g = CTGeometry((8, 8, 4), (1.0, 1.0, 1.0), (0, 0, 0), (nu, nv), (0.5, 1.0), (0.25, 0), 1000.0, 500.0, 1500.0,
                   circular_betas(3), flatPanel=flat)
    y = np.random.default_rng(nu).random(g.sino_shape, dtype=np.float32)
    got = FDK(g, "hann").filter(torch.from_numpy(y).cuda()).cpu().numpy().astype(np.float64)
    want = fdk_oracle.filtered_sinogram(y, g, "hann")
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
