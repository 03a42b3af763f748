"""The 3D Laplacian on both sides of the lines between its kernels (launch_march in
zm_stencil.cu): N = 256, block heights, vector lengths, row lengths, one rank per column."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL, rand_field, relerr, to_dev, to_host


@pytest.mark.gpu
@pytest.mark.parametrize("n,p,b", [(128, 2, 8), (128, 2, 32), (256, 1, 8), (256, 1, 16), (256, 2, 2), (256, 2, 4),
                                   (256, 2, 8), (256, 2, 64), (256, 4, 4), (256, 4, 8), (256, 8, 4)])
def test_laplacian_matches_fp64(n, p, b):
    from stencilfft_b200 import Plan
    x = rand_field(3, n, seed=n + 3 * b + p)
    lap = -6.0 * x
    for d in range(3):
        lap += np.roll(x, 1, d)
        lap += np.roll(x, -1, d)
    real, ref = O.natural_to_real_layout(x, b, p), O.natural_to_real_layout(lap, b, p)
    for dt in ("c128", "c64"):
        pl = Plan(3, n, b, p, dtype=dt)
        d_in = to_dev(real, dt)
        out = pl.empty()
        pl.laplace(d_in, out)
        assert relerr(to_host(out), ref) < TOL[dt]
        assert pl.device_status() == 0
