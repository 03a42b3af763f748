"""The 2D stencils' row kernels (one, two and four rows per thread) at every block size."""
import numpy as np
import pytest

import oracle as O
from helpers import rand_field, relerr, to_dev, to_host


def _diff(x, axis, delta):
    """dx.cu:26-79 / dy.cu:34-100 in the reference's operations and order, per component."""
    def one(f):
        s = 0.0 + np.roll(f, 1, axis) * -8.0
        s = s + np.roll(f, 2, axis)
        s = s + np.roll(f, -1, axis) * 8.0
        s = s - np.roll(f, -2, axis)
        return s / (12.0 * delta)
    out = np.empty_like(x)
    out.real, out.imag = one(x.real), one(x.imag)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("delta", [0.37, -1.0 / 64])
@pytest.mark.parametrize("n,b,p", [(64, 1, 4), (64, 2, 4), (64, 4, 4), (64, 8, 2), (64, 16, 2), (64, 64, 1)])
def test_stencils_bit_exact_at_every_block_size(n, b, p, delta):
    """One, two and four rows per thread: Laplacian (oracle), dx and dy (the reference's
    operations in numpy) of a complex128 field bit for bit, and of the complex64 field within
    its bar; the three in one launch equal their own kernels."""
    import torch
    from stencilfft_b200 import Plan
    x = rand_field(2, n, seed=b)
    buf = O.natural_to_real_layout(x, b, p)
    for dt in ("c128", "c64"):
        pl = Plan(2, n, b, p, dtype=dt)
        d = to_dev(buf, dt)
        ref = to_host(d)
        nat = O.real_layout_to_natural(ref, 2, n, b, p)
        want = [O.laplace(ref, 2, n, b, p)] + [O.natural_to_real_layout(_diff(nat, ax, delta), b, p) for ax in (1, 0)]
        got = [torch.empty_like(d) for _ in range(3)]
        pl.laplace(d, got[0]), pl.dx(d, got[1], delta=delta), pl.dy(d, got[2], delta=delta)
        one = [torch.empty_like(d) for _ in range(3)]
        pl.laplace_dx_dy(d, *one, delta=delta)
        for g, o, w in zip(got, one, want):
            assert torch.equal(g, o)
            if dt == "c128":
                assert np.array_equal(to_host(g).ravel(), np.asarray(w).ravel())
            else:
                assert relerr(to_host(g).ravel(), np.asarray(w).ravel()) < 1e-6
