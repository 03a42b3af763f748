"""Complex128 batch fields of N = 32, the smallest of the range: half the points of a batch
tile.  Every step of every call, alone and beside larger fields."""
import numpy as np
import pytest

import oracle as O
from helpers import TOL, relerr, to_host

pytestmark = pytest.mark.gpu

SMALL = [(32, 1, 1), (32, 8, 1), (32, 32, 1), (32, 1, 2), (32, 4, 2), (32, 8, 2), (32, 1, 4), (32, 2, 4)]


def _fp64_poisson(rhs, length):
    n = rhs.shape[0]
    k = np.fft.fftfreq(n, 1.0 / n) * (2 * np.pi / length)
    ksq = k[:, None] ** 2 + k[None, :] ** 2
    ksq[0, 0] = 1.0
    s = np.fft.fft2(rhs) / -ksq
    s[0, 0] = 0.0
    phi = np.fft.ifft2(s)
    lap = sum(np.roll(phi, d, a) for d in (1, -1) for a in (0, 1)) - 4 * phi
    return phi, lap * (n / length) ** 2 - rhs


@pytest.mark.parametrize("fields", [SMALL, [SMALL[4]], [(64, 4, 2), *SMALL, (256, 16, 2), SMALL[2]]],
                         ids=["layouts", "one", "mixed"])
def test_every_call_against_the_oracle(fields):
    import torch
    from stencilfft_b200 import Batch, Plan, abi
    bt = Batch(*zip(*fields), dtype="c128")
    bufs = [torch.full_like(bt.empty(), float("nan")) for _ in range(6)]
    x, spec, back, phi, res, work = bufs
    bt.fill(x, abi.ZM_FIELD_GAUSSIAN, 11)
    bt.forward_fft(x, spec)
    bt.inverse_fft(spec, back, work=work)
    bt.poisson(x, phi, res, work, length=2.0)
    assert bt.status() == 0
    for i, (n, b, p) in enumerate(fields):
        xi = to_host(bt.field(x, i))
        pl = Plan(2, n, b, p, dtype="c128")
        ref = pl.empty()
        pl.fill(ref, abi.ZM_FIELD_GAUSSIAN, 11 + i)
        assert np.array_equal(xi, to_host(ref)), i
        assert relerr(to_host(bt.field(spec, i)), O.forward_fft(xi, 2, n, b, p)) < TOL["c128"], i
        assert relerr(to_host(bt.field(back, i)), xi) < TOL["c128"], i
        phi_ref, res_ref = _fp64_poisson(O.real_layout_to_natural(xi, 2, n, b, p), 2.0)
        for got, want in ((phi, phi_ref), (res, res_ref)):
            nat = O.real_layout_to_natural(to_host(bt.field(got, i)), 2, n, b, p)
            assert relerr(nat, want) < TOL["c128"], i
    back.fill_(float("nan"))
    bt.inverse_fft(spec, back)          # the input as scratch
    for i in range(len(fields)):
        assert relerr(to_host(bt.field(back, i)), to_host(bt.field(x, i))) < TOL["c128"], i
