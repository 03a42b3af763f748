"""The grid-barrier probe runs on the kernels that the batch's calls use."""
import time

import pytest

import oracle as O
from helpers import TOL, relerr, to_host


# (fields, dtype, kernels): the axis tiles and the Poisson call's (its own, or the split's
# where VEC = 32), complex128's axis tiles, and the split tiles of N = 32
BATCHES = [([(64, 4, 2), (256, 32, 2)], "c64", 2), ([(64, 4, 2), (256, 4, 2)], "c64", 2),
           ([(64, 4, 2), (256, 32, 2)], "c128", 1), ([(32, 4, 2), (64, 4, 2)], "c128", 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("fields,dt,kernels", BATCHES)
def test_every_kernel_gives_up_and_recovers(fields, dt, kernels):
    """Each kernel's barrier waits its 2 s limit out once, the status reports it, and the next
    calls run to the end."""
    from stencilfft_b200 import Batch, abi, launch_count
    bt = Batch(*zip(*fields), dtype=dt)
    n0 = launch_count()
    bt.barrier_probe(0)
    assert bt.status() == 0 and launch_count() - n0 == kernels
    t0 = time.perf_counter()
    bt.barrier_probe(1)
    assert bt.status() == 1
    assert 1.9 * kernels < time.perf_counter() - t0 < 30
    assert bt.status() == 0
    x, y, z, w = (bt.empty() for _ in range(4))
    bt.fill(x, abi.ZM_FIELD_GAUSSIAN, 1)
    bt.forward_fft(x, y)
    bt.poisson(x, z, None, w)
    assert bt.status() == 0
    for i, (n, b, p) in enumerate(fields):
        xi = to_host(bt.field(x, i))
        assert relerr(to_host(bt.field(y, i)), O.forward_fft(xi, 2, n, b, p)) < TOL[dt]
