"""The Poisson call gives the same phi, bit for bit, with and without its residual, on every
kind of tile."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["c64", "c128"])
@pytest.mark.parametrize("fields", [[(64, 4, 2), (256, 32, 2), (512, 64, 2)],       # VEC = 8, 4, 4
                                    [(128, 4, 1), (1024, 16, 2)],                   # VEC = 32
                                    [(64, 64, 1), (256, 32, 2)]])                   # VEC = 1 and 4
def test_phi_does_not_depend_on_the_residual(fields, dt):
    import torch
    from stencilfft_b200 import Batch, abi
    bt = Batch(*zip(*fields), dtype=dt)
    rhs, phi, phi_res, res, work = (bt.empty().zero_() for _ in range(5))
    bt.fill(rhs, abi.ZM_FIELD_GAUSSIAN, 5)
    bt.poisson(rhs, phi, None, work)
    bt.poisson(rhs, phi_res, res, work)
    assert bt.status() == 0
    assert torch.equal(torch.view_as_real(phi), torch.view_as_real(phi_res))
    assert float(phi.abs().max()) > 0
