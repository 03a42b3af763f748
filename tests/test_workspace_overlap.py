"""A workspace that overlaps the input or the output: the 2D forward transform needs none and
runs as without one, the other transforms refuse it."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["c64", "c128"])
@pytest.mark.parametrize("n,b,p", [(16, 2, 2), (64, 4, 2), (512, 8, 4), (1024, 32, 2), (4096, 32, 4)])
def test_forward_2d_leaves_it_alone(n, b, p, dt):
    import torch
    from stencilfft_b200 import Plan, ZmError, abi
    pl = Plan(2, n, b, p, dtype=dt)
    x, want, out = pl.empty(), pl.empty(), pl.empty()
    pl.fill(x, abi.ZM_FIELD_GAUSSIAN, 3)
    kept = x.clone()
    pl.forward_fft(x, want)
    for work in (x, out):
        pl.forward_fft(x, out, work=work)
        assert torch.equal(out, want) and torch.equal(x, kept)
    with pytest.raises(ZmError):
        pl.inverse_fft(out, x, work=out)
    with pytest.raises(ZmError):
        pl.forward_fft(x, x)


@pytest.mark.gpu
@pytest.mark.parametrize("dim,n,b,p,dt", [(3, 32, 4, 2, "c64"), (2, 8192, 128, 2, "c64"), (2, 8192, 64, 2, "c64"),
                                          (2, 16384, 64, 4, "c64")])
def test_the_others_refuse_it(dim, n, b, p, dt):
    from stencilfft_b200 import Plan, ZmError
    pl = Plan(dim, n, b, p, dtype=dt)
    x, out = pl.empty(), pl.empty()
    for work in (x, out):
        with pytest.raises(ZmError):
            pl.forward_fft(x, out, work=work)
