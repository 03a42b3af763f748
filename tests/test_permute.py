"""The layout converters as bit permutations (zm_layout.cu) and the reciprocal-space operator
on every kind of layout: their tables on the CPU, the kernels on the GPU."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from helpers import rand_field, relerr, to_dev, to_host

ROOT = Path(__file__).resolve().parents[1]


def test_permutations_match_the_index_maps(tmp_path):
    from stencilfft_b200 import _build
    exe = tmp_path / "perm_map_check"
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.FLAGS, str(ROOT / "tests" / "native" / "perm_map_check.cu"),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


# fields smaller than a tile, of one tile and of many; VP = 1 and 2, VEC = P, B = 1
LAYOUTS = [(2, 4, 1, 2), (2, 8, 2, 2), (2, 16, 1, 4), (2, 16, 4, 2), (2, 32, 8, 1), (2, 64, 16, 2), (2, 64, 1, 8),
           (2, 512, 1, 4), (2, 512, 32, 4), (3, 4, 1, 2), (3, 8, 2, 2), (3, 16, 1, 4), (3, 32, 8, 2), (3, 64, 1, 4)]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["c128", "c64"])
@pytest.mark.parametrize("dim,n,b,p", LAYOUTS)
def test_converters_and_operator(dim, n, b, p, dt):
    """Converters move elements (exact); the Poisson operator is one rounded factor of an
    exact integer |k|^2 per element: a few ulp of the working precision."""
    import torch
    from stencilfft_b200 import Plan, abi
    pl = Plan(dim, n, b, p, dtype=dt)
    x = rand_field(dim, n, seed=n + b)
    nat = to_dev(x, dt).contiguous()
    xr = to_host(nat).reshape(x.shape)          # rounded to the plan's precision
    for to_inter, to_nat, ref in ((pl.natural_to_real, pl.real_to_natural, O.natural_to_real_layout),
                                  (pl.natural_to_reciprocal, pl.reciprocal_to_natural, O.natural_to_reciprocal_layout)):
        inter, back = torch.empty_like(nat), torch.empty_like(nat)
        to_inter(nat, inter)
        assert np.array_equal(to_host(inter).ravel(), ref(xr, b, p).ravel())
        to_nat(inter, back)
        assert torch.equal(back, nat)
    k = np.fft.fftfreq(n, 1.0 / n) ** 2
    k2 = sum(np.meshgrid(*([k] * dim), indexing="ij"))
    with np.errstate(divide="ignore"):
        f = np.where(k2 == 0, 0.0, -1.0 / (4.0 * k2))
    d = to_dev(O.natural_to_reciprocal_layout(xr, b, p), dt)
    pl.spectral_apply(d, abi.ZM_SPECTRAL_POISSON, 2.0)
    ref = O.natural_to_reciprocal_layout(xr * f, b, p)
    assert relerr(to_host(d).ravel(), ref.ravel()) < (1e-15 if dt == "c128" else 1e-6)
