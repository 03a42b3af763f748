"""The axis pass sized by N alone (zm_axis.cuh): its weight tables against the general
address formula on the CPU, and its transforms at every tile shape on the GPU."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from helpers import TOL, rand_field, relerr, to_dev, to_host

ROOT = Path(__file__).resolve().parents[1]


def test_weight_tables_match_the_general_addresses(tmp_path):
    from stencilfft_b200 import _build
    exe = tmp_path / "axis_map_check"
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.FLAGS, str(ROOT / "tests" / "native" / "axis_map_check.cu"),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


# every log2 N with a narrow and (3D) a wide tile, VEC at its ends: B = 1 (M = P) and
# B = N / P^2 (VEC = P), and P = 1 (VP = VEC; B = N: VEC = 1)
LAYOUTS = [(dim, n, b, p) for dim, sizes in ((2, (16, 32, 64, 128, 256, 512, 1024, 2048)), (3, (16, 32, 64, 128)))
           for n in sizes for p in (1, 2, 4) for b in {1, n // (p * p)} if (dim, p) != (3, 1) or n <= 32]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["c128", "c64"])
@pytest.mark.parametrize("dim,n,b,p", LAYOUTS)
def test_transforms_match_fp64(dim, n, b, p, dt):
    """Forward and inverse (complex scale) against numpy's FP64 FFT through the oracle's
    layouts, with a workspace and in place.  TOL is the suite's transform bar."""
    import torch
    from stencilfft_b200 import Plan
    x = rand_field(dim, n, seed=n + 3 * b + p)
    real = O.natural_to_real_layout(x, b, p)
    spec = O.natural_to_reciprocal_layout(np.fft.fftn(x), b, p)
    pl = Plan(dim, n, b, p, dtype=dt)
    d_in = to_dev(real, dt)
    keep, out, work = d_in.clone(), torch.empty_like(d_in), torch.empty_like(d_in)
    pl.forward_fft(d_in, out, work=work)
    assert relerr(to_host(out), spec) < TOL[dt]
    assert torch.equal(d_in, keep)
    scale = complex(1.0, -0.5) / n ** dim
    back = torch.empty_like(d_in)
    pl.inverse_fft(out, back, scale=scale, work=work)
    assert relerr(to_host(back), real * (scale * n ** dim)) < 2 * TOL[dt]   # two transforms
    pl.forward_fft(d_in, back)                                              # in place: d_in may be scratch
    assert relerr(to_host(back), spec) < TOL[dt]
    pl.inverse_fft(back, d_in, scale=1.0 / n ** dim)
    assert relerr(to_host(d_in), real) < 2 * TOL[dt]


@pytest.mark.gpu
@pytest.mark.parametrize("n,b,p,dt", [(4096, 1, 4, "c64"), (4096, 256, 4, "c128"), (8192, 512, 4, "c64"),
                                      (8192, 2, 2, "c128"), (16384, 16, 4, "c64")])
def test_large_lines_round_trip(n, b, p, dt):
    """One plane wave is one spike of n^2 (the two-sided tolerance is the suite's), and a
    Gaussian field survives forward + inverse."""
    import torch
    from stencilfft_b200 import Plan, abi
    pl = Plan(2, n, b, p, dtype=dt)
    x, y, w = pl.empty(), pl.empty(), pl.empty()
    kx, ky = 5, n - 3
    pl.fill_modes(x, [(kx, ky)], [(1.0, 0.0)], 0.0, 0)
    pl.forward_fft(x, y, work=w)
    rid, cid, lr, lc = pl.global_to_reciprocal(ky, kx)
    L = n // p
    spike = ((rid * p + cid) * L + lr) * L + lc
    assert abs(y[spike].item() / n ** 2 - 1) < TOL[dt]
    y[spike] = 0
    assert torch.linalg.vector_norm(y).item() / n ** 2 < TOL[dt]
    pl.fill(x, abi.ZM_FIELD_GAUSSIAN, 3)
    pl.forward_fft(x, y, work=w)
    pl.inverse_fft(y, w, scale=1.0 / n ** 2)
    err = torch.linalg.vector_norm(w - x) / torch.linalg.vector_norm(x)
    assert err.item() < 2 * TOL[dt]
