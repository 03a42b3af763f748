"""Batches on the split-digit tiles (zm_batch_exact.cu) and the residual step.

* on the CPU: the digit orders, stage twiddles and weight tables of the split-digit tiles;
* on the GPU: the complex64 Poisson call with a residual gives, bit for bit, what the split
  tiles give (a batch with one field that only those hold runs all its fields on them);
* on the GPU: the residual is the 5-point Laplacian of the phi returned, over the layouts.
"""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle as O
from helpers import to_host

ROOT = Path(__file__).resolve().parents[1]


def test_digits_twiddles_and_weights_on_the_host(tmp_path):
    from stencilfft_b200 import _build
    exe = tmp_path / "batch_exact_check"
    subprocess.run([_build.nvcc(), *_build.ARCH, *_build.FLAGS,
                    str(ROOT / "tests" / "native" / "batch_exact_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _poisson(fields, dt):
    """phi and residual of every field, N(0,1) right-hand sides from seeds 7, 8, ..."""
    from stencilfft_b200 import Batch, abi
    bt = Batch([f[0] for f in fields], [f[1] for f in fields], [f[2] for f in fields], dtype=dt)
    rhs, phi, res, work = bt.empty(), bt.empty(), bt.empty(), bt.empty()
    bt.fill(rhs, abi.ZM_FIELD_GAUSSIAN, 7)
    bt.poisson(rhs, phi, res, work)
    assert bt.status() == 0
    return [tuple(bt.field(t, i) for t in (rhs, phi, res)) for i in range(len(fields))]


# every (N, VEC) of the split-digit tiles
EXACT = [(n, n // (p * v), p) for n in (64, 128, 256, 512, 1024, 2048, 4096) for v in (2, 4, 8, 16) for p in (1, 2)
         if p <= v]


@pytest.mark.gpu
def test_split_digit_tiles_keep_every_bit():
    import torch
    alone = _poisson(EXACT, "c64")
    beside = _poisson(EXACT + [(64, 1, 2)], "c64")   # VEC = 32
    for f, a, b in zip(EXACT, alone, beside):
        for x, y in zip(a, b):
            assert torch.equal(torch.view_as_real(x), torch.view_as_real(y)), f


# P = 1 .. 8; VEC = 1, below a 16-byte access, and up to B = 1
LAYOUTS = [(n, b, p) for n in (64, 128, 512) for p in (1, 2, 4, 8)
           for b in {1, 2, 8, n // (2 * p * p), n // (p * p)} if b >= 1 and n % (p * p * b) == 0]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["c128", "c64"])
def test_residual_is_the_laplacian_of_phi(dt):
    """Against FP64 on the phi returned.  With u the unit roundoff, the five-term sum (terms
    of at most 4 max|phi|, partial sums of at most 8) is off by at most 8 * 8 u max|phi|, the
    scaling by N^2 and the difference with rhs add at most 3 u of their values."""
    u = 2.0 ** (-53 if dt == "c128" else -24)
    for (n, b, p), out in zip(LAYOUTS, _poisson(LAYOUTS, dt)):
        rhs, phi, res = (O.real_layout_to_natural(to_host(t), 2, n, b, p) for t in out)
        lap = (np.roll(phi, 1, 0) + np.roll(phi, -1, 0) + np.roll(phi, 1, 1) + np.roll(phi, -1, 1) - 4 * phi) * n ** 2
        top = np.abs(phi).max() * n ** 2
        assert np.abs(res - (lap - rhs)).max() < u * ((64 + 24) * top + 3 * np.abs(rhs).max()), (n, b, p)
