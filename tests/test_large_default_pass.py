"""Fields of 2^31 elements and more, which the axis pass (32-bit offsets) does not take: the
lines that had a size-specialised default pass still have one, and it transforms them."""
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "stencilfft_b200" / "csrc"
HBM = 180e9     # bytes; a transform needs two fields


@pytest.mark.parametrize("dt,eb", [("c64", 8), ("c128", 16)])
def test_specialised_lines_keep_a_default(dt, eb):
    assert "if (total >= int64_t{1} << 31) return false;" in (CSRC / "zm_axis.cu").read_text()
    fwd, inv = ((CSRC / f"zm_fft2_{dt}_{d}.cu").read_text() for d in ("fwd", "inv"))
    lines = re.findall(r"case \((\d) << 8\) \| (\d): return \d+;", fwd)
    assert len(lines) == 10
    for lv, lm in lines:
        ln = int(lv) + int(lm)
        for dim in (2, 3):
            total = 1 << (dim * ln)
            if total >= 1 << 31 and 2 * total * eb <= HBM:
                first = f"case ({lv} << 16) | ({lm} << 8) | 0: return launch_"
                assert first in fwd and first in inv, (dim, ln)


@pytest.mark.gpu
def test_3d_2048_c64_delta():
    """A unit impulse: its spectrum is one phase per frequency, read at sampled elements; the
    inverse transform brings it back.  Both fields together fill 137 GB."""
    import torch
    from stencilfft_b200 import Plan
    n, b, p = 2048, 32, 2
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 2 * 8 * n ** 3 + 2 ** 30:
        pytest.skip("needs 138 GB of free device memory")
    pl = Plan(3, n, b, p, dtype="c64")
    L = n // p

    def element(rid, cid, did, ld, lr, lc):
        return (((did * p + rid) * p + cid) * L ** 3) + (ld * L + lr) * L + lc
    at = (1234, 77, 2047)
    e0 = element(*pl.global_to_real(*at))
    x, y = torch.zeros(n ** 3, dtype=torch.complex64, device="cuda"), pl.empty()
    x[e0] = 1.0
    pl.forward_fft(x, y)
    rng = np.random.default_rng(1)
    idx, ref = [], []
    for _ in range(4000):
        rid, cid, did = (int(v) for v in rng.integers(0, p, 3))
        ld, lr, lc = (int(v) for v in rng.integers(0, L, 3))
        k = pl.reciprocal_to_global(rid, cid, lr, lc, did, ld)
        idx.append(element(rid, cid, did, ld, lr, lc))
        ref.append(np.exp(-2j * np.pi * (sum(i * q for i, q in zip(at, k)) % n) / n))
    got, ref = y[torch.tensor(idx, device="cuda")].cpu().numpy().astype(np.complex128), np.array(ref)
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-6
    x.zero_()
    pl.inverse_fft(y, x, scale=1.0 / float(n) ** 3)
    assert abs(complex(x[e0]) - 1.0) < 1e-6
    x[e0] = 0.0
    # the largest of 2^33 sums of as many rounded unit phases, over 2^33
    assert max(float(v.abs().max()) for v in torch.view_as_real(x).view(64, -1)) < 1e-6
    del x, y
    torch.cuda.empty_cache()
