"""Field data is read by coherent loads (ld_field, zm_common.cuh): a kernel launched overlapped
begins while the one before it still writes, and in-place passes write what they read.  The
rule on the CPU, from the sources; long chains of unsynchronised calls on the GPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "stencilfft_b200" / "csrc"
SOURCES = sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_non_coherent_loads_read_tables_only():
    # const + __restrict__ lets the compiler make any load a non-coherent one
    bad = [p.name for p in SOURCES if re.search(r"const\s+[\w:<>]+\s*\*\s*__restrict__", _code(p))]
    assert not bad, f"const __restrict__ pointers in {bad}"
    # twiddles (ldd2, ldtw), a batch's weight tables and its tile -> field table
    table = re.compile(r"__ldg\((p|t \+ i|reinterpret_cast<const (double2|float4) \*>\(t\) \+ i|"
                       r"reinterpret_cast<const (uint4|float2) \*>\(p\)|"     # ld_field<true>
                       r"m->(va|vs|fa|fs|fr) \+ i|&(map|m\.m)->lg|bp\.tile_field \+ tile( \+ hop)?)\)")
    for path in SOURCES:
        code = _code(path)
        assert len(re.findall(r"__ldg\(", code)) == len(table.findall(code)), path.name
        assert ".nc" not in code or path.name == "zm_common.cuh", path.name


def test_overlapped_kernels_wait_and_read_coherently():
    code = "\n".join(_code(p) for p in SOURCES)
    launched = set(re.findall(r"launch_overlapped\(\s*(\w+)", code)) - {"void"}
    assert {"kern", "ktm", "permute_kernel", "stencil_kernel", "stencil3d_lines_kernel"} <= launched
    # the kernels with non-coherent field loads
    for name in ("kconst", "stencil_rowsc_kernel"):
        assert name in code and name not in launched
    # every kernel of the files that launch overlapped waits, itself or in its body function
    for f in ("zm_axis.cuh", "zm_layout.cu", "zm_stencil.cu"):
        for m in re.finditer(r"__global__[^{;]*?(\w+)\((?:[^()]|\([^()]*\))*\)\s*\{(.*?)\n\}", _code(CSRC / f), re.S):
            name, body = m.groups()
            if name in ("fill_kernel", "modes_kernel"):       # plain launches
                continue
            assert "overlap_wait()" in body or "stencil_rows_body" in body, name


def _chain(pl, x, y, z, dim, n, steps, sync):
    """`steps` rounds in the in-place contract, the converters and the operator."""
    import torch
    from stencilfft_b200 import abi

    def call(f, *a, **k):
        f(*a, **k)
        if sync:
            torch.cuda.synchronize()
    for _ in range(steps):
        call(pl.forward_fft, x, y)
        call(pl.spectral_apply, y, abi.ZM_SPECTRAL_GAUSSIAN, n / 4.0)
        call(pl.inverse_fft, y, x, scale=1.0 / float(n) ** dim)
        call(pl.laplace, x, z, inv_h2=-0.0625)
        call(pl.real_to_natural, z, y)
        call(pl.natural_to_real, y, x)
        call(pl.forward_fft, x, z)
        call(pl.reciprocal_to_natural, z, y)
        call(pl.natural_to_reciprocal, y, x)
        call(pl.inverse_fft, x, y, scale=1.0 / float(n) ** dim)
        call(pl.natural_to_real, y, x)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["c64", "c128"])
@pytest.mark.parametrize("dim,n,b,p", [(3, 16, 4, 2), (3, 32, 2, 2), (3, 64, 8, 2), (2, 64, 4, 2), (2, 256, 16, 4),
                                       (2, 1024, 32, 2), (2, 8192, 32, 4)])
def test_unsynchronised_chain_is_bit_identical(dim, n, b, p, dt):
    """The same calls with and without a synchronise after each: the same bits."""
    import torch
    from stencilfft_b200 import Plan, abi
    pl = Plan(dim, n, b, p, dtype=dt)
    out = []
    for sync in (True, False):
        x, y, z = pl.empty(), pl.empty(), pl.empty()
        pl.fill(x, abi.ZM_FIELD_GAUSSIAN, n)
        torch.cuda.synchronize()
        _chain(pl, x, y, z, dim, n, 3 if n > 4096 else 20, sync)
        torch.cuda.synchronize()
        out.append((x, y, z))
    for a, c in zip(*out):
        assert torch.equal(torch.view_as_real(a), torch.view_as_real(c))
    assert bool(torch.isfinite(torch.view_as_real(out[0][0])).all())
