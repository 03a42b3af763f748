"""The calls that a program makes of this framework, as performance cases.

Each case is one dict of plain values; its "kind" names the sequence of public calls that
`run` makes:

  round_trip  forward_fft, then inverse_fft of the spectrum (scale 1 / N^dim), then the
              5/7-point Laplacian of the input: the reference drivers' test sequence
  step        forward_fft, inverse_fft, and laplace_dx_dy of the round-tripped field:
              the benchmark's step (2D)
  in_place    forward_fft and inverse_fft under the reference's own contract (no
              workspace, both buffers reused)
  filter      a field in natural order through the whole pipeline: natural_to_real,
              forward_fft, spectral_apply (Gaussian), inverse_fft, real_to_natural, and
              the unfiltered spectrum in natural order
  poisson     forward_fft, spectral_apply (Poisson), inverse_fft
  adjoint     loss gradient of Laplace(IFFT(G FFT(u))): the forward chain and its VJPs
  stencils    laplace, dx, dy of a complex field and dx, dy of a real one (2D)
  batch       Batch.poisson with its residual over 2D fields of uneven N
  batch_fft   Batch.forward_fft and Batch.inverse_fft over 2D fields of uneven N
"""
import math

import numpy as np
import torch

from stencilfft_b200 import Batch, Plan
from stencilfft_b200.abi import ZM_SPECTRAL_GAUSSIAN, ZM_SPECTRAL_POISSON

CDT = {"c64": torch.complex64, "c128": torch.complex128}
RDT = {"c64": torch.float32, "c128": torch.float64}


# ------------------------------------------------------------------ the cases
def _c(name, kind, dim, n, p, b, dtype, **more):
    return {"name": name, "kind": kind, "dim": dim, "n": n, "p": p, "b": b, "dtype": dtype, **more}


def listed():
    return [
        # the smallest field of the reference's 2D sweep: a call's fixed cost
        _c("rt_2d_n64_c128", "round_trip", 2, 64, 2, 4, "c128"),
        # the plain method at its small size, the reference's only precision
        _c("rt_2d_n1024_c128", "round_trip", 2, 1024, 2, 32, "c128"),
        # the benchmark's step: the large 2D field in the bulk precision
        _c("step_2d_n16384_c64", "step", 2, 16384, 4, 64, "c64"),
        # the same step on a large complex128 field
        _c("step_2d_n8192_c128", "step", 2, 8192, 4, 32, "c128"),
        # the 3D precision form at its size
        _c("rt_3d_n512_c64", "round_trip", 3, 512, 4, 32, "c64"),
        # a middle 3D field with short blocks, complex128
        _c("rt_3d_n256_c128", "round_trip", 3, 256, 4, 16, "c128"),
        # a small 3D field in the reference's own buffer contract (3D sweep)
        _c("inplace_3d_n64_c64", "in_place", 3, 64, 2, 8, "c64"),
        # gradient of a spectral-solve loss through the adjoint entry points
        _c("adjoint_2d_n4096_c64", "adjoint", 2, 4096, 4, 32, "c64"),
        # a user's natural-order array filtered on a layout of the 2D sweep's other blocks
        _c("filter_2d_n2048_c64", "filter", 2, 2048, 2, 16, "c64"),
        # finite differences alone, complex and real, as a time step without transforms has them
        _c("stencils_2d_n4096_c128", "stencils", 2, 4096, 4, 64, "c128"),
        # many small Poisson problems of uneven size in one call, blocks N / 8 at P = 2
        {"name": "batch_poisson96_c64", "kind": "batch", "dtype": "c64", "p": 2, "blocks": 8,
         "counts": "256:32,512:32,1024:24,2048:8"},
        # an odd number of uneven complex128 fields, short blocks on a wider grid
        {"name": "batch_fft29_c128", "kind": "batch_fft", "dtype": "c128", "p": 4, "blocks": 32,
         "counts": "128:9,256:11,512:6,1024:3"},
    ]


def draw(rng):
    kind = rng.choice(["round_trip", "round_trip", "round_trip", "step", "in_place", "filter", "poisson",
                       "adjoint", "stencils", "batch", "batch_fft"])
    dtype = rng.choice(["c64", "c128"])
    if kind in ("batch", "batch_fft"):
        # n / b = blocks, at least p^2 (the layout's constraint) and at most the smallest n
        p = rng.choice([1, 2, 2, 4])
        sizes = sorted(rng.sample([64, 128, 256, 512, 1024, 2048], rng.randint(1, 4)))
        blocks = 2 ** rng.randint(int(math.log2(p * p)), 6)
        parts = []
        for n in sizes:
            top = max(1, min(64, (1 << 24) // (n * n)))
            parts.append(f"{n}:{max(1, round(2 ** rng.uniform(0, math.log2(top))))}")
        return {"kind": kind, "dtype": dtype, "p": p, "blocks": blocks, "counts": ",".join(parts)}
    dim = 2 if kind in ("step", "stencils") else rng.choice([2, 2, 3])
    top = 13 if dtype == "c64" and kind != "adjoint" else 12     # (no dearer than the listed ones)
    n = 2 ** (rng.randint(6, top) if dim == 2 else rng.randint(4, 8))
    p = rng.choice([p for p in (1, 2, 2, 4, 4, 8) if p * p <= n])
    lo = 1 if kind in ("step", "stencils") else 0      # the reference's dx / dy take B >= 2
    hi = int(math.log2(n // (p * p)))
    b = 2 ** rng.randint(min(lo, hi), hi)
    if b < 2 and lo:                                   # (p too wide for a block of 2)
        p, b = 2, 2 ** rng.randint(1, int(math.log2(n // 4)))
    return {"kind": kind, "dim": dim, "n": n, "p": p, "b": b, "dtype": dtype}


# ------------------------------------------- the layouts, in plain torch (zmodel/utils.h)
def _to_real(x, dim, n, p, b):
    """natural (N,)*dim -> real-space layout: global index = (block cycle, rank, in block)."""
    v = n // (p * b)
    y = x.reshape(*([v, p, b] * dim))
    if dim == 2:
        return y.permute(1, 4, 0, 2, 5, 3).reshape(-1)
    return y.permute(1, 4, 7, 0, 2, 3, 5, 8, 6).reshape(-1)


def _to_recip(x, dim, n, p, b):
    """natural spectrum (N,)*dim -> reciprocal layout: frequency = (k1, rank, k2 in rank)."""
    m, vp = b * p, n // (p * b) // p
    y = x.reshape(*([m, p, vp] * dim))
    if dim == 2:
        return y.permute(1, 4, 3, 5, 0, 2).reshape(-1)
    return y.permute(1, 4, 7, 3, 5, 6, 8, 0, 2).reshape(-1)


def _k2(dim, n, dev):
    """|k|^2 of the signed integer frequencies on the natural grid."""
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev) ** 2
    return k[:, None] + k[None, :] if dim == 2 else k[:, None, None] + k[None, :, None] + k[None, None, :]


# -------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _gauss(case, seed, shape):
    """N(0, 1) real and imaginary parts in the case's precision."""
    return torch.randn(shape, dtype=CDT[case["dtype"]], device="cuda", generator=_gen(seed)) * math.sqrt(2.0)


def _modes(case, seed):
    """A sum of 32 seeded Fourier modes (|k| <= N / 8) plus 1e-3 noise, natural order."""
    n = case["n"]
    rng = np.random.default_rng(seed)
    x = torch.randn((n, n), dtype=CDT[case["dtype"]], device="cuda", generator=_gen(seed)) * (1e-3 * math.sqrt(2.0))
    i = torch.arange(n, device="cuda")
    one = torch.ones(n, dtype=torch.float64, device="cuda")

    def wave(k):
        return torch.polar(one, (int(k) * i % n).to(torch.float64) * (2 * math.pi / n))

    cols, rows = [], []
    for kx, ky in rng.integers(-(n // 8), n // 8 + 1, (32, 2)):
        rows.append(complex(rng.standard_normal(), rng.standard_normal()) * wave(ky))
        cols.append(wave(kx))
    x += (torch.stack(rows, 1) @ torch.stack(cols, 0)).to(x.dtype)
    return x


def _fields(case):
    """(ns, bs, ps) of a batch case."""
    ns = [int(n) for part in case["counts"].split(",") for n, c in [part.split(":")] for _ in range(int(c))]
    return ns, [n // case["blocks"] for n in ns], [case["p"]] * len(ns)


def _natural(case, seed):
    """The case's input field in natural order."""
    if case["kind"] == "step":
        return _modes(case, seed)
    return _gauss(case, seed, (case["n"],) * case["dim"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "batch_fft"):
        ns, bs, ps = _fields(case)
        bt = Batch(ns, bs, ps, dtype=case["dtype"])
        x = _gauss(case, seed, (bt.total,))
        return {"case": case, "batch": bt, "x": x, "a": bt.empty().zero_(), "b": bt.empty().zero_(),
                "work": bt.empty()}
    dim, n, p, b = case["dim"], case["n"], case["p"], case["b"]
    plan = Plan(dim, n, b, p, dtype=case["dtype"])
    st = {"case": case, "plan": plan, "scale": 1.0 / float(n) ** dim}
    x = _natural(case, seed)
    st["x"] = x if kind == "filter" else _to_real(x, dim, n, p, b).contiguous()
    del x
    bufs = {"round_trip": 4, "step": 6, "in_place": 1, "filter": 5, "poisson": 3, "adjoint": 5, "stencils": 3}
    st["bufs"] = [plan.empty() for _ in range(bufs[kind])]
    if kind == "adjoint":
        st["target"] = _gauss(case, seed + 1, (plan.total,))
    if kind == "stencils":
        st["r"] = torch.randn(plan.total, dtype=RDT[case["dtype"]], device="cuda", generator=_gen(seed + 1))
        st["rbufs"] = [plan.empty(real=True) for _ in range(2)]
    return st


# ---------------------------------------------------------------------- a pass
def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "batch":
        bt = state["batch"]
        bt.poisson(state["x"], state["a"], state["b"], state["work"], length=1.0)
        return [state["a"], state["b"]]
    if kind == "batch_fft":
        bt = state["batch"]
        bt.forward_fft(state["x"], state["a"])
        bt.inverse_fft(state["a"], state["b"], work=state["work"])
        return [state["a"], state["b"]]
    plan, x, bufs, scale, n = state["plan"], state["x"], state["bufs"], state["scale"], case["n"]
    if kind == "round_trip":
        spec, back, lap, work = bufs
        plan.forward_fft(x, spec, work=work)
        plan.inverse_fft(spec, back, scale=scale, work=work)
        plan.laplace(x, lap)
        return [spec, back, lap]
    if kind == "step":
        spec, back, lap, gx, gy, work = bufs
        plan.forward_fft(x, spec, work=work)
        plan.inverse_fft(spec, back, scale=scale, work=work)
        plan.laplace_dx_dy(back, lap, gx, gy, inv_h2=float(n) ** 2, delta=1.0 / n)
        return [spec, back, lap, gx, gy]
    if kind == "in_place":
        plan.forward_fft(x, bufs[0])
        plan.inverse_fft(bufs[0], x, scale=scale)
        return [x]
    if kind == "filter":
        real, spec, nat, back, work = bufs
        plan.natural_to_real(x, real)
        plan.forward_fft(real, spec, work=work)
        plan.reciprocal_to_natural(spec, nat)
        plan.spectral_apply(spec, ZM_SPECTRAL_GAUSSIAN, n / 16.0)
        plan.inverse_fft(spec, real, scale=scale, work=work)
        plan.real_to_natural(real, back)
        return [nat, back]
    if kind == "poisson":
        spec, phi, work = bufs
        plan.forward_fft(x, spec, work=work)
        plan.spectral_apply(spec, ZM_SPECTRAL_POISSON, 2.0 * math.pi)
        plan.inverse_fft(spec, phi, scale=scale, work=work)
        return [phi]
    if kind == "adjoint":
        # L = ||Lap(IFFT(G FFT(u))) - t||^2, dL/du = FFT^H G IFFT^H Lap^T (2 (y - t))
        spec, v, y, work, grad = bufs
        plan.forward_fft(x, spec, work=work)
        plan.spectral_apply(spec, ZM_SPECTRAL_GAUSSIAN, n / 16.0)
        plan.inverse_fft(spec, v, scale=scale, work=work)
        plan.laplace(v, y)
        torch.sub(y, state["target"], out=v)
        v.mul_(2.0)
        plan.laplace_vjp(v, grad)
        plan.inverse_fft_vjp(grad, spec, scale=scale, work=work)
        plan.spectral_apply_vjp(spec, ZM_SPECTRAL_GAUSSIAN, n / 16.0)
        plan.forward_fft_vjp(spec, grad, work=work)
        return [y, grad]
    lap, gx, gy = bufs
    rx, ry = state["rbufs"]
    plan.laplace(x, lap, inv_h2=float(n) ** 2)
    plan.dx(x, gx, delta=1.0 / n)
    plan.dy(x, gy, delta=1.0 / n)
    plan.dx(state["r"], rx, delta=1.0 / n)
    plan.dy(state["r"], ry, delta=1.0 / n)
    return [lap, gx, gy, rx, ry]


# ---------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    eb = 8 if case["dtype"] == "c64" else 16
    if kind in ("batch", "batch_fft"):
        ns = _fields(case)[0]
        elems = sum(n * n for n in ns)
        fft = sum(5.0 * n * n * math.log2(n * n) for n in ns)
        # one input, two outputs; two transforms (and the pointwise steps)
        return {"bytes": 3 * elems * eb, "flops": 2 * fft + (20.0 * elems if kind == "batch" else 2.0 * elems)}
    elems = case["n"] ** case["dim"]
    field = elems * eb
    fft = 5.0 * elems * math.log2(elems)
    lap = (10.0 if case["dim"] == 2 else 14.0) * elems
    diff = 12.0 * elems                      # one 4th-order difference of a complex field
    # (fields read and written, flops)
    fields, flops = {
        "round_trip": (4, 2 * fft + lap),
        "step": (6, 2 * fft + lap + 2 * diff),
        "in_place": (2, 2 * fft),
        "filter": (3, 2 * fft + 12.0 * elems),
        "poisson": (2, 2 * fft + 12.0 * elems),
        "adjoint": (4, 4 * fft + 2 * lap + 28.0 * elems),
        "stencils": (5.5, lap + 3 * diff),   # a complex field to three, a real one to two
    }[kind]
    return {"bytes": int(fields * field), "flops": flops}


# -------------------------------------------------------------- 64-bit values
def _lap(x):
    out = -2.0 * x.dim() * x
    for d in range(x.dim()):
        out += torch.roll(x, 1, d)
        out += torch.roll(x, -1, d)
    return out


def _diff(x, d, delta):
    """4th-order central difference along axis d."""
    y = torch.roll(x, 1, d).mul_(-8.0)
    y += torch.roll(x, -1, d).mul_(8.0)
    y += torch.roll(x, 2, d)
    y -= torch.roll(x, -2, d)
    return y.div_(12.0 * delta)


def _from_real(e, dim, n, p, b):
    """real-space layout -> natural, the inverse of _to_real."""
    v = n // (p * b)
    y = e.reshape(*([p] * dim), *([v, b] * (dim - 1)), b, v)
    if dim == 2:
        return y.permute(2, 0, 3, 5, 1, 4).reshape(n, n)
    return y.permute(3, 0, 4, 5, 1, 6, 8, 2, 7).reshape(n, n, n)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "batch_fft"):
        return _exact_batch(case, seed)
    dim, n, p, b = case["dim"], case["n"], case["p"], case["b"]
    x = _natural(case, seed).to(torch.complex128)
    axes = tuple(range(dim))

    def real(t):
        return _to_real(t, dim, n, p, b)

    if kind == "in_place":
        return [real(x)]
    if kind in ("round_trip", "step"):
        out = [_to_recip(torch.fft.fftn(x), dim, n, p, b), real(x)]
        if kind == "round_trip":
            return out + [real(_lap(x))]
        out.append(real(_lap(x).mul_(float(n) ** 2)))
        return out + [real(_diff(x, 1, 1.0 / n)), real(_diff(x, 0, 1.0 / n))]
    if kind == "stencils":
        r = torch.randn(n ** dim, dtype=RDT[case["dtype"]], device="cuda", generator=_gen(seed + 1))
        r = _from_real(r.to(torch.float64), dim, n, p, b)
        out = [real(_lap(x).mul_(float(n) ** 2))]
        for f in (x, r):
            out += [real(_diff(f, 1, 1.0 / n)), real(_diff(f, 0, 1.0 / n))]
        return out
    spec = torch.fft.fftn(x)
    k2 = _k2(dim, n, x.device)
    if kind == "poisson":
        k2 *= -(2.0 * math.pi) ** 2
        spec = spec / torch.where(k2 == 0, torch.ones_like(k2), k2)
        spec[(0,) * dim] = 0
        return [real(torch.fft.ifftn(spec))]
    g = torch.exp(-k2 / (2.0 * (n / 16.0) ** 2))
    if kind == "filter":
        return [spec.reshape(-1), torch.fft.ifftn(spec * g).reshape(-1)]
    y = _lap(torch.fft.ifftn(spec * g))
    t = _from_real(_gauss(case, seed + 1, (n ** dim,)).to(torch.complex128), dim, n, p, b)
    # every factor is self-adjoint up to the transforms' scales, which cancel
    grad = torch.fft.ifftn(torch.fft.fftn(_lap(2.0 * (y - t)), dim=axes) * g, dim=axes)
    return [real(y), real(grad)]


def _exact_batch(case, seed):
    """Field by field; elements between fields (alignment padding) stay zero."""
    ns, bs, ps = _fields(case)
    bt = Batch(ns, bs, ps, dtype=case["dtype"])
    offsets, total = [f["offset"] for f in bt.fields], bt.total
    bt.close()
    x = _gauss(case, seed, (total,)).to(torch.complex128)
    first, second = torch.zeros_like(x), torch.zeros_like(x)
    for n, b, p, o in zip(ns, bs, ps, offsets):
        f = x[o:o + n * n]
        if case["kind"] == "batch_fft":
            first[o:o + n * n] = _to_recip(torch.fft.fft2(_from_real(f, 2, n, p, b)), 2, n, p, b)
            second[o:o + n * n] = f
            continue
        r = _from_real(f, 2, n, p, b)
        k2 = _k2(2, n, x.device) * -(2.0 * math.pi) ** 2
        spec = torch.fft.fft2(r) / torch.where(k2 == 0, torch.ones_like(k2), k2)
        spec[0, 0] = 0
        phi = torch.fft.ifft2(spec)
        first[o:o + n * n] = _to_real(phi, 2, n, p, b)
        second[o:o + n * n] = _to_real(_lap(phi) * float(n) ** 2 - r, 2, n, p, b)
    return [first, second]
