"""Timed cases of the transform path: what programs built on pencil FFT plans
run, through the package's public entry points.

One pass is the loop body of such a program: a forward transform and its
normalised inverse (``mul_`` then ``ldiv_``, the reference's benchmark loop), a
spectral gradient or divergence, or one launch of a recorded batch.  Every
kind draws its sizes over the range that the framework plans in one go:
powers of two (the usual choice for turbulence boxes), smooth sizes (products
of 2, 3, 5 and 7) and arbitrary ones (primes included).
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "pencilffts.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import pencilffts_gb300 as P  # noqa: E402

T = P.Transforms
TWO_PI = 2 * math.pi

# FFTW kind codes of the real-to-real transforms, with the pairs that a
# Chebyshev, cosine or sine solver uses
R2R_KINDS = {"DHT": 2, "REDFT00": 3, "REDFT10": 5, "REDFT11": 6, "RODFT00": 7, "RODFT10": 9, "RODFT11": 10}


def _case(kind, dims, real, **more):
    return {"kind": kind, "dims": "x".join(map(str, dims)), "real": real, **more}


def _named(name, case):
    return {"name": name, **case}


def listed():
    return [
        # a small box, as in unit tests, tutorials and reduced-order models: every launch shows
        _named("rfft_f64_16x32x64", _case("rfft", (16, 32, 64), "f64")),
        # the headline of the reference's benchmark: a pseudo-spectral step's transform pair
        _named("rfft_f64_512", _case("rfft", (512, 512, 512), "f64")),
        # complex fields (Schroedinger, Gross-Pitaevskii solvers)
        _named("fft_c128_256", _case("fft", (256, 256, 256), "f64")),
        # single-precision turbulence box
        _named("rfft_f32_512", _case("rfft", (512, 512, 512), "f32")),
        # the largest box
        _named("rfft_f32_1024", _case("rfft", (1024, 1024, 1024), "f32")),
        # channel flow: two periodic directions and a Chebyshev one
        _named("channel_f64_512x512x257", _case("channel", (512, 512, 257), "f64", r2r="REDFT00")),
        # derivatives of a vector field, one per component
        _named("gradient_f32_384", _case("gradient", (384, 384, 384), "f32")),
        # a stack of unrelated fields recorded once and replayed (ensembles, patches of an adaptive grid)
        _named("batch_f32_16_uneven", _case("batch", (16,), "f32", low=48, high=192, draw=2024)),
        # in-place padded buffer at sizes picked for resolution and not for speed
        _named("rfft_inplace_f64_uneven", _case("rfft_inplace", (200, 180, 150), "f64")),
        # cosine solver (Neumann walls) on a vector field
        _named("dct_f64_vector_128x96x100", _case("r2r", (128, 96, 100), "f64", r2r="REDFT10", extra=3)),
        # long records: spectra of time series
        _named("rfft_f64_16384x4096", _case("rfft", (16384, 4096), "f64")),
        # incompressibility check / pressure source: divergence of a spectral vector field
        _named("divergence_f64_240", _case("divergence", (240, 240, 240), "f64")),
    ]


# ---------------------------------------------------------------------------
# Drawn sizes
# ---------------------------------------------------------------------------
def _smooth(n):
    """The 7-smooth size nearest to n."""
    def ok(k):
        for p in (2, 3, 5, 7):
            while k % p == 0:
                k //= p
        return k == 1
    for d in range(n):
        for k in (n - d, n + d):
            if k >= 2 and ok(k):
                return k
    return n


def _size(rng, style, low, high):
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    n = min(max(n, low), high)
    if style == "pow2":
        return 1 << max(3, int(round(math.log2(n))))
    if style == "smooth":
        return _smooth(n)
    return n


def _dims(rng, style, points):
    """Two or three dimensions of about `points` points."""
    nd = rng.choice((2, 3, 3, 3))
    side = points ** (1.0 / nd)
    dims, left = [], points
    for k in range(nd - 1):
        n = _size(rng, style, max(8, int(side / 2)), max(9, int(side * 2)))
        dims.append(n)
        left /= n
    last = max(8.0, min(left, 4096.0))
    dims.append(_size(rng, style, max(8, int(last * 0.9)), max(9, int(last * 1.1))))
    rng.shuffle(dims)
    return dims


def draw(rng):
    kind = rng.choice(("rfft", "rfft", "rfft", "fft", "fft", "rfft_inplace", "channel", "gradient", "r2r", "batch",
                       "divergence", "long"))
    real = rng.choice(("f32", "f64"))
    if kind == "batch":
        low = rng.randint(16, 64)
        return _case("batch", (rng.randint(4, 16),), "f32", low=low, high=low * rng.randint(2, 3), draw=rng.randrange(1 << 20))
    if kind == "long":
        n = _size(rng, rng.choice(("pow2", "smooth")), 4500, 65536)
        lines = int(math.exp(rng.uniform(math.log(16), math.log((1 << 25) / n))))
        return _case(rng.choice(("rfft", "fft")), (n, lines), real)
    style = rng.choice(("pow2", "pow2", "smooth", "smooth", "any"))
    most = {"pow2": 1 << 26, "smooth": 1 << 24, "any": 1 << 23}[style]
    if kind in ("channel", "gradient", "r2r", "divergence"):
        most >>= 2
    dims = _dims(rng, style, math.exp(rng.uniform(math.log(1 << 13), math.log(most))))
    if kind in ("gradient", "divergence", "channel") and len(dims) == 2:
        dims = [dims[0], dims[1], 8]
    if kind == "channel":
        dims[2] = rng.choice((17, 33, 65, 129, 97))
        return _case(kind, dims, real, r2r="REDFT00")
    if kind == "r2r":
        return _case(kind, dims, real, r2r=rng.choice(sorted(R2R_KINDS)), extra=rng.choice((1, 3)))
    return _case(kind, dims, real)


# ---------------------------------------------------------------------------
# Inputs, plans and passes
# ---------------------------------------------------------------------------
def _parse(case):
    dims = tuple(int(x) for x in case["dims"].split("x"))
    return dims, (np.float64 if case["real"] == "f64" else np.float32), (torch.float64 if case["real"] == "f64" else torch.float32)


def _batch_dims(case):
    r = np.random.default_rng(case["draw"])
    return [tuple(int(s) for s in r.integers(case["low"], case["high"] + 1, 3)) for _ in range(_parse(case)[0][0])]


def _normal(shape, dtype, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.randn(shape, generator=g, dtype=dtype, device="cuda")


def _complex_dtype(dtype):
    return torch.complex128 if dtype == torch.float64 else torch.complex64


def _field(shape, dtype, seed, cplx):
    """A field in memory order (dimension 1 fastest): N(0, 1), as velocity and
    scalar fields are after scaling."""
    if not cplx:
        return _normal(shape, dtype, seed)
    return torch.view_as_complex(_normal(tuple(shape) + (2,), dtype, seed))


def _transforms(case):
    kind = case["kind"]
    if kind in ("rfft", "gradient", "divergence", "batch"):
        return T.RFFT()
    if kind == "fft":
        return T.FFT()
    if kind == "rfft_inplace":
        return T.RFFT_()
    r = T.R2R(R2R_KINDS[case["r2r"]])
    return (T.RFFT(), T.FFT(), r) if kind == "channel" else r


def _extra(case):
    return (case["extra"],) if case.get("extra", 1) > 1 else ()


def _memory_shape(dims, extra=()):
    return tuple(reversed(tuple(dims) + tuple(extra)))


def prepare(case, seed):
    dims, real, dtype = _parse(case)
    kind = case["kind"]
    if kind == "batch":
        ops, fields = [], []
        for k, d in enumerate(_batch_dims(case)):
            plan = P.PencilFFTPlan(d, T.RFFT(), real)
            u, v, w = plan.allocate_input(), plan.allocate_output(), plan.allocate_input()
            u.data.copy_(_field(_memory_shape(d), dtype, seed * 131 + k, False))
            ops += [(P.mul_, v, plan, u), (P.ldiv_, w, plan, v)]
            fields.append((v, w))
        return {"kind": kind, "batch": P.Batch(ops), "fields": fields}
    plan = P.PencilFFTPlan(dims, _transforms(case), real, extra_dims=_extra(case))
    st = {"kind": kind, "plan": plan}
    if kind == "rfft_inplace":
        st["u"] = plan.allocate_input()
        st["u"].first().data[..., :dims[0]].copy_(_field(_memory_shape(dims), dtype, seed, False))
    elif kind == "gradient":
        st["u"], st["v"], st["w"] = plan.allocate_input(P.Val(3)), plan.allocate_output(P.Val(3)), plan.allocate_input(P.Val(3))
        for c in range(3):
            st["u"][c].data.copy_(_field(_memory_shape(dims), dtype, seed * 3 + c, False))
    elif kind == "divergence":
        # the solver's state: spectra of a real vector field
        st["v"], st["w"] = plan.allocate_output(P.Val(3)), plan.allocate_input()
        for c in range(3):
            st["v"][c].data.copy_(_spectrum(case, seed * 3 + c).to(st["v"][c].data.dtype))
    else:
        st["u"], st["v"], st["w"] = plan.allocate_input(), plan.allocate_output(), plan.allocate_input()
        st["u"].data.copy_(_field(_memory_shape(dims, _extra(case)), dtype, seed, kind == "fft"))
    return st


def run(st):
    kind = st["kind"]
    if kind == "batch":
        st["batch"].launch()
        return [(v.data, w.data) for v, w in st["fields"]]
    plan = st["plan"]
    if kind == "rfft_inplace":
        P.mul_(st["u"], plan, st["u"])
        P.ldiv_(st["u"], plan, st["u"])
        return st["u"].first().logical()
    if kind == "gradient":
        for c in range(3):
            P.mul_(st["v"][c], plan, st["u"][c])
            P.ldiv_(st["w"][c], plan, st["v"][c], deriv=(c + 1, TWO_PI))
        return [(v.data, w.data) for v, w in zip(st["v"], st["w"])]
    if kind == "divergence":
        P.ldiv_divergence_(st["w"], plan, st["v"], (TWO_PI, TWO_PI, TWO_PI))
        return st["w"].data
    P.mul_(st["v"], plan, st["u"])
    P.ldiv_(st["w"], plan, st["v"])
    return st["v"].data, st["w"].data


# ---------------------------------------------------------------------------
# Bytes and operations that a pass cannot do without
# ---------------------------------------------------------------------------
def _fft_flops(points, cplx):
    return (5.0 if cplx else 2.5) * points * math.log2(max(2, points))


def work(case):
    dims, real, dtype = _parse(case)
    kind, rb = case["kind"], np.dtype(real).itemsize
    if kind == "batch":
        every = [work({**case, "kind": "rfft", "dims": "x".join(map(str, d))}) for d in _batch_dims(case)]
        return {k: sum(w[k] for w in every) for k in ("bytes", "flops")}
    n = math.prod(dims) * case.get("extra", 1)
    half = (dims[0] // 2 + 1) * (n // dims[0])
    if kind == "fft":
        return {"bytes": 8 * rb * n, "flops": 2 * _fft_flops(n, True)}
    if kind == "r2r":
        return {"bytes": 4 * rb * n, "flops": 2 * _fft_flops(n, False)}
    if kind == "rfft_inplace":
        return {"bytes": 2 * (rb * n + 2 * rb * half), "flops": 2 * _fft_flops(n, False)}
    if kind == "divergence":
        return {"bytes": 3 * 2 * rb * half + rb * n, "flops": _fft_flops(n, False) + 3 * 8.0 * half}
    times = 3 if kind == "gradient" else 1
    return {"bytes": times * (2 * rb * n + 4 * rb * half), "flops": times * 2 * _fft_flops(n, False)}


# ---------------------------------------------------------------------------
# The same in 64 bits, with torch alone
# ---------------------------------------------------------------------------
def _r2r_matrix(kind, n):
    """The n x n matrix of FFTW's definition of an unnormalised real-to-real kind."""
    j = torch.arange(n, dtype=torch.int64, device="cuda")[None, :]
    k = torch.arange(n, dtype=torch.int64, device="cuda")[:, None]

    def cos(num, den):  # cos(pi num / den), the argument reduced exactly
        return torch.cos(math.pi * ((num % (2 * den)).double() / den))

    def sin(num, den):
        return torch.sin(math.pi * ((num % (2 * den)).double() / den))

    if kind == 2:
        return cos(2 * j * k, n) + sin(2 * j * k, n)
    if kind == 3:
        m = 2 * cos(j * k, n - 1)
        m[:, 0] /= 2
        m[:, -1] /= 2
        return m
    if kind == 5:
        return 2 * cos((2 * j + 1) * k, 2 * n)
    if kind == 6:
        return 2 * cos((2 * j + 1) * (2 * k + 1), 4 * n)
    if kind == 7:
        return 2 * sin((j + 1) * (k + 1), n + 1)
    if kind == 9:
        return 2 * sin((2 * j + 1) * (k + 1), 2 * n)
    if kind == 10:
        return 2 * sin((2 * j + 1) * (2 * k + 1), 4 * n)
    raise ValueError(kind)


def _apply_matrix(m, x, axis):
    """m along an axis of a real or complex tensor, in 64 bits."""
    x = x.movedim(axis, -1)
    if x.is_complex():
        y = torch.complex(x.real @ m.T, x.imag @ m.T)
    else:
        y = x @ m.T
    return y.movedim(-1, axis)


def _reverse(x, n):
    """The memory order of the plan's output: the transformed dimensions reversed."""
    lead = x.dim() - n
    return x.permute(*range(lead), *reversed(range(lead, x.dim()))).contiguous()


def _spectrum(case, seed):
    """The 64-bit spectrum of a real field, in the order of the plan's output."""
    dims, _, dtype = _parse(case)
    u = _field(_memory_shape(dims), dtype, seed, False).double()
    return _reverse(torch.fft.fftn(torch.fft.rfft(u, dim=-1), dim=tuple(range(len(dims) - 1))), len(dims))


def _forward64(x, nd):
    """rfft (real x) or fft over the last nd axes of a memory-order field."""
    axes = tuple(range(-nd, 0))
    if x.is_complex():
        return torch.fft.fftn(x, dim=axes)
    y = torch.fft.rfft(x, dim=-1)
    return torch.fft.fftn(y, dim=axes[:-1]) if nd > 1 else y


def _derivative64(dims, c, spec):
    """i k_c times a memory-order half spectrum of a 2 pi-periodic field."""
    n = dims[c]
    k = torch.fft.rfftfreq(n, 1.0 / n) if c == 0 else torch.fft.fftfreq(n, 1.0 / n)
    shape = [1] * len(dims)
    shape[len(dims) - 1 - c] = k.numel()
    return spec * (1j * k.double().to("cuda").reshape(shape))


def _inverse64(dims, spec):
    nd = len(dims)
    y = torch.fft.ifftn(spec, dim=tuple(range(-nd, -1))) if nd > 1 else spec.clone()
    y.imag[..., 0] = 0  # FFTW's c2r reads the real part of these two only
    if dims[0] % 2 == 0:
        y.imag[..., -1] = 0
    return torch.fft.irfft(y, n=dims[0], dim=-1)


def exact(case, seed):
    dims, real, dtype = _parse(case)
    kind, nd = case["kind"], len(dims)
    if kind == "batch":
        out = []
        for k, d in enumerate(_batch_dims(case)):
            u = _field(_memory_shape(d), dtype, seed * 131 + k, False).double()
            out.append((_reverse(_forward64(u, len(d)), len(d)), u))
        return out
    if kind == "gradient":
        out = []
        for c in range(3):
            u = _field(_memory_shape(dims), dtype, seed * 3 + c, False).double()
            s = _forward64(u, nd)
            out.append((_reverse(s, nd), _inverse64(dims, _derivative64(dims, c, s))))
        return out
    if kind == "divergence":
        cd = _complex_dtype(dtype)
        s = sum(_derivative64(dims, c, _reverse(_spectrum(case, seed * 3 + c).to(cd).to(torch.complex128), nd))
                for c in range(3))
        return _inverse64(dims, s)
    extra = _extra(case)
    u = _field(_memory_shape(dims, extra), dtype, seed, kind == "fft")
    u = u.to(torch.complex128) if u.is_complex() else u.double()
    if kind == "rfft_inplace":
        return u.permute(*reversed(range(nd)))
    if kind in ("rfft", "fft"):
        return _reverse(_forward64(u, nd), nd), u
    if kind == "channel":
        y = torch.fft.fft(torch.fft.rfft(u, dim=-1), dim=-2)
        return _reverse(_apply_matrix(_r2r_matrix(R2R_KINDS[case["r2r"]], dims[2]), y, 0), nd), u
    y = u
    for d in range(nd):
        y = _apply_matrix(_r2r_matrix(R2R_KINDS[case["r2r"]], dims[d]), y, u.dim() - 1 - d)
    return _reverse(y, nd), u
