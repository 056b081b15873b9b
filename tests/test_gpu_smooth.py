"""Smooth-length pass (sm_pass): lengths of 2, 3, 5 and 7 only, against the
oracle at the repository's bounds (Float64 1e-13, Float32 2e-6)."""
import numpy as np
import pytest

import pencilffts_gb300 as P
from helpers import TOL, oracle_plan, random_input, rel
from oracle import pencilfft_oracle as O
from test_gpu_parity import check_plan


T = P.Transforms
pytestmark = pytest.mark.gpu
F32, F64 = np.float32, np.float64


def kernels(plan):
    A, B = plan.allocate_input(), None
    A.fill_(0)
    plan.set_timing(True)
    B = plan * A
    plan.ldiv(B)
    k = {e["kernel"].split("<")[0] for e in plan.get_timing()}
    plan.set_timing(False)
    return k


# one stage; every radix; odd, prime powers; five and six stages; above 2048
# points: Float32 lines only (and 2560, five times a power of two); the longest
@pytest.mark.parametrize("real", [F64, F32])
@pytest.mark.parametrize("n", [6, 9, 10, 14, 15, 18, 25, 35, 49, 60, 100, 135, 243, 343, 700, 729, 1000, 1215, 2025,
                               2187, 2560, 3456, 4050, 4032])
def test_sm_lines(cuda, real, n):
    """Contiguous and strided lines, both output orders, r2c / c2r and c2c;
    34 and 19 real lines (an odd pair, partial tiles)."""
    for tr in (T.FFT(), T.RFFT()):
        for dims, trs in (((n, 34), (tr, T.NoTransform())), ((19, n, 2), (T.NoTransform(), tr, T.NoTransform()))):
            for permute in (True, False):
                plan = P.PencilFFTPlan(dims, trs, real, permute_dims=permute)
                check_plan(plan, seed=n)
                assert ("sm_pass" in kernels(plan)) == (n <= 2048 or (real == F32) == (n != 2560))


@pytest.mark.parametrize("lines,few", [(15, True), (16, False), (17, False)])
def test_sm_line_count(cuda, lines, few):
    plan = P.PencilFFTPlan((100,), T.FFT(), F64, extra_dims=(lines,))
    check_plan(plan, seed=lines)
    assert kernels(plan) == {"bs_pass" if few else "sm_pass"}


@pytest.mark.parametrize("real", [F64, F32])
@pytest.mark.parametrize("dims", [(20, 18, 30), (45, 14, 20), (36, 50, 7)])
def test_sm_spectral_operators(cuda, real, dims):
    """i k on the input (each dimension: along, beside and outside the tile),
    on the output, and a divergence, on smooth lines."""
    plan = P.PencilFFTPlan(dims, T.RFFT(), real)
    orc = oracle_plan(plan)
    L = (2 * np.pi, 3.0, 5.0)
    xs = [random_input(plan, 7 + c) for c in range(3)]
    specs = [orc.forward(x) for x in xs]
    uF = []
    for s in specs:
        S = plan.allocate_output()
        S.copy_from_logical(s)
        uF.append(S)
    for d in range(3):
        U = plan.allocate_input()
        P.ldiv_(U, plan, uF[d], deriv=(d + 1, L[d]))
        assert rel(U.to_logical(), orc.ldiv(O.wavenumbers(orc, d, L[d]) * specs[d])) <= TOL[np.dtype(real)]
        A, B = plan.allocate_input(), plan.allocate_output()
        A.copy_from_logical(xs[d])
        P.mul_(B, plan, A, deriv=(d + 1, L[d]))
        assert rel(B.to_logical(), O.wavenumbers(orc, d, L[d]) * specs[d]) <= TOL[np.dtype(real)]
    div = plan.allocate_input()
    P.ldiv_divergence_(div, plan, uF, L)
    ref = orc.ldiv(sum(O.wavenumbers(orc, d, L[d]) * specs[d] for d in range(3)))
    assert rel(div.to_logical(), ref) <= TOL[np.dtype(real)]


def test_sm_lines_of_every_scale(cuda):
    """Float64 lines of very different magnitude in one tile, and one with a NaN."""
    n = 90
    rng = np.random.default_rng(2)
    x = rng.standard_normal((n, 20)) + 1j * rng.standard_normal((n, 20))
    x *= 10.0 ** np.linspace(-280, 290, 20)
    x[:, 7] = 0
    x[3, 11] = np.nan
    for strided in (False, True):
        a = x.T.copy() if strided else x
        trs = (T.NoTransform(), T.FFT()) if strided else (T.FFT(), T.NoTransform())
        plan = P.PencilFFTPlan(a.shape, trs, F64)
        u = plan.allocate_input()
        u.copy_from_logical(a)
        y = (plan * u).to_logical()
        y = y.T if strided else y
        for i in range(20):
            if i == 11:
                assert not np.isfinite(y[:, i]).any()
                continue
            s = 10.0 ** -np.linspace(-280, 290, 20)[i]
            ref = np.fft.fft(x[:, i] * s)
            assert np.linalg.norm(y[:, i] * s - ref) <= 2e-14 * np.linalg.norm(ref), i


def test_sm_in_place_and_batch(cuda):
    check_plan(P.PencilFFTPlan((45, 36, 20), T.RFFT_(), F64), seed=4)
    check_plan(P.PencilFFTPlan((60, 50), T.FFT_(), F32), seed=5)
    rng = np.random.default_rng(1)
    for form in ("graph", "persistent"):
        plans = [P.PencilFFTPlan(d, T.RFFT(), F32) for d in ((50, 60, 20), (63, 36, 45))]
        ops, keep = [], []
        for p in plans:
            u, v, w = p.allocate_input(), p.allocate_output(), p.allocate_input()
            x = rng.standard_normal(p.size()).astype(F32)
            u.copy_from_logical(x)
            ops += [(P.mul_, v, p, u), (P.ldiv_, w, p, v)]
            keep.append((p, x, v, w))
        b = P.Batch(ops, form=form)
        b.launch()
        for p, x, v, w in keep:
            assert rel(v.to_logical(), oracle_plan(p).forward(x)) <= 2e-6
            assert rel(w.to_logical(), x) <= 2e-6


# D2 / D3 (odd and even n), X and D4 lines: DFTs of 6 points to the longest of
# each type, odd extensions' zeros, one and several stages
@pytest.mark.parametrize("real", [F64, F32])
@pytest.mark.parametrize("kind,sizes", [(T.REDFT10, (6, 9, 25, 60, 100, 343, 1000)),
                                        (T.RODFT10, (6, 7, 63, 96, 500)),
                                        (T.REDFT01, (7, 10, 45, 120, 960)),
                                        (T.RODFT01, (6, 15, 50, 243)),
                                        (T.DHT, (6, 12, 35, 200, 2025)),
                                        (T.REDFT00, (4, 46, 97, 501, 1001)),
                                        (T.RODFT00, (2, 5, 44, 299, 999)),
                                        (T.REDFT11, (3, 5, 50, 105, 1000)),
                                        (T.RODFT11, (3, 6, 75, 1000))])
def test_sm_r2r_lines(cuda, real, kind, sizes):
    r = T.R2R(kind)
    for n in sizes + ((3000,) if real == F32 and kind in (T.REDFT10, T.RODFT01) else ()):
        for dims, trs in (((n, 19), (r, T.NoTransform())), ((18, n, 2), (T.NoTransform(), r, T.NoTransform())),
                          ((9, n), (T.FFT(), r)), ((n, 10), (r, T.FFT()))):
            plan = P.PencilFFTPlan(dims, trs, real, permute_dims=n % 2 == 0)
            check_plan(plan, seed=n)
            assert "sm_pass" in kernels(plan)


def test_sm_r2r_spectral_operator(cuda):
    """A derivative along a Fourier dimension, fused into the R2R pass at the
    plan's end (Float64), on its output and on its input."""
    plan = P.PencilFFTPlan((20, 18, 25), (T.RFFT(), T.FFT(), T.R2R(T.REDFT10)), F64)
    orc = oracle_plan(plan)
    x = random_input(plan, 3)
    spec = orc.forward(x)
    S = plan.allocate_output()
    S.copy_from_logical(spec)
    for d, L in ((0, 2 * np.pi), (1, 3.0)):
        A, B = plan.allocate_input(), plan.allocate_output()
        A.copy_from_logical(x)
        P.mul_(B, plan, A, deriv=(d + 1, L))
        assert rel(B.to_logical(), O.wavenumbers(orc, d, L) * spec) <= 1e-13
        P.ldiv_(A, plan, S, deriv=(d + 1, L))
        assert rel(A.to_logical(), orc.ldiv(O.wavenumbers(orc, d, L) * spec)) <= 1e-13
