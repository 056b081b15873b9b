"""Float64 lines that do not grow like noise (a dominant mean, a ramp, a tone, few
points among zeros) on the integer-float stages, power-of-two and smooth
lengths, every operation of those passes.  Bound per line: the double-float
stages' error of such lines, 1.3e-14 at most (tests/test_xf_lines.py, which
holds the integer-float ones below it), and two conversions of 2^-50: 1.5e-14;
R2R lines have twiddles at their ends as well: 2e-14.  Spectra of fields with a
mean, power-of-two lines: sqrt(n) 2^-50 and the conversions."""
import numpy as np
import pytest

import pencilffts_gb300 as P
from helpers import oracle_plan

T = P.Transforms
pytestmark = pytest.mark.gpu


def _lines(n, cplx):
    """One line of each kind, along axis 0."""
    rng = np.random.default_rng(n)
    j = np.arange(n)
    noise = rng.standard_normal((n, 7))
    if cplx:
        noise = noise + 1j * rng.standard_normal((n, 7))
    x = noise.copy()
    x[:, 0] += 10
    x[:, 1] += 1000
    x[:, 2] = j / n
    x[:, 3] += 30 * (np.exp(2j * np.pi * 3 * j / n) if cplx else np.cos(2 * np.pi * 3 * j / n))
    x[:, 4] = np.where(j == n // 3, noise[:, 4], 0)
    x[:, 5] = np.where(j % (n // 8 + 1) == 0, noise[:, 5], 0)
    return x


def _apply(tr, x, permute):
    plan = P.PencilFFTPlan(x.shape, (tr, T.NoTransform()), np.float64, permute_dims=permute, extra_dims=(4,))
    u = plan.allocate_input()
    u.copy_from_logical(np.stack([x] * 4, axis=2))  # 28 lines: the smooth-length pass from 16 complex ones on
    return plan, (plan * u).to_logical()


def _check(y, ref, bound, what):
    for c in range(4):
        err = np.linalg.norm(y[:, :, c] - ref, axis=0) / np.linalg.norm(ref, axis=0)
        assert (err <= bound).all(), (what, c, err)


@pytest.mark.parametrize("n", [128, 512, 1000, 1024, 2048, 4096, 243, 729, 2025, 2560])
def test_xf_lines_that_do_not_grow_like_noise(cuda, n):
    x, r = _lines(n, True), _lines(n, False)
    for permute in (True, False):
        _check(_apply(T.FFT(), x, permute)[1], np.fft.fft(x, axis=0), 1.5e-14, "c2c")
        plan, y = _apply(T.RFFT(), np.repeat(r, 2, axis=1), permute)
        _check(y, np.repeat(np.fft.rfft(r, axis=0), 2, axis=1), 1.5e-14, "r2c")
        # c2r: the same kinds of lines as half spectra
        s = x[: n // 2 + 1].copy()
        s[0] = s[0].real
        if n % 2 == 0:
            s[-1] = s[-1].real
        S = plan.allocate_output()
        S.copy_from_logical(np.stack([np.repeat(s, 2, axis=1)] * 4, axis=2))
        _check(plan.ldiv(S).to_logical(), np.repeat(np.fft.irfft(s, n, axis=0), 2, axis=1), 1.5e-14, "c2r")


@pytest.mark.parametrize("n", [64, 256, 512, 1024, 4096])
def test_xf_spectra_of_fields_with_a_mean(cuda, n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 12)) + np.repeat([10.0, 1000.0, 0.5], 4)
    x[:, 8:] = rng.random((n, 4))
    for tr in (T.FFT(), T.RFFT()):
        f = x.astype(complex) if isinstance(tr, T.FFT) else x
        plan = P.PencilFFTPlan(x.shape, (tr, T.NoTransform()), np.float64)
        S = plan.allocate_output()
        S.copy_from_logical(np.fft.fft(f, axis=0) if isinstance(tr, T.FFT) else np.fft.rfft(f, axis=0))
        _check(plan.ldiv(S).to_logical()[:, :, None].repeat(4, axis=2), f, (n ** 0.5 + 2) * 2.0 ** -50, tr)


@pytest.mark.parametrize("kind,n", [(T.REDFT10, 729), (T.RODFT10, 1000), (T.REDFT01, 729), (T.DHT, 1215), (T.REDFT00, 730),
                                    (T.RODFT00, 999), (T.REDFT11, 500), (T.REDFT11, 1024), (T.REDFT10, 4096),
                                    (T.REDFT01, 4096), (T.REDFT00, 2049)])
def test_xf_r2r_lines_that_do_not_grow_like_noise(cuda, kind, n):
    r = np.repeat(_lines(n, False), 2, axis=1)  # (two real lines share a unit)
    plan, y = _apply(T.R2R(kind), r, False)
    ref = oracle_plan(plan).forward(np.stack([r] * 4, axis=2))
    _check(y, ref[:, :, 0], 2e-14, kind)
