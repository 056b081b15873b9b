"""Float64 power-of-two lines in the integer-float stages (pfgb_xf.cuh): lines
of different kinds side by side in one tile, along a contiguous and along a
strided axis.  Bound per line: 2^-47 for the stages (tests/test_xf_arith.py)
plus two conversions of at most 2^-50 each: 1e-14."""
import numpy as np
import pytest

import pencilffts_gb300 as P

T = P.Transforms
pytestmark = pytest.mark.gpu

KINDS = ("noise", "tone", "point", "zero", "large", "small", "nan", "inf")


def _lines(n, rng):
    """One line of each kind; their count (8) is not a multiple of every tile."""
    j = np.arange(n)
    noise = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    point = np.zeros(n, complex)
    point[n // 3] = 0.3 - 1.1j
    bad = noise.copy()
    bad[n // 2] = np.nan
    inf = noise.copy()
    inf[1] = np.inf
    return {"noise": noise, "tone": np.exp(2j * np.pi * ((3 * j) % n) / n) * 1e-3, "point": point,
            "zero": np.zeros(n, complex), "large": noise * 1e300, "small": noise * 1e-290, "nan": bad, "inf": inf}


@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("n", [8, 16, 64, 128, 512, 1024, 4096])
def test_xf_lines_of_every_kind(cuda, n, strided):
    lines = _lines(n, np.random.default_rng(n))
    x = np.stack([lines[k] for k in KINDS], axis=0 if strided else 1)
    tr = (T.NoTransform(), T.FFT()) if strided else (T.FFT(), T.NoTransform())
    for permute in (False, True):
        plan = P.PencilFFTPlan(x.shape, tr, np.float64, permute_dims=permute)
        u = plan.allocate_input()
        u.copy_from_logical(x)
        y = (plan * u).to_logical()
        for i, k in enumerate(KINDS):
            got = y[i] if strided else y[:, i]
            if k in ("nan", "inf"):
                assert not np.isfinite(got).any(), (n, k)
                continue
            s = 1e-300 if k == "large" else 1e290 if k == "small" else 1.0
            ref = np.fft.fft(lines[k] * s)
            err = np.linalg.norm(got * s - ref)
            assert err <= 1e-14 * np.linalg.norm(ref), (n, k, permute, err / max(np.linalg.norm(ref), 1e-300))


@pytest.mark.parametrize("dims", [(16, 6, 10), (64, 5, 3), (512, 3, 2)])
def test_xf_normalisation_that_is_no_power_of_two(cuda, dims):
    """The ldiv! factor as a product in xf: 1 / (n1 n2 n3) with odd factors on
    the double outputs of a c2r pass and of a c2c pass."""
    rng = np.random.default_rng(3)
    for tr in (T.RFFT(), T.FFT()):
        plan = P.PencilFFTPlan(dims, tr, np.float64)
        x = rng.standard_normal(dims)
        if isinstance(tr, T.FFT):
            x = x + 1j * rng.standard_normal(dims)
        u = plan.allocate_input()
        u.copy_from_logical(x)
        back = plan.ldiv(plan * u).to_logical()
        assert np.linalg.norm(back - x) <= 1e-13 * np.linalg.norm(x)
