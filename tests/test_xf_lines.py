"""Integer-float lines (pfgb_xf.cuh) against the double-float stages they stand
for, on the host: the stages of power-of-two and of smooth lengths compiled with
g++ from the same headers, over lines whose values do not grow like noise.

A double-float value keeps 48 bits of itself, an integer-float one a fraction of
the unit its whole line shares, so a dominant mean, a ramp or a few points among
zeros are where the second could lose.  Required: per kind of line, a relative
L2 error against long double no larger than that of the double-float stages on
the same lines (their rms over four lines a kind).

The spectrum of a field with a mean is one large value among small ones, and its
transform does not grow.  Its unit is the large value's 2^-26 to 2^-27, and a stage's
roundings (four of 2^-25 unit a value, 2^-50 of the large value together) add up
over the values that an output sums: M 2^-102 from the input, M/8 2^-100 (1 + 1/8 +
...) from the radix-8 stages, 0.63 sqrt(M) 2^-50 in all; double-float has about
2^-47.  Required of the power-of-two lines: sqrt(M) 2^-50."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pencilffts.jl_gb300" / "csrc"

DRIVER = r"""
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <random>
#include <type_traits>
#include <vector>
#include "pfgb_xf.cuh"
using namespace pfgb;
typedef long double ld;
typedef std::complex<ld> cld;
static const ld PI = acosl(-1.0L);
template <typename R> struct C { R re, im; };
template <typename R> C<R> operator+(C<R> a, C<R> b) { return {a.re + b.re, a.im + b.im}; }
template <typename R> C<R> operator-(C<R> a, C<R> b) { return {a.re - b.re, a.im - b.im}; }
template <typename R> C<R> mmi(C<R> a) { return {a.im, -a.re}; }
static ld val(xf a) { return (ld)a.h + (ld)a.l; }
static ld val(dd a) { return (ld)a.h + (ld)a.l; }
static xf mulc(xf a, double c) { return xf_mulc(a, c); }
static dd mulc(dd a, double c) { return a * dd(c); }
static xf half_root(xf a) { return a * xf(0.70710678118654752440); }
static dd half_root(dd a) { return a * dd(0.70710678118654752440); }
template <typename R> C<R> mulc(C<R> a, double c) { return {mulc(a.re, c), mulc(a.im, c)}; }

template <typename R> void dft4(C<R>& a, C<R>& b, C<R>& c, C<R>& d) {
  const C<R> t0 = a + c, t1 = a - c, t2 = b + d, t3 = mmi(b - d);
  a = t0 + t2; c = t0 - t2; b = t1 + t3; d = t1 - t3;
}
template <typename R> void dft3(C<R>& v0, C<R>& v1, C<R>& v2) {
  const C<R> t = v1 + v2, d = mmi(mulc(v1 - v2, sqrt(0.75))), m = v0 + mulc(t, -0.5);
  v0 = v0 + t; v1 = m + d; v2 = m - d;
}
template <typename R> void dft(C<R>* v, int r) {
  if (r == 2) {
    const C<R> t = v[0];
    v[0] = t + v[1]; v[1] = t - v[1];
  } else if (r == 3) {
    dft3(v[0], v[1], v[2]);
  } else if (r == 4) {
    dft4(v[0], v[1], v[2], v[3]);
  } else if (r == 6) {  // 2 x 3, prime factor map
    C<R> a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
    for (int n = 0; n < 3; ++n) { const C<R> t = a[n]; a[n] = t + b[n]; b[n] = t - b[n]; }
    dft3(a[0], a[1], a[2]); dft3(b[0], b[1], b[2]);
    v[0] = a[0]; v[4] = a[1]; v[2] = a[2];
    v[3] = b[0]; v[1] = b[1]; v[5] = b[2];
  } else if (r == 8) {
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    const C<R> a = v[3], b = v[7];
    v[3] = {half_root(a.re + a.im), half_root(a.im - a.re)};
    v[5] = mmi(v[5]);
    v[7] = {half_root(b.im - b.re), half_root(-b.re - b.im)};
    C<R> y[8];
    for (int k = 0; k < 4; ++k) { y[k] = v[2 * k] + v[2 * k + 1]; y[k + 4] = v[2 * k] - v[2 * k + 1]; }
    std::copy(y, y + 8, v);
  } else {  // 5 and 7: paired sums
    const int H = r / 2;
    C<R> s[3], d[3], y[7];
    y[0] = v[0];
    for (int j = 1; j <= H; ++j) { s[j - 1] = v[j] + v[r - j]; d[j - 1] = v[j] - v[r - j]; y[0] = y[0] + s[j - 1]; }
    for (int k = 1; k <= H; ++k) {
      C<R> a = v[0], b = mulc(d[0], (double)sinl(2 * PI * k / r));
      for (int j = 1; j <= H; ++j) {
        a = a + mulc(s[j - 1], (double)cosl(2 * PI * (j * k % r) / r));
        if (j > 1) b = b + mulc(d[j - 1], (double)sinl(2 * PI * (j * k % r) / r));
      }
      y[k] = a + mmi(b); y[r - k] = a - mmi(b);
    }
    std::copy(y, y + r, v);
  }
}
static xf_tw entry(cld w, int s) {
  std::vector<float> t;
  push_xf_twiddle(t, w, s);
  xf_tw e;
  memcpy(&e, t.data(), sizeof e);
  return e;
}
template <bool ROUND> void twiddle(C<xf>& v, cld w, int q, int sh, int up) {
  if (up) v = {xf_up(v.re, up), xf_up(v.im, up)};
  if (q == 0) v = {xf_shift<ROUND>(v.re, sh), xf_shift<ROUND>(v.im, sh)};
  else xf_twiddle<false, ROUND>(v.re, v.im, entry(w, sh));
}
static dd split(ld x) { const float h = (float)x; return dd(h, (float)(x - h)); }
// Stockham stages in place of x; returns the bits that xf values went down
template <typename R> int stages(std::vector<C<R>>& x, const std::vector<int>& rad, bool rounds) {
  const int M = x.size();
  std::vector<C<R>> y(M);
  int Ls = 1, shifts = 0;
  for (const int& r : rad) {
    int sh = 0, up = 0;
    if constexpr (std::is_same<R, xf>::value) if (Ls > 1) {
      unsigned m = 0;
      for (auto& v : x) m = std::max({m, (unsigned)(v.re.h ^ (v.re.h >> 31)), (unsigned)(v.im.h ^ (v.im.h >> 31))});
      const int excess = M & (M - 1) ? xf_excess(m, r) : xf_excess_pow2(m, r == 8 ? 3 : r == 4 ? 2 : 1);
      sh = xf_shift_of(excess);
      up = xf_up_of(excess, xf_slack(r));
      shifts += sh - up;
    }
    for (int b = 0; b < M / r; ++b) {
      const int j = b % Ls;
      C<R> v[8];
      for (int q = 0; q < r; ++q) {
        v[q] = x[b + q * (M / r)];
        if (Ls == 1) continue;
        const cld w = std::polar((ld)1, -2 * PI * q * j / (r * Ls));
        if constexpr (std::is_same<R, xf>::value) {
          if (rounds && (int)(&r - rad.data()) + 2 >= (int)rad.size()) twiddle<true>(v[q], w, q, sh, up);
          else twiddle<false>(v[q], w, q, sh, up);
        } else if (q) {
          const dd wr = split(w.real()), wi = split(w.imag());
          v[q] = {v[q].re * wr - v[q].im * wi, v[q].re * wi + v[q].im * wr};
        }
      }
      dft(v, r);
      for (int q = 0; q < r; ++q) y[(b - j) * r + j + q * Ls] = v[q];
    }
    x.swap(y);
    Ls *= r;
  }
  return shifts;
}
static void fft(std::vector<cld>& x) {
  const int n = x.size();
  if (n == 1) return;
  int p = 2;
  while (n % p) ++p;
  std::vector<std::vector<cld>> s(p, std::vector<cld>(n / p));
  for (int i = 0; i < n; ++i) s[i % p][i / p] = x[i];
  for (auto& q : s) fft(q);
  static std::map<int, std::vector<cld>> table;
  auto& w = table[n];
  if (w.empty()) for (int i = 0; i < n; ++i) w.push_back(std::polar((ld)1, -2 * PI * i / n));
  for (int k = 0; k < n; ++k) {
    cld a = 0;
    for (int j = 0; j < p; ++j) a += w[(long long)j * k % n] * s[j][k % (n / p)];
    x[k] = a;
  }
}
static xf to_xf(ld p) {  // toward zero, as d2xf
  const ld a = fabsl(p), f = floorl(a);
  return p < 0 ? xf(-(int)f, -(float)(a - f)) : xf((int)f, (float)(a - f));
}
static ld error(const std::vector<cld>& y, const std::vector<cld>& e) {
  ld n = 0, d = 0;
  for (size_t i = 0; i < e.size(); ++i) { n += std::norm(y[i] - e[i]); d += std::norm(e[i]); }
  return n / d;
}
int main(int argc, char** argv) {  // length, radices
  const int M = atoi(argv[1]);
  std::vector<int> rad;
  for (const char* q = argv[2]; *q; ++q) rad.push_back(*q - '0');
  std::mt19937_64 g(M);
  std::normal_distribution<double> un(0, 1);
  const char* names[] = {"noise", "mean 1", "mean 10", "mean 1000", "ramp", "tone", "corner", "point", "two points", "eight points", "k^-2",
                         "spectrum 10", "spectrum 1000", "spectrum uniform"};
  for (int kind = 0; kind < 14; ++kind) {
    ld ex = 0, ed = 0;
    for (int rep = 0; rep < 4; ++rep) {
      std::vector<cld> x(M);
      const int k0 = 1 + g() % (M - 1);
      const ld scale = 0.5L + (g() % 1000) / 999.0L;
      for (int i = 0; i < M; ++i) {
        const cld n(un(g), un(g));
        const ld t = 2 * PI * ((long long)i * k0 % M) / M;
        x[i] = kind == 0   ? n
               : kind <= 3 ? n + powl(10, kind - 1 + (kind == 3)) * (rep % 2 ? cld(0.8L, -0.6L) : cld(1, 0))
               : kind == 4 ? cld((ld)i / M, rep % 2 ? 0 : 1 - (ld)i / M)
               : kind == 5 ? n + std::polar((ld)30, t)
               : kind == 6 ? cld(1, 1) * std::polar((ld)1, PI / 2 * (i * rep % 4))
               : kind == 7 ? (i == k0 ? n : cld(0))
               : kind == 8 ? (i == k0 || i == (k0 * 3 + 1) % M ? n : cld(0))
               : kind == 9 ? (i % (M / 8 + 1) == 0 ? n : cld(0))
               : kind == 11 ? n + (ld)10
               : kind == 12 ? n + (ld)1000
               : kind == 13 ? cld((ld)(g() >> 11) * 0x1p-53L)
                           : n / (ld)((1 + std::min(i, M - i)) * (1 + std::min(i, M - i)));
        x[i] *= scale;
      }
      if (kind >= 10) fft(x);
      ld mx = 0;
      for (auto& v : x) {
        v = cld((double)v.real(), (double)v.imag());
        mx = std::max({mx, fabsl(v.real()), fabsl(v.imag())});
      }
      std::vector<cld> e = x, y(M);
      fft(e);
      const ld f = ldexpl(1, -ilogbl(mx)), fx = ldexpl(f, 26);
      std::vector<C<xf>> a(M);
      std::vector<C<dd>> b(M);
      for (int i = 0; i < M; ++i) {
        a[i] = {to_xf(x[i].real() * fx), to_xf(x[i].imag() * fx)};
        b[i] = {split(x[i].real() * f), split(x[i].imag() * f)};
      }
      const int logm = 31 - __builtin_clz(M);
      const bool rounds = !(M & (M - 1)) && xf_rounds(logm);  // smooth lines: never
      const int s = stages(a, rad, rounds);
      for (int i = 0; i < M; ++i) y[i] = cld(val(a[i].re), val(a[i].im)) * ldexpl(1, s) / fx;
      ex += error(y, e);
      stages(b, rad, false);
      for (int i = 0; i < M; ++i) y[i] = cld(val(b[i].re), val(b[i].im)) / f;
      ed += error(y, e);
    }
    std::printf("%s: %.2Le %.2Le %d\n", names[kind], sqrtl(ex / 4), sqrtl(ed / 4), (int)(ex <= ed));
  }
  // the halved sum of the r2c split, at the ends of the range
  for (int q : {2040109465, -2040109465, 7, -8}) for (int r : {2040109464, -2040109465, 3}) {
    const xf a(q, 0.3f), b(r, -2.7f);
    if (!(fabsl(val(xf_half_sum(a, b)) - (val(a) + val(b)) / 2) <= ldexpl(1, -22))) std::printf("half sum: %d %d 0\n", q, r);
  }
}
"""


def radices(n):
    """Of the power-of-two lines, and of the Float64 smooth-length pass."""
    if n & (n - 1) == 0:
        out = []
        while n >= 8:
            out.append(8)
            n //= 8
        return out + [n] * (n > 1)
    if n > 2048:
        return radices(n // 8) + [4, 2]
    best = None

    def search(m, cur, start):
        nonlocal best
        if m == 1:
            if best is None or (len(cur), sum(cur)) < (len(best), sum(best)):
                best = list(cur)
            return
        for r in range(start, 1, -1):
            if m % r == 0 and len(cur) < 6:
                search(m // r, cur + [r], r)

    search(n, [], 8)
    return best


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("xf")
    (d / "xf.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), str(d / "xf.cpp"), "-o", str(d / "xf")], check=True)
    return d / "xf"


# every power of two, every radix, the longest stage lists and lines
@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 45, 49, 100, 243, 343, 360, 384, 729, 1000,
                               1029, 1215, 1458, 1536, 1701, 2025, 2560])
def test_xf_lines_are_no_less_exact_than_double_float(driver, n):
    out = subprocess.run([str(driver), str(n), "".join(map(str, radices(n)))], check=True, capture_output=True,
                         text=True).stdout
    lines = out.splitlines()
    assert len(lines) == 14 and all(line.endswith(" 1") for line in lines[:11]), out


@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024, 2048, 4096])
def test_xf_lines_of_one_large_value(driver, n):
    out = subprocess.run([str(driver), str(n), "".join(map(str, radices(n)))], check=True, capture_output=True,
                         text=True).stdout
    errors = [float(line.split()[-3]) for line in out.splitlines()[11:]]
    assert len(errors) == 3 and max(errors) <= n ** 0.5 * 2.0 ** -50, out
