"""Integer-float arithmetic of the Float64 register stages (pfgb_xf.cuh),
compiled for the host with g++ from the same header and checked against long
double:

* a product with a twiddle of any shift, and with a constant, is within
  2^-20 units of the exact one (values up to 2^28 units, fractions up to 4:
  four roundings of terms below 8 units at 2^-24 each);
* the shift of a stage keeps a radix-8 butterfly's sums below 2^31, and is at
  most one bit above what the line's largest component needs;
* line DFTs of 8 to 4096 points, of noise, one tone and one point: relative
  L2 error below 2^-47 (the double-float stages: 2^-46).
"""
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
#include <random>
#include <vector>
#include "pfgb_xf.cuh"
using namespace pfgb;
typedef long double ld;
typedef std::complex<ld> cld;
struct C { xf re, im; };
static C add(C a, C b) { return {a.re + b.re, a.im + b.im}; }
static C sub(C a, C b) { return {a.re - b.re, a.im - b.im}; }
static C mmi(C a) { return {a.im, -a.re}; }
static const xf H(0.70710678118654752440);
static void dft4(C& a, C& b, C& c, C& d) {
  const C t0 = add(a, c), t1 = sub(a, c), t2 = add(b, d), t3 = mmi(sub(b, d));
  a = add(t0, t2); c = sub(t0, t2); b = add(t1, t3); d = sub(t1, t3);
}
static void dft8(C* v) {
  dft4(v[0], v[2], v[4], v[6]);
  dft4(v[1], v[3], v[5], v[7]);
  v[3] = {(v[3].re + v[3].im) * H, (v[3].im - v[3].re) * H};
  v[5] = mmi(v[5]);
  v[7] = {(v[7].im - v[7].re) * H, (-v[7].re - v[7].im) * H};
  C y[8];
  for (int k = 0; k < 4; ++k) { y[k] = add(v[2 * k], v[2 * k + 1]); y[k + 4] = sub(v[2 * k], v[2 * k + 1]); }
  std::copy(y, y + 8, v);
}
static ld val(xf a) { return (ld)a.h + (ld)a.l; }
static xf_tw entry(cld w, int s) {
  std::vector<float> t;
  push_xf_twiddle(t, w, s);
  xf_tw e;
  memcpy(&e, t.data(), sizeof e);
  return e;
}
int main() {
  std::mt19937_64 g(5);
  std::normal_distribution<double> un(0, 1);
  std::uniform_real_distribution<double> u1(-1, 1);
  ld wt = 0, wm = 0, ws = 0;
  for (int k = 0; k < 300000; ++k) {
    xf a((int)(u1(g) * 268435456.0), (float)(4 * u1(g))), b((int)(u1(g) * 268435456.0), (float)(4 * u1(g)));
    wm = std::max(wm, fabsl(val(a * H) - val(a) * sqrtl(0.5L)));
    const ld th = k % 7 == 0 ? acosl(-1.0L) * (k % 4) / 2 : (ld)un(g) * 3, c = cosl(th), s = sinl(th);
    const int sh = 1 + k % 3;
    const ld A = val(a), B = val(b), q = 1 << sh;
    ws = std::max(ws, fabsl(val(xf_shift(a, sh)) - A / q));
    xf re = a, im = b;
    xf_twiddle<false>(re, im, entry(cld(c, s), sh));
    wt = std::max({wt, fabsl(val(re) - (A * c - B * s) / q), fabsl(val(im) - (A * s + B * c) / q)});
    re = a, im = b;
    xf_twiddle<true>(re, im, entry(cld(c, s), sh));
    wt = std::max({wt, fabsl(val(re) - (A * c + B * s) / q), fabsl(val(im) - (B * c - A * s) / q)});
  }
  long bad = !(wt < ldexpl(1, -20)) + !(wm < ldexpl(1, -20)) + !(ws < ldexpl(1, -20));
  for (int lr = 1; lr <= 4; ++lr)
    for (int bit = 0; bit < 31; ++bit)
      for (unsigned m : {1u << bit, (2u << bit) - 1}) {
        const int s = xf_stage_shift(m, lr);
        if (s < 1 || s > kXfShifts) ++bad;
        if (bit < 30 && lr <= 3 && (ld)m / (1 << s) * (1 << lr) * sqrtl(2) >= 2147483648.0L) ++bad;
        if (s > 1 && (ld)(m + 1) / (1 << (s - 1)) * (1 << lr) <= 1073741824.0L) ++bad;
      }
  ld worst = 0;
  for (int lg = 3; lg <= 12; ++lg)
    for (int kind = 0; kind < 3; ++kind) {
      const int M = 1 << lg;
      std::vector<cld> x0(M);
      for (int i = 0; i < M; ++i)
        x0[i] = kind == 0 ? cld(un(g), un(g))
                : kind == 1 ? std::polar((ld)1.3L, 2 * acosl(-1.0L) * ((3 * i) % M) / M)
                            : cld(i == 3 ? 0.9L : 0, i == 3 ? -0.4L : 0);
      ld mx = 0;
      for (auto& v : x0) mx = std::max({mx, fabsl(v.real()), fabsl(v.imag())});
      const ld f = ldexpl(1, 26 - ilogbl(mx));
      std::vector<C> x(M), y(M);
      std::vector<cld> r(M);
      for (int i = 0; i < M; ++i) {
        const ld p = x0[i].real() * f, q = x0[i].imag() * f;
        x[i].re = xf((int)llrintl(p), (float)(p - llrintl(p)));
        x[i].im = xf((int)llrintl(q), (float)(q - llrintl(q)));
        r[i] = cld(val(x[i].re), val(x[i].im));
      }
      int shifts = 0;
      for (int Ls = 1; Ls < M;) {
        const int R = std::min(8, M / Ls), lr = R == 8 ? 3 : R == 4 ? 2 : 1;
        int sh = 0;
        if (Ls > 1) {
          unsigned m = 0;
          for (auto& v : x) m = std::max({m, (unsigned)(v.re.h ^ (v.re.h >> 31)), (unsigned)(v.im.h ^ (v.im.h >> 31))});
          sh = xf_stage_shift(m, lr);
          shifts += sh;
        }
        for (int b = 0; b < M / R; ++b) {
          const int j = b % Ls;
          C v[8];
          for (int k = 0; k < R; ++k) {
            v[k] = x[b + k * (M / R)];
            if (sh && k == 0) v[0] = {xf_shift(v[0].re, sh), xf_shift(v[0].im, sh)};
            if (sh && k) {
              const ld an = -2 * acosl(-1.0L) * ((ld)k * j) / (R * Ls);
              xf_twiddle<false>(v[k].re, v[k].im, entry(cld(cosl(an), sinl(an)), sh));
            }
          }
          if (R == 8) dft8(v);
          else if (R == 4) dft4(v[0], v[1], v[2], v[3]);
          else { const C t = v[0]; v[0] = add(t, v[1]); v[1] = sub(t, v[1]); }
          for (int k = 0; k < R; ++k) y[(b - j) * R + j + k * Ls] = v[k];
        }
        x.swap(y);
        Ls *= R;
      }
      std::vector<cld> o(M);
      for (int i = 0; i < M; ++i) {
        int q = 0;
        for (int k = 0; k < lg; ++k) if (i >> k & 1) q |= 1 << (lg - 1 - k);
        o[q] = r[i];
      }
      for (int len = 2; len <= M; len *= 2)
        for (int s = 0; s < M; s += len)
          for (int k = 0; k < len / 2; ++k) {
            const cld w = std::polar((ld)1, -2 * acosl(-1.0L) * k / len);
            const cld u = o[s + k], t = o[s + k + len / 2] * w;
            o[s + k] = u + t;
            o[s + k + len / 2] = u - t;
          }
      ld num = 0, den = 0;
      for (int i = 0; i < M; ++i) {
        const cld q = o[i] * ldexpl(1, -shifts);
        num += std::norm(cld(val(x[i].re), val(x[i].im)) - q);
        den += std::norm(q);
      }
      worst = std::max(worst, sqrtl(num / den));
    }
  if (!(worst < ldexpl(1, -47))) ++bad;
  std::printf("%ld twiddle %.3Le constant %.3Le shift %.3Le dft %.3Le\n", bad, wt, wm, ws, worst);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_xf_arithmetic_against_long_double(tmp_path):
    src = tmp_path / "xf.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "xf"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split()[0] == "0", out
