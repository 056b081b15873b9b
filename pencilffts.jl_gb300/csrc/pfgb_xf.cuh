// Integer-float pairs ("xf"): the arithmetic of the register stages of
// Float64 (double-float) lines.
//
// A double-float (dd) sum costs eight FP32 instructions, and sums are most
// of an FFT.  Inside the stages of one line a value is held as h + l instead:
// h a 32-bit integer count of the line's unit q, l a float holding the
// fraction below it (|l| of a few units).  Sums are one integer and one float
// addition, exact in h.  A product with a twiddle w, |w| <= 1, is a 32 x 32
// -> 64-bit integer product with W = round(w 2^(32 - s)): its high word, to
// nearest, is the new h, in units 2^s q, its low word the new fraction; the
// rest of w (o = w 2^(32 - s) - W) and the product of l go into the fraction in
// float.
//
// Range: a line's complex values stay within 0.95 2^31 / r units in modulus
// before a radix-r butterfly, r <= 8, and so within 0.95 2^31 after it: h cannot
// overflow.  The line enters with components below 2^27 (its largest in
// [2^26, 2^27)), and the twiddles of each later stage carry the shift s = 1, 2
// or 3 that the line's largest component after the previous butterfly asks for
// (xf_excess, xf_shift_of; s = 3 always suffices).  The tables hold all three
// forms, so the shift costs no instruction.  A line that grew too little for
// s = 1 (few non-zero points, small radices) goes up by some bits first
// (xf_up_of).
//
// Cost: 512^3 Float64 round trip 4.14 ms with dd stages, 3.30 ms with these;
// 256^3 complex 0.945 and 0.757 ms.
//
// Precision: each operation rounds the fraction at about 2^-24 unit, whatever the
// value, where a dd stage's error follows the single value.  Lines of noise have
// a third of dd's error.  The line that can lose is the one whose sum grows with
// its length (a large mean, a ramp): its small outputs carry the error that goes
// with the large one, as sqrt(M).  tests/test_xf_lines.py holds such lines, and
// those of few points, below dd's error at all lengths; what that took, as
// multiples of dd's error:
//   4096 points, mean 10 and noise: 1.7 with high words rounded down in every
//     stage and a bit of the range unused, 0.8 as it is (xf_rounds, xf_excess);
//   512 points, mean 1000 and noise, r2c: 1.6 with one bit of the range kept free
//     for the split's sum, 0.8 with the sum halved (xf_half_sum);
//   729 points of which 8 are not zero: 2.8 without going up, 0.5 with it.
// What dd does better is the line of one large value among small ones, such as the
// spectrum of a field with a mean: its transform does not grow, so a unit of the
// large value's 2^-27 is all there is, and the error is up to 0.63 sqrt(M) 2^-50 of
// the line (2.5 times dd's at 512 points, 5 times at 4096; 5.6 and 11 without going
// up).  A round trip of such a field stays below dd's error at 512^3 (mean 10 and unit
// noise 1.6e-14 against 2.8e-14), 1.4 times above it at 4096^2 (3.6e-14 against 2.6e-14).
#pragma once

#include <stdint.h>
#include <string.h>

#include "pfgb_dd.cuh"
#if defined(__CUDACC__)
#include "pfgb_device.cuh"
#endif

namespace pfgb {

struct xf {
  int h;
  float l;
  xf() = default;
  PFGB_HD constexpr xf(int hh, float ll) : h(hh), l(ll) {}
  // a constant c in (0.5, 1.5), the right-hand operand of a product:
  // c = 1 + (h + l) 2^-32
  PFGB_HD constexpr explicit xf(double c)
      : h((int)((c - 1.0) * 4294967296.0)),
        l((float)((c - 1.0) * 4294967296.0 - (double)(int)((c - 1.0) * 4294967296.0))) {}
};

PFGB_HD xf operator+(xf a, xf b) { return xf(a.h + b.h, f_add(a.l, b.l)); }
PFGB_HD xf operator-(xf a, xf b) { return xf(a.h - b.h, f_sub(a.l, b.l)); }
PFGB_HD xf operator-(xf a) { return xf(-a.h, -a.l); }

PFGB_HD float xf_i2f(int x) {
#if defined(__CUDA_ARCH__)
  return __int2float_rn(x);
#else
  return (float)x;
#endif
}

// u 2^-32 + f for the low word u of a product whose high word was rounded down
PFGB_HD float xf_frac(uint32_t u, float f) {
#if defined(__CUDA_ARCH__)
  return f_fma(__uint2float_rn(u), 0x1p-32f, f);
#else
  return f_fma((float)u, 0x1p-32f, f);
#endif
}
// p 2^-32 + f for a product p: its high word rounded down, or to nearest
// (ROUND: the low word is a signed fraction then, and its top bit the carry).
// Fractions rounded down do not cancel in the butterflies' sums: 1.2 to 1.9
// times the error.
template <bool ROUND>
PFGB_HD xf xf_product(uint64_t p, float f) {
  const uint32_t u = (uint32_t)p;
  if (ROUND) return xf((int)(p >> 32) + (int)(u >> 31), f_fma(xf_i2f((int)u), 0x1p-32f, f));
  return xf((int)(p >> 32), xf_frac(u, f));
}
// Power-of-two lines that need it, in their last two stages (an earlier stage's
// error counts an eighth of the next one's): 4096^2 complex round trip 873 us
// without, 891 us, 930 us with every stage rounded.  Smooth lines, up to 2048
// points but for 2560, stay below dd's error without.
PFGB_HD constexpr bool xf_rounds(int logm) { return logm > 10; }
// Slack of a stage of radix r (xf_up_of).  Lines of noise never come to 0 before
// a radix of 7 or 8, so a line that does is one that the sums do not grow (the
// spectrum of a field with a mean: its error is halved); before the smaller ones
// they do, and going up each time costs (243^3 Float64 1.73 ms instead of 1.57 with
// 2 for radix 3).
PFGB_HD constexpr int xf_slack(int r) { return r > 6 ? 0 : r > 3 ? 2 : 3; }

// a c, in a's unit
PFGB_HD xf operator*(xf a, xf c) {
  const float cf = f_fma((float)c.h, 0x1p-32f, 1.0f);
  const uint64_t p = (uint64_t)((int64_t)a.h * c.h);
  const float f = f_fma(xf_i2f(a.h), c.l * 0x1p-32f, f_mul(a.l, cf));
  return xf(a.h + (int)(p >> 32), xf_frac((uint32_t)p, f));
}

// a c for a compile-time constant |c| <= 1, in a's unit
PFGB_HD xf xf_mulc(xf a, double c) {
  const int base = c > 0.5 ? 1 : c < -0.5 ? -1 : 0;
  const double r = (c - base) * 4294967296.0;
  const int w = (int)(r < -2147483648.0 ? -2147483648.0 : r > 2147483647.0 ? 2147483647.0 : r);
  const uint64_t p = (uint64_t)((int64_t)a.h * w);
  const float f = f_fma(xf_i2f(a.h), (float)((r - w) * 0x1p-32), f_mul(a.l, (float)c));
  const int b = base > 0 ? a.h : base < 0 ? -a.h : 0;
  return xf(b + (int)(p >> 32), xf_frac((uint32_t)p, f));
}

// (a + b) / 2 where a + b may be beyond 2^31
PFGB_HD xf xf_half_sum(xf a, xf b) {
  const int x = a.h ^ b.h;
  return xf((a.h & b.h) + (x >> 1), f_fma(f_add(a.l, b.l), 0.5f, x & 1 ? 0.5f : 0.0f));
}

// a c for a factor c in [1/2, 1) given as w = round(c 2^31), o = (c 2^31 - w)
// 2^-32 and f = c / 2, in units 2 times larger (the ldiv! normalisation).
PFGB_HD xf xf_scaled(xf a, int w, float o, float f) {
  const uint64_t p = (uint64_t)((int64_t)a.h * w);
  return xf((int)(p >> 32), xf_frac((uint32_t)p, f_fma(xf_i2f(a.h), o, f_mul(a.l, f))));
}

// Table entry of a twiddle w for the shift s: round(w 2^(32 - s)) (clamped to
// 31 bits) and the rest, per part.
struct xf_tw {
  int wr, wi;
  float orr, oi;
};

// shifts 1 .. kXfShifts: one table each, one after the other
constexpr int kXfShifts = 3;
// a twiddle (parts of magnitude at most 1) as doubles and what they leave; once
// for all shifts, since the Arm host's long double is software
struct xf_tw_parts {
  double hi[2], lo[2];
};
template <typename C>
inline xf_tw_parts split_twiddle(const C& w) {
  const auto x = w.real(), y = w.imag();
  const double h[2] = {(double)x, (double)y};
  return {{h[0], h[1]}, {(double)(x - h[0]), (double)(y - h[1])}};
}
// appends the entry of w for the shift s to a table of 32-bit words
template <typename V>
inline void push_xf_twiddle(V& t, const xf_tw_parts& w, int s) {
  const double q = (double)(1ll << (32 - s));
  const double c[2] = {w.hi[0] * q, w.hi[1] * q};
  const double rest[2] = {w.lo[0] * q, w.lo[1] * q};
  float o[2];
  for (int i = 0; i < 2; ++i) {
    const long long r = (long long)(c[i] < 0 ? c[i] - 0.5 : c[i] + 0.5);
    const int n = (int)(r > 0x7FFFFFFFll ? 0x7FFFFFFFll : r < -0x7FFFFFFFll ? -0x7FFFFFFFll : r);
    float f;
    memcpy(&f, &n, sizeof f);
    t.push_back(f);
    o[i] = (float)((c[i] - n) + rest[i]);
  }
  t.push_back(o[0]);
  t.push_back(o[1]);
}

template <typename V, typename C>
inline void push_xf_twiddle(V& t, const C& w, int s) {
  push_xf_twiddle(t, split_twiddle(w), s);
}

// (re, im) times w (CONJ: times its conjugate), in units 2^s times larger.
template <bool CONJ, bool ROUND = false>
PFGB_HD void xf_twiddle(xf& re, xf& im, xf_tw w) {
  const int wi = CONJ ? -w.wi : w.wi, mwi = CONJ ? w.wi : -w.wi;
  const float oi = CONJ ? -w.oi : w.oi;
  const uint64_t pr = (uint64_t)((int64_t)re.h * w.wr) + (uint64_t)((int64_t)im.h * mwi);
  const uint64_t pi = (uint64_t)((int64_t)re.h * wi) + (uint64_t)((int64_t)im.h * w.wr);
  const float wrf = xf_i2f(w.wr), wif = xf_i2f(wi), hr = xf_i2f(re.h), hi = xf_i2f(im.h);
  const float ar = f_fma(re.l, wrf, f_fma(-im.l, wif, f_fma(-hi, oi, f_mul(hr, w.orr))));
  const float ai = f_fma(re.l, wif, f_fma(im.l, wrf, f_fma(hi, w.orr, f_mul(hr, oi))));
  re = xf_product<ROUND>(pr, f_mul(ar, 0x1p-32f));
  im = xf_product<ROUND>(pi, f_mul(ai, 0x1p-32f));
}

// a in units 2^s times larger
template <bool ROUND = false>
PFGB_HD xf xf_shift(xf a, int s) {
#if defined(__CUDA_ARCH__)
  const float f = __uint_as_float((unsigned)(127 - s) << 23);
#else
  const float f = 1.0f / (float)(1 << s);
#endif
  if (ROUND) {
    const int h = (a.h + (1 << (s - 1))) >> s;
    return xf(h, f_mul(f, f_add(a.l, xf_i2f(a.h - (h << s)))));
  }
  return xf(a.h >> s, f_mul(f, f_add(a.l, xf_i2f(a.h & ((1 << s) - 1)))));
}
// a in units 2^u times smaller
PFGB_HD xf xf_up(xf a, int u) {
#if defined(__CUDA_ARCH__)
  const float t = f_mul(a.l, __uint_as_float((unsigned)(127 + u) << 23));
  const int i = __float2int_rn(t);
#else
  const float t = f_mul(a.l, (float)(1 << u));
  const int i = (int)__builtin_rintf(t);
#endif
  return xf((int)((unsigned)a.h << u) + i, f_sub(t, xf_i2f(i)));
}

// Bits of a line with largest h or ~h m beyond what a butterfly of radix r <= 8
// takes: 1.5 r m (1.5 and not sqrt 2 for the complex moduli, and for what the
// fractions add) is to stay below 2^31.
PFGB_HD int xf_bits(unsigned m) {
#if defined(__CUDA_ARCH__)
  return 32 - __clz((int)m);
#else
  return m ? 32 - __builtin_clz(m) : 0;
#endif
}
PFGB_HD int xf_excess(unsigned m, int r) { return xf_bits(((m >> 4) + 1u) * (3u * (unsigned)r)) - 28; }
// Shift of the twiddles before that butterfly, within 1 .. 3: with moduli up to
// 0.95 2^31 three are enough.
PFGB_HD int xf_shift_of(int excess) { return excess < 1 ? 1 : excess > kXfShifts ? kXfShifts : excess; }
// Bits that the line's values go up by before the shift of 1: 0 unless that
// shift would leave slack + 1 bits free, then all of them, at most 4.  A line of
// zeros (the rest of a last tile: far below any other) stays.
PFGB_HD int xf_up_of(int excess, int slack) {
  return (unsigned)(-slack - excess) > 13u ? 0 : excess < -3 ? 4 : 1 - excess;
}
// r = 2^lr: one instruction less
PFGB_HD int xf_excess_pow2(unsigned m, int lr) { return xf_bits(m + (m >> 1)) - 31 + lr; }
PFGB_HD int xf_stage_shift(unsigned m, int lr) { return xf_shift_of(xf_excess_pow2(m, lr)); }

// A dd line in xf units: from the float bits m of its largest |high part|, the
// scale 2^(153 - e), e the biased exponent of m, at least 27 (a line below
// 2^-100 keeps fewer bits, as its dd low parts do), that takes the largest
// component to [2^26, 2^27).  A NaN or an infinity among the high parts gives
// a NaN (or infinite) fraction, which every sum carries to all of the line.
PFGB_HD unsigned xf_line_exp(unsigned m) {
  const unsigned e = m >> 23;
  return e < 27u ? 27u : e;
}

#if defined(__CUDACC__)
__device__ __forceinline__ float xf_scale_in(unsigned e) {
  return __uint_as_float((280u - e) << 23);
}
// biased float exponent of the unit in the dd line's scale, before any shift
__device__ __forceinline__ int xf_unit_exp(unsigned e) { return (int)min(e, 254u) - 26; }

__device__ __forceinline__ xf dd2xf(dd a, float f) {
  const float hs = f_mul(a.h, f);
  const int h = __float2int_rn(hs);
  return xf(h, f_fma(a.l, f, f_sub(hs, __int2float_rn(h))));
}
// a as the unevaluated sum hi + lo, hi = h rounded to float
__device__ __forceinline__ void xf_split(xf a, float& hi, float& lo) {
  hi = __int2float_rn(a.h);
  lo = f_add(a.l, __int2float_rn(a.h - __float2int_rn(hi)));
}
// a 2^(ue - 127): ue the unit's biased exponent, above -23 (below 1 for lines
// near the bottom of the dd range that went up)
__device__ __forceinline__ dd xf2dd(xf a, int ue) {
  const float g = __uint_as_float(ue > 0 ? (unsigned)ue << 23 : 0x800000u >> (1 - ue));
  float hi, lo;
  xf_split(a, hi, lo);
  return dd(f_mul(hi, g), f_mul(lo, g));
}

// x as a count of 2^(emax - 1023 - B) (20 < B <= 27 bits; emax: the line's largest
// biased exponent), fs = xf_frac_scale(emax): the 53-bit significand shifted
// right in 64 bits, its low word as the fraction.  Zeros and subnormals give
// zero; a line with a NaN or an infinity gets NaN fractions.  No branch, where
// the conversion to dd needs one for its rare cases.
__device__ __forceinline__ float xf_frac_scale(int emax) {
  return __uint_as_float(emax >= 0x7FF ? 0x7FC00000u : 0x2F800000u);  // 2^-32
}
__device__ __forceinline__ xf d2xf(double x, int emax, float fs, int B) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned hi32 = (unsigned)(b >> 32), lo32 = (unsigned)b;
  const int e = (int)((hi32 >> 20) & 0x7FF);
  const unsigned mh = (hi32 & 0xFFFFFu) | 0x100000u;
  const unsigned long long m = (unsigned long long)__funnelshift_l(lo32, mh, B - 20) << 32 | (lo32 << (B - 20));
  const unsigned long long f = m >> (e == 0 ? 63 : min(emax - e, 63));
  const int s = (int)hi32 >> 31;
  const float l = __uint2float_rn((unsigned)f) * __uint_as_float(__float_as_uint(fs) | (hi32 & 0x80000000u));
  return xf(((int)(f >> 32) ^ s) - s, l);
}
template <int B>
__device__ __forceinline__ xf d2xf(double x, int emax, float fs) {
  return d2xf(x, emax, fs, B);
}

// A rare result of xf2d: zero, NaN (a NaN or infinite fraction, overflow).
static __device__ __noinline__ double xf2d_rare(float s, int off) {
  const unsigned sb = __float_as_uint(s);
  const int es = (int)(sb >> 23) & 255;
  if (es == 255 || es + off >= 0x7FF) return __longlong_as_double(0x7FF8000000000000ll);
  return __longlong_as_double((long long)((unsigned long long)(sb & 0x80000000u) << 32));
}
// (re, im) 2^(off - 896) as doubles (off: the unit's biased exponent plus the
// line's biased double exponent minus 254), within one unit in the last
// place.  h + l as s + e with s rounded toward zero, so that e has its sign
// and counts up from s's bit pattern: s gives the high word and the top three
// bits of the low one, e in units of the double's last place the other 29.
__device__ __forceinline__ void xf2d(Cx<xf> x, int off, double& re, double& im) {
  int lo = max(1 - off, 1), hi = min(2046 - off, 254);
  if (hi < lo) lo = hi = 512;  // no result in the double range
  bool ok = true;
  float sv[2];
  double r[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float a, b;
    xf_split(i ? x.im : x.re, a, b);
    const float s = __fadd_rz(a, b);
    const float e = __fsub_rn(b, __fsub_rn(s, a));
    const unsigned sb = __float_as_uint(s);
    const unsigned esx = sb & 0x7F800000u;
    ok = ok && (unsigned)((int)(esx >> 23) - lo) <= (unsigned)(hi - lo);
    const float sux = __uint_as_float(0x99000000u - max(esx, 52u << 23));  // 2^(179 - es)
    const unsigned li = (unsigned)min(__float2int_rz(__fmul_rn(fabsf(e), sux)), 0x1FFFFFFF);
    const unsigned hw = (((unsigned)((int)sb >> 3)) & 0x8FFFFFFFu) + ((unsigned)off << 20);
    r[i] = __hiloint2double((int)hw, (int)((sb << 29) | li));
    sv[i] = s;
  }
  if (!ok) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int es = (int)(__float_as_uint(sv[i]) >> 23) & 255;
      if ((unsigned)(es - lo) > (unsigned)(hi - lo)) r[i] = xf2d_rare(sv[i], off);
    }
  }
  re = r[0];
  im = r[1];
}
#endif

}  // namespace pfgb
