// Smooth-length pass: lines of M points, M a product of 2, 3, 5 and 7 that no
// power-of-two pass takes, for c2c, r2c, c2r and the R2R kinds (SmMode), any
// input / output layout, in FP32 or (Float64 data) in integer-float pairs,
// doubles in and out.
//
// A tile of TW lines goes through nst Stockham stages of mixed radix between
// two shared-memory buffers.  A thread owns one line of the tile (p = thread
// mod TW) and every K-th butterfly of each stage: its loads, twiddles and
// stores need no division, its line's scale is its own, and the pitch leaves the
// fewest bank conflicts for the tile's width (sm_best_pitch).  Radices up to 16
// (Float32) or 8 (Float64, whose range bound is a growth of 8 per stage) leave
// two to four stages for most lengths.
//
// Bound by issue slots (125 to 155 instructions a point in Float32, half of
// them integer, before addresses were stepped in bytes) and the shared-memory
// pipe together: 360^3 Float32 round trip 930 -> 834 us, Float64 2514 -> 2421 us
// with byte steps, walks of their own for lanes across the lines, and the
// pitch.  Float64: 330 to 450 instructions a point at 24 warps an SM (80
// registers).  A derivative on the input or output multiplies in FP64 (in1k),
// whose unit then bounds the pass: 329 us for the first pass of a 240^3
// divergence, where a pass without takes 107.
//
// Against the Bluestein tile, which takes these lengths through two
// power-of-two transforms of at least twice the length: see sm_form in
// pfgb_plan.cu for the measured times.
#pragma once

#include "pfgb_fast.cuh"

namespace pfgb {

// threads of a tile: its lines times the butterfly step, at most this many
constexpr int kSmThreads = 256;

// a c for a compile-time constant |c| <= 1, in a's unit
__device__ __forceinline__ float mulc(float a, double c) { return a * (float)c; }
__device__ __forceinline__ xf mulc(xf a, double c) { return xf_mulc(a, c); }
template <typename R>
__device__ __forceinline__ Cx<R> mulc(Cx<R> a, double c) { return mk(mulc(a.re, c), mulc(a.im, c)); }

// y_k = sum_j v_j exp(SIGN 2 pi i j k / RAD) in place, the roots of unity as
// compile-time constants
template <int SIGN, typename R>
__device__ __forceinline__ void sm_dft3(Cx<R>& v0, Cx<R>& v1, Cx<R>& v2) {
  const Cx<R> t = v1 + v2, d = mul_w4<SIGN>(mulc(v1 - v2, 0.86602540378443864676));
  const Cx<R> m = v0 + mulc(t, -0.5);
  v0 = v0 + t;
  v1 = m + d;
  v2 = m - d;
}
template <int SIGN, typename R>
__device__ __forceinline__ void sm_dft5(Cx<R>& v0, Cx<R>& v1, Cx<R>& v2, Cx<R>& v3, Cx<R>& v4) {
  const Cx<R> a1 = v1 + v4, a2 = v2 + v3, b1 = v1 - v4, b2 = v2 - v3, t = a1 + a2;
  Cx<R> A1, A2;
  if constexpr (std::is_same<R, float>::value) {  // as many instructions, one rounding less
    A1 = v0 + mulc(a1, 0.30901699437494742410) + mulc(a2, -0.80901699437494742410);
    A2 = v0 + mulc(a1, -0.80901699437494742410) + mulc(a2, 0.30901699437494742410);
  } else {
    const Cx<R> m = v0 + mulc(t, -0.25), q = mulc(a1 - a2, 0.55901699437494742410);  // sqrt(5) / 4
    A1 = m + q;
    A2 = m - q;
  }
  const Cx<R> B1 = mul_w4<SIGN>(mulc(b1, 0.95105651629515357212) + mulc(b2, 0.58778525229247312917));
  const Cx<R> B2 = mul_w4<SIGN>(mulc(b1, 0.58778525229247312917) - mulc(b2, 0.95105651629515357212));
  v0 = v0 + t;
  v1 = A1 + B1;
  v4 = A1 - B1;
  v2 = A2 + B2;
  v3 = A2 - B2;
}
template <int SIGN, typename R>
__device__ __forceinline__ void sm_dft7(Cx<R>& v0, Cx<R>& v1, Cx<R>& v2, Cx<R>& v3, Cx<R>& v4, Cx<R>& v5, Cx<R>& v6) {
  constexpr double c1 = 0.62348980185873353053, c2 = -0.22252093395631440429, c3 = -0.90096886790241912624;
  constexpr double s1 = 0.78183148246802980871, s2 = 0.97492791218182360702, s3 = 0.43388373911755812048;
  const Cx<R> a1 = v1 + v6, a2 = v2 + v5, a3 = v3 + v4, b1 = v1 - v6, b2 = v2 - v5, b3 = v3 - v4;
  const Cx<R> A1 = v0 + mulc(a1, c1) + mulc(a2, c2) + mulc(a3, c3);
  const Cx<R> A2 = v0 + mulc(a1, c2) + mulc(a2, c3) + mulc(a3, c1);
  const Cx<R> A3 = v0 + mulc(a1, c3) + mulc(a2, c1) + mulc(a3, c2);
  const Cx<R> B1 = mul_w4<SIGN>(mulc(b1, s1) + mulc(b2, s2) + mulc(b3, s3));
  const Cx<R> B2 = mul_w4<SIGN>(mulc(b1, s2) - mulc(b2, s3) - mulc(b3, s1));
  const Cx<R> B3 = mul_w4<SIGN>(mulc(b1, s3) - mulc(b2, s1) + mulc(b3, s2));
  v0 = v0 + a1 + a2 + a3;
  v1 = A1 + B1;
  v6 = A1 - B1;
  v2 = A2 + B2;
  v5 = A2 - B2;
  v3 = A3 + B3;
  v4 = A3 - B3;
}
__host__ __device__ constexpr int sm_inv(int a, int n) {  // a^-1 mod n
  for (int x = 1; x < n; ++x)
    if (a * x % n == 1) return x;
  return 1;
}
template <int RAD, int SIGN, typename R>
__device__ __forceinline__ void sm_dft(Cx<R> (&v)[RAD]);
// RAD = N1 N2, coprime: the prime factor map (no twiddles)
template <int N1, int N2, int SIGN, typename R>
__device__ __forceinline__ void sm_pfa(Cx<R> (&v)[N1 * N2]) {
  constexpr int N = N1 * N2;
  Cx<R> t[N2][N1];
#pragma unroll
  for (int n2 = 0; n2 < N2; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) t[n2][n1] = v[(N2 * n1 + N1 * n2) % N];
    sm_dft<N1, SIGN>(t[n2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) {
    Cx<R> u[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) u[n2] = t[n2][k1];
    sm_dft<N2, SIGN>(u);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) v[(N2 * sm_inv(N2 % N1, N1) * k1 + N1 * sm_inv(N1 % N2, N2) * k2) % N] = u[k2];
  }
}
template <int RAD, int SIGN, typename R>
__device__ __forceinline__ void sm_dft(Cx<R> (&v)[RAD]) {
  if constexpr (RAD == 2) dft2<SIGN>(v[0], v[1]);
  else if constexpr (RAD == 3) sm_dft3<SIGN>(v[0], v[1], v[2]);
  else if constexpr (RAD == 4) dft4<SIGN>(v[0], v[1], v[2], v[3]);
  else if constexpr (RAD == 5) sm_dft5<SIGN>(v[0], v[1], v[2], v[3], v[4]);
  else if constexpr (RAD == 6) sm_pfa<2, 3, SIGN>(v);
  else if constexpr (RAD == 7) sm_dft7<SIGN>(v[0], v[1], v[2], v[3], v[4], v[5], v[6]);
  else if constexpr (RAD == 8) dft8<SIGN>(v);
  else if constexpr (RAD == 10) sm_pfa<2, 5, SIGN>(v);
  else if constexpr (RAD == 12) sm_pfa<4, 3, SIGN>(v);
  else if constexpr (RAD == 15) sm_pfa<3, 5, SIGN>(v);
  else if constexpr (RAD == 16) dft16<SIGN>(v);
  else {
    static_assert(RAD == 9, "no butterfly of this radix");
    // n = n1 + 3 n2, k = k2 + 3 k1
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) sm_dft3<SIGN>(v[n1], v[n1 + 3], v[n1 + 6]);
    constexpr double c[3] = {0.76604444311897803520, 0.17364817766693034885, -0.93969262078590838405};
    constexpr double s[3] = {0.64278760968653932632, 0.98480775301220805937, 0.34202014332566873304};
    auto rot = [&](Cx<R> x, int i) {  // x exp(SIGN 2 pi i m / 9), m = 1, 2, 4
      const double sn = SIGN < 0 ? -s[i] : s[i];
      return mk(mulc(x.re, c[i]) - mulc(x.im, sn), mulc(x.im, c[i]) + mulc(x.re, sn));
    };
    v[4] = rot(v[4], 0);  // n1 = 1, k2 = 1
    v[7] = rot(v[7], 1);  // n1 = 1, k2 = 2
    v[5] = rot(v[5], 1);  // n1 = 2, k2 = 1
    v[8] = rot(v[8], 2);  // n1 = 2, k2 = 2
    Cx<R> y[9];
#pragma unroll
    for (int k2 = 0; k2 < 3; ++k2) {
      Cx<R> a0 = v[3 * k2], a1 = v[3 * k2 + 1], a2 = v[3 * k2 + 2];
      sm_dft3<SIGN>(a0, a1, a2);
      y[k2] = a0;
      y[k2 + 3] = a1;
      y[k2 + 6] = a2;
    }
#pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = y[i];
  }
}

// The tile's two buffers (by index, so that accesses stay in the shared space)
template <typename R>
__device__ __forceinline__ Cx<R>* sm_z() {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  return reinterpret_cast<Cx<R>*>(smem_raw);
}
// A thread's walk over the points of the tile's lines, at array offset off and
// element at of the buffer.  ACROSS: along its own line in steps of the
// butterfly step (lanes side by side on different lines); else along the lines
// one after the other.  The array's contiguous dimension decides.  One
// division a tile, none a point.
template <bool ACROSS>
struct SmWalk {
  int i, k, left, at;  // line, point, points left to this thread
  int64_t off;
  int di, dk, dat, n, pitch;
  int64_t step, turn;
  __device__ __forceinline__ SmWalk(int points, Div31 d, int tw, int pitch_, int p, int b0, int step_b, int64_t base,
                                    int64_t sa, int64_t st) {
    const int nt = blockDim.x, tid = threadIdx.x;
    n = points;
    pitch = pitch_;
    if constexpr (ACROSS) {
      i = p;
      k = b0;
      left = (n - b0 + step_b - 1) / step_b;
      di = 0;
      dk = step_b;
    } else {
      i = (int)div31((unsigned)tid, d);
      k = tid - i * n;
      left = (tw * n - tid + nt - 1) / nt;
      di = (int)div31((unsigned)nt, d);
      dk = nt - di * n;
    }
    at = i * pitch + k;
    dat = di * pitch + dk;
    off = base + k * sa + i * st;
    step = dk * sa + di * st;
    turn = st - n * sa;
  }
  __device__ __forceinline__ void next() {
    k += dk;
    at += dat;
    off += step;
    if constexpr (!ACROSS) {
      i += di;
      if (k >= n) {
        k -= n;
        at += pitch - n;
        ++i;
        off += turn;
      }
    }
  }
};

// Where a thread stands in its tile.
struct SmThread {
  int p, b0, k;        // line, first butterfly and butterfly step
  int zi, zo;          // the thread's line in the stage's input and output buffer
  int sh;              // xf: shift of the stage's twiddles
  unsigned m;          // xf: largest component of the thread's outputs
};

// Stage s of radix RAD on the thread's butterflies; FIRST: the inputs come
// from ld(position), else from the line's input buffer times the twiddles.
template <typename R, int RAD, int SIGN, bool FIRST, typename LD>
__device__ __forceinline__ void sm_stage(const FastArgs& a, int s, SmThread& t, int Ls, LD ld) {
  constexpr bool XF = std::is_same<R, xf>::value;
  const int T = a.sm_m / RAD;
  Cx<R>* z = sm_z<R>();
  const void* tw = a.tw;
  if constexpr (XF) tw = reinterpret_cast<const int4*>(a.tw) + (t.sh - 1) * a.sm_ntw;
  int hi = 0, lo = 0;
  // byte steps between a butterfly's inputs, outputs and twiddles (one
  // multiply-add an access: a third of the instructions were addresses)
  constexpr unsigned EB = sizeof(Cx<R>);
  const unsigned dT = T * EB, dL = Ls * EB;
#pragma unroll 1
  for (int b = t.b0; b < T; b += t.k) {
    Cx<R> v[RAD];
    int j = 0;
    if constexpr (FIRST) {
#pragma unroll
      for (int q = 0; q < RAD; ++q) v[q] = ld(b, q, T);
    } else {
      j = b - (int)div31((unsigned)b, a.sm_ls[s]) * Ls;
      const char* zr = reinterpret_cast<const char*>(z + t.zi + b);
      const char* tp = reinterpret_cast<const char*>(tw) + (size_t)(unsigned)(a.sm_tw0[s] + j) * EB;
#pragma unroll
      for (int q = 0; q < RAD; ++q) v[q] = *reinterpret_cast<const Cx<R>*>(zr + q * dT);
#pragma unroll
      for (int q = 1; q < RAD; ++q) v[q] = tw_mul<R, SIGN>(v[q], tp + (size_t)(q - 1) * dL, 0);
      if constexpr (XF) v[0] = mk(xf_shift(v[0].re, t.sh), xf_shift(v[0].im, t.sh));
    }
    sm_dft<RAD, SIGN>(v);
    char* zw = reinterpret_cast<char*>(z + t.zo + (b - j) * RAD + j);
#pragma unroll
    for (int q = 0; q < RAD; ++q) *reinterpret_cast<Cx<R>*>(zw + q * dL) = v[q];
    if constexpr (XF) {
#pragma unroll
      for (int q = 0; q < RAD; ++q) {
        hi = __vimax3_s32(hi, v[q].re.h, v[q].im.h);
        lo = __vimin3_s32(lo, v[q].re.h, v[q].im.h);
      }
    }
  }
  t.m = (unsigned)max(hi, ~lo);
}
// The inputs of the thread's butterflies go up by some bits (xf_up), in place:
// no other thread reads them.  Out of the stage's loop, where the branch costs more
// (240^3 Float64 round trip 646 us; here 637; nowhere 630).
__device__ __forceinline__ void sm_up(Cx<xf>* z, const SmThread& t, int T, int M, int up) {
#pragma unroll 1
  for (int b = t.b0; b < T; b += t.k)
#pragma unroll 1
    for (int i = b; i < M; i += T) z[i] = mk(xf_up(z[i].re, up), xf_up(z[i].im, up));
}
template <typename R, int SIGN, bool FIRST, typename LD>
__device__ __forceinline__ void sm_radix(const FastArgs& a, int s, SmThread& t, int Ls, LD ld) {
  switch (a.sm_r[s]) {
    case 2: sm_stage<R, 2, SIGN, FIRST>(a, s, t, Ls, ld); break;
    case 3: sm_stage<R, 3, SIGN, FIRST>(a, s, t, Ls, ld); break;
    case 4: sm_stage<R, 4, SIGN, FIRST>(a, s, t, Ls, ld); break;
    case 5: sm_stage<R, 5, SIGN, FIRST>(a, s, t, Ls, ld); break;
    case 6: sm_stage<R, 6, SIGN, FIRST>(a, s, t, Ls, ld); break;
    case 7: sm_stage<R, 7, SIGN, FIRST>(a, s, t, Ls, ld); break;
    case 8: sm_stage<R, 8, SIGN, FIRST>(a, s, t, Ls, ld); break;
    default:
      if constexpr (std::is_same<R, float>::value) {
        switch (a.sm_r[s]) {
          case 9: sm_stage<R, 9, SIGN, FIRST>(a, s, t, Ls, ld); break;
          case 10: sm_stage<R, 10, SIGN, FIRST>(a, s, t, Ls, ld); break;
          case 12: sm_stage<R, 12, SIGN, FIRST>(a, s, t, Ls, ld); break;
          case 15: sm_stage<R, 15, SIGN, FIRST>(a, s, t, Ls, ld); break;
          default: sm_stage<R, 16, SIGN, FIRST>(a, s, t, Ls, ld); break;
        }
      }
  }
}

// frequency times k0 of index idx along a derivative dimension, in FP64
__device__ __forceinline__ double sm_k(int64_t idx, int half, int64_t n, float k0h, float k0l) {
  const int64_t f = (half || idx <= (n - 1) / 2) ? idx : idx - n;
  return ((double)k0h + (double)k0l) * (double)f;
}

// TW lines at a time; CTAs per SM: 64 registers a thread for Float32, 80 for
// Float64.
template <typename R, int SIGN, int OP>
__global__ void __launch_bounds__(kSmThreads, std::is_same<R, xf>::value ? 3 : 4) sm_pass(const FastArgs a) {
  pass_enter();
  constexpr bool XF = std::is_same<R, xf>::value;
  using MR = typename std::conditional<XF, double, float>::type;
  using MC = typename std::conditional<XF, double2, float2>::type;
  // xf: bits of the largest component at the first stage, below 27 by one for
  // c2r's sum of two spectra (the r2c split halves its sums)
  constexpr bool R2R = OP == OP_R2R_C || OP == OP_R2R_R;
  constexpr bool CIN = OP == OP_C2C || OP == OP_R2R_C;  // complex elements in and out
  // (D2: for its sum of two outputs; D4: one above, its first twiddles shift by one)
  const int head = R2R && a.sm_mode == SM_D2 ? 1 : 0;
  const int bits = !R2R ? 26 - (OP == OP_C2R ? 1 : 0) : a.sm_mode == SM_D2 ? 25 : a.sm_mode == SM_D4 ? 27 : 26;
  constexpr bool packed = !CIN;
  __shared__ unsigned lm[kSmStages][kSmLines];  // xf: per line, the input's largest exponent, then the stages' components
  __shared__ int loff[kSmLines];
  const int TW = a.sm_tw, M = a.sm_m, pitch = a.sm_pitch, NT = blockDim.x, tid = threadIdx.x;
  Cx<R>* z = sm_z<R>();
  const int z1 = TW * pitch;  // the second buffer
  const int lines = packed ? 2 * TW : TW;
  const TileOrigin o = tile_origin(a, blockIdx.x, lines);
  const int nvalid = (int)min((int64_t)lines, a.nt - o.t0);
  const int64_t ssa = a.in_sa, sst = a.in_st, ioff = o.ioff;
  SmThread t;
  t.k = NT / TW;
  t.b0 = tid / TW;
  t.p = tid - t.b0 * TW;
  t.sh = 1;
  if constexpr (XF) {
    for (int i = tid; i < kSmStages * kSmLines; i += NT) (&lm[0][0])[i] = 0;
    __syncthreads();
  }
  const bool lanes = a.lmap_tile != 0;

  // one input value at offset off: a complex element of line i, or the two
  // real lines' elements
  auto in1 = [&](int i, int64_t off) {
    MC x{0, 0};
    if constexpr (CIN) {
      if (i < nvalid) x = reinterpret_cast<const MC*>(a.in)[off];
    } else {
      const MR* in = reinterpret_cast<const MR*>(a.in) + off;
      if (2 * i < nvalid) x.x = in[0];
      if (2 * i + 1 < nvalid) x.y = in[sst];
    }
    return x;
  };
  // with a derivative on the input: i k src, or the sum of i k_t src_t
  const bool spectral = CIN && (a.nterm > 0 || a.deriv == 1);
  auto in1k = [&](int i, int pos, int64_t off) {
    MC x{0, 0};
    if (i >= nvalid) return x;
    const int n = a.nterm > 0 ? a.nterm : 1;
    for (int q = 0; q < n; ++q) {
      const bool sum = a.nterm > 0;
      const MC y = reinterpret_cast<const MC*>(sum ? a.tsrc[q] : a.in)[off];
      const int role = sum ? a.trole[q] : a.deriv_role;
      const int64_t idx = role == 0   ? (int64_t)pos
                          : role == 1 ? o.t0 + i
                          : sum       ? outer_index(a, blockIdx.x, role - 2)
                                      : o.didx;
      const int half = sum ? a.thalf[q] : a.deriv_half;
      const int64_t dn = sum ? a.tn[q] : a.deriv_n;
      const float kh = sum ? a.tk0_h[q] : a.k0_h, kl = sum ? a.tk0_l[q] : a.k0_l;
      if constexpr (XF) {
        const double k = sm_k(idx, half, dn, kh, kl);
        x = MC{x.x - y.y * k, x.y + y.x * k};
      } else {
        const Cx<float> w = mul_ik(mk(y.x, y.y), idx, half, dn, kh, kl);
        x = MC{x.x + w.re, x.y + w.im};
      }
    }
    return x;
  };
  const int m = M / 2 + 1;  // half spectrum of a c2r line
  const int n = a.n_in, odd = a.r2r_odd;  // R2R lines
  // where point k of an R2R line goes before a D2 transform, and where it comes
  // from after a D3 one
  auto even_odd = [&](int k) { return k & 1 ? n - ((k + 1) >> 1) : k >> 1; };
  // point k of the array line to the tile's line
  auto put = [&](MC* zl, int k, MC x) {
    if constexpr (!R2R) {
      zl[k] = x;
    } else if (a.sm_mode == SM_D2) {
      if (odd == 1 && (k & 1)) x = MC{-x.x, -x.y};
      zl[odd == 2 ? k : even_odd(k)] = x;
    } else if (a.sm_mode == SM_D3) {
      zl[odd ? n - 1 - k : k] = x;
    } else if (a.sm_mode == SM_X) {
      if (odd) {
        zl[k + 1] = x;
        zl[M - 1 - k] = MC{-x.x, -x.y};
      } else {
        zl[k] = x;
        if (k >= 1 && k <= n - 2) zl[M - k] = x;
      }
    } else {
      zl[k] = x;
    }
  };
  const bool pre = R2R && (a.sm_mode == SM_D3 || a.sm_mode == SM_D4);  // twiddles before the first stage

  // ---- first stage, its inputs copied to z1 where the lanes read along the
  // line (or the values need their line's exponent, or mirror a half
  // spectrum), else straight from memory ----
  t.zo = t.p * pitch;
  const int zc = z1 + t.p * pitch;
  bool direct = false;
  if constexpr (!XF && OP != OP_C2R && !R2R) {
    direct = lanes && !spectral;
    if (direct) {
      const int64_t off = ioff + (t.p * (packed ? 2 : 1)) * sst;
      sm_radix<R, SIGN, true>(a, 0, t, 1, [&](int b, int q, int T) {
        const MC x = in1(t.p, off + b * ssa + q * (T * ssa));
        return mk(x.x, x.y);
      });
    }
  }
  if (!direct) {
    MC* zr = reinterpret_cast<MC*>(z) + z1;  // raw values (xf: doubles, converted at the first stage)
    const int points = OP == OP_C2R ? m : R2R ? n : M;
    unsigned emx = 0;
    if constexpr (R2R) {
      if (a.sm_mode == SM_X && odd && t.b0 == 0) zr[t.p * pitch] = zr[t.p * pitch + M / 2] = MC{0, 0};
    }
    auto load = [&](auto w) {
      if constexpr (OP == OP_C2R) {
        const MC* in = reinterpret_cast<const MC*>(a.in);
#pragma unroll 2
        for (; w.left > 0; --w.left, w.next()) {
          const int k = w.k;
          MC A{0, 0}, B{0, 0};
          if (2 * w.i < nvalid) A = in[w.off];
          if (2 * w.i + 1 < nvalid) B = in[w.off + sst];
          MC* zk = zr + w.at;
          if constexpr (XF) {
            zk[0] = A;
            zk[m] = B;
            emx = max(emx, max(max(dexp_u(A.x), dexp_u(A.y)), max(dexp_u(B.x), dexp_u(B.y))));
          } else if (k == 0 || 2 * k == M) {
            zk[0] = MC{A.x, B.x};
          } else {  // A + i B, and conj(A) + i conj(B) at M - k
            zk[0] = MC{A.x - B.y, A.y + B.x};
            zk[M - 2 * k] = MC{A.x + B.y, B.x - A.y};
          }
        }
      } else if (spectral) {
#pragma unroll 1
        for (; w.left > 0; --w.left, w.next()) {
          const MC x = in1k(w.i, w.k, w.off);
          put(zr + w.at - w.k, w.k, x);
          if constexpr (XF) emx = max(emx, max(dexp_u(x.x), dexp_u(x.y)));
        }
      } else {
        constexpr int U = XF ? 4 : 8;  // loads in flight a thread
#pragma unroll 1
        while (w.left > 0) {
          MC x[U];
          int at[U], pt[U];
#pragma unroll
          for (int q = 0; q < U; ++q) {
            const bool ok = w.left > q;
            at[q] = ok ? w.at : -1;
            pt[q] = w.k;
            x[q] = in1(ok ? w.i : nvalid, w.off);
            w.next();
          }
          w.left -= U;
#pragma unroll
          for (int q = 0; q < U; ++q) {
            if (at[q] >= 0) put(zr + at[q] - pt[q], pt[q], x[q]);
            if constexpr (XF) emx = max(emx, max(dexp_u(x[q].x), dexp_u(x[q].y)));
          }
        }
      }
    };
    if (lanes) load(SmWalk<true>(points, a.sm_din, TW, pitch, t.p, t.b0, t.k, ioff, ssa, packed ? 2 * sst : sst));
    else load(SmWalk<false>(points, a.sm_din, TW, pitch, t.p, t.b0, t.k, ioff, ssa, packed ? 2 * sst : sst));
    if constexpr (XF) {
      if (!lanes) {  // lines along the lanes: each line's own threads look it over
        __syncthreads();
        emx = 0;
        const MC* zl = zr + t.p * pitch;
        const int held = OP == OP_C2R ? 2 * m : R2R && a.sm_mode == SM_D4 ? n : M;
        for (int q = t.b0; q < held; q += t.k) {
          const MC x = zl[q];
          emx = max(emx, max(dexp_u(x.x), dexp_u(x.y)));
        }
      }
      atomicMax(&lm[0][t.p], emx);
    }
    __syncthreads();
    if constexpr (R2R) {
      if (pre) {  // in place: a thread holds both points of each pair
        const MC* zl = reinterpret_cast<const MC*>(z) + zc;
        const int emax = XF ? (int)lm[0][t.p] : 0;
        const float fs = XF ? xf_frac_scale(emax) : 0.0f;
        auto val = [&](MC x) {
          if constexpr (XF) return mk(d2xf(x.x, emax, fs, bits), d2xf(x.y, emax, fs, bits));
          else return mk(x.x, x.y);
        };
        if (a.sm_mode == SM_D3) {  // conj(w_k) (x[k] - i x[n - k])
          for (int k = t.b0; 2 * k <= n; k += t.k) {
            const Cx<R> A = val(zl[k]);
            if (k == 0) {
              if constexpr (XF) z[zc] = mk(xf_shift(A.re, 1), xf_shift(A.im, 1));
              else z[zc] = A;
            } else {
              const Cx<R> B = val(zl[n - k]);
              z[zc + k] = tw_mul<R, 1>(A + mul_mi(B), a.d23_tab, k);
              if (2 * k != n) z[zc + n - k] = tw_mul<R, 1>(B + mul_mi(A), a.d23_tab, n - k);
            }
          }
        } else {
          for (int j = t.b0; j < n; j += t.k) {
            const Cx<R> A = val(zl[j]);
            const Cx<R> B = tw_mul<R, -1>(A, a.d23_tab, 2 * n - 1 - j);
            z[zc + j] = tw_mul<R, -1>(A, a.d23_tab, j);
            z[zc + 2 * n - 1 - j] = odd ? B : -B;
          }
        }
        __syncthreads();
      }
    }
    if constexpr (XF) {
      const int emax = (int)lm[0][t.p];
      const float fs = xf_frac_scale(emax);
      const MC* zl = reinterpret_cast<const MC*>(z) + zc;
      sm_radix<R, SIGN, true>(a, 0, t, 1, [&](int b, int q, int T) {
        const int pos = b + q * T;
        if constexpr (OP == OP_C2R) {
          const int k = pos < m ? pos : M - pos;
          const MC qa = zl[k], qb = zl[m + k];
          Cx<R> A = mk(d2xf(qa.x, emax, fs, bits), d2xf(qa.y, emax, fs, bits));
          Cx<R> B = mk(d2xf(qb.x, emax, fs, bits), d2xf(qb.y, emax, fs, bits));
          if (k == 0 || 2 * k == M) { A.im = xf(0, 0.0f); B.im = xf(0, 0.0f); }
          if (pos >= m) { A.im = -A.im; B.im = -B.im; }
          return mk(A.re - B.im, A.im + B.re);
        } else {
          if (R2R && pre) return z[zc + pos];
          const MC x = zl[pos];
          return mk(d2xf(x.x, emax, fs, bits), d2xf(x.y, emax, fs, bits));
        }
      });
    } else {
      sm_radix<R, SIGN, true>(a, 0, t, 1, [&](int b, int q, int T) { return z[zc + b + q * T]; });
    }
  }

  // ---- the other stages ----
  int Ls = a.sm_r[0], shifts = pre ? 1 : 0;
  int za = 0, zb = z1;  // output of the last stage, the other buffer
#pragma unroll 1
  for (int s = 1; s < a.sm_nst; ++s) {
    if constexpr (XF) atomicMax(&lm[s][t.p], t.m);
    __syncthreads();
    if constexpr (XF) {
      const int r = a.sm_r[s], excess = xf_excess(lm[s][t.p], r) + head;
      t.sh = xf_shift_of(excess);
      shifts += t.sh;
      if (const int up = xf_up_of(excess, xf_slack(r))) {
        sm_up(z + za + t.p * pitch, t, M / r, M, up);
        shifts -= up;
      }
    }
    t.zi = za + t.p * pitch;
    t.zo = zb + t.p * pitch;
    sm_radix<R, SIGN, false>(a, s, t, Ls, [](int, int, int) { return mk(R(), R()); });
    Ls *= a.sm_r[s];
    const int x = za;
    za = zb;
    zb = x;
  }
  if constexpr (XF && R2R) shifts += a.sm_mode == SM_D2 || a.sm_mode == SM_D4 ? 1 : 0;  // twiddles after the last
  if constexpr (XF) {
    // the unit's exponent with the line's, and the normalisation's
    if (t.b0 == 0) loff[t.p] = 127 - bits + shifts + (int)lm[0][t.p] + a.emax_shift - 254 + a.scale_xe;
  }
  __syncthreads();

  // ---- store ----
  auto out1 = [&](Cx<R> y, int i) {
    MC q;
    if constexpr (XF) {
      if (a.scale_on) y = mk(xf_scaled(y.re, a.scale_xw, a.scale_xo, a.scale_xf), xf_scaled(y.im, a.scale_xw, a.scale_xo, a.scale_xf));
      xf2d(y, loff[i], q.x, q.y);
    } else {
      y = apply_scale(y, a);
      q = MC{y.re, y.im};
    }
    return q;
  };
  // output k of an R2R line
  auto post = [&](const Cx<R>* zl, int k) {
    if (a.sm_mode == SM_D2) {
      const int q = odd == 1 ? n - 1 - k : k;
      const Cx<R> V = zl[q], W = zl[q == 0 ? 0 : n - q], S = V + W, D = V - W;
      return mk(tw_mul<R, -1>(mk(S.re, D.im), a.d23_tab, q).re, tw_mul<R, -1>(mk(S.im, -D.re), a.d23_tab, q).re);
    }
    if (a.sm_mode == SM_D3) {  // the DFT of the other sign: outputs backwards
      const int q = even_odd(k);
      const Cx<R> y = zl[q == 0 ? 0 : n - q];
      return odd && (k & 1) ? -y : y;
    }
    const Cx<R> y = a.sm_mode == SM_X ? zl[k + (odd ? 1 : 0)] : tw_mul<R, -1>(zl[k], a.d23_tab, 2 * n + k);
    return odd ? mul_i(y) : y;
  };
  auto store = [&](auto w) {
#pragma unroll 2
    for (; w.left > 0; --w.left, w.next()) {
      const int i = w.i, k = w.k;
      const Cx<R>* zl = z + za + w.at - k;
      if constexpr (CIN) {
        if (i >= nvalid) continue;
        MC y = out1(R2R ? post(zl, k) : zl[k], i);
        if (a.deriv == 2) {  // fused spectral derivative on the output
          const int64_t idx = a.deriv_role == 0 ? (int64_t)k : a.deriv_role == 1 ? o.t0 + i : o.didx;
          if constexpr (XF) {
            const double kk = sm_k(idx, a.deriv_half, a.deriv_n, a.k0_h, a.k0_l);
            y = MC{-y.y * kk, y.x * kk};
          } else {
            const Cx<float> q = mul_ik(mk(y.x, y.y), idx, a.deriv_half, a.deriv_n, a.k0_h, a.k0_l);
            y = MC{q.re, q.im};
          }
        }
        reinterpret_cast<MC*>(a.out)[w.off] = y;
      } else if constexpr (OP == OP_R2C) {
        const Cx<R> f = zl[k], g = conj(zl[k == 0 ? 0 : M - k]);
        Cx<R> A, B;
        if constexpr (XF) {
          A = xf_half_sum(f, g);
          B = mul_mi(xf_half_sum(f, -g));
        } else {
          A = f + g;
          B = mul_mi(f - g);
          A = mk(half(A.re), half(A.im));
          B = mk(half(B.re), half(B.im));
        }
        MC* out = reinterpret_cast<MC*>(a.out) + w.off;
        if (2 * i < nvalid) out[0] = out1(A, i);
        if (2 * i + 1 < nvalid) out[a.out_st] = out1(B, i);
      } else {  // real outputs of lines 2 i and 2 i + 1
        const MC y = out1(R2R ? post(zl, k) : zl[k], i);
        MR* out = reinterpret_cast<MR*>(a.out) + w.off;
        if (2 * i < nvalid) out[0] = y.x;
        if (2 * i + 1 < nvalid) out[a.out_st] = y.y;
      }
    }
  };
  const int outs = OP == OP_R2C ? m : R2R ? n : M;
  const int64_t ost = packed ? 2 * a.out_st : a.out_st;
  if (a.out_tfast) store(SmWalk<true>(outs, a.sm_dout, TW, pitch, t.p, t.b0, t.k, o.ooff, a.out_sa, ost));
  else store(SmWalk<false>(outs, a.sm_dout, TW, pitch, t.p, t.b0, t.k, o.ooff, a.out_sa, ost));
}

int fail_cuda(cudaError_t e, const char* what);

// grid == 0 only sets the shared-memory attribute
template <typename R, int SIGN, int OP>
static int launch_sm_one(const FastArgs& A, int64_t grid, int threads, size_t smem, cudaStream_t s) {
  static bool configured[kMaxDevicesConfigured] = {};
  int rc = ensure_smem_attr(sm_pass<R, SIGN, OP>, kSmMaxSmem, configured, "cudaFuncSetAttribute(sm_pass)");
  if (rc || grid == 0) return rc;
  const cudaError_t e = launch_pass_kernel(sm_pass<R, SIGN, OP>, grid, threads, smem, s, A);
  if (e != cudaSuccess) return fail_cuda(e, "sm_pass launch");
  return PFGB_OK;
}

}  // namespace pfgb
