// Register pass for mixed-radix lines of M = R0 * N points (R0 = 3 or 5,
// N = 2^LOGN >= 8): one 1D transform per line, any input / output layout,
// the pencil re-layout fused into the store.
//
// Decomposition n = n1 + N n2 (n1 < N, n2 < R0), k = k2 + R0 k1:
//   X[k2 + R0 k1] = sum_n1 W_N^(n1 k1) [ W_M^(n1 k2) sum_n2 x[n1 + N n2] W_R0^(n2 k2) ].
// Phase A: thread (line p, index b) holds the positions n1 = b + r N/8
// (r < 8) of its line; for each r it loads the R0 inputs x[n1 + N n2],
// computes their R0-point DFT in registers (symmetric split; roots of unity
// from the first R0 entries of tw2), multiplies by the twiddles W_M^(n1 k2)
// (its other entries, consecutive for consecutive n1) and parks value k2 in
// sub-line k2 of shared memory.  Phase B: each sub-line is an
// N-point transform computed by the power-of-two register stages
// (fast_stages), its outputs X[k2 + R0 k1] left in the sub-line at k1.
// Store: one loop over the tile's outputs through shared memory (c2c, the
// r2c split of two packed real lines, or the two real outputs of a c2r
// line), coalesced along the output's contiguous dimension.
//
// Float64 data compute phase A in double-float (dd) and phase B in integer-float
// pairs (fast_stages), with one power-of-two scale per complex line (its largest
// input exponent), doubles in and out; Float32 in FP32.  Float64 lines come here
// in plans of fewer than 16 complex lines; the others take sm_pass.
#pragma once

#include "pfgb_fast.cuh"

namespace pfgb {

// threads per CTA and lines (complex) per tile
template <typename R>
__host__ __device__ constexpr int mr_threads(int logn) {
  return ((1 << logn) / 8) > 256 ? (1 << logn) / 8 : 256;
}
template <typename R>
__host__ __device__ constexpr int mr_tw(int logn) {
  return mr_threads<R>(logn) / ((1 << logn) / 8);
}
// sub-line pitch in elements (the exchange layout of fast_stages)
template <typename R, int LOGN, int OP>
__host__ __device__ constexpr int mr_pitch() {
  return fast_pitch<R>(LOGN, OP);
}
template <typename R>
__host__ __device__ constexpr size_t mr_smem(int r0, int logn, int op) {
  return (size_t)r0 * mr_tw<R>(logn) * fast_pitch<R>(logn, op) * sizeof(Cx<R>);
}

// y_k = sum_j v_j exp(SIGN 2 pi i j k / R0) for odd R0, from the R0-th roots
// exp(-2 pi i m / R0) (the first R0 entries of tw2)
template <int R0, int SIGN, typename R>
__device__ __forceinline__ void mr_dft_odd(Cx<R> (&v)[R0], const void* tw2) {
  constexpr int H = (R0 - 1) / 2;
  Cx<R> s[H], d[H];
  Cx<R> y0 = v[0];
#pragma unroll
  for (int j = 1; j <= H; ++j) {
    s[j - 1] = v[j] + v[R0 - j];
    d[j - 1] = v[j] - v[R0 - j];
    y0 = y0 + s[j - 1];
  }
  Cx<R> y[R0];
  y[0] = y0;
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    Cx<R> a = v[0], b = mk(R(0), R(0));
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      const Cx<R> w = ldg_tw<R>(tw2, (j * k) % R0);  // (cos t, -sin t)
      a = a + mk(s[j - 1].re * w.re, s[j - 1].im * w.re);
      b = b - mk(d[j - 1].re * w.im, d[j - 1].im * w.im);  // sum d_j sin t
    }
    const Cx<R> ib = mul_i(b);
    if (SIGN < 0) {
      y[k] = a - ib;
      y[R0 - k] = a + ib;
    } else {
      y[k] = a + ib;
      y[R0 - k] = a - ib;
    }
  }
#pragma unroll
  for (int i = 0; i < R0; ++i) v[i] = y[i];
}

// NT threads (mr_threads by default; the persistent batch kernel runs the
// tile with its own CTA size), NT / (N / 8) complex lines a tile.
template <typename R, int R0, int LOGN, int SIGN, int OP, int NT = mr_threads<R>(LOGN)>
__device__ __forceinline__ void mr_tile(const FastArgs& a, int64_t bid, Cx<R>* z) {
  using IO = FastIO<R>;
  using MR = typename IO::MR;
  using MC = typename IO::MC;
  constexpr int N = 1 << LOGN;
  constexpr int M = R0 * N;
  constexpr int T = N / 8;
  constexpr int TW = NT / T;
  static_assert(NT % T == 0 && TW >= 1, "mr_tile: threads must hold whole lines");
  constexpr int PITCH = mr_pitch<R, LOGN, OP>();
  constexpr bool packed = OP == OP_R2C || OP == OP_C2R;

  const int tid = threadIdx.x;
  int p, b;
  if (a.lmap_tile) { p = tid % TW; b = tid / TW; } else { b = tid % T; p = tid / T; }
  const int lines = packed ? 2 * TW : TW;
  const TileOrigin o = tile_origin(a, (unsigned)bid, lines);
  const int64_t t0 = o.t0, ooff = o.ooff, ioff = o.ioff, didx = o.didx;
  const int nvalid = (int)min((int64_t)lines, a.nt - t0);
  const int ncl_valid = packed ? (nvalid + 1) / 2 : nvalid;
  const int64_t ssa = a.in_sa, sst = a.in_st;
  auto sub = [&](int s) { return z + (size_t)s * TW * PITCH; };  // sub-line region s

  // ---- line exponent (dd): largest input exponent of the complex line ----
  int emax = 0;
  __shared__ int lexp[TW];
  if constexpr (IO::kDD) {
    unsigned emx = 0;
#pragma unroll 1
    for (int r = 0; r < 8; ++r) {
#pragma unroll
      for (int n2 = 0; n2 < R0; ++n2) {
        const int n = b + r * T + N * n2;
        if constexpr (OP == OP_C2C) {
          for (int t = 0; t < (a.nterm > 0 ? a.nterm : 1); ++t) {
            const void* src = a.nterm > 0 ? a.tsrc[t] : a.in;
            const MC q = p < nvalid ? reinterpret_cast<const MC*>(src)[ioff + (int64_t)n * ssa + (int64_t)p * sst] : MC{0, 0};
            emx = max(emx, max(dexp_u(q.x), dexp_u(q.y)));
          }
        } else if constexpr (OP == OP_R2C) {
          const MR* in = reinterpret_cast<const MR*>(a.in) + ioff + (int64_t)n * ssa;
          const MR qa = 2 * p < nvalid ? in[(int64_t)(2 * p) * sst] : MR(0);
          const MR qb = 2 * p + 1 < nvalid ? in[(int64_t)(2 * p + 1) * sst] : MR(0);
          emx = max(emx, max(dexp_u(qa), dexp_u(qb)));
        } else {
          const int k = n <= M / 2 ? n : M - n;
          const MC* in = reinterpret_cast<const MC*>(a.in) + ioff + (int64_t)k * ssa;
          const MC qa = 2 * p < nvalid ? in[(int64_t)(2 * p) * sst] : MC{0, 0};
          const MC qb = 2 * p + 1 < nvalid ? in[(int64_t)(2 * p + 1) * sst] : MC{0, 0};
          emx = max(emx, max(max(dexp_u(qa.x), dexp_u(qa.y)), max(dexp_u(qb.x), dexp_u(qb.y))));
        }
      }
    }
    emax = line_exponent<R, LOGN, OP>(emx, a, (unsigned)bid, t0, p, ncl_valid, a.lmap_tile != 0);
    if (b == 0) lexp[p] = emax;
  }

  // ---- phase A: R0-point DFTs, twiddles, park in the sub-lines (a loop:
  // nothing is held in registers across its rounds).  The loads of a round's
  // BA positions are issued before its stores to shared memory, which the
  // compiler does not move them over: with one position a round the Float32
  // 384-point passes waited for memory 8 times a tile (3 x 384^3 gradient
  // 2.69 -> 2.59 ms) ----
  constexpr bool MIRROR = OP == OP_C2R && !IO::kDD;
  if constexpr (MIRROR) {
    // Half spectra: positions n1 = g and N - g need the same R0 pairs (A, B), at
    // k = g + N j and (N - g) + N j, and take them as A + i B up to M / 2 and
    // conj(A) + i conj(B) beyond.  One thread does both, so each input is loaded
    // once (each position on its own loaded them twice: the 384^3 c2r pass
    // 195 -> 144 us).  Position 0 stands alone, as does N / 2.
    constexpr int HU = (R0 + 1) / 2, G = 2;  // groups whose loads are issued together
    const MC* in = reinterpret_cast<const MC*>(a.in) + ioff + (2 * p) * sst;
    const bool ok0 = 2 * p < nvalid, ok1 = 2 * p + 1 < nvalid;
    auto load = [&](int g, MC (&A)[R0], MC (&B)[R0]) {
#pragma unroll
      for (int j = 0; j < R0; ++j) {
        const int k = j < HU ? g + N * j : N - g + N * (j - HU);
        A[j] = B[j] = MC{0, 0};
        if (ok0) A[j] = in[k * ssa];
        if (ok1) B[j] = in[k * ssa + sst];
      }
    };
    auto position = [&](int n1, bool second, const MC (&A)[R0], const MC (&B)[R0]) {
      Cx<R> u[R0];
#pragma unroll
      for (int n2 = 0; n2 < R0; ++n2) {
        // first: U_n2 below M / 2, then V mirrored; second: V_n2, then U mirrored
        const int e = second ? (n2 < R0 - HU ? HU + n2 : R0 - 1 - n2) : (n2 < HU ? n2 : HU + R0 - 1 - n2);
        const bool mirror = second ? n2 >= R0 - HU : n2 >= HU;
        const int k = mirror ? M - n1 - N * n2 : n1 + N * n2;
        MC x = A[e], y = B[e];
        if (k == 0 || 2 * k == M) x.y = y.y = 0;
        u[n2] = mirror ? mk(x.x + y.y, y.x - x.y) : mk(x.x - y.y, x.y + y.x);
      }
      mr_dft_odd<R0, SIGN>(u, a.tw2);
#pragma unroll
      for (int k2 = 0; k2 < R0; ++k2)
        sub(k2)[sidx<R, LOGN, OP>(p, n1)] = k2 == 0 ? u[0] : tw_mul<R, SIGN>(u[k2], a.tw2, R0 + (k2 - 1) * N + n1);
    };
#pragma unroll 1
    for (int r = 0; r < 4; r += G) {
      MC A[G][R0], B[G][R0];
#pragma unroll
      for (int q = 0; q < G; ++q) load(b + (r + q) * T, A[q], B[q]);
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int g = b + (r + q) * T;
        position(g, false, A[q], B[q]);
        if (g != 0) position(N - g, true, A[q], B[q]);
      }
    }
    if (b == 0) {
      MC A[R0], B[R0];
      load(N / 2, A, B);
      position(N / 2, false, A, B);
    }
    line_sync<R, LOGN, OP>(a.lmap_tile != 0, p);
  } else {
    constexpr int BA = IO::kDD ? 1 : 4;
#pragma unroll 1
    for (int r0 = 0; r0 < 8; r0 += BA) {
      MC ra[BA][R0], rb[BA][R0];
      if (OP != OP_C2C || a.nterm == 0) {
#pragma unroll
        for (int q = 0; q < BA; ++q)
#pragma unroll
          for (int n2 = 0; n2 < R0; ++n2) {
            const int n = b + (r0 + q) * T + N * n2;
            ra[q][n2] = rb[q][n2] = MC{0, 0};
            if constexpr (OP == OP_C2C) {
              if (p < nvalid) ra[q][n2] = reinterpret_cast<const MC*>(a.in)[ioff + n * ssa + p * sst];
            } else if constexpr (OP == OP_R2C) {
              const MR* in = reinterpret_cast<const MR*>(a.in) + ioff + n * ssa;
              if (2 * p < nvalid) ra[q][n2].x = in[(2 * p) * sst];
              if (2 * p + 1 < nvalid) ra[q][n2].y = in[(2 * p + 1) * sst];
            } else {  // C2R: Hermitian extension of two half spectra (m = M/2 + 1 inputs)
              const MC* in = reinterpret_cast<const MC*>(a.in) + ioff + (n <= M / 2 ? n : M - n) * ssa;
              if (2 * p < nvalid) ra[q][n2] = in[(2 * p) * sst];
              if (2 * p + 1 < nvalid) rb[q][n2] = in[(2 * p + 1) * sst];
            }
          }
      }
#pragma unroll
      for (int q = 0; q < BA; ++q) {
        const int n1 = b + (r0 + q) * T;
        Cx<R> u[R0];
#pragma unroll
        for (int n2 = 0; n2 < R0; ++n2) {
          const int n = n1 + N * n2;
          u[n2] = mk(mkr<R>(ra[q][n2].x, emax), mkr<R>(ra[q][n2].y, emax));
          if constexpr (OP == OP_C2C) {
            if (a.nterm > 0) {  // sum of i k_t src_t (fused divergence / curl)
              u[n2] = mk(R(0), R(0));
              for (int t = 0; t < a.nterm; ++t) {
                const MC x = p < nvalid ? reinterpret_cast<const MC*>(a.tsrc[t])[ioff + n * ssa + p * sst] : MC{0, 0};
                const int64_t idx = a.trole[t] == 0   ? (int64_t)n
                                    : a.trole[t] == 1 ? t0 + p
                                                      : outer_index(a, (unsigned)bid, a.trole[t] - 2);
                u[n2] = u[n2] + mul_ik(mk(mkr<R>(x.x, emax), mkr<R>(x.y, emax)), idx, a.thalf[t], a.tn[t],
                                       a.tk0_h[t], a.tk0_l[t]);
              }
            }
            if (a.deriv == 1) {
              const int64_t idx = a.deriv_role == 0 ? (int64_t)n : a.deriv_role == 1 ? t0 + p : didx;
              u[n2] = mul_ik(u[n2], idx, a.deriv_half, a.deriv_n, a.k0_h, a.k0_l);
            }
          } else if constexpr (OP == OP_C2R) {
            Cx<R> B = mk(mkr<R>(rb[q][n2].x, emax), mkr<R>(rb[q][n2].y, emax));
            if (n == 0 || 2 * n == M) { u[n2].im = R(0); B.im = R(0); }
            if (n > M / 2) { u[n2].im = -u[n2].im; B.im = -B.im; }
            u[n2] = mk(u[n2].re - B.im, u[n2].im + B.re);
          }
        }
        mr_dft_odd<R0, SIGN>(u, a.tw2);
#pragma unroll
        for (int k2 = 0; k2 < R0; ++k2) {
          const Cx<R> y = k2 == 0 ? u[0] : tw_mul<R, SIGN>(u[k2], a.tw2, R0 + (k2 - 1) * N + n1);
          sub(k2)[sidx<R, LOGN, OP>(p, n1)] = y;
        }
      }
    }
  }

  // ---- phase B: the N-point transform of each sub-line ----
#pragma unroll 1
  for (int s = 0; s < R0; ++s) {
    Cx<R>* zs = sub(s);
    Cx<R> v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = zs[sidx<R, LOGN, OP>(p, b + r * T)];
    // every thread of the line has read its inputs before the first exchange writes
    line_sync<R, LOGN, OP>(a.lmap_tile != 0, p);
    fast_stages<R, LOGN, SIGN, OP>(v, zs, p, b, a.tw, a.lmap_tile != 0);
    // fast_stages ends after a barrier that follows the last exchange read:
    // the outputs X[s + R0 k1], k1 = b + r T, overwrite the sub-line
#pragma unroll
    for (int r = 0; r < 8; ++r) zs[sidx<R, LOGN, OP>(p, b + r * T)] = v[r];
  }
  __syncthreads();

  // ---- store: element k of line i is sub-line k mod R0 at k / R0 ----
  auto at = [&](int i, int k) { return sub(k % R0)[sidx<R, LOGN, OP>(i, k / R0)]; };
  auto eo = [&](int i) { return IO::kDD ? lexp[i] + a.emax_shift : 0; };
  // all M outputs of each line, 8 R0 a thread.  Along the lines: stepped without
  // divisions (k = s + R0 k1; 384^3 c2c pass 142 -> 133 us); across them a point's
  // line and position are a mask and a shift.
  auto each = [&](auto put) {
    const int64_t sto = OP == OP_C2R ? 2 * a.out_st : a.out_st;
    if (a.out_tfast) {
#pragma unroll 1
      for (int e = tid; e < TW * M; e += NT) {
        const int i = e % TW, k = e / TW;
        put(i, k, apply_scale(at(i, k), a), ooff + k * a.out_sa + i * sto);
      }
    } else {
      const int k0 = tid % M;
      int i = tid / M, k1 = k0 / R0, s = k0 % R0;
      constexpr int dk = NT % M, di = NT / M;
      int64_t off = ooff + k0 * a.out_sa + i * sto;
      const int64_t step = dk * a.out_sa + di * sto, turn = sto - M * a.out_sa;
#pragma unroll 4
      for (int e = 0; e < 8 * R0; ++e) {
        put(i, s + R0 * k1, apply_scale(sub(s)[sidx<R, LOGN, OP>(i, k1)], a), off);
        off += step;
        i += di;
        k1 += dk / R0;
        s += dk % R0;
        if (s >= R0) { s -= R0; ++k1; }
        if (k1 >= N) { k1 -= N; ++i; off += turn; }
      }
    }
  };
  if constexpr (OP == OP_C2C) {
    each([&](int i, int k, Cx<R> y, int64_t off) {
      if (i >= nvalid) return;
      if (a.deriv == 2) {
        const int64_t idx = a.deriv_role == 0 ? (int64_t)k : a.deriv_role == 1 ? t0 + i : didx;
        y = mul_ik(y, idx, a.deriv_half, a.deriv_n, a.k0_h, a.k0_l);
      }
      MC q;
      q.x = outr<R>(y.re, eo(i));
      q.y = outr<R>(y.im, eo(i));
      reinterpret_cast<MC*>(a.out)[off] = q;
    });
  } else if constexpr (OP == OP_R2C) {
    MC* out = reinterpret_cast<MC*>(a.out) + ooff;
    constexpr int m = M / 2 + 1;
    constexpr int tot = TW * m;
    for (int e = tid; e < tot; e += NT) {
      int q, k;
      if (a.out_tfast) { q = e % TW; k = e / TW; } else { k = e % m; q = e / m; }
      const Cx<R> f = at(q, k);
      const Cx<R> g = conj(at(q, k == 0 ? 0 : M - k));
      Cx<R> A = f + g, B = mul_mi(f - g);
      A = apply_scale(mk(half(A.re), half(A.im)), a);
      B = apply_scale(mk(half(B.re), half(B.im)), a);
      const int i0 = 2 * q, i1 = 2 * q + 1;
      const int64_t off = (int64_t)k * a.out_sa;
      if (i0 < nvalid) {
        MC w;
        w.x = outr<R>(A.re, eo(q));
        w.y = outr<R>(A.im, eo(q));
        out[off + (int64_t)i0 * a.out_st] = w;
      }
      if (i1 < nvalid) {
        MC w;
        w.x = outr<R>(B.re, eo(q));
        w.y = outr<R>(B.im, eo(q));
        out[off + (int64_t)i1 * a.out_st] = w;
      }
    }
  } else {  // C2R: real outputs of lines 2q and 2q + 1
    each([&](int q, int, Cx<R> y, int64_t off) {
      MR* out = reinterpret_cast<MR*>(a.out) + off;
      if (2 * q < nvalid) out[0] = outr<R>(y.re, eo(q));
      if (2 * q + 1 < nvalid) out[a.out_st] = outr<R>(y.im, eo(q));
    });
  }
}

template <typename R, int R0, int LOGN, int SIGN, int OP>
__global__ void __launch_bounds__(mr_threads<R>(LOGN)) mr_pass(const FastArgs a) {
  pass_enter();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  mr_tile<R, R0, LOGN, SIGN, OP>(a, blockIdx.x, reinterpret_cast<Cx<R>*>(smem_raw));
}

// Launchers; grid == 0 only sets the shared-memory attribute.  Line lengths:
// R0 = 3 and 5 with N = 8 .. 512.
int fail_cuda(cudaError_t e, const char* what);

template <typename R, int R0, int LOGN, int SIGN, int OP>
static int launch_mr_one(const FastArgs& A, int64_t grid, cudaStream_t s) {
  static bool configured[kMaxDevicesConfigured] = {};
  const size_t smem = mr_smem<R>(R0, LOGN, OP);
  int rc = ensure_smem_attr(mr_pass<R, R0, LOGN, SIGN, OP>, (int)smem, configured, "cudaFuncSetAttribute(mr_pass)");
  if (rc || grid == 0) return rc;
  const cudaError_t e = launch_pass_kernel(mr_pass<R, R0, LOGN, SIGN, OP>, grid, mr_threads<R>(LOGN), smem, s, A);
  if (e != cudaSuccess) return fail_cuda(e, "mr_pass launch");
  return PFGB_OK;
}

template <typename R, int R0, int SIGN, int OP>
static int launch_mr_n(int logn, const FastArgs& A, int64_t grid, cudaStream_t s) {
  switch (logn) {
    case 3: return launch_mr_one<R, R0, 3, SIGN, OP>(A, grid, s);
    case 4: return launch_mr_one<R, R0, 4, SIGN, OP>(A, grid, s);
    case 5: return launch_mr_one<R, R0, 5, SIGN, OP>(A, grid, s);
    case 6: return launch_mr_one<R, R0, 6, SIGN, OP>(A, grid, s);
    case 7: return launch_mr_one<R, R0, 7, SIGN, OP>(A, grid, s);
    case 8: return launch_mr_one<R, R0, 8, SIGN, OP>(A, grid, s);
    case 9: return launch_mr_one<R, R0, 9, SIGN, OP>(A, grid, s);
    default: return PFGB_ERR_UNSUPPORTED;
  }
}

template <typename R, int R0, int OP>
static int launch_mr_r0(int logn, int sign, const FastArgs& A, int64_t grid, cudaStream_t s) {
  return sign < 0 ? launch_mr_n<R, R0, -1, OP>(logn, A, grid, s) : launch_mr_n<R, R0, 1, OP>(logn, A, grid, s);
}

}  // namespace pfgb
