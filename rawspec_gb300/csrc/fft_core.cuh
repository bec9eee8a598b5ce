// fft_core.cuh -- the FFT engine of the spectrometer kernels.
//
// Two levels:
//   * dft_regs<R>: an R-point DFT (R a power of two <= 32) held entirely in
//     registers; radix-2 decimation in time, natural order in and out, every
//     twiddle multiplication fused into its butterfly.
//   * GroupFFT<N, R>: an N-point FFT computed by a group of T = N/R threads,
//     each holding R values of two vectors in lockstep, which share every
//     twiddle.  Stockham auto-sort passes of radix R (a smaller radix for the
//     last pass when N is not a power of R), with one shared-memory exchange
//     between passes.  On entry thread j holds x[j + m*T] in v[m]; on exit it
//     holds X[j + m*T].  The formulation is the classic per-thread Stockham
//     iteration (Govindaraju et al., SC08).
//
// All FFTs here are forward, exp(-2 pi i k n / N), unnormalised; the inverse
// transform is obtained by the index reversal X_inv[k] = X_fwd[(N-k) mod N]
// applied where results are stored.
//
// Butterflies.  The kernels are bound by the FMA pipe (on which a packed
// f32x2 instruction takes two issue slots of a scalar one), so the engine
// counts pipe slots.  a +- w b with w = c (1 - i t), t = tan of the angle, is
// six fused multiply-adds,
//   u = b.re + t b.im,  v = b.im - t b.re,  a +- c (u + i v),
// against eight operations for a product followed by two sums (the form of
// Linzer and Feig, "Implementation of efficient FFT algorithms on fused
// multiply-add architectures", IEEE Trans. Signal Processing 41, 1993).  In a
// twiddled pass the input factors w^r, r < R, need no multiplications of
// their own: the stage of length L of a decimation-in-time DFT takes
// w^(R/L) W_L^q, and q and q + L/4 differ by -i only, so a radix-R pass costs
// 6 operations per butterfly and R/2 table entries (16 points: 192 operations
// and 8 entries; separate factors: 228 and 15).
//
// Two vectors in lockstep (the two polarisations of a spectrum, or two
// spectra, columns or rows of one polarisation) run on the packed
// FP32 instructions of sm_100 and later (add/sub/fma .f32x2, each lane
// rounded exactly as the scalar _rn operation): element m of both vectors is
// held as a cpair {re: (x0.re, x1.re), im: (x0.im, x1.im)}, so that one
// instruction does the work of two, with the twiddles shared by both lanes.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace rsg {

// ---- packed pairs -----------------------------------------------------------
__device__ __forceinline__ float2 f2add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 f2mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 f2sub(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 ra, rb, rr;\n\t"
      "mov.b64 ra, {%2, %3};\n\t"
      "mov.b64 rb, {%4, %5};\n\t"
      "sub.rn.f32x2 rr, ra, rb;\n\t"
      "mov.b64 {%0, %1}, rr;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 f2dup(float x) { return make_float2(x, x); }

// Elements of the engine (two vectors in lockstep): sums, differences and a
// multiply-add by a factor common to the lanes.
__device__ __forceinline__ float2 eadd(float2 a, float2 b) { return f2add(a, b); }
__device__ __forceinline__ float2 esub(float2 a, float2 b) { return f2sub(a, b); }
__device__ __forceinline__ float2 esubk(float2 a, float k) { return f2add(a, f2dup(-k)); }
__device__ __forceinline__ float2 efma(float2 a, float k, float2 c) { return f2fma(a, f2dup(k), c); }

template <typename E>
struct cx {
  E re, im;
};
using cpair = cx<float2>;  // lane 0: vector 0, lane 1: vector 1

// a * w for one twiddle w shared by both lanes
__device__ __forceinline__ cpair pmul(const cpair& a, float2 w) {
  const float2 c = f2dup(w.x), s = f2dup(w.y), ns = f2dup(-w.y);
  return {f2fma(a.im, ns, f2mul(a.re, c)), f2fma(a.re, s, f2mul(a.im, c))};
}
__device__ __forceinline__ cpair pack2(float2 x0, float2 x1) { return {make_float2(x0.x, x1.x), make_float2(x0.y, x1.y)}; }
__device__ __forceinline__ float2 lane0(const cpair& p) { return make_float2(p.re.x, p.im.x); }
__device__ __forceinline__ float2 lane1(const cpair& p) { return make_float2(p.re.y, p.im.y); }

// The four components of a word of 8-bit codes, (re, im) of lane 0 then of
// lane 1, as a pair that carries kCodeBias.
__device__ __forceinline__ cpair unpack_biased(uint32_t w) {
  const uint32_t u = offset_codes(w);
  return {make_float2(code_float<0>(u), code_float<2>(u)), make_float2(code_float<1>(u), code_float<3>(u))};
}

// ---- butterflies: (a, b) -> (a + w b, a - w b) ------------------------------
// w b = m (u + i v), or -i times that (MI).
template <typename E>
__device__ __forceinline__ void bfly_uv(cx<E>& a, cx<E>& b, E u, E v, float m, bool mi) {
  const cx<E> x = a;
  if (!mi) {
    a = {efma(u, m, x.re), efma(v, m, x.im)};
    b = {efma(u, -m, x.re), efma(v, -m, x.im)};
  } else {
    a = {efma(v, m, x.re), efma(u, -m, x.im)};
    b = {efma(v, -m, x.re), efma(u, m, x.im)};
  }
}

// w = exp(-2 pi i q / len), 0 <= q < len/2, len a power of two <= 32; q and
// len are compile-time constants after unrolling.
template <typename E>
__device__ __forceinline__ void bfly_const(cx<E>& a, cx<E>& b, int q, int len) {
  const int t = (32 / len) * q;  // angle = pi t / 16
  const bool mi = t >= 8;
  const int r = t & 7;           // remaining angle below pi/2
  const cx<E> x = a, y = b;
  if (r == 0) {
    if (!mi) {
      a = {eadd(x.re, y.re), eadd(x.im, y.im)};
      b = {esub(x.re, y.re), esub(x.im, y.im)};
    } else {
      a = {eadd(x.re, y.im), esub(x.im, y.re)};
      b = {esub(x.re, y.im), eadd(x.im, y.re)};
    }
    return;
  }
  if (r == 4) {  // (1 - i) / sqrt(2)
    bfly_uv(a, b, eadd(y.re, y.im), esub(y.im, y.re), 0.70710678118654752f, mi);
    return;
  }
  // (tangents of the rounded cosine, as in the tables)
  const float c = (float)cos_pi16(r), s = (float)sin_pi16(r);
  if (r < 4) {  // c (1 - i tan)
    const float k = (float)(sin_pi16(r) / (double)c);
    bfly_uv(a, b, efma(y.im, k, y.re), efma(y.re, -k, y.im), c, mi);
  } else {      // s (cot - i)
    const float k = (float)(cos_pi16(r) / (double)s);
    const E u = efma(y.re, k, y.im), nv = efma(y.im, -k, y.re);  // w y = s (u - i nv)
    if (!mi) {
      a = {efma(u, s, x.re), efma(nv, -s, x.im)};
      b = {efma(u, -s, x.re), efma(nv, s, x.im)};
    } else {
      a = {efma(nv, -s, x.re), efma(u, -s, x.im)};
      b = {efma(nv, s, x.re), efma(u, s, x.im)};
    }
  }
}

// w = c (1 - i t) from a table entry (c, t), times -i if mi.
template <typename E>
__device__ __forceinline__ void bfly_tab(cx<E>& a, cx<E>& b, float2 ct, bool mi) {
  const cx<E> y = b;
  bfly_uv(a, b, efma(y.im, ct.y, y.re), efma(y.re, -ct.y, y.im), ct.x, mi);
}

__host__ __device__ constexpr int ilog2(int n) {
  int l = 0;
  while ((2 << l) <= n) ++l;
  return l;
}
// x with its low `bits` (<= 5) bits reversed (no loop, so that a constant
// argument always folds)
__host__ __device__ constexpr int bitrev(int x, int bits) {
  return (((x & 1) << 4) | ((x & 2) << 2) | (x & 4) | ((x & 8) >> 2) | ((x & 16) >> 4)) >> (5 - bits);
}

// In-register DFT over the RP elements v[off + s*STRIDE] (RP <= 32), natural
// order in and out.  tw(i): twiddle entry i of the pass for this butterfly
// (stage L = 2: i = 0; stage L >= 4: i = L/4 + q, q < L/4); NoTwiddle: no
// input factors.
struct NoTwiddle {};
struct TableTwiddle {  // entries `stride` apart
  const float2* __restrict__ p;
  int stride;
  __device__ __forceinline__ float2 operator()(int i) const { return p[i * stride]; }
};
template <int RP, int STRIDE, typename Tw, typename E, int R>
__device__ __forceinline__ void dft_subset(cx<E> (&v)[R], int off, const Tw& tw) {
  if constexpr (RP > 1) {
    constexpr int LOG = ilog2(RP);
    cx<E> t[RP];
#pragma unroll
    for (int s = 0; s < RP; ++s) t[s] = v[off + bitrev(s, LOG) * STRIDE];
#pragma unroll
    for (int l = 1; l <= LOG; ++l) {
      const int len = 1 << l, half = len >> 1;
      if constexpr (!std::is_same_v<Tw, NoTwiddle>) {
        const int nq = len >= 4 ? len / 4 : 1;
#pragma unroll
        for (int q = 0; q < nq; ++q) {
          const float2 ct = tw(len >= 4 ? len / 4 + q : 0);
#pragma unroll
          for (int i = 0; i < RP; i += len) {
            bfly_tab(t[i + q], t[i + q + half], ct, false);
            if (len >= 4) bfly_tab(t[i + q + len / 4], t[i + q + len / 4 + half], ct, true);
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < RP; i += len)
#pragma unroll
          for (int q = 0; q < half; ++q) bfly_const(t[i + q], t[i + q + half], q, len);
      }
    }
#pragma unroll
    for (int s = 0; s < RP; ++s) v[off + s * STRIDE] = t[s];
  }
}

// Shared-memory positions of the exchanges, with a padding element every
// 2^PS elements (PS = log2 R, 4 at least), which keeps the strided writes of
// the Stockham passes free of bank conflicts: element e lives at
// e + (e >> PS).  GroupFFT computes these positions as a per-thread base plus
// compile-time offsets, which is exact because every pass's write stride
// Ns*R and read stride T are powers of two.
__host__ __device__ constexpr int smem_padded_len(int n) { return n + (n >> 4) + 1; }

// Number of radix-R passes and the radix of the trailing pass.
template <int N, int R>
struct FftShape {
  static constexpr int T = N / R;                       // threads per FFT
  static constexpr int LOGN = ilog2(N);
  static constexpr int LOGR = ilog2(R);
  static constexpr int FULL = (LOGR == 0) ? 0 : LOGN / LOGR;     // radix-R passes
  static constexpr int RLAST = (LOGR == 0) ? 1 : (1 << (LOGN - FULL * LOGR));
  static constexpr int PASSES = FULL + (RLAST > 1 ? 1 : 0);
};

// Twiddle table of a GroupFFT<N, R>, one block per twiddled pass, laid out so
// that the lanes of a warp read consecutive (or identical) entries.  Entry
// (i, k) of a pass of radix P after passes of total length M (M = R^p for the
// full passes p >= 1, N/RL for the trailing one of radix RL) is (cos, tan) of
// the angle 2 pi (k + q M) / (M L), with (L, q) of index i as in dft_subset:
//   full pass p:    [i][k], i < R/2,  k < M
//   trailing pass:  [i][k], i < RL/2, k < M
// stockham_tw_offset(N, R, p) is the start of pass p's block.
__host__ __device__ constexpr int stockham_tw_offset(int N, int R, int p) {
  // blocks of passes 1 .. p-1
  int off = 0, Ns = R;
  for (int q = 1; q < p; ++q) {
    off += (R / 2) * Ns;
    Ns *= R;
  }
  return off;
}
__host__ __device__ constexpr int stockham_tw_size(int N, int R) {
  if (R <= 1 || N <= R) return 0;
  int full = 0, Ns = 1;
  while (Ns * R <= N) {
    Ns *= R;
    ++full;
  }
  const int rl = N / Ns;
  return stockham_tw_offset(N, R, full) + (rl > 1 ? (rl / 2) * (N / rl) : 0);
}

// Group FFT.  tw: the pass-ordered twiddle table described above (shared or
// global memory).  sm: this group's exchange buffers, two buffers (the re and
// the im parts) of smem_padded_len(N) elements each, `sm_stride` elements
// apart.  SYNC is a functor performing the barrier required between the
// group's threads.
template <int N, int R>
struct GroupFFT {
  using S = FftShape<N, R>;
  static constexpr int T = S::T;
  static constexpr int PS = R >= 32 ? 5 : 4;
  using E = float2;

  template <bool BIASED>
  static __device__ __forceinline__ void first_pass(cx<E> (&v)[R]) {
    dft_subset<R, 1>(v, 0, NoTwiddle{});
    if constexpr (BIASED) {
      v[0].re = esubk(v[0].re, R * kCodeBias);
      v[0].im = esubk(v[0].im, R * kCodeBias);
    }
  }

  // SPLIT: one exchange buffer only (sm_stride unused), the re parts and then
  // the im parts passing through it (twice the barriers, half the shared
  // memory).  BIASED: the input values carry kCodeBias.  sync(first, last) is
  // told whether the barrier is the transform's first (every thread of the
  // group has taken its input) or its last.
  template <bool SPLIT = false, bool BIASED = false, typename Sync>
  static __device__ __forceinline__ void run_packed(cx<E> (&v)[R], int j, E* sm, int sm_stride,
                                                    const float2* __restrict__ tw, Sync sync) {
    if constexpr (T == 1) {
      first_pass<BIASED>(v);
    } else {
      int Ns = 1;
#pragma unroll
      for (int p = 0; p < S::FULL; ++p) {
        if (p == 0) {
          first_pass<BIASED>(v);
        } else {
          const int k = j & (Ns - 1);
          dft_subset<R, 1>(v, 0, TableTwiddle{tw + stockham_tw_offset(N, R, p) + k, Ns});
        }
        const bool last = (p == S::FULL - 1) && (S::RLAST == 1);
        if (!last) {
          const int lo = j & (Ns - 1);
          const int hi = j / Ns;
          const int idxD = hi * Ns * R + lo;
          const int wbase = idxD + ((hi * Ns * R) >> PS) + (Ns >> PS ? (lo >> PS) : 0);
          const int rbase = j + (T >> PS ? (j >> PS) : 0);
          if constexpr (SPLIT) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const int off = Ns >> PS ? r * (Ns + (Ns >> PS)) : r * Ns + ((r * Ns) >> PS);
                sm[wbase + off] = h == 0 ? v[r].re : v[r].im;
              }
              sync(p == 0 && h == 0, false);
#pragma unroll
              for (int m = 0; m < R; ++m) {
                const int off = T >> PS ? m * (T + (T >> PS)) : m * T + ((m * T) >> PS);
                if (h == 0) v[m].re = sm[rbase + off]; else v[m].im = sm[rbase + off];
              }
              sync(false, h == 1 && p == S::PASSES - 2);
            }
          } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const int off = Ns >> PS ? r * (Ns + (Ns >> PS)) : r * Ns + ((r * Ns) >> PS);
              sm[wbase + off] = v[r].re;
              sm[sm_stride + wbase + off] = v[r].im;
            }
            sync(p == 0, false);
#pragma unroll
            for (int m = 0; m < R; ++m) {
              const int off = T >> PS ? m * (T + (T >> PS)) : m * T + ((m * T) >> PS);
              v[m].re = sm[rbase + off];
              v[m].im = sm[sm_stride + rbase + off];
            }
            sync(false, p == S::PASSES - 2);
          }
        }
        Ns *= R;
      }
      if constexpr (S::RLAST > 1) {
        // Trailing pass of radix RL < R: thread j computes Q = R/RL
        // butterflies b = j + q*T on elements m = q + r*Q.
        constexpr int RL = S::RLAST;
        constexpr int Q = R / RL;
        constexpr int NSL = N / RL;
        const float2* twl = tw + stockham_tw_offset(N, R, S::FULL) + j;
#pragma unroll
        for (int qb = 0; qb < Q; ++qb) dft_subset<RL, Q>(v, qb, TableTwiddle{twl + qb * T, NSL});
      }
    }
  }
};

}  // namespace rsg
