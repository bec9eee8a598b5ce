// k_small.cu -- fused spectrometer kernel for FFT lengths N <= 4096.
//
// One launch per output product and input buffer replaces the reference's
// per-(product, batch, pol) cufftExecC2C calls with their texture load
// callback and read-modify-write store callbacks (rawspec_gpu.cu:1555-1569,
// :133-267), the sub-integration `accumulate` kernel (:297-318, :1588-1601)
// and the FFT-shifting device-to-host copies (:1647-1697):
//
//   int8/int16 load + exact integer unpack -> Stockham FFT in registers and
//   shared memory (both polarisations together) -> detection -> accumulation
//   of the unit's spectra in registers -> reduction across the CTA's thread
//   groups -> SNORM scale and FFT-shifted store into the dump buffer
//   [Nd][|P|][Nc][N] (or partial sums when one unit is spread over CTAs).
//
// Nothing but the raw voltages is read and nothing but integrated spectra is
// written.
#include <algorithm>
#include <atomic>
#include <cmath>

#include "detect.cuh"
#include "fft_core.cuh"
#include "internal.h"
#include "small_split.h"

namespace rsg {

__host__ __device__ constexpr int small_r(int N, int NP) {
  const int most = NP == 1 && (N == 32 || N == 512 || N == 1024) ? 32 : 16;
  return N < most ? N : most;
}
// The smallest number >= x that is r modulo m.
__host__ __device__ constexpr int pad_mod(int x, int m, int r) { return x + ((r - x) % m + m) % m; }

// Geometry of a configuration.
//
// Vectors in lockstep: the two polarisations of a spectrum, or (one
// polarisation, PAIR) two spectra of the unit, so that every transform runs
// on the packed instructions.
//
// R, the values per thread per vector: as many as the accumulators leave
// registers for, since every halving of the passes removes a trip through
// shared memory, whose bandwidth is the bound next to the FMA pipe.  Total
// power (one accumulator per bin): 32 where that leaves one exchange (N =
// 512, 1024: 32 x 16, 32 x 32) or none (N = 32), else 16.  Four planes: 16.
//
// MINB: resident CTAs per SM the register budget is cut for: 168 registers a
// thread for R = 32 and for the four planes at R = 16, 128 otherwise, and for
// 4096 points in four planes, whose 256-thread CTAs would be alone on their
// SM (410 us per 64 Mi samples; two of them with spills: 367).
template <int N, int FMT, int NV, int POL>
struct SmallCfg {
  static constexpr int NP = PolOut<POL>::NP;
  static constexpr int R = small_r(N, NP);
  static constexpr int T = N / R;            // threads per FFT
  static constexpr bool PAIR = NV == 1;      // spectra (not polarisations) in lockstep
  static constexpr int SPI = PAIR ? 2 : 1;   // spectra a group takes per iteration
  static constexpr int REGS = R >= 32 || (NP == 4 && R == 16 && T <= 128) ? 168 : 128;
  static constexpr int TPB = T > 128 ? T : 128;
  static constexpr int G = TPB / T;          // FFT groups per CTA
  static constexpr int MINB = 65536 / (TPB * REGS);
  static constexpr int TW = stockham_tw_size(N, R);  // twiddle table entries
  // Staged input (N >= 16): every group copies its next spectrum into shared
  // memory with cp.async while it transforms the current one, so that no
  // registers hold words in flight.  Spectra are RAW bytes apart, the groups
  // of a warp in different banks.
  static constexpr bool STAGED = N >= 16;
  using W = typename SampleWord<FMT, NV>::type;
  static constexpr int RAW = N * (int)sizeof(W) + (T >= 32 ? 0 : (T * (int)sizeof(W) + 15) / 16 * 16);
  static constexpr int RAW_GROUP = STAGED ? RAW * SPI : 0;
  // Exchange: re and im parts through one buffer in turn (SPLIT) where the
  // group is within a warp, whose barriers cost next to nothing.
  static constexpr bool SPLIT = T <= 32;
  static constexpr int PLANE = smem_padded_len(N);
  // Elements between the groups' exchange buffers: the groups of a half-warp
  // start T elements apart modulo 16, so that they use different banks.
  static constexpr int XCH = T == 1 ? 0 : pad_mod(SPLIT ? PLANE : 2 * PLANE, 16, T < 16 ? T : 0);
  // Floats between the groups' slices of the reduction area (NP R T floats
  // each): the groups of a warp start T banks apart.
  static constexpr int RED = T >= 32 ? NP * R * T : pad_mod(NP * R * T, 32, T);
  // Shared memory: the twiddle table, then the staged input and the exchange
  // buffers of the groups, or the reduction area.
  static constexpr size_t TW_BYTES = (size_t)((TW + 1) & ~1) * sizeof(float2);
  static constexpr size_t WORK = (size_t)G * (RAW_GROUP + XCH * sizeof(float2));
  static constexpr size_t REDUCE = (size_t)G * RED * sizeof(float);
  static constexpr size_t SMEM = TW_BYTES + (WORK > REDUCE ? WORK : REDUCE);
};

// Barrier of one transform group that spans whole warps (named barrier
// 1 + group, `threads` = the group's thread count), so that the groups of a
// CTA progress independently.
__device__ __forceinline__ void group_barrier(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <int V>
using Int = std::integral_constant<int, V>;

// The cluster's size and its barrier.
__device__ __forceinline__ uint32_t cluster_ctas() {
  uint32_t n;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The cluster address of `addr` of CTA `rank`'s shared memory, and its float.
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float cluster_load(uint32_t addr) {
  float f;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f) : "r"(addr) : "memory");
  return f;
}

// The same through L1 (neighbouring copies share a 32-byte sector).
__device__ __forceinline__ void cp_async16_l1(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
// 8 bytes (twiddle tables need not start or end on 16).
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}

// The kernel body for CTA `bid` of launch `a` (k_small: one launch;
// k_small_group: several launches of the same configuration, e.g. the
// buffers of several jobs, in one grid).
template <int N, int FMT, int NV, int POL>
__device__ __forceinline__ void small_body(const SmallLaunch& a, const int bid) {
  using C = SmallCfg<N, FMT, NV, POL>;
  using W = typename C::W;
  constexpr int NP = C::NP, R = C::R, T = C::T, G = C::G, TPB = C::TPB, SPI = C::SPI;
  extern __shared__ __align__(16) unsigned char smem_raw[];

  float2* tw_s = reinterpret_cast<float2*>(smem_raw);
  unsigned char* work = smem_raw + C::TW_BYTES;
  float* red = reinterpret_cast<float*>(work);

  const int tid = threadIdx.x;
  const int g = tid / T;   // group within the CTA
  const int j = tid % T;   // thread within the group

  // The twiddle table and the first spectra are requested together: one trip
  // to memory before the first transform, not two.
#pragma unroll 4
  for (int i = tid; i < C::TW; i += TPB) cp_async8(tw_s + i, a.tw + i);

  // Which unit / spectra this group works on.  The CTA covers `sets` units
  // (gps groups each) and one chunk of spc spectra of each of them.
  const int gps = G / a.sets;           // groups per set
  const int set = g / gps;
  const int gi = g % gps;
  const int ublock = bid / a.chunks;
  const int chunk = bid % a.chunks;
  const int unit = a.unit0 + ublock * a.sets + set;
  const int s_begin = chunk * a.spc;
  const int s_end = min(a.M, s_begin + a.spc);
  const bool unit_ok = unit < a.unit0 + a.unit_count;
  const int c = unit_ok ? unit / a.units_per_chan : 0;
  const int d = unit_ok ? unit % a.units_per_chan : 0;
  const int iters = (a.spc + gps * SPI - 1) / (gps * SPI);
  const float im_sign = a.conj ? -1.0f : 1.0f;
  const W* const unit_src = reinterpret_cast<const W*>(a.in) + (long long)c * a.chan_stride + (long long)d * a.M * N;
  auto spec_of = [&](int it) { return s_begin + (gi + it * gps) * SPI; };

  // Accumulators.  Total power: one sum per bin over both lanes.  Four
  // planes: the first two as one packed pair, the cross terms Re and Im(X0
  // X1*) as another.
  float tp[NP == 1 ? R : 1];
  float2 pw[NP == 4 ? R : 1], xr[NP == 4 ? R : 1];
#pragma unroll
  for (int m = 0; m < (NP == 1 ? R : 1); ++m) tp[m] = 0.0f;
#pragma unroll
  for (int m = 0; m < (NP == 4 ? R : 1); ++m) pw[m] = xr[m] = make_float2(0.f, 0.f);

  unsigned char* const raw = work + (size_t)g * C::RAW_GROUP;
  float2* const xch = reinterpret_cast<float2*>(work + (size_t)G * C::RAW_GROUP) + (size_t)g * C::XCH;

  // Requests the group's spectra of iteration `it` (those that exist).
  auto stage = [&](int it) {
#pragma unroll
    for (int q = 0; q < SPI; ++q) {
      const int s = spec_of(it) + q;
      if (!(unit_ok && s < s_end)) break;
      const W* src = unit_src + (long long)s * N;
      unsigned char* dst = raw + q * C::RAW;
      if (a.vec16) {
#pragma unroll
        for (int i = 0; i < N * (int)sizeof(W) / 16; i += T) {
          if (N * (int)sizeof(W) / 16 % T == 0 || i + j < N * (int)sizeof(W) / 16) {
            if constexpr (T == 1) cp_async16_l1(dst + (i + j) * 16, reinterpret_cast<const char*>(src) + (i + j) * 16);
            else cp_async16(dst + (i + j) * 16, reinterpret_cast<const char*>(src) + (i + j) * 16);
          }
        }
      } else {
#pragma unroll 4
        for (int i = j; i < N; i += T) reinterpret_cast<W*>(dst)[i] = __ldg(src + i);
      }
    }
  };
  // Words of the staged spectrum q of this group, or of spectrum s in global
  // memory (short transforms, one thread each).
  auto take = [&](int q, W (&w)[R]) {
    const unsigned char* src = raw + q * C::RAW;
    if constexpr (T == 1) {
#pragma unroll
      for (int i = 0; i < (int)(R * sizeof(W) / 16); ++i) {
        const uint4 u = reinterpret_cast<const uint4*>(src)[i];
        memcpy(reinterpret_cast<char*>(w) + 16 * i, &u, 16);
      }
    } else {
#pragma unroll
      for (int m = 0; m < R; ++m) w[m] = reinterpret_cast<const W*>(src)[j + m * T];
    }
  };
  constexpr bool kBiased = FMT == FMT_I8;  // 8-bit codes carry kCodeBias into the first pass
  constexpr bool kVec = (R * sizeof(W)) % 16 == 0;
  auto fetch = [&](int it, int q, W (&w)[R]) {
    const int s = spec_of(it) + q;
    if (!(unit_ok && s < s_end)) {
#pragma unroll
      for (int m = 0; m < R; ++m) w[m] = W{};
      return;
    }
    const W* src = unit_src + (long long)s * N + j;
    if (kVec && a.vec16) {
      const uint4* s4 = reinterpret_cast<const uint4*>(src);
#pragma unroll
      for (int i = 0; i < (int)(R * sizeof(W) / 16); ++i) {
        const uint4 u = __ldg(s4 + i);
        memcpy(reinterpret_cast<char*>(w) + 16 * i, &u, 16);
      }
    } else {
#pragma unroll
      for (int m = 0; m < R; ++m) w[m] = __ldg(src + m * T);
    }
  };
  W wn[SPI][C::STAGED ? 1 : R];
  if constexpr (C::STAGED) {
    stage(0);
    if constexpr (C::TW > 0) {
      cp_async_wait();
      __syncthreads();
    }
  } else {
    static_assert(C::TW == 0, "unstaged transforms use no table");
#pragma unroll
    for (int q = 0; q < SPI; ++q) fetch(0, q, wn[q]);
  }

  for (int it = 0; it < iters; ++it) {
    const int s_local = spec_of(it);
    const bool valid = unit_ok && s_local < s_end;
    const bool valid1 = unit_ok && s_local + 1 < s_end;  // PAIR: the second spectrum
    cpair v[R];
    {
      W w[SPI][R];
      if constexpr (C::STAGED) {
        if constexpr (T <= 32) {
          cp_async_wait();
          __syncwarp();
        }
#pragma unroll
        for (int q = 0; q < SPI; ++q) take(q, w[q]);
        if constexpr (T <= 32) {
          __syncwarp();
          stage(it + 1);
        }
      } else {
#pragma unroll
        for (int q = 0; q < SPI; ++q) {
#pragma unroll
          for (int m = 0; m < R; ++m) w[q][m] = wn[q][m];
          if (it + 1 < iters) fetch(it + 1, q, wn[q]);
        }
      }
#pragma unroll
      for (int m = 0; m < R; ++m) {
        if constexpr (kBiased) {
          uint32_t both = w[0][m];
          if constexpr (C::PAIR) both |= valid1 ? (uint32_t)w[1][m] << 16 : 0u;
          v[m] = unpack_biased(both);
        } else if constexpr (C::PAIR) {
          float2 s0[1], s1[1];
          Unpack<FMT, 1>::run(w[0][m], s0);
          Unpack<FMT, 1>::run(valid1 ? w[1][m] : W{}, s1);
          v[m] = pack2(s0[0], s1[0]);
        } else {
          float2 smp[2];
          Unpack<FMT, 2>::run(w[0][m], smp);
          v[m] = pack2(smp[0], smp[1]);
        }
      }
    }
    // Within a warp: the warp's barrier.  Larger groups request the next
    // spectrum once everyone has taken the current one, and wait for their
    // part of it before the transform's last barrier, which publishes it.
    auto sync = [&](bool first, bool last) {
      if constexpr (T <= 32) {
        __syncwarp();
      } else {
        if (last) cp_async_wait();
        group_barrier(1 + g, T);
        if (first) stage(it + 1);
      }
    };
    static_assert(T <= 32 || FftShape<N, R>::PASSES >= 3, "a group's copies span two exchanges");
    static_assert(G <= 15 || T <= 32, "one named barrier per group");
    GroupFFT<N, R>::template run_packed<C::SPLIT, kBiased>(v, j, xch, C::PLANE, tw_s, sync);
    if (valid) {
#pragma unroll
      for (int m = 0; m < R; ++m) {
        if constexpr (NP == 1) {
          tp[m] += both_powers(v[m]);
        } else {
          add_planes<POL>(v[m], pw[m], xr[m]);
        }
      }
    }
  }

  // Bin j + m T of plane p as this thread summed it.
  auto sum_of = [&](int p, int m) -> float {
    if constexpr (NP == 1) return tp[m];
    else return p == 0 ? pw[m].x : p == 1 ? pw[m].y : p == 2 ? xr[m].x : xr[m].y * im_sign;
  };
  const bool clustered = cluster_ctas() > 1;
  // The sums of the CTA's units are shared out over its threads: to those of
  // the unit's own groups, or where it has fewer units than sets, to 2, 4, ...
  // times as many (one unit of four spectra of 32 points in four planes, 8 and
  // all of 128 threads: 7.9 and 5.8 us).
  const int here = min(a.sets, a.unit0 + a.unit_count - (unit - set));
  int set_threads = gps * T;
  while (2 * here * set_threads <= TPB) set_threads *= 2;
  const int sum_set = tid / set_threads, t_in_set = tid % set_threads;
  const int sum_unit = unit - set + sum_set;
  const bool sum_ok = sum_set < here;
  // A unit's result (its plane 0), and the place of bin k in a plane (out_pos).
  auto result = [&](int u) {
    return a.out + ((size_t)(u % a.units_per_chan) * NP * a.Nc + u / a.units_per_chan) * N;
  };
  const size_t plane = (size_t)a.Nc * N;
  const int dir = a.inverse ? -1 : 1;
  auto place = [&](int k) { return ((k * dir) & (N - 1)) ^ (N >> 1); };
  // Writes s[i], or adds it, to the addresses at(i), i < n (the old values are
  // requested before the first is written).
  auto store = [&](auto& s, int n, auto at) {
    constexpr int U = sizeof(s) / sizeof(float);
    if (a.mode == ACC_ADD) {
      float old[U];
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (i < n) old[i] = *at(i);
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (i < n) *at(i) = __fmaf_rn(s[i], a.scale, old[i]);
    } else {
#pragma unroll
      for (int i = 0; i < U; ++i)
        if (i < n) *at(i) = s[i] * a.scale;
    }
  };
  // Where unit u's sums go, the result or the chunk's partial sums, and bins k +
  // i step, i < n, of its plane p.
  auto target = [&](int u) {
    return a.chunks == 1 ? result(u) : a.partial + ((size_t)u * a.chunks + chunk) * NP * N;
  };
  auto store_or_part = [&](float* to, auto& s, int n, int p, int k, int step) {
    if (a.chunks == 1) {
      float* const o = to + p * plane;
      store(s, n, [&](int i) { return o + place(k + i * step); });
      return;
    }
    float* const o = to + p * N + k;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(s) / sizeof(float)); ++i)
      if (i < n) __stcg(o + i * step, s[i]);
  };

  // What follows runs once a CTA, often with one warp to a scheduler, so that
  // its time is its instructions': addresses move by additions.
  cp_async_wait();  // none is in flight after the last iteration; nothing lands in the reduction area any more
  float* const red_set = red + sum_set * gps * C::RED;
  constexpr bool kDirect = R < 32;
  if (kDirect && gps == 1 && !clustered) {
    // One group a unit: its threads hold the sums.  (Of 32 values each they go
    // through shared memory all the same, eight at a time: with this branch the
    // transforms' loop takes 5 % longer.)
    if (unit_ok) {
      float* const to = target(unit);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        float s[R];
#pragma unroll
        for (int m = 0; m < R; ++m) s[m] = sum_of(p, m);
        store_or_part(to, s, R, p, j, T);
      }
    }
  } else {
    // Reduce across the groups of each set: red[g][p][m][j] = red[g][p][k].
    __syncthreads();
#pragma unroll
    for (int m = 0; m < R; ++m)
#pragma unroll
      for (int p = 0; p < NP; ++p) red[g * C::RED + (p * R + m) * T + j] = sum_of(p, m);
    __syncthreads();
    float* const to = target(sum_unit);
    const int kstep = min(set_threads, N), pstep = max(1, set_threads / N);
    // U bins at a time, Q groups at a time (a divisor of their number)
    auto sum_groups = [&](auto u_, auto q_) {
      constexpr int U = decltype(u_)::value, Q = decltype(q_)::value;
      for (int p = t_in_set / N; p < NP; p += pstep) {
        for (int k = t_in_set % N; k < N; k += U * kstep) {
          const int n = U == 1 ? 1 : (N - 1 - k) / kstep + 1;
          float* const src = red_set + p * N + k;
          float s[U] = {};
          for (int q = 0; q < gps; q += Q)
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (u < n) {
                const float* f = src + q * C::RED + u * kstep;
                s[u] += Q == 1 ? f[0] : Q == 2 ? f[0] + f[C::RED] : (f[0] + f[C::RED]) + (f[2 * C::RED] + f[3 * C::RED]);
              }
          if (clustered) {
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (u < n) src[u * kstep] = s[u];
          } else {
            store_or_part(to, s, n, p, k, kstep);
          }
        }
      }
    };
    // (a cluster's CTA of one group has its sums where they belong)
    if (sum_ok && gps > 4) sum_groups(Int<1>{}, Int<4>{});
    else if (sum_ok && gps > 1) sum_groups(Int<(NP * R >= 16 ? 4 : 1)>{}, Int<2>{});
    else if (!kDirect && sum_ok && !clustered) sum_groups(Int<8>{}, Int<1>{});
  }
  if (a.chunks == 1 || a.finalize) return;

  // Units spread over the CTAs of a cluster: every CTA keeps its sums where
  // the first group's were, and sums a share of the outputs over the chunks,
  // in chunk order, from the others' shared memory.  By the last CTA alone
  // (below) four units of 8 x 2048 points in four planes take 27.7 us, so
  // 11.3; 64 Mi samples of 4096 points in four planes 390, so 353.
  if (clustered) {
    cluster_sync();
    constexpr int U = NP * N >= 1024 ? 4 : 1;
    uint32_t from[kSmallCluster];
#pragma unroll
    for (int q = 0; q < kSmallCluster; ++q)
      if (q < a.chunks) from[q] = cluster_map(static_cast<uint32_t>(__cvta_generic_to_shared(red_set)), q);
    const int step = set_threads * a.chunks;
    float* const out = result(sum_unit);
    for (int o = sum_ok ? t_in_set + chunk * set_threads : NP * N; o < NP * N; o += U * step) {
      const int n = (NP * N - 1 - o) / step + 1;
      float f[U][kSmallCluster], s[U] = {};
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < kSmallCluster; ++q)
          if (u < n && q < a.chunks) f[u][q] = cluster_load(from[q] + (o + u * step) * sizeof(float));
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < kSmallCluster; ++q)
          if (u < n && q < a.chunks) s[u] += f[u][q];
      store(s, n, [&](int u) { return out + (o + u * step) / N * plane + place(o + u * step); });
    }
    cluster_sync();  // no CTA leaves before its sums are read
    return;
  }

  // Units spread over more CTAs than a cluster holds, and the launches that
  // share a grid: the last CTA of the block of units to arrive sums
  // the chunks' partials in chunk order (the same order whichever CTA it is)
  // and leaves the arrival counter zeroed for the next launch.  A kernel of its
  // own for this sum costs a launch and a drained GPU, and is left for sums that
  // take one CTA longer (SplitCost).
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    s_last = atomicAdd(a.arrived + ublock, 1u) == (unsigned)a.chunks - 1;
    if (s_last) a.arrived[ublock] = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (!sum_ok) return;
  // U accesses of V outputs a thread and Q chunks at a time: the sum is a
  // chain of trips to L2 otherwise (four planes of 4096 points in 4 chunks: 64
  // trips, 12 us).
  constexpr int V = NP * N % 4 == 0 ? 4 : 1, U = NP * N >= 2048 ? 4 : 1, Q = U == 4 ? 2 : 8;
  const int step = set_threads * V;
  const float* const base = a.partial + (size_t)sum_unit * a.chunks * NP * N;
  float* const out = result(sum_unit);
  for (int o = t_in_set * V; o < NP * N; o += step * U) {
    float s[U][V] = {};
    for (int q0 = 0; q0 < a.chunks; q0 += Q) {
      float f[Q][U][V];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (q0 + q >= a.chunks || o + u * step >= NP * N) continue;
          const float* src = base + (size_t)(q0 + q) * NP * N + o + u * step;
          if constexpr (V == 4) {
            const float4 w = __ldcg(reinterpret_cast<const float4*>(src));
            f[q][u][0] = w.x, f[q][u][1] = w.y, f[q][u][2] = w.z, f[q][u][3] = w.w;
          } else {
            f[q][u][0] = __ldcg(src);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (q0 + q >= a.chunks) break;
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
          for (int i = 0; i < V; ++i) s[u][i] += f[q][u][i];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int at = o + u * step;
      if (at >= NP * N) break;
      store(s[u], V, [&](int i) { return out + (at + i) / N * plane + place(at + i); });
    }
  }
}

template <int N, int FMT, int NV, int POL>
__global__ void __launch_bounds__(SmallCfg<N, FMT, NV, POL>::TPB, SmallCfg<N, FMT, NV, POL>::MINB)
k_small(const __grid_constant__ SmallLaunch a) {
  small_body<N, FMT, NV, POL>(a, blockIdx.x);
}

// Several launches of one configuration in one grid: CTA b belongs to the
// launch k whose range [end[k-1], end[k]) holds it.
template <int N, int FMT, int NV, int POL>
__global__ void __launch_bounds__(SmallCfg<N, FMT, NV, POL>::TPB, SmallCfg<N, FMT, NV, POL>::MINB)
k_small_group(const __grid_constant__ SmallGroup g) {
  int k = 0;
  while (k + 1 < g.n && (int)blockIdx.x >= g.end[k]) ++k;
  small_body<N, FMT, NV, POL>(g.e[k], (int)blockIdx.x - (k ? g.end[k - 1] : 0));
}

// Finalisation of chunked units: fixed-order sum of the chunks' partials,
// SNORM scale and FFT-shifted store.
__global__ void k_finalize(FinalizeLaunch a) {
  const long long total = (long long)a.n_units * a.np * a.N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i % a.N);
    const long long up = i / a.N;
    const int p = (int)(up % a.np);
    const int unit = a.unit0 + (int)(up / a.np);
    const float* src = a.partial + ((size_t)unit * a.chunks * a.np + p) * a.N + k;
    float s = 0.0f;
    for (int q = 0; q < a.chunks; ++q) s += src[(size_t)q * a.np * a.N];
    const int c = unit / a.units_per_chan;
    const int d = unit % a.units_per_chan;
    float* dst = a.out + (((size_t)d * a.np + p) * a.Nc + c) * a.N + out_pos(k, a.N, a.inverse);
    if (a.mode == ACC_ADD) *dst = __fmaf_rn(s, a.scale, *dst); else *dst = s * a.scale;
  }
}

// ---------------------------------------------------------------------------
// Host side: configuration and dispatch.
// ---------------------------------------------------------------------------
namespace {

struct SmallInfo {
  int R, T, TPB, G, SPI;
  size_t smem;
};

int small_grid(const SmallLaunch& L) { return ((L.unit_count + L.sets - 1) / L.sets) * L.chunks; }

// op: 0 launch, 1 allow the dynamic shared memory, 2 also report the
// resident CTAs per SM in *occ, 3 launch the group *grp (entries of L's
// configuration), 4 report the geometry in *info.
template <int N, int FMT, int NV, int POL>
cudaError_t launch_t(const SmallLaunch& L, cudaStream_t s, int op, int* occ, const SmallGroup* grp, SmallInfo* info) {
  using C = SmallCfg<N, FMT, NV, POL>;
  auto k = k_small<N, FMT, NV, POL>;
  if (op == 4) {
    *info = SmallInfo{C::R, C::T, C::TPB, C::G, C::SPI, C::SMEM};
    return cudaSuccess;
  }
  if (op == 3) {
    auto kg = k_small_group<N, FMT, NV, POL>;
    cudaError_t e = cudaFuncSetAttribute(kg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
    if (e != cudaSuccess) return e;
    const int grid = grp->end[grp->n - 1];
    if (grid < 1) return cudaSuccess;
    kg<<<grid, C::TPB, L.smem, s>>>(*grp);
    return cudaGetLastError();
  }
  if (op != 0) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
    if (e != cudaSuccess || op == 1) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k, C::TPB, L.smem);
  }
  const int grid = small_grid(L);
  if (grid < 1) return cudaSuccess;
  if (!L.finalize && small_clustered(L.chunks, grid, L.sms)) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(C::TPB);
    cfg.dynamicSmemBytes = L.smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = L.chunks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, L);
  }
  k<<<grid, C::TPB, L.smem, s>>>(L);
  return cudaGetLastError();
}

template <int N, int FMT>
cudaError_t launch_pol(const SmallLaunch& L, cudaStream_t s, int op, int* occ, const SmallGroup* grp, SmallInfo* info) {
  if (L.nv == 1) return launch_t<N, FMT, 1, POL_TP>(L, s, op, occ, grp, info);
  switch (L.pol) {
    case POL_FULL: return launch_t<N, FMT, 2, POL_FULL>(L, s, op, occ, grp, info);
    case POL_STOKES: return launch_t<N, FMT, 2, POL_STOKES>(L, s, op, occ, grp, info);
    default: return launch_t<N, FMT, 2, POL_TP>(L, s, op, occ, grp, info);
  }
}

template <int N>
cudaError_t launch_fmt(const SmallLaunch& L, cudaStream_t s, int op, int* occ, const SmallGroup* grp, SmallInfo* info) {
  return L.fmt == FMT_I16 ? launch_pol<N, FMT_I16>(L, s, op, occ, grp, info) : launch_pol<N, FMT_I8>(L, s, op, occ, grp, info);
}

cudaError_t small_dispatch(const SmallLaunch& L, cudaStream_t s, int op, int* occ = nullptr,
                           const SmallGroup* grp = nullptr, SmallInfo* info = nullptr) {
  switch (L.logN) {
    case 0: return launch_fmt<1>(L, s, op, occ, grp, info);
    case 1: return launch_fmt<2>(L, s, op, occ, grp, info);
    case 2: return launch_fmt<4>(L, s, op, occ, grp, info);
    case 3: return launch_fmt<8>(L, s, op, occ, grp, info);
    case 4: return launch_fmt<16>(L, s, op, occ, grp, info);
    case 5: return launch_fmt<32>(L, s, op, occ, grp, info);
    case 6: return launch_fmt<64>(L, s, op, occ, grp, info);
    case 7: return launch_fmt<128>(L, s, op, occ, grp, info);
    case 8: return launch_fmt<256>(L, s, op, occ, grp, info);
    case 9: return launch_fmt<512>(L, s, op, occ, grp, info);
    case 10: return launch_fmt<1024>(L, s, op, occ, grp, info);
    case 11: return launch_fmt<2048>(L, s, op, occ, grp, info);
    case 12: return launch_fmt<4096>(L, s, op, occ, grp, info);
    default: return cudaErrorInvalidValue;
  }
}

// Resident CTAs per SM of the configuration and SMs of the current device, with
// the kernel's dynamic shared-memory limit raised; asked of the runtime once
// per configuration and device (it takes longer than a small launch).  0
// CTAs if it cannot say.
void resident_ctas(const SmallLaunch& L, int* occ, int* sms) {
  constexpr int kDevices = 64, kConfigs = 13 * 2 * 4;
  static std::atomic<int> known[kDevices][kConfigs];  // occ + 1
  static std::atomic<int> known_sms[kDevices];
  *occ = *sms = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return;
  const int mode = L.nv == 1 ? 0 : L.pol == POL_FULL ? 1 : L.pol == POL_STOKES ? 2 : 3;
  const int key = (L.logN * 2 + (L.fmt == FMT_I16 ? 1 : 0)) * 4 + mode;
  const bool cached = dev < kDevices;
  if (cached && known[dev][key].load() > 0) {
    *occ = known[dev][key].load() - 1;
    *sms = known_sms[dev].load();
    return;
  }
  if (cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      small_dispatch(L, nullptr, 2, occ) != cudaSuccess) {
    *occ = 0;
    return;
  }
  if (cached) {
    known_sms[dev].store(*sms);
    known[dev][key].store(*occ + 1);
  }
}

}  // namespace

int small_radix(int logN, int pol) { return small_r(1 << logN, pol == POL_TP ? 1 : 4); }

int small_configure(SmallLaunch& L, int target_ctas, size_t* partial_floats, int pipe_groups, size_t max_partial,
                    bool counters) {
  if (L.logN < 0 || L.logN > 12 || L.M < 1 || L.n_units < 1) return -1;
  SmallInfo si{};
  if (small_dispatch(L, nullptr, 4, nullptr, nullptr, &si) != cudaSuccess) return -1;
  L.smem = si.smem;
  const int G = si.G;
  const int np = L.pol == POL_TP ? 1 : 4;
  int occ = 0, sms = 0;
  resident_ctas(L, &occ, &sms);
  L.sms = sms;
  SplitProblem p;
  p.turns = (L.M + si.SPI - 1) / si.SPI;
  p.units = p.all_units = L.n_units;
  p.groups = G;
  p.planes = np;
  p.n = 1 << L.logN;
  p.radix = si.R;
  p.threads = si.TPB;
  p.target_ctas = target_ctas;
  p.sms = sms;
  p.occ = occ;
  // a sample of both lanes takes about 2.3 ps of the GPU
  p.unit_us = si.TPB * si.R * sms * 2.3e-6;
  p.max_partial = max_partial;
  p.counters = counters;
  const Split all = split_groups_and_chunks(p);
  auto take = [&](const Split& s, int* spc, int* chunks, int* finalize) {
    const int per = (p.turns + s.chunks - 1) / s.chunks;  // iterations' worth of spectra per chunk
    *spc = std::min(L.M, per * si.SPI);
    *chunks = (p.turns + per - 1) / per;
    *finalize = s.finalize && *chunks > 1;
  };
  L.sets = G / all.gps;
  const int ublocks = (L.n_units + L.sets - 1) / L.sets;
  take(all, &L.spc, &L.chunks, &L.finalize);
  // the same for a launch over 1/pipe_groups of the units
  p.units = std::max(1, L.n_units / std::max(1, pipe_groups));
  take(p.units == p.all_units ? all : split_chunks(p, all.gps), &L.spc_pipe, &L.chunks_pipe,
       &L.finalize_pipe);
  const int cmax = std::max(L.chunks, L.chunks_pipe);
  *partial_floats = cmax > 1 ? (size_t)L.n_units * cmax * np * ((size_t)1 << L.logN) : 0;
  L.arrivals = counters && cmax > 1 ? ublocks : 0;
  L.unit0 = 0;
  L.unit_count = L.n_units;
  const long long wbytes = (L.fmt == FMT_I16 ? 4 : 2) * L.nv;
  L.vec16 = ((L.chan_stride * wbytes) % 16 == 0) && ((reinterpret_cast<uintptr_t>(L.in) & 15) == 0);
  return 0;
}

cudaError_t small_prepare(const SmallLaunch& L) { return small_dispatch(L, nullptr, 1); }
cudaError_t small_launch(const SmallLaunch& L, cudaStream_t s) { return small_dispatch(L, s, 0); }

bool small_same_kernel(const SmallLaunch& a, const SmallLaunch& b) {
  return a.logN == b.logN && a.fmt == b.fmt && a.nv == b.nv && (a.nv == 1 || a.pol == b.pol) && a.smem == b.smem;
}

cudaError_t small_launch_group(const SmallLaunch* L, int n, cudaStream_t s) {
  if (n < 1 || n > kSmallGroupMax) return cudaErrorInvalidValue;
  SmallGroup g;
  g.n = n;
  int end = 0;
  for (int k = 0; k < n; ++k) {
    if (!small_same_kernel(L[0], L[k])) return cudaErrorInvalidValue;
    g.e[k] = L[k];
    end += std::max(0, small_grid(L[k]));
    g.end[k] = end;
  }
  return small_dispatch(L[0], s, 3, nullptr, &g);
}

cudaError_t finalize_launch(const FinalizeLaunch& L, cudaStream_t s) {
  const long long total = (long long)L.n_units * L.np * L.N;
  int blocks = (int)std::min<long long>((total + 255) / 256, 152LL * 16);
  if (blocks < 1) blocks = 1;
  k_finalize<<<blocks, 256, 0, s>>>(L);
  return cudaGetLastError();
}

}  // namespace rsg
