// k_large.cu -- four-step FFT spectrometer for 4096 < N <= 2^24.
//
// Replaces the reference's cuFFT plan for long transforms (one
// cufftExecC2C per product, channel batch and polarisation with load/store
// callbacks, rawspec_gpu.cu:1182-1195, :1555-1569) by two kernels:
//
//   pass A  N2-point FFTs down the columns of x[n1 + N1*n2] (both
//           polarisations), twiddled by W_N^(n1*k2), written to scratch as
//           [slab][k2][n1] -- the only intermediate that touches global
//           memory;
//   pass B  N1-point FFTs along the rows k2 of that scratch, detection of
//           the output bins X[k2 + N2*k1], integration over the unit's
//           spectra in registers, SNORM scale and the FFT-shifted store (or
//           add).
//
// X[k2 + N2 k1] = sum_n1 W_N1^(n1 k1) W_N^(n1 k2) sum_n2 x[n1 + N1 n2] W_N2^(n2 k2).
#include <algorithm>
#include <cmath>

#include "detect.cuh"
#include "fft_core.cuh"
#include "internal.h"

namespace rsg {

namespace {

// Both passes run two lanes in lockstep on the packed instructions: the two
// polarisations of a value (NV = 2), or, of one polarisation, neighbouring
// columns n1 in pass A and neighbouring rows k2 in pass B.  In pass A a lane
// pair is one word of the input either way (two polarisations of a sample,
// or two samples).
//
// What bounds them is HBM and how well its lines are used: pass A moves 20 bytes
// a sample of both polarisations (4 in, 16 out), pass B 16 and the result.
//   * Pass A: CTAs of 128 threads, C neighbouring columns each, whose
//     words come through shared memory (cp.async, 16 bytes of a row a copy) one
//     tile ahead of the transforms, where a CTA has whole sectors (32 bytes) of
//     a row: of half ones the copies fetch every sector twice (2^22 points of 16
//     bits, columns of 2048: 2055 us copied, 1186 read directly, 1815 with 256
//     threads and a polarisation at a time).  16 values per thread up to 256
//     points, 32 for 512 and 1024 (one exchange).
//   * Pass B: 16 values per thread and two neighbouring rows across the lanes,
//     so that a warp's load takes 256 contiguous bytes of each row; with
//     eight rows (64 bytes) a load it took 333 us per 64 Mi samples, with two
//     186 (65536 points, Nint 16).  Results are staged in shared memory until
//     a CTA has ROWS_OUT neighbouring rows, 32 bytes of a line in total power.
// With 256 threads, each polarisation in a plane of its own and eight rows
// across the lanes, 65536 points at Nint 16 took 446 + 344 us.
template <int NSUB, int FMT>
struct ColumnCfg {
  static constexpr int R = NSUB == 512 || NSUB == 1024 ? 32 : 16;
  static constexpr int T = NSUB / R;              // threads per column
  static constexpr int TPB = T <= 32 ? 128 : 256;
  static constexpr int C = TPB / T;               // columns (lane pairs) per CTA
  static constexpr int REGS = R == 32 ? 168 : 128;
  static constexpr int MINB = 65536 / (TPB * REGS);
  static constexpr int TW = stockham_tw_size(NSUB, R);
  static constexpr bool SPLIT = R == 32;          // one exchange buffer: three CTAs fit an SM
  static constexpr int WB = FMT == FMT_I16 ? 8 : 4;
  static constexpr bool STAGED = C * WB >= 32;
  static constexpr int STAGE = STAGED ? NSUB * C * WB : 0;
};
// OUT: results staged until a CTA has several neighbouring rows (units of one
// or two spectra, whose output is as large as their input).
template <int NSUB, int NV, int POL, bool OUT>
struct RowCfg {
  static constexpr int NP = PolOut<POL>::NP;
  static constexpr int R = POL == POL_TP || NSUB <= 1024 ? 16 : 8;
  static constexpr int T = NSUB / R;
  static constexpr int TPB = T <= 64 ? 128 : T <= 256 ? 256 : T;
  static constexpr int C = TPB / T;               // transforms per CTA
  static constexpr int CR = C < 2 ? C : 2;        // of them neighbouring lanes
  static constexpr int ROWS = NV == 2 ? 1 : 2;    // rows per transform
  static constexpr int REGS = POL != POL_TP && R == 16 ? 168 : 128;
  static constexpr int MINB = 65536 / (TPB * REGS);
  static constexpr int TW = stockham_tw_size(NSUB, R);
  // rows staged before they are written: eight, within 32 KiB
  static constexpr int FIT = 32768 / (NP * NSUB * 4);
  static constexpr int WANT = FIT < 8 ? FIT : 8;
  static constexpr int GROUPS = !OUT || C * ROWS >= WANT ? 1 : WANT / (C * ROWS);
  static constexpr int ROWS_OUT = C * ROWS * GROUPS;
};

// *p += v for four floats, without a round trip.
__device__ __forceinline__ void red_add4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

struct BlockSyncL {
  __device__ __forceinline__ void operator()(bool, bool) const { __syncthreads(); }
};

// Elements between the exchange areas of neighbouring transforms (BUFS buffers
// of smem_padded_len(N) each): at least their size, and chosen so that the C
// transforms served by one half-warp start in different banks (their start
// offsets modulo 16 are multiples of 16 / C).
template <int N, int C, int BUFS>
__host__ __device__ constexpr int sub_stride() {
  int base = BUFS * smem_padded_len(N);
  const int cp = C < 16 ? C : 16;
  const int want = (16 / cp) % 16;
  while (base % 16 != want) ++base;
  return base;
}

template <int N2, int FMT>
constexpr size_t passA_smem() {
  using Cf = ColumnCfg<N2, FMT>;
  return (size_t)((Cf::TW + 1) & ~1) * sizeof(float2) + Cf::STAGE +
         (size_t)Cf::C * sub_stride<N2, Cf::C, Cf::SPLIT ? 1 : 2>() * sizeof(float2);
}

template <int N1, int NV, int POL, bool OUT>
constexpr size_t passB_smem() {
  using Cf = RowCfg<N1, NV, POL, OUT>;
  return (size_t)((Cf::TW + 1) & ~1) * sizeof(float2) + (OUT ? (size_t)Cf::NP * N1 * Cf::ROWS_OUT * sizeof(float) : 0) +
         (size_t)Cf::C * sub_stride<N1, Cf::CR, 2>() * sizeof(float2);
}

// a * (w0, w1), one twiddle per lane
__device__ __forceinline__ cpair pmul2(const cpair& a, float2 w0, float2 w1) {
  const float2 c = make_float2(w0.x, w1.x), s = make_float2(w0.y, w1.y), ns = make_float2(-w0.y, -w1.y);
  return {f2fma(a.im, ns, f2mul(a.re, c)), f2fma(a.re, s, f2mul(a.im, c))};
}

}  // namespace

template <int N2, int FMT, int NV>
__global__ void __launch_bounds__(ColumnCfg<N2, FMT>::TPB, ColumnCfg<N2, FMT>::MINB)
k_large_a(const __grid_constant__ LargeLaunch a) {
  using Cf = ColumnCfg<N2, FMT>;
  constexpr int R = Cf::R, T = Cf::T, C = Cf::C, TPB = Cf::TPB;
  constexpr int XS = sub_stride<N2, C, Cf::SPLIT ? 1 : 2>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw_s = reinterpret_cast<float2*>(smem_raw);
  unsigned char* const stage = smem_raw + (size_t)((Cf::TW + 1) & ~1) * sizeof(float2);
  float2* const xch = reinterpret_cast<float2*>(stage + Cf::STAGE);

  const int tid = threadIdx.x;
  for (int i = tid; i < Cf::TW; i += TPB) tw_s[i] = a.twN2[i];

  const int N1 = 1 << a.logN1;
  const int NW = NV == 2 ? N1 : N1 / 2;  // lane pairs per row of the input
  const int tiles = NW / C;              // per slab
  const int first = blockIdx.x * a.tiles_a, last = min(first + a.tiles_a, tiles * a.S);
  const int col = tid % C;
  const int j = tid / C;

  using W = typename SampleWord<FMT, 2>::type;
  // Word 0 of column 0 of a tile (tiles are counted over the slabs).
  auto tile_src = [&](int tile) {
    const int slab = a.slab0 + tile / tiles;
    return reinterpret_cast<const W*>(a.in) +
           ((long long)(slab / a.Nss) * a.chan_stride + (long long)(slab % a.Nss) * (N1 * (long long)N2)) / (NV == 2 ? 1 : 2) +
           (tile % tiles) * C;
  };
  auto request = [&](int tile) {
    if constexpr (Cf::STAGED) {
      constexpr int PER = C * Cf::WB / 16;  // copies per row
      const char* src = reinterpret_cast<const char*>(tile_src(tile));
#pragma unroll
      for (int i = 0; i < N2 * PER / TPB; ++i) {
        const int e = i * TPB + tid;
        cp_async16(stage + e * 16, src + (long long)(e / PER) * NW * Cf::WB + (e % PER) * 16);
      }
    }
  };
  // W_N^e from the two-level table.
  auto level2 = [&](int e) {
    return cmul(__ldg(a.twLo + (e & ((1 << a.h) - 1))), __ldg(a.twHi + (e >> a.h)));
  };

  if (first < last) request(first);
  for (int tile = first; tile < last; ++tile) {
    const int slab = a.slab0 + tile / tiles;
    const int wc = (tile % tiles) * C + col;
    // W_N^(n1*j) of the lanes' columns
    const int n1 = NV == 2 ? wc : 2 * wc;
    const float2 w0 = level2(n1 * j);
    const float2 w1 = NV == 2 ? w0 : level2((n1 + 1) * j);
    cpair v[R];
    {
      W w[R];
      if constexpr (Cf::STAGED) {
        cp_async_wait();
        __syncthreads();  // every thread's copies have landed (and the twiddle table)
#pragma unroll
        for (int m = 0; m < R; ++m) w[m] = reinterpret_cast<const W*>(stage)[tid + m * T * C];
      } else {
        const W* src = tile_src(tile) + col + (long long)NW * j;
#pragma unroll
        for (int m = 0; m < R; ++m) w[m] = __ldg(src + (long long)NW * T * m);
        __syncthreads();
      }
#pragma unroll
      for (int m = 0; m < R; ++m) {
        if constexpr (FMT == FMT_I8) {
          v[m] = unpack_biased(w[m]);
        } else {
          float2 smp[2];
          Unpack<FMT, 2>::run(w[m], smp);
          v[m] = pack2(smp[0], smp[1]);
        }
      }
    }
    // the next tile is requested when every thread has taken this one's words
    GroupFFT<N2, R>::template run_packed<Cf::SPLIT, FMT == FMT_I8>(
        v, j, xch + (size_t)col * XS, smem_padded_len(N2), tw_s, [&](bool taken, bool) {
          __syncthreads();
          if (taken && tile + 1 < last) request(tile + 1);
        });

    // Output k2 = j + m*T: W_N^(n1*k2) = W_N^(n1*j) * W_N^(n1*m*T).  Elements of
    // 16 bytes, [slab][k2][lane pair]: both polarisations (re, re, im, im), or
    // two columns (re, im, re, im).
    float4* dst = reinterpret_cast<float4*>(a.scratch) + ((size_t)slab * N2 + j) * NW + wc;
    const float2* twm = a.twM + n1;
#pragma unroll
    for (int m = 0; m < R; ++m) {
      float4 o;
      if constexpr (NV == 2) {
        const cpair x = pmul(v[m], m == 0 ? w0 : cmul(w0, __ldg(twm + (size_t)m * N1)));
        o = make_float4(x.re.x, x.re.y, x.im.x, x.im.y);
      } else {
        float2 wa = w0, wb = w1;
        if (m > 0) {
          const float4 t = __ldg(reinterpret_cast<const float4*>(twm + (size_t)m * N1));
          wa = cmul(w0, make_float2(t.x, t.y));
          wb = cmul(w1, make_float2(t.z, t.w));
        }
        const cpair x = pmul2(v[m], wa, wb);
        o = make_float4(x.re.x, x.im.x, x.re.y, x.im.y);
      }
      dst[(size_t)m * T * NW] = o;
    }
  }
}

template <int N1, int NV, int POL, bool OUT>
__global__ void __launch_bounds__(RowCfg<N1, NV, POL, OUT>::TPB, RowCfg<N1, NV, POL, OUT>::MINB)
k_large_b(const __grid_constant__ LargeLaunch a) {
  using Cf = RowCfg<N1, NV, POL, OUT>;
  constexpr int R = Cf::R, T = Cf::T, C = Cf::C, CR = Cf::CR, TPB = Cf::TPB;
  constexpr int NP = Cf::NP, ROWS = Cf::ROWS, ROWS_OUT = Cf::ROWS_OUT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw_s = reinterpret_cast<float2*>(smem_raw);
  float* const outs = reinterpret_cast<float*>(tw_s + ((Cf::TW + 1) & ~1));  // [plane][k1][ROWS_OUT]
  float2* const xch = reinterpret_cast<float2*>(outs + (OUT ? NP * N1 * ROWS_OUT : 0));

  const int tid = threadIdx.x;
  for (int i = tid; i < Cf::TW; i += TPB) tw_s[i] = a.twN1[i];
  __syncthreads();

  const int N2 = 1 << a.logN2;
  const int N = N1 * N2;
  const int tiles = N2 / ROWS_OUT;
  const int tile = blockIdx.x % tiles;
  const int uc = blockIdx.x / tiles;
  const int unit = a.unit0 + uc / a.chunks;
  const int chunk = uc % a.chunks;
  const int c = unit / a.units_per_chan;
  const int d = unit % a.units_per_chan;
  const int row = tid % CR + CR * (tid / (CR * T));  // transform of the CTA
  const int j = tid / CR % T;
  const int s_begin = chunk * a.spc;
  const int s_end = min(a.M, s_begin + a.spc);
  const float im_sign = a.conj ? -1.0f : 1.0f;

  // Row k2 holds bins k2 + N2*k1: of the partial sums in bin order, or of the
  // dump buffer.
  const bool part = a.chunks > 1;
  float* const obase = part ? a.partial + ((size_t)unit * a.chunks + chunk) * NP * N : a.out + ((size_t)d * NP * a.Nc + c) * N;
  const size_t plane = part ? (size_t)N : (size_t)a.Nc * N;
  const float scale = part ? 1.0f : a.scale;
  const bool add = !part && a.mode == ACC_ADD;

  float2* const my_xch = xch + (size_t)row * sub_stride<N1, CR, 2>();
#pragma unroll 1
  for (int g = 0; g < Cf::GROUPS; ++g) {
    const int r0 = (g * C + row) * ROWS;    // the transform's first row of the CTA's
    const int k2 = tile * ROWS_OUT + r0;
    // total power: per lane (a row each) of one polarisation, else their sum
    float2 acc[NP == 4 || NV == 1 ? R : 1], xr[NP == 4 ? R : 1];
    float tp[NP == 1 && NV == 2 ? R : 1];
#pragma unroll
    for (int m = 0; m < R; ++m) {
      if constexpr (NP == 4 || NV == 1) acc[m] = make_float2(0.f, 0.f);
      if constexpr (NP == 4) xr[m] = make_float2(0.f, 0.f);
      if constexpr (NP == 1 && NV == 2) tp[m] = 0.0f;
    }

    for (int sl = s_begin; sl < s_end; ++sl) {
      const int slab = c * a.Nss + d * a.M + sl;
      cpair v[R];
      if constexpr (NV == 2) {
        const float4* src = reinterpret_cast<const float4*>(a.scratch) + ((size_t)slab * N2 + k2) * N1 + j;
#pragma unroll
        for (int m = 0; m < R; ++m) {
          const float4 f = __ldcs(src + m * T);
          v[m] = cpair{make_float2(f.x, f.y), make_float2(f.z, f.w)};
        }
      } else {
        const float2* src = a.scratch + ((size_t)slab * N2 + k2) * N1 + j;
#pragma unroll
        for (int m = 0; m < R; ++m) v[m] = pack2(__ldcs(src + m * T), __ldcs(src + N1 + m * T));
      }
      GroupFFT<N1, R>::template run_packed<false>(v, j, my_xch, smem_padded_len(N1), tw_s, BlockSyncL{});
#pragma unroll
      for (int m = 0; m < R; ++m) {
        if constexpr (NP == 4) {
          add_planes<POL>(v[m], acc[m], xr[m]);
        } else if constexpr (NV == 1) {
          acc[m] = f2add(acc[m], powers(v[m]));
        } else {
          tp[m] += both_powers(v[m]);
        }
      }
    }
    // value (plane p, or the lanes' rows) of element m
    auto result = [&](int m, int p, int lane) -> float {
      if constexpr (NP == 4) {
        if (p == 2) return xr[m].x;
        if (p == 3) return xr[m].y * im_sign;
        return p == 0 ? acc[m].x : acc[m].y;
      } else if constexpr (NV == 1) {
        return lane == 0 ? acc[m].x : acc[m].y;
      } else {
        return tp[m];
      }
    };

    if constexpr (OUT) {  // k1 = j + m*T of the rows into the staging area
#pragma unroll
      for (int m = 0; m < R; ++m)
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int l = 0; l < ROWS; ++l) outs[((size_t)p * N1 + j + m * T) * ROWS_OUT + r0 + l] = result(m, p, l);
    } else {
#pragma unroll
      for (int m = 0; m < R; ++m)
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
          for (int l = 0; l < ROWS; ++l) {
            const int k = k2 + l + N2 * (j + m * T);
            float* o = obase + p * plane + (part ? k : out_pos(k, N, a.inverse));
            const float x = result(m, p, l) * scale;
            if (add) atomicAdd(o, x);  // each element once per launch: a plain add, without a round trip (with: 2^19 points 258 -> 314 us)
            else *o = x;
          }
    }
  }
  if constexpr (!OUT) return;
  __syncthreads();

  // Neighbouring rows are neighbouring bins.
  constexpr int V = ROWS_OUT % 4 == 0 ? 4 : 1;
  const int k20 = tile * ROWS_OUT;
  for (int e = tid * V; e < NP * N1 * ROWS_OUT; e += TPB * V) {
    const int r = e % ROWS_OUT, k1 = e / ROWS_OUT % N1, p = e / (ROWS_OUT * N1);
    const int k = k20 + r + N2 * k1;
    float* o = obase + p * plane;
    if (V == 4 && (part || !a.inverse)) {
      float4 x = *reinterpret_cast<const float4*>(outs + e);
      x = make_float4(x.x * scale, x.y * scale, x.z * scale, x.w * scale);
      o += part ? k : out_pos(k, N, 0);
      if (add) red_add4(o, x);
      else *reinterpret_cast<float4*>(o) = x;
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float* q = o + (part ? k + i : out_pos(k + i, N, a.inverse));
        if (add) atomicAdd(q, outs[e + i] * scale);  // each element once per launch
        else *q = outs[e + i] * scale;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
namespace {

template <int N2, int FMT, int NV>
cudaError_t launch_a_t(const LargeLaunch& L, cudaStream_t s, bool prep) {
  using Cf = ColumnCfg<N2, FMT>;
  auto k = k_large_a<N2, FMT, NV>;
  const size_t smem = passA_smem<N2, FMT>();
  if (prep) return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int N1 = 1 << L.logN1;
  const long long tiles = (long long)(N1 / (NV == 2 ? 1 : 2) / Cf::C) * L.S;
  if (tiles < 1) return cudaSuccess;
  // Tiles per CTA: as many as leave four CTAs for every resident one, eight at
  // most (the first tile of a CTA is not copied ahead of time).
  LargeLaunch l = L;
  l.tiles_a = Cf::STAGED ? (int)std::max<long long>(1, std::min<long long>(8, tiles / (4ll * 152 * Cf::MINB))) : 1;
  k<<<(unsigned)((tiles + l.tiles_a - 1) / l.tiles_a), Cf::TPB, smem, s>>>(l);
  return cudaGetLastError();
}

// Units of at most this many spectra in a buffer stage their results: one
// spectrum, 2^16 points 319 -> 270 us, 2^18 496 -> 375; with 16 the staging
// costs more than it gives (2^18 237 -> 311).
constexpr int kStageOutSpectra = 2;
bool stage_out(const LargeLaunch& L) { return L.M <= kStageOutSpectra; }

template <int N1, int NV, int POL, bool OUT>
cudaError_t launch_b_o(const LargeLaunch& L, cudaStream_t s, bool prep) {
  using Cf = RowCfg<N1, NV, POL, OUT>;
  auto k = k_large_b<N1, NV, POL, OUT>;
  const size_t smem = passB_smem<N1, NV, POL, OUT>();
  if (prep) return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int N2 = 1 << L.logN2;
  const long long grid = (long long)(N2 / Cf::ROWS_OUT) * L.unit_count * L.chunks;
  if (grid < 1) return cudaSuccess;
  k<<<(unsigned)grid, Cf::TPB, smem, s>>>(L);
  return cudaGetLastError();
}

template <int N1, int NV, int POL>
cudaError_t launch_b_t(const LargeLaunch& L, cudaStream_t s, bool prep) {
  return stage_out(L) ? launch_b_o<N1, NV, POL, true>(L, s, prep) : launch_b_o<N1, NV, POL, false>(L, s, prep);
}

template <int N2>
cudaError_t launch_a_n(const LargeLaunch& L, cudaStream_t s, bool prep) {
  if (L.fmt == FMT_I16) return L.nv == 1 ? launch_a_t<N2, FMT_I16, 1>(L, s, prep) : launch_a_t<N2, FMT_I16, 2>(L, s, prep);
  return L.nv == 1 ? launch_a_t<N2, FMT_I8, 1>(L, s, prep) : launch_a_t<N2, FMT_I8, 2>(L, s, prep);
}

template <int N1>
cudaError_t launch_b_n(const LargeLaunch& L, cudaStream_t s, bool prep) {
  if (L.nv == 1) return launch_b_t<N1, 1, POL_TP>(L, s, prep);
  switch (L.pol) {
    case POL_FULL: return launch_b_t<N1, 2, POL_FULL>(L, s, prep);
    case POL_STOKES: return launch_b_t<N1, 2, POL_STOKES>(L, s, prep);
    default: return launch_b_t<N1, 2, POL_TP>(L, s, prep);
  }
}

cudaError_t dispatch_a(const LargeLaunch& L, cudaStream_t s, bool prep) {
  switch (L.logN2) {
    case 7: return launch_a_n<128>(L, s, prep);
    case 8: return launch_a_n<256>(L, s, prep);
    case 9: return launch_a_n<512>(L, s, prep);
    case 10: return launch_a_n<1024>(L, s, prep);
    case 11: return launch_a_n<2048>(L, s, prep);
    case 12: return launch_a_n<4096>(L, s, prep);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t dispatch_b(const LargeLaunch& L, cudaStream_t s, bool prep) {
  switch (L.logN1) {
    case 6: return launch_b_n<64>(L, s, prep);
    case 7: return launch_b_n<128>(L, s, prep);
    case 8: return launch_b_n<256>(L, s, prep);
    case 9: return launch_b_n<512>(L, s, prep);
    case 10: return launch_b_n<1024>(L, s, prep);
    case 11: return launch_b_n<2048>(L, s, prep);
    case 12: return launch_b_n<4096>(L, s, prep);
    default: return cudaErrorInvalidValue;
  }
}

template <int N1, int NV, int POL>
void row_geometry_t(bool out, int* radix, int* rows) {
  *radix = RowCfg<N1, NV, POL, false>::R;
  *rows = out ? RowCfg<N1, NV, POL, true>::ROWS_OUT : RowCfg<N1, NV, POL, false>::ROWS_OUT;
}
template <int N1>
void row_geometry(const LargeLaunch& L, int* radix, int* rows) {
  if (L.pol != POL_TP) row_geometry_t<N1, 2, POL_FULL>(stage_out(L), radix, rows);
  else if (L.nv == 2) row_geometry_t<N1, 2, POL_TP>(stage_out(L), radix, rows);
  else row_geometry_t<N1, 1, POL_TP>(stage_out(L), radix, rows);
}

// Radix and rows per CTA of pass B.
void pass_b_geometry(const LargeLaunch& L, int* radix, int* rows) {
  switch (L.logN1) {
    case 6: return row_geometry<64>(L, radix, rows);
    case 7: return row_geometry<128>(L, radix, rows);
    case 8: return row_geometry<256>(L, radix, rows);
    case 9: return row_geometry<512>(L, radix, rows);
    case 10: return row_geometry<1024>(L, radix, rows);
    case 11: return row_geometry<2048>(L, radix, rows);
    default: return row_geometry<4096>(L, radix, rows);
  }
}

}  // namespace

int large_pass_a_radix(const LargeLaunch& L) { return L.logN2 == 9 || L.logN2 == 10 ? 32 : 16; }
int large_pass_b_radix(const LargeLaunch& L) {
  int r, c;
  pass_b_geometry(L, &r, &c);
  return r;
}
int stockham_table_size(int N, int R) { return stockham_tw_size(N, R); }

// N2 of N1 * N2.  Pass A is fastest at 256 points (eight columns a CTA: 250 us
// per 64 Mi samples of two polarisations; 512 points 295, 1024, with four
// columns, 490), pass B between 128 and 512 (185-240; 1024 250, 2048 340, 4096
// 410 with 16 spectra a unit): 2^16 247 + 190, 2^18 as 256 x 1024 249 + 246,
// as 512 x 512 294 + 240; 2^20 in total power 512 x 2048 300 + 338, 1024 x 1024
// 502 + 276.  The four planes and one polarisation pay more for long rows
// (2^20: 760 and 307 with 2048, 441 and 243 with 1024).
static int split_log_n2(const LargeLaunch& L) {
  const bool pair = L.pol == POL_TP && L.nv == 2;  // total power of two polarisations
  switch (L.logN) {
    case 13: case 14: return 7;
    case 15: case 16: case 18: return 8;
    case 17: case 19: return 9;
    case 20: return pair ? 9 : 10;
    case 21: return pair ? 9 : L.nv == 1 ? 10 : 11;
    case 22: return L.nv == 1 ? 10 : 11;
    default: return 12;
  }
}

int large_configure(LargeLaunch& L, int target_ctas, size_t* scratch_float2, size_t* partial_floats) {
  if (L.logN < 13 || L.logN > 24) return -1;
  L.logN2 = split_log_n2(L);
  L.logN1 = L.logN - L.logN2;
  L.h = (L.logN + 1) / 2;
  const int N2 = 1 << L.logN2;
  const int np = L.pol == POL_TP ? 1 : 4;
  // Chunks of a unit's spectra across CTAs: where a unit's spectra one after
  // another (about 1.5 us each in a CTA) would take longer than the pass's
  // traffic, by more than the sum of the partials costs (a launch and its
  // traffic: 21 channels x 16384 points, Nint 8: whole units 39 us, halves
  // 35 + 14; 8 channels, Nint 32: whole 50, quarters 23 + 6).
  int radix, rows;
  pass_b_geometry(L, &radix, &rows);
  const long long base = (long long)(N2 / rows) * L.n_units;  // CTAs per chunk
  const double bytes = (double)L.n_units * L.M * ((size_t)8 * L.nv << L.logN);
  const double partial_us = (double)L.n_units * np * ((size_t)8 << L.logN) / 4e6;
  int chunks = 1;
  double best = 1e300;
  for (int c = 1; c <= L.M && (c == 1 || base * c <= 2ll * target_ctas); ++c) {
    const double serial = std::ceil((double)L.M / c) * 1.5 * std::max(1.0, (double)base * c / target_ctas);
    const double t = std::max(bytes / 5.5e6, serial) + (c > 1 ? 6.0 + c * partial_us : 0.0);
    if (t < best * 0.95) {
      best = t;
      chunks = c;
    }
  }
  L.spc = (L.M + chunks - 1) / chunks;
  L.chunks = (L.M + L.spc - 1) / L.spc;
  *scratch_float2 = (size_t)L.Nc * L.Nss * L.nv * ((size_t)1 << L.logN);
  *partial_floats = L.chunks > 1 ? (size_t)L.n_units * L.chunks * np * ((size_t)1 << L.logN) : 0;
  L.slab0 = 0;
  L.S = L.Nc * L.Nss;
  L.unit0 = 0;
  L.unit_count = L.n_units;
  return 0;
}

cudaError_t large_prepare(const LargeLaunch& L) {
  cudaError_t e = dispatch_a(L, nullptr, true);
  if (e != cudaSuccess) return e;
  return dispatch_b(L, nullptr, true);
}

cudaError_t large_launch_a(const LargeLaunch& L, cudaStream_t s) { return dispatch_a(L, s, false); }
cudaError_t large_launch_b(const LargeLaunch& L, cudaStream_t s) { return dispatch_b(L, s, false); }

}  // namespace rsg
