// detect.cuh -- detection of the two polarisations' spectra into the output
// products, accumulated in registers.
//
// Formulas follow the reference's cuFFT store callbacks:
//   total power (Npolout 1)  P  += |X0|^2 (+ |X1|^2)          rawspec_gpu.cu:153-161
//   full pol    (Npolout +4) XX += |X0|^2, YY += |X1|^2,
//                            re += Re(X0 X1*), im += Im(X0 X1*) rawspec_gpu.cu:223-267
//   Stokes      (Npolout -4) I  += |X0|^2 + |X1|^2, Q += |X0|^2 - |X1|^2,
//                            U  += Re(X0 X1*), V += Im(X0 X1*)  rawspec_gpu.cu:167-218
// with the imaginary cross term negated when the input is conjugated.
#pragma once

#include "common.cuh"
#include "fft_core.cuh"
#include "internal.h"

namespace rsg {

template <int POL>
struct PolOut {
  static constexpr int NP = (POL == POL_TP) ? 1 : 4;
};

// |X|^2 of both lanes, and their sum.  A spectrum's power is formed first and
// enters a sum over spectra with one rounding.
__device__ __forceinline__ float2 powers(const cpair& v) { return f2fma(v.re, v.re, f2mul(v.im, v.im)); }
__device__ __forceinline__ float both_powers(const cpair& v) {
  return __fmaf_rn(v.im.y, v.im.y, __fmaf_rn(v.re.y, v.re.y, __fmaf_rn(v.im.x, v.im.x, v.re.x * v.re.x)));
}

// Adds one spectrum's bin of both polarisations to the sums of the four
// planes: pw the planes 0 and 1, xr Re and Im of X0 X1* (its sign for
// conjugated input comes after the last spectrum, being linear).  Stokes Q is summed as the
// difference of every spectrum, not as the difference of two large sums.
template <int POL>
__device__ __forceinline__ void add_planes(const cpair& v, float2& pw, float2& xr) {
  const float2 p = powers(v);
  pw = f2add(pw, POL == POL_STOKES ? make_float2(p.x + p.y, p.x - p.y) : p);
  const float2 x0 = lane0(v), x1 = lane1(v);
  xr = f2add(xr, make_float2(__fmaf_rn(x0.x, x1.x, x0.y * x1.y), __fmaf_rn(x0.y, x1.x, -(x0.x * x1.y))));
}

// Position of forward-FFT bin k in the FFT-shifted output of an N-point
// transform in the requested direction: inverse transforms read bin -k, and
// the shift puts bin 0 at N/2 (rawspec_gpu.cu:1659-1691).
__device__ __forceinline__ int out_pos(int k, int N, int inverse) {
  const int kr = inverse ? ((N - k) & (N - 1)) : k;
  return (kr + (N >> 1)) & (N - 1);
}

}  // namespace rsg
