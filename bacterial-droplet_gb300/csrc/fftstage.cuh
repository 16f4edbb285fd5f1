// fftstage.cuh — FP32 butterflies of a radix plan's stages (factors 2, 3, 4, 5), shared by the any-size
// FFT kernels (fft.cu, fftplan_impl.cuh).
#pragma once
#include "common.cuh"

namespace ttsh {

// a b in FP32: one product of each part is rounded, the other joins it in a fused multiply-add. INV (the
// inverse transform, run on conjugated values) fuses the other product of the imaginary part: the
// choice the compiler makes for a times a conjugated twiddle, which the results have always had.
template <bool INV>
__device__ __forceinline__ float2 stage_cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), INV ? fmaf(a.y, b.x, a.x * b.y) : fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 stage_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 stage_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

template <class T> constexpr int fft_min_ctas() { return sizeof(T) == 4 ? 3 : 2; }

// FP32: one butterfly of the radix plan, in place: the twiddles w^(r k ts) of its stage, then the DFT
// of R = 2, 4 in butterflies, of R = 3, 5 as the sum that defines it (its roots of unity from the
// table).
template <bool INV, int R>
__device__ __forceinline__ void plan_butterfly(float2* v, const float2* tw, int N, int k, int ts) {
  if (k > 0) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = stage_cmul<INV>(v[r], __ldg(tw + r * k * ts));
  }
  if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = stage_add(a, b);
    v[1] = stage_sub(a, b);
  } else if constexpr (R == 4) {
    const float2 a = stage_add(v[0], v[2]), b = stage_sub(v[0], v[2]), c = stage_add(v[1], v[3]), d = stage_sub(v[1], v[3]);
    const float2 dd = make_float2(d.y, -d.x);
    v[0] = stage_add(a, c);
    v[2] = stage_sub(a, c);
    v[1] = stage_add(b, dd);
    v[3] = stage_sub(b, dd);
  } else {
    float2 o[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      float2 acc = v[0];
#pragma unroll
      for (int r = 1; r < R; ++r) acc = stage_add(acc, (q * r) % R ? stage_cmul<INV>(v[r], __ldg(tw + ((q * r) % R) * (N / R))) : v[r]);
      o[q] = acc;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = o[q];
  }
}
}  // namespace ttsh
