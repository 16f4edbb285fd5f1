// fftreg.cuh — register-resident two-level FFT passes (the fast path of fft.cu's passes).
//
// A line of length N = N1*N2 is transformed as in the "four-step" factorisation:
//   Y[k1][n2] = DFT_N1 over n1 of x[N2*n1 + n2]                 (thread n2 holds x[N2*n1+n2])
//   X[k1 + N1*k2] = DFT_N2 over n2 of w_N^(n2*k1) * Y[k1][n2]    (after one shared-memory transpose)
// and the inverse runs the same steps backwards. Each thread keeps its N1 (or N2) values in
// registers; small DFTs are expanded at compile time by mixed-radix decimation in time
// (FP32: radix 4, 2, and 3 and 5 as the sums that define them; FP64: dft.cuh), with twiddles from the FP64-built table
// exp(-2 pi i k / N).
// The z pass goes forward, applies the Poisson multiplier and goes back without leaving the
// CTA: two shared-memory transposes for the whole forward-divide-inverse sequence.
#pragma once
#include "common.cuh"
#include "dft.cuh"

namespace ttsh {
namespace fftreg {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  float2 r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
// FP32: one packed instruction (add/sub .f32x2: two IEEE FP32 operations, round to nearest, the
// results of the two scalar ones) per complex add or subtract.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  float2 d;
  asm("sub.rn.f32x2 %0, %1, %2;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<const unsigned long long*>(&a)), "l"(*reinterpret_cast<const unsigned long long*>(&b)));
  return d;
}
// exp(-+2 pi i k / N) from the table; conjugate for the inverse.
template <class C, bool INV>
__device__ __forceinline__ C tw(const C* t, int k) {
  C w = __ldg(t + k);
  if (INV) w.y = -w.y;
  return w;
}

constexpr int first_radix(int L) { return L % 4 == 0 ? 4 : (L % 2 == 0 ? 2 : (L % 3 == 0 ? 3 : 5)); }

// exp(-2 pi i k / NF) from the __constant__ copy of the size-NF table (defined per size by
// fftreg_impl.cuh): with a compile-time k it is a constant-bank operand, not a load.
template <class C, int NF>
__device__ C ctw(int k);

// ... conjugate for the inverse
template <bool INV, int NF>
__device__ __forceinline__ float2 twx(int k) {
  float2 w = ctw<float2, NF>(k);
  if (INV) w.y = -w.y;
  return w;
}

// FP32: in-place DFT of v[0..L) (natural order in and out), a factor of a line of length NF. `step` = NF / L, so
// that w_L^m is entry m step of the line's table.
template <int L, bool INV, int NF>
struct Dft {
  typedef float2 C;
  static __device__ __forceinline__ void run(C* v, int step) {
    constexpr int R = first_radix(L);
    constexpr int M = L / R;
    if constexpr (L == 1) {
      return;
    } else if constexpr (L == 2) {
      C a = v[0], b = v[1];
      v[0] = cadd(a, b);
      v[1] = csub(a, b);
    } else if constexpr (L == 4) {
      C a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
      C dd;
      if (INV) { dd.x = -d.y; dd.y = d.x; } else { dd.x = d.y; dd.y = -d.x; }
      v[0] = cadd(a, c);
      v[2] = csub(a, c);
      v[1] = cadd(b, dd);
      v[3] = csub(b, dd);
    } else if constexpr (L == 3 || L == 5) {
      C o[L];
#pragma unroll
      for (int q = 0; q < L; ++q) {
        C acc = v[0];
#pragma unroll
        for (int r = 1; r < L; ++r) acc = cadd(acc, cmul(v[r], twx<INV, NF>(((q * r) % L) * step)));
        o[q] = acc;
      }
#pragma unroll
      for (int q = 0; q < L; ++q) v[q] = o[q];
    } else {
      // decimation in time: R sub-sequences v[r + R*m], each a DFT of length M
      C u[R][M];
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int m = 0; m < M; ++m) u[r][m] = v[r + R * m];
        Dft<M, INV, NF>::run(u[r], step * R);
      }
#pragma unroll
      for (int k0 = 0; k0 < M; ++k0) {
        C t[R];
#pragma unroll
        for (int r = 0; r < R; ++r) t[r] = (r > 0 && k0 > 0) ? cmul(u[r][k0], twx<INV, NF>(r * k0 * step)) : u[r][k0];
        Dft<R, INV, NF>::run(t, step * M);
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) v[k0 + M * k1] = t[k1];
      }
    }
  }
};

// -F / k^2 of getStream mode 1 (:672-683) with k2 from initPoissonSolver (:1088-1124), along the z
// line at (x, y). In FP64 k2 is the host's kx*kx + ky*ky + kz*kz bit for bit (rounded squares, no
// contraction); the spectrum is multiplied by one reciprocal instead of divided twice (an FP64
// division takes about ten operations).
template <class T>
struct Poisson {
  T a, b, c;
  bool line0;  // x = y = 0
  __device__ __forceinline__ Poisson(const InstDev<T>& I, int x, int y) {
    line0 = (x | y) == 0;
    if (I.k2mode == 0) {
      a = sum(I.k2t[x], I.k2t[y]);
      b = c = T(0);
    } else {
      a = I.St[x] * I.Ct[y];
      b = I.Ct[x] * I.St[y];
      c = I.Ct[x] * I.Ct[y];
    }
  }
  static __device__ __forceinline__ double sum(double u, double v) { return __dadd_rn(u, v); }
  static __device__ __forceinline__ float sum(float u, float v) { return __fadd_rn(u, v); }
  static __device__ __forceinline__ double reciprocal(double v) { return 1.0 / v; }
  static __device__ __forceinline__ float reciprocal(float v) { return __frcp_rn(v); }  // the value of 1.f / v
  template <class C>
  __device__ __forceinline__ C operator()(C v, const InstDev<T>& I, int z) const {
    T k2;
    C o;
    if (I.k2mode == 0) {
      k2 = sum(a, I.k2t[z]);
      if (line0 && z == 0) k2 = T(1);  // k2[0] = 1 (:1120)
    } else {
      const T ct = I.Ct[z], Kx = a * ct, Ky = b * ct, Kz = c * I.St[z];
      k2 = Kx * Kx + Ky * Ky + Kz * Kz;
      if (k2 < T(1e-8) / (I.ph.h * I.ph.h)) {
        o.x = o.y = T(0);
        return o;
      }
    }
    const T f = -reciprocal(k2);
    o.x = v.x * f;
    o.y = v.y * f;
    return o;
  }
};

// getStream mode 2 (:684-690): times 1/N^3 (exact where N is a power of two)
__device__ __forceinline__ double2 scale_n3(double2 v, const InstDev<double>& I) {
  return make_double2(v.x * I.ph.invN3, v.y * I.ph.invN3);
}
__device__ __forceinline__ float2 scale_n3(float2 v, const InstDev<float>& I) {
  return make_float2(v.x * I.ph.invN3, v.y * I.ph.invN3);
}

}  // namespace fftreg
}  // namespace ttsh
