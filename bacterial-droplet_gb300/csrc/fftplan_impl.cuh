// fftplan_impl.cuh — the any-size FFT of fft.cu built per size: the steps, strides, lines per CTA and
// index arithmetic of a size are compile-time constants, the values the same bits. The kernel for any
// size spends most of its issue slots on that arithmetic (FP32 at N = 288: 190 instructions per value
// and 1-D transform, of which the butterflies are about 60), and in a launch of few CTAs on fetching
// the code of every step. Sizes without a kernel here, explicit lines per CTA and other radix plans run
// there. One Poisson solve (three launches), kernel for any size -> per size: FP32 2 x 288^3 2.27 -> 1.12
// ms, 4 x 100^3 250 -> 110 us, 200^3 482 -> 252, 9 x 20^3 54 -> 26; FP64 4 x 100^3 1.26 -> 1.19 ms (bound by
// the FP64 pipe either way).
#pragma once
#include <stdexcept>
#include <string>

#include "common.cuh"
#include "dft.cuh"
#include "fftplan.h"
#include "fftreg.cuh"
#include "fftstage.cuh"
#include "kernels.h"

namespace ttsh {
namespace fftplan {

template <class T, int N, bool SMALL>
struct Plan {
  static constexpr Steps S = SMALL ? small_steps(N) : default_steps<T>(N);
  static constexpr int LB = SMALL ? small_lb(N) : default_lb<T>(N), NG = N / LB, PC = cluster_parts(NG), THREADS = threads_for(S, N, LB);
  static constexpr int HALF = LB * x_pitch(N);  // values of one buffer
  static_assert(N % LB == 0 && 2 * HALF * 2 * sizeof(T) <= 227 * 1024, "lines per CTA");
  static constexpr int ops(int pass) { return pass_steps<T>(S.n, pass); }
  static constexpr size_t smem(int pass) {
    return (size_t)(ops(pass) < 2 ? 0 : (ops(pass) == 2 ? 1 : 2)) * HALF * sizeof(typename CxT<T>::type);
  }
  // operation q of a pass: its step, and the product of the radices before it. The inverse x and y
  // transforms of a small size go through the steps backwards, as the register kernels do.
  static constexpr bool back(int q, int pass) { return sizeof(T) == 8 && (q >= S.n || (SMALL && pass >= 3)); }
  static constexpr int step_of(int q, int pass) {
    if (pass != 2) return back(q, pass) ? S.n - 1 - q : q;
    return q < S.n ? q : (back(q, pass) ? 2 * S.n - 2 - q : q - S.n);
  }
  static constexpr int before(int q, int pass) {
    int p = 1;
    if (back(q, pass)) {
      for (int i = S.n - 1; i > step_of(q, pass); --i) p *= S.radix(i);
    } else {
      for (int i = 0; i < step_of(q, pass); ++i) p *= S.radix(i);
    }
    return p;
  }
};

// Operation Q of a pass and the ones after it, on the lines whose first element is at W + base.
template <class T, int N, bool SMALL, int PASS, int Q>
__device__ __forceinline__ void run_ops(const InstDev<T>& I, size_t base, int x0, int y, typename CxT<T>::type* buf) {
  typedef typename CxT<T>::type C;
  typedef Plan<T, N, SMALL> P;
  constexpr int OPS = P::ops(PASS), IDX = P::step_of(Q, PASS), A = P::S.a[IDX], B = P::S.b[IDX], R = A * B, M = N / R, NS = P::before(Q, PASS);
  constexpr bool XAXIS = PASS == 0 || PASS == 4, FIRST = Q == 0, LAST = Q == OPS - 1, DIVIDE = PASS == 2 && Q == P::S.n - 1;
  constexpr bool INV = PASS >= 3 || Q >= P::S.n;
  constexpr size_t STRIDE = XAXIS ? 1 : (PASS == 2 ? (size_t)N * N : N), LSTRIDE = XAXIS ? N : 1;
  const C* src = buf + (Q % 2 ? 0 : P::HALF);
  C* dst = buf + (Q % 2 ? P::HALF : 0);
  auto spos = [](int l, int e) { return XAXIS ? l * x_pitch(N) + e + (e >> 3) : e * P::LB + l; };
  const C* __restrict__ tw = I.tw;
#pragma unroll 1
  for (int b = threadIdx.x; b < P::LB * M; b += P::THREADS) {
    const int l = XAXIS ? b / M : b % P::LB, j = XAXIS ? b % M : b / P::LB;
    C* const w = I.W + base + (size_t)l * LSTRIDE;
    C v[R];
    if constexpr (FIRST) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = w[(size_t)(j + r * M) * STRIDE];
      if constexpr (PASS >= 3) {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r].y = -v[r].y;
      }
      if constexpr (PASS == 0 && sizeof(T) == 4) {
        if (I.wmax) {
          const T su = pow2_norm(I.wmax[0]), sp = pow2_norm(I.wmax[1]);
#pragma unroll
          for (int r = 0; r < R; ++r) { v[r].x *= su; v[r].y *= sp; }
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = src[spos(l, j + r * M)];
    }
    const int k = NS == 1 ? 0 : j % NS;
    // element of output r of the step: e0 + oe(r)
    int e0 = (j / NS) * (NS * R) + k;
    constexpr bool TURN = DIVIDE && sizeof(T) == 8;
    if constexpr (sizeof(T) == 8) {
      if constexpr (NS > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = dft::mul(v[r], __ldg(tw + r * (N / (NS * R)) * k));
      }
      dft::Dft<R>::run(v);
      if constexpr (TURN) {
        const fftreg::Poisson<T> pm(I, x0 + l, y);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = dft::conj(pm(v[r], I, j + r * M));
        dft::Dft<R>::run(v);
        e0 = j * R;
      }
    } else {
#pragma unroll
      for (int q = 0; q < B; ++q) {
        C u[A];
#pragma unroll
        for (int r = 0; r < A; ++r) u[r] = v[r * B + q];
        plan_butterfly<INV, A>(u, tw, N, k, N / (NS * A));
#pragma unroll
        for (int r = 0; r < A; ++r) v[r * B + q] = u[r];
      }
      if constexpr (B > 1) {
#pragma unroll
        for (int r = 0; r < A; ++r) {
          C u[B];
#pragma unroll
          for (int q = 0; q < B; ++q) u[q] = v[r * B + q];
          plan_butterfly<INV, B>(u, tw, N, k + r * NS, N / (NS * R));
#pragma unroll
          for (int q = 0; q < B; ++q) v[r * B + q] = u[q];
        }
      }
      if constexpr (DIVIDE) {
        const fftreg::Poisson<T> pm(I, x0 + l, y);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = dft::conj(pm(v[r], I, e0 + (r / B + r % B * A) * NS));
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int e = e0 + (TURN ? r : (r / B + r % B * A) * NS);
      if constexpr (LAST) {
        C o = v[r];
        if constexpr (PASS >= 2) o.y = -o.y;
        if constexpr (PASS == 4) o = fftreg::scale_n3(o, I);
        w[(size_t)e * STRIDE] = o;
      } else {
        dst[spos(l, e)] = v[r];
      }
    }
  }
  if constexpr (!LAST) {
    __syncthreads();
    run_ops<T, N, SMALL, PASS, Q + 1>(I, base, x0, y, buf);
  }
}

// Line group g of a pass.
template <class T, int N, bool SMALL, int PASS>
__device__ __forceinline__ void run_group(const InstDev<T>& I, int g, typename CxT<T>::type* buf) {
  typedef Plan<T, N, SMALL> P;
  if constexpr (PASS == 0 || PASS == 4) {
    run_ops<T, N, SMALL, PASS, 0>(I, (size_t)g * P::LB * N, 0, 0, buf);
  } else {
    const int outer = g / P::NG, x0 = (g - outer * P::NG) * P::LB;
    run_ops<T, N, SMALL, PASS, 0>(I, (size_t)outer * (PASS == 2 ? N : N * N) + x0, x0, outer, buf);
  }
}

template <class T>
constexpr int min_ctas() { return sizeof(T) == 4 ? 3 : 2; }

// z lines
template <class T, int N, bool SMALL>
__global__ void __launch_bounds__(Plan<T, N, SMALL>::THREADS, min_ctas<T>()) k_plan_z(const InstDev<T>* __restrict__ insts) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  run_group<T, N, SMALL, 2>(insts[blockIdx.y], blockIdx.x, reinterpret_cast<typename CxT<T>::type*>(smem_raw));
}
// Both in-plane axes of a z-plane, one cluster per plane (as k_fft_plane): FIRST pass, then SECOND.
template <class T, int N, bool SMALL, int FIRST, int SECOND>
__global__ void __cluster_dims__(Plan<T, N, SMALL>::PC, 1, 1) __launch_bounds__(Plan<T, N, SMALL>::THREADS, min_ctas<T>())
    k_plan_plane(const InstDev<T>* __restrict__ insts) {
  typedef Plan<T, N, SMALL> P;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto* buf = reinterpret_cast<typename CxT<T>::type*>(smem_raw);
  const InstDev<T>& I = insts[blockIdx.y];
  const int z = blockIdx.x / P::PC, part = blockIdx.x % P::PC;
#pragma unroll 1
  for (int gg = part; gg < P::NG; gg += P::PC) {
    run_group<T, N, SMALL, FIRST>(I, z * P::NG + gg, buf);
    __syncthreads();  // the next group reuses the buffers
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
#pragma unroll 1
  for (int gg = part; gg < P::NG; gg += P::PC) {
    run_group<T, N, SMALL, SECOND>(I, z * P::NG + gg, buf);
    __syncthreads();
  }
}

template <class T, int N, bool SMALL>
void prepare_one() {
  typedef Plan<T, N, SMALL> P;
  const std::pair<const void*, size_t> k[] = {{(const void*)k_plan_z<T, N, SMALL>, P::smem(2)},
                                              {(const void*)k_plan_plane<T, N, SMALL, 0, 1>, P::smem(0)},
                                              {(const void*)k_plan_plane<T, N, SMALL, 3, 4>, P::smem(3)}};
  for (const auto& f : k) {
    const cudaError_t e = cudaFuncSetAttribute(f.first, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.second);
    if (e != cudaSuccess) throw std::runtime_error(std::string("fft (plan) smem attribute: ") + cudaGetErrorString(e));
  }
}

// pass 2: the z lines; 0: forward x + y of every plane; 4: inverse y + x
template <class T, int N, bool SMALL>
void launch_size(const Group<T>& g, int pass, cudaStream_t st) {
  typedef Plan<T, N, SMALL> P;
  if (pass == 2) k_plan_z<T, N, SMALL><<<dim3(N * P::NG, g.n), P::THREADS, P::smem(2), st>>>(g.d_inst);
  else if (pass == 0) k_plan_plane<T, N, SMALL, 0, 1><<<dim3(N * P::PC, g.n), P::THREADS, P::smem(0), st>>>(g.d_inst);
  else k_plan_plane<T, N, SMALL, 3, 4><<<dim3(N * P::PC, g.n), P::THREADS, P::smem(3), st>>>(g.d_inst);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("fft (plan) launch: ") + cudaGetErrorString(e));
}

}  // namespace fftplan

// The sizes of one translation unit (several build in parallel): NAME_launch / NAME_prepare return false
// where the size is not among them.
#define TTSH_FFTPLAN_UNIT(NAME, T, SIZES)                                     \
  bool NAME##_launch(const Group<T>& g, int pass, cudaStream_t st) {          \
    switch (g.N) {                                                            \
      SIZES(TTSH_FFTPLAN_LAUNCH)                                              \
      default: return false;                                                  \
    }                                                                         \
  }                                                                           \
  bool NAME##_prepare(int N) {                                                \
    switch (N) {                                                              \
      SIZES(TTSH_FFTPLAN_PREPARE)                                             \
      default: return false;                                                  \
    }                                                                         \
  }
#ifndef TTSH_FFTPLAN_SMALL
#define TTSH_FFTPLAN_SMALL false
#endif
#define TTSH_FFTPLAN_LAUNCH(n) case n: fftplan::launch_size<TTSH_FFTPLAN_T, n, TTSH_FFTPLAN_SMALL>(g, pass, st); return true;
#define TTSH_FFTPLAN_PREPARE(n) case n: fftplan::prepare_one<TTSH_FFTPLAN_T, n, TTSH_FFTPLAN_SMALL>(); return true;

// The products of 2, 3 and 5 up to 500 without a register kernel (fftreg_impl.cuh).
#define TTSH_FFTPLAN_A(X) X(9) X(10) X(12) X(15) X(18) X(20) X(25) X(27) X(30) X(36) X(40) X(45) X(50) X(54) X(60) X(72)
#define TTSH_FFTPLAN_B(X) X(75) X(80) X(81) X(90) X(100) X(108) X(120) X(125) X(135) X(144) X(150) X(162) X(180) X(200) X(216)
#define TTSH_FFTPLAN_C(X) \
  X(225) X(240) X(243) X(250) X(270) X(288) X(300) X(320) X(324) X(360) X(375) X(384) X(400) X(405) X(432) X(450) X(480) X(486) X(500)
// The small sizes of the register kernels in FP64 (small_steps): 8 and 16 gain nothing.
#define TTSH_FFTPLAN_S(X) X(24) X(32) X(48)

}  // namespace ttsh
