// fft.cu — hand-written batched 3D FFT Poisson solve for any N = 2^a 3^b 5^c (replaces the
// reference's cufftExecZ2Z forward/inverse pair and getStream modes 1 and 2, TTSH3D.cu:635-691);
// the sizes of the register table (fftreg_impl.cuh) use its kernels instead.
//
// Both projections of a step are solved with ONE complex transform: the packed
// field W = div(u*)/dt + i div(P*)/dt is transformed, multiplied by the real, even
// multiplier -1/k^2, and transformed back, so Re W = p_v and Im W = p_p (the
// multiplier keeps the Hermitian symmetry of each real part separately).
//
// A CTA takes LB lines. The transform of a line is a Stockham autosort FFT (the formulation of
// Govindaraju et al., SC'08). The first step reads its values from global memory and the last one
// writes its results there, in the same coalesced pattern, so a line goes through shared memory once
// per pair of steps. Passes:
//   0 forward x   1 forward y   2 forward z -> divide -> inverse z
//   3 inverse y   4 inverse x, scaled by 1/N^3 (getStream mode 2, :684-690)
// The inverse transform is the forward one between conjugations.
//   FP64 (bound by the FP64 pipe): steps of radix 2 .. 16 with the small DFTs of dft.cuh, chosen by
//     size (N = 100 is 10 x 10, N = 320 is 10 x 8 x 4); a radix-5 butterfly is 36 operations instead of
//     the 120 of the sum that defines it. Pass 2 multiplies by -1/k^2 and begins the inverse in the
//     registers of the forward transform's last step, whose outputs (elements j + r N/R) are the
//     inputs of a first step of the same radix.
//   FP32 (bound by latency and issue): the stages of the radix plan (4, 2, 3, 5), up to two of them
//     in registers per step: the butterflies of one stage feed those of the next within a thread, so
//     the arithmetic is the plan's, stage by stage, with half the trips through shared memory. Few line
//     groups, one launch per axis: one stage per step (k_fft_smem).
// Twiddles between steps come from a table exp(-2 pi i k/N) built on the host in FP64.
#include <algorithm>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>

#include "common.cuh"
#include "dft.cuh"
#include "fftplan.h"
#include "fftreg.cuh"
#include "fftstage.cuh"
#include "kernels.h"

namespace ttsh {

using fftreg::scale_n3;
using namespace fftplan;

namespace {

constexpr int FFT_THREADS = fftplan::kThreads;

// The smem position of element e of line l. Lines along x (contiguous in memory) are one after
// another, elements spread by one in eight so that a step's stride-R writes use more banks; lines
// along y and z (adjacent in x) are interleaved.
template <bool XAXIS>
__device__ __forceinline__ int spos(int l, int e, int LB, int pitch) {
  return XAXIS ? l * pitch + e + (e >> 3) : e * LB + l;
}

// One line group of a pass: where its lines are.
struct Lines {
  int LB, pitch;
  size_t base, stride;  // element e of line l: base + e stride + l lstride
  size_t lstride;
  int x0, y;            // z lines: the first line's x, their y
};

// Where a step reads and writes: the first step of a pass from_w, the last one to_w.
template <class C>
struct Io {
  const C* src;
  C* dst;
  bool from_w, to_w;
};

// v[r] <- element j + r M of line l, r < R; the first step of an inverse pass conjugates, the first
// forward pass in FP32 brings both parts of the packed source to the same size (pow2_norm).
template <class T, bool XAXIS, int R, class C>
__device__ __forceinline__ void load(C* v, const InstDev<T>& I, int pass, const Lines& L, const Io<C>& io, int l, int j, int M) {
  if (io.from_w) {
    const C* p = I.W + L.base + (size_t)l * L.lstride + (size_t)j * L.stride;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = p[(size_t)(r * M) * L.stride];
    if (pass >= 3) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r].y = -v[r].y;
    }
    if constexpr (sizeof(T) == 4) {
      if (pass == 0 && I.wmax) {
        const T su = pow2_norm(I.wmax[0]), sp = pow2_norm(I.wmax[1]);
#pragma unroll
        for (int r = 0; r < R; ++r) { v[r].x *= su; v[r].y *= sp; }
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = io.src[spos<XAXIS>(l, j + r * M, L.LB, L.pitch)];
  }
}
// element e of line l <- o; the last step of a pass with an inverse transform conjugates
template <class T, bool XAXIS, class C>
__device__ __forceinline__ void store(C o, const InstDev<T>& I, int pass, const Lines& L, const Io<C>& io, int l, int e) {
  if (io.to_w) {
    if (pass >= 2) o.y = -o.y;
    if (pass == 4) o = scale_n3(o, I);
    I.W[L.base + (size_t)l * L.lstride + (size_t)e * L.stride] = o;
  } else {
    io.dst[spos<XAXIS>(l, e, L.LB, L.pitch)] = o;
  }
}

// FP64: one step of radix R. turn: the last forward step of pass 2, which goes on with the divide and
// the first inverse step.
template <bool XAXIS, int R>
__device__ __forceinline__ void fft_step(const InstDev<double>& I, int pass, const Lines& L, const Io<double2>& io, int Ns, bool turn) {
  const int N = I.N, M = N / R, total = L.LB * M, ts = N / (Ns * R);
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    int l, j;
    if (XAXIS) { l = b / M; j = b - l * M; } else { j = b / L.LB; l = b - j * L.LB; }
    double2 v[R];
    load<double, XAXIS, R>(v, I, pass, L, io, l, j, M);
    const int k = j % Ns;
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = dft::mul(v[r], __ldg(I.tw + r * k * ts));
    }
    dft::Dft<R>::run(v);
    int e0 = (j / Ns) * Ns * R + k, de = Ns;
    if (!XAXIS && turn) {
      // v[r] is the spectrum at z = j + r M: divide, and the inverse transform's first step
      const fftreg::Poisson<double> pm(I, L.x0 + l, L.y);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = dft::conj(pm(v[r], I, j + r * M));
      dft::Dft<R>::run(v);
      e0 = j * R;
      de = 1;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) store<double, XAXIS>(v[r], I, pass, L, io, l, e0 + r * de);
  }
}

// FP32: the plan's stages R1 and (R2 > 1) R2 in one step. With P = N / (R1 R2), the thread of base j
// holds the elements j + (r R2 + q) P: for each q the inputs (over r) of stage R1's butterfly j + q P,
// whose outputs r are, for each r, the inputs (over q) of the stage-R2 butterfly (j / Ns) Ns R1 + k + r Ns.
// divide: the last forward step of pass 2.
template <bool XAXIS, bool INV, int R1, int R2>
__device__ __forceinline__ void fft_step(const InstDev<float>& I, int pass, const Lines& L, const Io<float2>& io, int Ns, bool divide) {
  constexpr int R = R1 * R2;
  const int N = I.N, P = N / R, total = L.LB * P;
  for (int b = threadIdx.x; b < total; b += blockDim.x) {
    int l, j;
    if (XAXIS) { l = b / P; j = b - l * P; } else { j = b / L.LB; l = b - j * L.LB; }
    float2 v[R];
    load<float, XAXIS, R>(v, I, pass, L, io, l, j, P);
    const int k = j % Ns, e0 = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int q = 0; q < R2; ++q) {
      float2 u[R1];
#pragma unroll
      for (int r = 0; r < R1; ++r) u[r] = v[r * R2 + q];
      plan_butterfly<INV, R1>(u, I.tw, N, k, N / (Ns * R1));
#pragma unroll
      for (int r = 0; r < R1; ++r) v[r * R2 + q] = u[r];
    }
    if constexpr (R2 > 1) {
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        float2 u[R2];
#pragma unroll
        for (int q = 0; q < R2; ++q) u[q] = v[r * R2 + q];
        plan_butterfly<INV, R2>(u, I.tw, N, k + r * Ns, N / (Ns * R));
#pragma unroll
        for (int q = 0; q < R2; ++q) v[r * R2 + q] = u[q];
      }
    }
    // v[r R2 + q] is element e0 + (r + q R1) Ns
    if (!XAXIS && !INV && divide) {
      const fftreg::Poisson<float> pm(I, L.x0 + l, L.y);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = dft::conj(pm(v[r], I, e0 + (r / R2 + r % R2 * R1) * Ns));
    }
#pragma unroll
    for (int r = 0; r < R; ++r) store<float, XAXIS>(v[r], I, pass, L, io, l, e0 + (r / R2 + r % R2 * R1) * Ns);
  }
}

// The steps InstDev::step holds: FP64 the radix, FP32 R1 + 8 R2 of a stage pair (R2 = 1: one stage).
constexpr int pair_code(int r1, int r2) { return r1 + 8 * r2; }
template <bool XAXIS>
__device__ __forceinline__ void run_step(int s, const InstDev<double>& I, int pass, const Lines& L, const Io<double2>& io, int Ns, bool turn,
                                         bool) {
  switch (s) {
#define X(R) case R: fft_step<XAXIS, R>(I, pass, L, io, Ns, turn); break;
    X(2) X(3) X(4) X(5) X(6) X(8) X(9) X(10) X(12) X(15) X(16)
#undef X
    default: break;
  }
}
template <bool XAXIS>
__device__ __forceinline__ void run_step(int s, const InstDev<float>& I, int pass, const Lines& L, const Io<float2>& io, int Ns, bool divide,
                                         bool inv) {
  if (inv) {
    switch (s) {
#define X(R1, R2) case pair_code(R1, R2): fft_step<XAXIS, true, R1, R2>(I, pass, L, io, Ns, false); break;
      TTSH_STAGE_PAIRS(X)
#undef X
      default: break;
    }
  } else {
    switch (s) {
#define X(R1, R2) case pair_code(R1, R2): fft_step<XAXIS, false, R1, R2>(I, pass, L, io, Ns, divide); break;
      TTSH_STAGE_PAIRS(X)
#undef X
      default: break;
    }
  }
}
template <class T>
__device__ __forceinline__ int step_radix(int s) { return sizeof(T) == 8 ? s : (s & 7) * (s >> 3); }
// Line group g of a pass. buf: two buffers of `half` values (the second unused by two steps or fewer).
template <class T, bool XAXIS>
__device__ __forceinline__ void fft_group(const InstDev<T>& I, int pass, int g, int LB, typename CxT<T>::type* buf, int half) {
  typedef typename CxT<T>::type C;
  const int N = I.N;
  const size_t NN = (size_t)N * N;
  Lines L;
  L.LB = LB;
  L.pitch = x_pitch(N);
  L.x0 = L.y = 0;
  if (XAXIS) {
    L.base = (size_t)g * LB * N;
    L.stride = 1;
    L.lstride = N;
  } else {
    const int ng = N / LB, outer = g / ng;
    L.x0 = (g - outer * ng) * LB;
    L.lstride = 1;
    if (pass == 2) { L.base = (size_t)outer * N + L.x0; L.stride = NN; L.y = outer; }
    else { L.base = (size_t)outer * NN + L.x0; L.stride = N; }
  }
  const int n = I.nsteps, nops = pass_steps<T>(n, pass);
  C *src = buf + half, *dst = buf;
  int Ns = 1;
  for (int q = 0; q < nops; ++q) {
    const int s = I.step[q < n ? q : (sizeof(T) == 8 ? 2 * n - 2 - q : q - n)];
    if (q == n) Ns = sizeof(T) == 8 ? step_radix<T>(I.step[n - 1]) : 1;
    const bool last = q == nops - 1;
    run_step<XAXIS>(s, I, pass, L, Io<C>{src, dst, q == 0, last}, Ns, pass == 2 && q == n - 1, pass >= 3 || q >= n);
    Ns *= step_radix<T>(s);
    if (!last) __syncthreads();
    C* t = src;
    src = dst;
    dst = t;
  }
}

// One pass: XAXIS passes 0 and 4, else 1, 2, 3.
template <class T, bool XAXIS>
__global__ void __launch_bounds__(FFT_THREADS, fft_min_ctas<T>()) k_fft(const InstDev<T>* __restrict__ insts, int pass, int LB,
                                                                         int half) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  fft_group<T, XAXIS>(insts[blockIdx.y], pass, blockIdx.x, LB, reinterpret_cast<typename CxT<T>::type*>(smem_raw), half);
}

// FP32, a grid of few CTAs (in_smem): a line group is copied to shared memory, each stage of the plan goes from
// one buffer to the other, and the result is copied back. A step of fft_group has a thread for every two
// stages, 20 values at N = 20, and the code of 13 stage pairs is fetched from cold caches; here every stage has a
// thread for each of its butterflies. The same stages in the same order, so the same bits.
template <int R, bool INV>
__device__ __forceinline__ void smem_stage(const float2* src, float2* dst, int N, int LB, int Ns, const float2* tw) {
  const int M = N / R, pitch = N + 1, ts = N / (Ns * R);
  for (int b = threadIdx.x; b < LB * M; b += blockDim.x) {
    const int l = b / M, j = b - l * M, k = j % Ns;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[l * pitch + j + r * M];
    plan_butterfly<INV, R>(v, tw, N, k, ts);
    float2* d = dst + l * pitch + (j / Ns) * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) d[r * Ns] = v[r];
  }
}
template <bool INV>
__device__ __forceinline__ void smem_fft(float2*& a, float2*& b, const InstDev<float>& I, int LB) {
  int Ns = 1;
  for (int s = 0; s < I.nstages; ++s) {
    const int R = I.radix[s];
    if (R == 4) smem_stage<4, INV>(a, b, I.N, LB, Ns, I.tw);
    else if (R == 2) smem_stage<2, INV>(a, b, I.N, LB, Ns, I.tw);
    else if (R == 3) smem_stage<3, INV>(a, b, I.N, LB, Ns, I.tw);
    else smem_stage<5, INV>(a, b, I.N, LB, Ns, I.tw);
    __syncthreads();
    float2* t = a;
    a = b;
    b = t;
    Ns *= R;
  }
}
template <int PASS>
__global__ void __launch_bounds__(FFT_THREADS) k_fft_smem(const InstDev<float>* __restrict__ insts, int LB) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool XAXIS = PASS == 0 || PASS == 4;
  const InstDev<float>& I = insts[blockIdx.y];
  const int N = I.N, NN = N * N, pitch = N + 1;
  float2 *a = reinterpret_cast<float2*>(smem_raw), *b = a + LB * pitch;
  // this group's lines: x rows one after another, or y or z lines adjacent in x
  const int ng = N / LB, outer = XAXIS ? 0 : blockIdx.x / ng, x0 = XAXIS ? 0 : (blockIdx.x - outer * ng) * LB;
  float2* const w = I.W + (XAXIS ? blockIdx.x * LB * N : (PASS == 2 ? outer * N : outer * NN) + x0);
  const int stride = PASS == 2 ? NN : N;
  // the forward passes, first: both parts of the packed source brought to the same size (pow2_norm)
  const float su = PASS == 0 && I.wmax ? pow2_norm(I.wmax[0]) : 1.f, sp = PASS == 0 && I.wmax ? pow2_norm(I.wmax[1]) : 1.f;
  for (int t = threadIdx.x; t < LB * N; t += blockDim.x) {
    const int e = XAXIS ? t % N : t / LB, l = XAXIS ? t / N : t % LB;
    float2 v = w[XAXIS ? t : e * stride + l];
    if (PASS == 0) { v.x *= su; v.y *= sp; }
    if (PASS >= 3) v.y = -v.y;
    a[l * pitch + e] = v;
  }
  __syncthreads();
  smem_fft<(PASS >= 3)>(a, b, I, LB);
  if constexpr (PASS == 2) {
    for (int t = threadIdx.x; t < LB * N; t += blockDim.x) {
      const int l = t / N, e = t - l * N;
      const fftreg::Poisson<float> pm(I, x0 + l, outer);
      a[l * pitch + e] = dft::conj(pm(a[l * pitch + e], I, e));
    }
    __syncthreads();
    smem_fft<true>(a, b, I, LB);
  }
  for (int t = threadIdx.x; t < LB * N; t += blockDim.x) {
    const int e = XAXIS ? t % N : t / LB, l = XAXIS ? t / N : t % LB;
    float2 o = a[l * pitch + e];
    if (PASS >= 2) o.y = -o.y;
    if (PASS == 4) o = scale_n3(o, I);
    w[XAXIS ? t : e * stride + l] = o;
  }
}

// Both in-plane axes of a z-plane, one thread-block cluster per plane: dir 0 forward x then forward
// y, dir 1 inverse y then inverse x. As in fftreg_impl.cuh: each CTA of the cluster takes every
// clusterDim-th line group of the first axis, the cluster barrier (release / acquire) makes the
// plane's results visible to all its CTAs, then each takes every clusterDim-th of the second; the
// plane's intermediate is read back from L2.
template <class T>
__global__ void __launch_bounds__(FFT_THREADS, fft_min_ctas<T>()) k_fft_plane(const InstDev<T>* __restrict__ insts, int dir,
                                                                               int LB, int half, int parts) {
  typedef typename CxT<T>::type C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* const buf = reinterpret_cast<C*>(smem_raw);
  const InstDev<T>& I = insts[blockIdx.y];
  const int z = blockIdx.x / parts, part = blockIdx.x - z * parts, ng = I.N / LB;
  // the line groups of plane z are z ng .. z ng + ng - 1 of each axis; a barrier between groups, since
  // the next one reuses the buffers
  for (int gg = part; gg < ng; gg += parts) {
    if (dir == 0) fft_group<T, true>(I, 0, z * ng + gg, LB, buf, half);
    else fft_group<T, false>(I, 3, z * ng + gg, LB, buf, half);
    __syncthreads();
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  for (int gg = part; gg < ng; gg += parts) {
    if (dir == 0) fft_group<T, false>(I, 1, z * ng + gg, LB, buf, half);
    else fft_group<T, true>(I, 4, z * ng + gg, LB, buf, half);
    __syncthreads();
  }
}

// ---- host side -----------------------------------------------------------------------------

// The steps of a plan, as InstDev::step holds them: the best ones for N when the plan is the default
// order, else (FP64) reversed for the reverse order or consecutive factors merged.
std::vector<int> encode(const Steps& st, bool f64) {
  std::vector<int> s;
  for (int i = 0; i < st.n; ++i) s.push_back(f64 ? st.a[i] : pair_code(st.a[i], st.b[i]));
  return s;
}
Radices radices(const std::vector<int>& plan) {
  Radices p;
  for (int r : plan) p.add(r);
  return p;
}
bool is_default(int N, const std::vector<int>& plan) {
  const Radices d = default_plan(N);
  return plan == std::vector<int>(d.r, d.r + d.n);
}
std::vector<int> plan_steps(float, int, const std::vector<int>& plan) { return encode(stage_steps(radices(plan)), false); }
std::vector<int> plan_steps(double, int N, const std::vector<int>& plan) {
  std::vector<int> s = encode(default_steps<double>(N), true);
  if (is_default(N, plan)) return s;
  if (is_default(N, std::vector<int>(plan.rbegin(), plan.rend()))) return std::vector<int>(s.rbegin(), s.rend());
  s.clear();
  for (int r : plan) {
    if (!s.empty() && is_radix(s.back() * r)) s.back() *= r;
    else s.push_back(r);
  }
  return s;
}

// Shared memory of a pass over LB lines: none, one or two buffers of half_values by its steps.
int half_values(int N, int LB) { return LB * x_pitch(N); }
template <class T>
size_t smem_of(const Group<T>& g, int LB, int pass) {
  const int nops = pass_steps<T>(g.fft_nsteps > 0 ? g.fft_nsteps : 3, pass);
  return (size_t)(nops < 2 ? 0 : (nops == 2 ? 1 : 2)) * half_values(g.N, LB) * sizeof(typename CxT<T>::type);
}
constexpr size_t kFftSmem = 227 * 1024;

// Largest power-of-two LB (the explicit choices of a tuning): its two buffers fit in kFftSmem.
int pow2_lb(int N, size_t csize) {
  int lb = 16;
  while (lb > 1 && (N % lb != 0 || 2 * (size_t)lb * (N + 1) * csize > 200 * 1024)) lb >>= 1;
  return lb;
}

template <class T>
int threads_of(const Group<T>& g, int LB) { return threads_for(default_steps<T>(g.N), g.N, LB); }

inline void check_fft(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// Lines per CTA of k_fft_smem for this group, 0 where it is not used: boxes up to 64^3 whose grid of
// power-of-two line groups (the explicit choices, else the largest) has at most five CTAs per SM. FFT of a step
// (five launches), us, k_fft / this: one 8^3 37.9 / 32.6, one 20^3 60.1 / 36.3, 4 x 20^3 60.7 / 37.0, 16 x 12^3 45.6 /
// 36.1, one 32^3 48.7 / 41.0, one 48^3 55.5 / 43.0, one 64^3 60.7 / 48.0; against the rule 4 x 18^3 43.9 / 49.0; beyond it
// 4 x 64^3 81 / 87, one 72^3 55 / 71, 16 x 24^3 47 / 55, 4 x 36^3 53 / 63.
int smem_lines(const Group<float>& g) {
  const int lb = g.fft_lb ? fft_lines(g) : pow2_lb(g.N, sizeof(float2));
  return g.N <= 64 && (long)g.N * (g.N / lb) * g.n <= 5L * g.sms ? lb : 0;
}
template <class T>
bool launch_smem(const Group<T>&, int, cudaStream_t) { return false; }
template <>
bool launch_smem<float>(const Group<float>& g, int pass, cudaStream_t st) {
  const int lb = smem_lines(g);
  if (!lb) return false;
  const size_t smem = 2 * (size_t)lb * (g.N + 1) * sizeof(float2);
  const dim3 grid(g.N * (g.N / lb), g.n);
  switch (pass) {
#define X(P) case P: k_fft_smem<P><<<grid, FFT_THREADS, smem, st>>>(g.d_inst, lb); break;
    X(0) X(1) X(2) X(3) X(4)
#undef X
  }
  check_fft("fft launch");
  return true;
}

template <class T>
void launch_one(const Group<T>& g, int pass, cudaStream_t st) {
  if (launch_smem<T>(g, pass, st)) return;
  const int N = g.N, LB = fft_lines(g), half = half_values(N, LB);
  const size_t smem = smem_of(g, LB, pass);
  const dim3 grid((N / LB) * N, g.n);
  if (pass == 0 || pass == 4) k_fft<T, true><<<grid, threads_of(g, LB), smem, st>>>(g.d_inst, pass, LB, half);
  else k_fft<T, false><<<grid, threads_of(g, LB), smem, st>>>(g.d_inst, pass, LB, half);
  check_fft("fft launch");
}

}  // namespace

template <> bool fftplan_launch<float>(const Group<float>&, int, cudaStream_t);
template <> bool fftplan_launch<double>(const Group<double>&, int, cudaStream_t);
template <> void fftplan_prepare<float>(int);
template <> void fftplan_prepare<double>(int);

template <class T>
void fft_steps(int N, const std::vector<int>& plan, int* step, int* nsteps) {
  const std::vector<int> s = plan_steps(T(0), N, plan);
  *nsteps = (int)s.size();
  for (size_t k = 0; k < s.size(); ++k) step[k] = s[k];
}

// fft_kind 2: by plane at the sizes of the register kernels (which have their own lines and plan) and with the
// default lines per CTA and, in FP32, the default plan. An explicit choice goes per axis: a plane's cluster has
// at most eight CTAs, too few for the short lines of the small choices. A step, us, by plane / per axis: FP32 one
// 25^3 with one line 123 / 47, one 50^3 with two 129 / 94, 16 x 60^3 with four 952 / 881, one 20^3 with the reverse plan
// 47 / 35; FP64 one 30^3 with two lines 138 / 91; against the rule FP64 16 x 12^3 with four 0.97. In FP64 the reverse
// plan is as fast by plane (one 50^3 0.98).
template <class T>
bool fft_by_plane(const Group<T>& g) {
  return g.fft_kind == 2 && (fftreg_has<T>(g.N) || (g.fft_lb == 0 && (sizeof(T) == 8 || g.fft_default)));
}

template <class T>
void launch_fft_plane(const Group<T>& g, int dir, cudaStream_t st) {
  // the per-size kernels come first: in FP64 the small sizes of the register kernels have them too
  if (fftplan_launch<T>(g, dir == 0 ? 0 : 4, st) || fftreg_plane_launch<T>(g, dir, st)) return;
  const int N = g.N, LB = fft_lines(g), half = half_values(N, LB), ng = N / LB;
  const int parts = cluster_parts(ng);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(N * parts, g.n);
  cfg.blockDim = dim3(threads_of(g, LB));
  cfg.dynamicSmemBytes = smem_of(g, LB, 0);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = parts;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_fft_plane<T>, (const InstDev<T>*)g.d_inst, dir, LB, half, parts);
  if (e != cudaSuccess) throw std::runtime_error(std::string("fft (plane) launch: ") + cudaGetErrorString(e));
}

// The per-size kernels, in three translation units per type.
#define X(NAME, T)                                            \
  bool NAME##_launch(const Group<T>&, int, cudaStream_t);     \
  bool NAME##_prepare(int);
X(fftplan_f32_a, float) X(fftplan_f32_b, float) X(fftplan_f32_c, float)
X(fftplan_f64_a, double) X(fftplan_f64_b, double) X(fftplan_f64_c, double) X(fftplan_f64_s, double)
#undef X
template <>
bool fftplan_launch<float>(const Group<float>& g, int pass, cudaStream_t st) {
  if (g.fft_kind != 2 || g.fft_lb != 0 || !g.fft_default) return false;
  return fftplan_f32_a_launch(g, pass, st) || fftplan_f32_b_launch(g, pass, st) || fftplan_f32_c_launch(g, pass, st);
}
template <>
bool fftplan_launch<double>(const Group<double>& g, int pass, cudaStream_t st) {
  if (g.fft_kind != 2 || g.fft_lb != 0 || !g.fft_default) return false;
  return fftplan_f64_s_launch(g, pass, st) || fftplan_f64_a_launch(g, pass, st) || fftplan_f64_b_launch(g, pass, st) || fftplan_f64_c_launch(g, pass, st);
}
template <>
void fftplan_prepare<float>(int N) {
  if (!fftplan_f32_a_prepare(N) && !fftplan_f32_b_prepare(N)) fftplan_f32_c_prepare(N);
}
template <>
void fftplan_prepare<double>(int N) {
  fftplan_f64_s_prepare(N);
  if (!fftplan_f64_a_prepare(N) && !fftplan_f64_b_prepare(N)) fftplan_f64_c_prepare(N);
}

// One kernel serves every size, so its shared-memory limit is set once for all.
template <class T>
void fft_prepare(int N) {
  fftreg_prepare<T>(N);
  fftplan_prepare<T>(N);
  for (const void* f : {(const void*)k_fft<T, true>, (const void*)k_fft<T, false>, (const void*)k_fft_plane<T>}) {
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFftSmem);
    if (e != cudaSuccess) throw std::runtime_error(std::string("fft smem attribute: ") + cudaGetErrorString(e));
  }
}

template <class T>
std::vector<int> fft_lb_candidates(int N) {
  typedef typename CxT<T>::type C;
  std::vector<int> r;
  for (int lb = pow2_lb(N, sizeof(C)); lb >= 1; lb >>= 1)
    if (N % lb == 0) r.push_back(lb);
  return r;
}

template <class T>
int fft_lines(const Group<T>& g) {
  if (g.fft_lb == 0) {
    static thread_local int last_n = 0, last = 0;
    if (last_n != g.N) {
      last = default_lb<T>(g.N);
      last_n = g.N;
    }
    return last;
  }
  if (g.fft_lb < 1 || g.fft_lb > pow2_lb(g.N, sizeof(typename CxT<T>::type)) || g.N % g.fft_lb != 0)
    throw std::runtime_error("fft: bad lines per CTA");
  return g.fft_lb;
}

template <class T>
void launch_fft_pass(const Group<T>& g, int pass, cudaStream_t st) {
  if (pass < 0 || pass > 4) throw std::runtime_error("bad fft pass");
  if ((pass == 2 && fftplan_launch<T>(g, pass, st)) || fftreg_launch<T>(g, pass, st)) return;
  launch_one<T>(g, pass, st);
}

template void fft_steps<float>(int, const std::vector<int>&, int*, int*);
template void fft_steps<double>(int, const std::vector<int>&, int*, int*);
template std::vector<int> fft_lb_candidates<float>(int);
template std::vector<int> fft_lb_candidates<double>(int);
template int fft_lines<float>(const Group<float>&);
template int fft_lines<double>(const Group<double>&);
template void launch_fft_pass<float>(const Group<float>&, int, cudaStream_t);
template void launch_fft_pass<double>(const Group<double>&, int, cudaStream_t);
template bool fft_by_plane<float>(const Group<float>&);
template bool fft_by_plane<double>(const Group<double>&);
template void launch_fft_plane<float>(const Group<float>&, int, cudaStream_t);
template void launch_fft_plane<double>(const Group<double>&, int, cudaStream_t);
template void fft_prepare<float>(int);
template void fft_prepare<double>(int);

}  // namespace ttsh
