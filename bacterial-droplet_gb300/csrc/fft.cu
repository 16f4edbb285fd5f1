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
//     size (N = 100 is 10 x 10, N = 320 is 8 x 8 x 5); a radix-5 butterfly is 36 operations instead of
//     the 120 of the sum that defines it. Pass 2 multiplies by -1/k^2 and begins the inverse in the
//     registers of the forward transform's last step, whose outputs (elements j + r N/R) are the
//     inputs of a first step of the same radix.
//   FP32 (bound by latency and issue): the stages of the radix plan (4, 2, 3, 5), up to two of them
//     in registers per step: the butterflies of one stage feed those of the next within a thread, so
//     the arithmetic is the plan's, stage by stage, with half the trips through shared memory.
// Twiddles between steps come from a table exp(-2 pi i k/N) built on the host in FP64.
#include <algorithm>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>

#include "common.cuh"
#include "dft.cuh"
#include "fftreg.cuh"
#include "kernels.h"

namespace ttsh {

using fftreg::scale_n3;

namespace {

constexpr int FFT_THREADS = 256;

// a b in FP32: one product of each part is rounded, the other joins it in a fused multiply-add. INV (the
// inverse transform, run on conjugated values) fuses the other product of the imaginary part: the
// choice the compiler makes for a times a conjugated twiddle, which the results have always had.
template <bool INV>
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), INV ? fmaf(a.y, b.x, a.x * b.y) : fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

template <class T> constexpr int fft_min_ctas() { return sizeof(T) == 4 ? 3 : 2; }

// The smem position of element e of line l. Lines along x (contiguous in memory) are one after
// another, elements spread by one in eight so that a step's stride-R writes use more banks; lines
// along y and z (adjacent in x) are interleaved.
template <bool XAXIS>
__device__ __forceinline__ int spos(int l, int e, int LB, int pitch) {
  return XAXIS ? l * pitch + e + (e >> 3) : e * LB + l;
}
inline int x_pitch(int N) { return N + N / 8 + 1; }

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

// FP32: one butterfly of the radix plan, in place: the twiddles w^(r k ts) of its stage, then the DFT
// of R = 2, 4 in butterflies, of R = 3, 5 as the sum that defines it (its roots of unity from the
// table).
template <bool INV, int R>
__device__ __forceinline__ void plan_butterfly(float2* v, const float2* tw, int N, int k, int ts) {
  if (k > 0) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul<INV>(v[r], __ldg(tw + r * k * ts));
  }
  if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    const float2 dd = make_float2(d.y, -d.x);
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = cadd(b, dd);
    v[3] = csub(b, dd);
  } else {
    float2 o[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      float2 acc = v[0];
#pragma unroll
      for (int r = 1; r < R; ++r) acc = cadd(acc, cmul<INV>(v[r], __ldg(tw + ((q * r) % R) * (N / R))));
      o[q] = acc;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = o[q];
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
    const fftreg::Poisson<float> pm(I, XAXIS ? 0 : L.x0 + l, XAXIS ? 0 : L.y);
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      float2 u[R2];
#pragma unroll
      for (int q = 0; q < R2; ++q) u[q] = v[r * R2 + q];
      if constexpr (R2 > 1) plan_butterfly<INV, R2>(u, I.tw, N, k + r * Ns, N / (Ns * R));
#pragma unroll
      for (int q = 0; q < R2; ++q) {
        const int e = e0 + r * Ns + q * Ns * R1;
        if (!XAXIS && divide) u[q] = dft::conj(pm(u[q], I, e));
        store<float, XAXIS>(u[q], I, pass, L, io, l, e);
      }
    }
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
#define TTSH_STAGE_PAIRS(X) \
  X(2, 1) X(3, 1) X(4, 1) X(5, 1) X(4, 4) X(4, 2) X(4, 3) X(4, 5) X(2, 3) X(2, 5) X(3, 3) X(3, 5) X(5, 5)
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
// Steps of a pass: FP64 the divide's step is the last forward and the first inverse one, and the
// inverse goes through the steps backwards; FP32 the inverse runs the plan from its start.
template <class T>
__host__ __device__ __forceinline__ int pass_steps(int n, int pass) { return pass != 2 ? n : (sizeof(T) == 8 ? 2 * n - 1 : 2 * n); }

// Line group g of a pass. buf: two buffers of `half` values (the second unused by two steps or fewer).
template <class T, bool XAXIS>
__device__ __forceinline__ void fft_group(const InstDev<T>& I, int pass, int g, int LB, typename CxT<T>::type* buf, int half) {
  typedef typename CxT<T>::type C;
  const int N = I.N;
  const size_t NN = (size_t)N * N;
  Lines L;
  L.LB = LB;
  L.pitch = N + N / 8 + 1;
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

constexpr int kRadix[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
bool is_radix(int r) { return std::find(std::begin(kRadix), std::end(kRadix), r) != std::end(kRadix); }

// Real operations per value of a radix-R step (the DFT of dft.cuh and its twiddles).
double step_cost(int R) {
  double c = 0;
  switch (R) {
    case 2: c = 2; break;
    case 3: c = 4; break;
    case 4: c = 4; break;
    case 5: c = 7.2; break;
    case 6: c = 6; break;
    case 8: c = 6.5; break;
    case 9: c = 9.8; break;
    case 10: c = 9.2; break;
    case 12: c = 8; break;
    case 15: c = 11.2; break;
    default: c = 10; break;
  }
  return c + 4.0 * (R - 1) / R;
}

// The steps for size N: fewest first (each boundary is a trip through shared memory), then fewest
// operations; larger radices first.
void best_steps(int N, int most, std::vector<int>& cur, std::vector<int>& best, double cost, double& best_cost) {
  if (N == 1) {
    if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && cost < best_cost)) {
      best = cur;
      best_cost = cost;
    }
    return;
  }
  if (!best.empty() && cur.size() >= best.size()) return;
  for (int r : kRadix)
    if (r <= most && N % r == 0) {
      cur.push_back(r);
      best_steps(N / r, r, cur, best, cost + step_cost(r), best_cost);
      cur.pop_back();
    }
}
std::vector<int> size_steps(int N) {
  std::vector<int> cur, best;
  double c = 0;
  best_steps(N, 16, cur, best, 0, c);
  return best;
}
// The default radix plan.
std::vector<int> default_plan(int N) {
  std::vector<int> p;
  for (int r : {4, 2, 3, 5})
    while (N % r == 0) { p.push_back(r); N /= r; }
  return p;
}
bool is_pair(int r1, int r2) {
#define X(A, B) if (r1 == A && r2 == B) return true;
  TTSH_STAGE_PAIRS(X)
#undef X
  return false;
}
// The steps of a plan, as InstDev::step holds them.
std::vector<int> plan_steps(float, int, const std::vector<int>& plan) {
  std::vector<int> s;
  for (size_t k = 0; k < plan.size(); ++k) {
    if (k + 1 < plan.size() && is_pair(plan[k], plan[k + 1])) {
      s.push_back(pair_code(plan[k], plan[k + 1]));
      ++k;
    } else {
      s.push_back(pair_code(plan[k], 1));
    }
  }
  return s;
}
std::vector<int> plan_steps(double, int N, const std::vector<int>& plan) {
  std::vector<int> s = size_steps(N);
  const std::vector<int> d = default_plan(N);
  if (plan == d) return s;
  if (plan == std::vector<int>(d.rbegin(), d.rend())) return std::vector<int>(s.rbegin(), s.rend());
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

// Default lines per CTA: the divisor of N whose steps, counted in whole warps per line, cost least,
// among those that leave two CTAs' buffers on an SM (three for FP32) and whose rows along x are at
// least 64 bytes where N allows. N = 100 in FP64: 25 lines (250 radix-10 butterflies in 8 warps; 4
// lines, the largest power of two dividing 100, would fill 40 of 64 lanes).
template <class T>
int default_lb(int N) {
  constexpr size_t csize = sizeof(typename CxT<T>::type);
  const std::vector<int> st = plan_steps(T(0), N, default_plan(N));
  const size_t room = (sizeof(T) == 4 ? 227 / 3 : 227 / 2) * 1024 - 1024;
  int best = 0;
  double cost = 0;
  for (int lb = 1; lb <= std::min(N, 64); ++lb) {
    if (N % lb != 0) continue;
    if (lb > 1 && 2 * (size_t)half_values(N, lb) * csize > room) break;
    double c = 0;
    for (int s : st) {
      const int r = sizeof(T) == 8 ? s : (s & 7) * (s >> 3);
      const int warps = (lb * (N / r) + 31) / 32;
      const int rounds = (warps + FFT_THREADS / 32 - 1) / (FFT_THREADS / 32);
      // whole warps, and (a tenth of the weight) whole rounds of the CTA
      c += (sizeof(T) == 8 ? step_cost(r) : 10.0) * r * (warps + 0.1 * (rounds * (FFT_THREADS / 32) - warps));
    }
    c /= lb;
    if (lb * csize < 64) c *= 1.0 + 0.1 * (64.0 / (lb * csize) - 1);  // short rows along x
    if (!best || c < cost * 0.999) {
      best = lb;
      cost = c;
    }
  }
  return best;
}

template <class T>
int threads_of(const Group<T>& g, int LB) {
  int most = 0;
  for (int s : plan_steps(T(0), g.N, default_plan(g.N))) {
    const int r = sizeof(T) == 8 ? s : (s & 7) * (s >> 3);
    most = std::max(most, LB * (g.N / r));
  }
  return std::min(FFT_THREADS, (most + 31) / 32 * 32);
}

inline void check_fft(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

template <class T>
void launch_one(const Group<T>& g, int pass, cudaStream_t st) {
  const int N = g.N, LB = fft_lines(g), half = half_values(N, LB);
  const size_t smem = smem_of(g, LB, pass);
  const dim3 grid((N / LB) * N, g.n);
  if (pass == 0 || pass == 4) k_fft<T, true><<<grid, threads_of(g, LB), smem, st>>>(g.d_inst, pass, LB, half);
  else k_fft<T, false><<<grid, threads_of(g, LB), smem, st>>>(g.d_inst, pass, LB, half);
  check_fft("fft launch");
}

}  // namespace

template <class T>
void fft_steps(int N, const std::vector<int>& plan, int* step, int* nsteps) {
  const std::vector<int> s = plan_steps(T(0), N, plan);
  *nsteps = (int)s.size();
  for (size_t k = 0; k < s.size(); ++k) step[k] = s[k];
}

template <class T>
void launch_fft_plane(const Group<T>& g, int dir, cudaStream_t st) {
  if (fftreg_plane_launch<T>(g, dir, st)) return;
  const int N = g.N, LB = fft_lines(g), half = half_values(N, LB), ng = N / LB;
  int parts = 8;  // the cluster (8 CTAs at most is portable) splits a plane's line groups evenly
  while (ng % parts != 0) --parts;
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

// One kernel serves every size, so its shared-memory limit is set once for all.
template <class T>
void fft_prepare(int N) {
  fftreg_prepare<T>(N);
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
  if (fftreg_launch<T>(g, pass, st)) return;
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
template void launch_fft_plane<float>(const Group<float>&, int, cudaStream_t);
template void launch_fft_plane<double>(const Group<double>&, int, cudaStream_t);
template void fft_prepare<float>(int);
template void fft_prepare<double>(int);

}  // namespace ttsh
