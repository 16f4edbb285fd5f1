// plain.cu — the FP32 plain form of the TTSH3D step: one thread per lattice site, the
// reference's stencils evaluated in its arithmetic order, global intermediates (sizes that are no
// multiple of 32, and cross-checks). plain64.cu is the FP64 form; the fused FP32 kernels in fused.cu
// replace stage1/stage2/div for speed. The diagnostics serve every form.
//
//   stage1  <- getTempVari_1 + getTempVari_2 (TTSH3D.cu:537-605): mu_0, mu_b, sigma_ab
//   stage2  <- getDtF + getVStar + phi update of getVNew (:608-632, :471-491, :515)
//   div     <- getStream mode 0 for both fields (:664-670), packed as one complex field
//   correct <- getVNew (:494-516), pressures read from the packed complex field
//   stats   <- new FP64 diagnostics (mass, max |div u|, non-finite watchdog)
#include <algorithm>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>

#include "common.cuh"
#include "kernels.h"

namespace ttsh {

namespace {

constexpr int BX = 32, BY = 8;

inline void check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    char buf[256];
    snprintf(buf, sizeof(buf), "%s launch failed: %s", what, cudaGetErrorString(e));
    throw std::runtime_error(buf);
  }
}

// ---- staged planes ---------------------------------------------------------------------------
// The kernels evaluate the reference's stencils in its arithmetic order, one thread per site of a
// 32 x 8 column tile, and march along z: the planes z-1, z, z+1 of every field a kernel's stencils
// read (tile + 1) lie in a ring of planes in shared memory, into which the next ones are copied
// (cp.async) meanwhile. With each neighbour read from global memory instead, a site of k_stage2
// loaded some 600 values through L1, each with its own 64-bit address: 4 x 100^3, us per launch,
// k_stage1 144 -> 126, k_stage2 1178 -> 519, k_div 311 -> 114, k_correct 125 -> 81. They are now bound by
// shared-memory reads (79 - 91 % of the pipe). All of a site's arithmetic follows one barrier, so that
// it stays one expression with the roundings it has always had.
constexpr int SX = BX + 2, SYR = BY + 2, SPL = SX * SYR, NT = BX * BY;

// NF fields of elements E (float; float2: an interleaved complex field), RING slots.
template <class E, int NF, int RING>
struct Planes {
  E* sm;               // [RING][NF][SPL]
  int N, NN, z0, tid;
  int go[2];           // this thread's staged points (two at most): offset within a plane, or -1
  bool out[2];         // ... beyond the boundary in x or y
  int lx, ly, x, y;

  static constexpr size_t bytes() { return (size_t)RING * NF * SPL * sizeof(E); }
  __device__ __forceinline__ Planes(unsigned char* m, int N_, int z0_) : sm(reinterpret_cast<E*>(m)), N(N_), NN(N_ * N_), z0(z0_) {
    tid = threadIdx.x;
    lx = tid & 31;
    ly = tid >> 5;
    const int x0 = blockIdx.x * BX, y0 = blockIdx.y * BY;
    x = x0 + lx;
    y = y0 + ly;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = tid + k * NT, r = i / SX, gx = x0 - 1 + i - r * SX, gy = y0 - 1 + r;
      // a partial tile's points beyond its halo wrap too (small boxes more than once); they are not used
      go[k] = i < SPL ? wrapi(gy, N) % N * N + wrapi(gx, N) % N : -1;
      out[k] = gx < 0 || gx >= N || gy < 0 || gy >= N;
    }
  }
  __device__ __forceinline__ bool on() const { return x < N && y < N; }
  __device__ __forceinline__ int slot(int z) const { return (z - z0 + 1) % RING; }
  // copies plane z; src(f, beyond) is the array field f's values come from, `beyond` where the point lies
  // beyond the boundary
  template <class F>
  __device__ __forceinline__ void stage(int z, F&& src, bool any) const {
    const size_t zo = (size_t)wrapi(z, N) * NN;
    const bool zw = z < 0 || z >= N;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (go[k] < 0 || !any) continue;
      E* d = sm + (size_t)slot(z) * NF * SPL + tid + k * NT;
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const E* g = src(f, zw || out[k]) + zo + go[k];
        const unsigned a = (unsigned)__cvta_generic_to_shared(d + f * SPL);
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(a), "l"(g), "n"(sizeof(E)) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  // body(z) for the planes z0 .. z1 - 1, each after its neighbours have arrived
  template <class F, class G>
  __device__ __forceinline__ void march(int z1, F&& src, G&& body) const {
#pragma unroll 1
    for (int z = z0 - 1; z < z0 + RING - 2; ++z) stage(z <= z1 ? z : z1, src, z <= z1);
    for (int z = z0; z < z1; ++z) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(RING - 4) : "memory");  // planes up to z + 1
      __syncthreads();  // the planes of every thread; and plane z - 2 has been read
      stage(z + RING - 2, src, z + RING - 2 <= z1);
      if (on()) body(z);
    }
  }
  // this thread's site in field 0 of plane z
  __device__ __forceinline__ const E* at(int z) const { return sm + (size_t)slot(z) * NF * SPL + (ly + 1) * SX + lx + 1; }
};

// Accessors of staged fields for st_dx .. st_lap: p[1 + dz] is the site in the planes z-1, z, z+1; or
// the 27 values in registers.
struct AccS {
  const float* p[3];
  __device__ __forceinline__ float operator()(int dx, int dy, int dz) const { return p[dz + 1][dy * SX + dx]; }
};
struct AccV {
  float v[27];
  __device__ __forceinline__ float operator()(int dx, int dy, int dz) const { return v[(dz + 1) * 9 + (dy + 1) * 3 + dx + 1]; }
};
// the pointwise product phi * Pa * Pb (build-defined active stress)
struct AccProd {
  AccS phi, pa, pb;
  __device__ __forceinline__ float operator()(int dx, int dy, int dz) const { return phi(dx, dy, dz) * pa(dx, dy, dz) * pb(dx, dy, dz); }
};
template <int NF, int RING>
__device__ __forceinline__ AccS field(const Planes<float, NF, RING>& P, int z, int f) {
  return AccS{{P.at(z - 1) + f * SPL, P.at(z) + f * SPL, P.at(z + 1) + f * SPL}};
}

typedef InstDev<float> Inst;
typedef float T;

__global__ void __launch_bounds__(NT, 4) k_stage1(const Inst* __restrict__ insts, int par, int nchunk, int zc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / nchunk];
  // this step's maxima of the Poisson source start from zero (k_div records them)
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)
    for (int i = threadIdx.x; i < 2 * (int)(gridDim.z / nchunk); i += blockDim.x) insts[i >> 1].wmax[i & 1] = 0;
  const int z0 = (blockIdx.z % nchunk) * zc;
  const Planes<float, 4, 7> S(smem_raw, N, z0);
  const Phys<T>& p = I.ph;
  auto src = [&](int f, bool) -> const float* { return f == 0 ? I.phi[par] : I.P[f - 1]; };
  S.march(min(z0 + zc, N), src, [&](int z) {
    const int i = z * S.NN + S.y * N + S.x;
    const AccS phi = field(S, z, 0);
    const T ph = phi(0, 0, 0);
    // mu_0 (TTSH3D.cu:567)
    const T mu0 = p.aPhi2 * (ph - 3 * ph * ph + 2 * ph * ph * ph) - p.kPhi * st_lap<T>(phi, p);
    T mu[3], sig[9];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const AccS F = field(S, z, b + 1);
      // mu_b (:571-573)
      mu[b] = ph * F(0, 0, 0) + p.La2 * st_lap<T>(F, p);
      // sigma_ab = phi * D_a P_b (:587-595; the 1/28 term is an integer-division zero)
      sig[0 * 3 + b] = ph * st_dx<T>(F, p.c2h);
      sig[1 * 3 + b] = ph * st_dy<T>(F, p.c2h);
      sig[2 * 3 + b] = ph * st_dz<T>(F, p.c2h);
    }
    // the stores after the last stencil: a store may alias the staged values, which are then read again
    I.mu0[i] = mu0;
#pragma unroll
    for (int b = 0; b < 3; ++b) I.mu[b][i] = mu[b];
#pragma unroll
    for (int b = 0; b < 9; ++b) I.sig[b][i] = sig[b];
  });
}

// fields: phi, P (1 + b), u (4 + b), mu_0 (7), mu_b (8 + b), sigma_ab (11 + 3 a + b)
__global__ void __launch_bounds__(NT, 2) k_stage2(const Inst* __restrict__ insts, int par, int nchunk, int zc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / nchunk];
  const int z0 = (blockIdx.z % nchunk) * zc;
  const Planes<float, 20, 4> S(smem_raw, N, z0);
  const Phys<T>& p = I.ph;
  auto src = [&](int f, bool) -> const float* {
    return f == 0 ? I.phi[par] : (f < 4 ? I.P[f - 1] : (f < 7 ? I.U[f - 4] : (f == 7 ? I.mu0 : (f < 11 ? I.mu[f - 8] : I.sig[f - 11]))));
  };
  S.march(min(z0 + zc, N), src, [&](int z) {
    const int i = z * S.NN + S.y * N + S.x;
    auto F = [&](int f) { return field(S, z, f); };
    const AccS Fphi = F(0);
    const T dphi[3] = {st_dx<T>(Fphi, p.c2h), st_dy<T>(Fphi, p.c2h), st_dz<T>(Fphi, p.c2h)};
    const T vx = F(4)(0, 0, 0), vy = F(5)(0, 0, 0), vz = F(6)(0, 0, 0);
    const T px = F(1)(0, 0, 0), py = F(2)(0, 0, 0), pz = F(3)(0, 0, 0), ph = Fphi(0, 0, 0);
    const T P2 = px * px + py * py + pz * pz;
    const T dPhi2 = dphi[0] * dphi[0] + dphi[1] * dphi[1] + dphi[2] * dphi[2];
    const T mu0 = F(7)(0, 0, 0);
    T us[3], ps[3];
    // getDtF, velocity (TTSH3D.cu:617-621) and getVStar (:480-482)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const AccS Fv = F(4 + b);
      T r = -vx * st_dx<T>(Fv, p.c2h) - vy * st_dy<T>(Fv, p.c2h) - vz * st_dz<T>(Fv, p.c2h) + p.mu * st_lap<T>(Fv, p) +
            mu0 * dphi[b] +
            p.cA * (st_dx<T>(F(11 + b), p.c2h) + st_dy<T>(F(14 + b), p.c2h) + st_dz<T>(F(17 + b), p.c2h));
      if (p.zeta != T(0)) {
        r = r - p.zeta * (st_dx<T>(AccProd{Fphi, F(1), F(1 + b)}, p.c2h) + st_dy<T>(AccProd{Fphi, F(2), F(1 + b)}, p.c2h) +
                          st_dz<T>(AccProd{Fphi, F(3), F(1 + b)}, p.c2h));
      }
      const T u = b == 0 ? vx : (b == 1 ? vy : vz);
      us[b] = u + p.dt * r;
    }
    // getDtF, polarisation (:623-629) and getVStar (:486-488)
    const T pb[3] = {px, py, pz};
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const AccS Fp = F(1 + b);
      const T dxp = st_dx<T>(Fp, p.c2h), dyp = st_dy<T>(Fp, p.c2h), dzp = st_dz<T>(Fp, p.c2h);
      T cub;
      if (b == 0) cub = px * px * px + px * py * py + px * pz * pz;
      else if (b == 1) cub = px * py * px + py * py * py + py * pz * pz;
      else cub = px * pz * px + py * pz * py + pz * pz * pz;
      const T Ab = dphi[0] * dphi[b] * px + dphi[1] * dphi[b] * py + dphi[2] * dphi[b] * pz;
      // OP_b + kappa*phi*DP_b are integer-division zeros in the reference (:579-585).
      const T r = -vx * dxp - vy * dyp - vz * dzp - p.alpha * ph * pb[b] - p.beta * P2 * pb[b] +
                  p.eta * st_lap<T>(F(8 + b), p) - p.lambda0 * (px * dxp + py * dyp + pz * dzp) -
                  p.A * (dPhi2 * cub + sqrt(P2) * Ab);
      ps[b] = pb[b] + p.dt * r;
    }
    // dtphi (:631) and the phi update of getVNew (:515)
    const T dtphi = -vx * dphi[0] - vy * dphi[1] - vz * dphi[2] + p.gamma * (st_lap<T>(F(7), p));
    I.phi[par ^ 1][i] = ph + p.dt * dtphi;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      I.Us[par ^ 1][b][i] = us[b];
      I.Ps[par ^ 1][b][i] = ps[b];
    }
  });
}

// fields: u*_a (a), P*_a (3 + a); beyond the boundary the previous step's (quirk Q2 of the reference:
// the halo of u*, P* is refreshed at the start of getRHS, TTSH3D.cu:369-371 and :405-407, before
// getVStar rewrites the interior, :471-491)
__global__ void __launch_bounds__(NT, 4) k_div(const Inst* __restrict__ insts, int par, int nchunk, int zc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / nchunk];
  const int z0 = (blockIdx.z % nchunk) * zc;
  const Planes<float, 6, 6> S(smem_raw, N, z0);
  const Phys<T>& p = I.ph;
  const bool stale = I.stale;
  auto src = [&](int f, bool beyond) -> const float* {
    const int q = stale && beyond ? par : par ^ 1;
    return f < 3 ? I.Us[q][f] : I.Ps[q][f - 3];
  };
  T mx = 0, my = 0;
  S.march(min(z0 + zc, N), src, [&](int z) {
    T d[2];
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const T a = st_dx<T>(field(S, z, 3 * f), p.c2h);
      const T b = st_dy<T>(field(S, z, 3 * f + 1), p.c2h);
      const T c = st_dz<T>(field(S, z, 3 * f + 2), p.c2h);
      d[f] = (a + b + c) * p.inv_dt;  // getStream mode 0 (:666-668)
    }
    I.W[z * S.NN + S.y * N + S.x] = make_float2(d[0], d[1]);
    mx = fmaxf(mx, fabsf(d[0]));
    my = fmaxf(my, fabsf(d[1]));
  });
  record_wmax(I.wmax, mx, my);
}

__global__ void __launch_bounds__(NT, 5) k_correct(const Inst* __restrict__ insts, int par, int nchunk, int zc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / nchunk];
  const int z0 = (blockIdx.z % nchunk) * zc;
  const Planes<float2, 1, 8> S(smem_raw, N, z0);
  const Phys<T>& p = I.ph;
  // the pressures come out of the FFT scaled by powers of two (pow2_norm); undo it exactly
  const T du = pow2_denorm(I.wmax[0]), dp = pow2_denorm(I.wmax[1]);
  auto src = [&](int, bool) -> const float2* { return I.W; };
  S.march(min(z0 + zc, N), src, [&](int z) {
    const int i = z * S.NN + S.y * N + S.x;
    // both pressures of a neighbour by one 8-byte load
    AccV Fv, Fp;
#pragma unroll
    for (int k = 0; k < 27; ++k) {
      const float2 w = S.at(z - 1 + k / 9)[(k / 3 % 3 - 1) * SX + k % 3 - 1];
      Fv.v[k] = w.x;
      Fp.v[k] = w.y;
    }
    // getVNew (TTSH3D.cu:505-511)
    const T u[3] = {I.Us[par ^ 1][0][i] - p.dt * (st_dx<T>(Fv, p.c2h) * du), I.Us[par ^ 1][1][i] - p.dt * (st_dy<T>(Fv, p.c2h) * du),
                    I.Us[par ^ 1][2][i] - p.dt * (st_dz<T>(Fv, p.c2h) * du)};
    const T P[3] = {I.Ps[par ^ 1][0][i] - p.dt * (st_dx<T>(Fp, p.c2h) * dp), I.Ps[par ^ 1][1][i] - p.dt * (st_dy<T>(Fp, p.c2h) * dp),
                    I.Ps[par ^ 1][2][i] - p.dt * (st_dz<T>(Fp, p.c2h) * dp)};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      I.U[k][i] = u[k];
      I.P[k][i] = P[k];
    }
  });
}

// Planes per CTA: 16 (three planes beyond them are staged), halved while the grid has fewer than
// four CTAs per SM.
template <class K>
void launch_planes(K kernel, size_t smem, const Group<float>& g, int par, cudaStream_t st, const char* what) {
  if ((long)g.N * g.n > 65535) throw std::runtime_error("too many instances of this size in one group");
  const int nx = (g.N + BX - 1) / BX, ny = (g.N + BY - 1) / BY;
  int zc = std::min(16, g.N);
  while (zc > 1 && (long)nx * ny * g.n * ((g.N + zc - 1) / zc) < 4 * g.sms) zc /= 2;
  const int nchunk = (g.N + zc - 1) / zc;
  kernel<<<dim3(nx, ny, nchunk * g.n), NT, smem, st>>>(g.d_inst, par, nchunk, zc);
  check_launch(what);
}

constexpr int STATS_THREADS = 256;

// Diagnostics of the current state (phi[par], u, P): per block, sum(phi), max |D.u|, max |u|, and
// a non-finite count; the sum is combined across threads and blocks in FP64 in a fixed order. FP64 fields
// are summed in FP64. FP32 fields are summed by each thread in FP32 with Kahan's compensated
// summation (error of order one rounding of the thread's partial, instead of one per term) and
// only the per-thread partials are combined in FP64: the GPU's FP64 rate is a small fraction of
// its FP32 rate, and an FP64 add per site would cost more than the step's stencils for a mass
// read-back after every step. The maxima are exact in either precision.
template <class V>
struct MassAcc;
template <>
struct MassAcc<double> {
  double s = 0;
  __device__ __forceinline__ void add(double v) { s += v; }
  __device__ __forceinline__ double total() const { return s; }
};
template <>
struct MassAcc<float> {
  float s = 0.f, c = 0.f;  // Kahan: c carries the low part lost by the last addition
  __device__ __forceinline__ void add(float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double total() const { return (double)s - (double)c; }
};

// Block reduction of the four per-thread diagnostics (fixed order) into the block's partials.
template <class T>
__device__ __forceinline__ void stats_finish(const InstDev<T>& I, double sum, double mdiv, double mu, double bad) {
  __shared__ double sh[4][STATS_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_down_sync(0xffffffffu, sum, o);
    mdiv = fmax(mdiv, __shfl_down_sync(0xffffffffu, mdiv, o));
    mu = fmax(mu, __shfl_down_sync(0xffffffffu, mu, o));
    bad += __shfl_down_sync(0xffffffffu, bad, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sh[0][w] = sum; sh[1][w] = mdiv; sh[2][w] = mu; sh[3][w] = bad; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, b = 0, c = 0, e = 0;
    for (int k = 0; k < STATS_THREADS / 32; ++k) {
      a += sh[0][k]; b = fmax(b, sh[1][k]); c = fmax(c, sh[2][k]); e += sh[3][k];
    }
    double* out = I.red + 4 * blockIdx.x;
    out[0] = a; out[1] = b; out[2] = c; out[3] = e;
  }
}

// 16-byte vectors of T (the mass pass reads phi with them).
template <class T> struct Vec16;
template <> struct Vec16<float> { typedef float4 type; };
template <> struct Vec16<double> { typedef double2 type; };

// Sum of phi over this thread's share of the sites (fixed order) and the count of non-finite
// values: 16-byte loads, four in flight per thread, and one compensated accumulator per vector
// lane, so that the pass streams phi at HBM speed (one 4-byte load per thread in flight had kept
// it at a few hundred GB/s). Both diagnostics modes take the mass from here, so they agree.
template <class T>
__device__ __forceinline__ double mass_pass(const T* __restrict__ phi, long n, int& badn) {
  typedef typename Vec16<T>::type V;
  constexpr int W = (int)(sizeof(V) / sizeof(T));
  const long nv = n / W, stride = (long)gridDim.x * blockDim.x;
  const V* __restrict__ pv = reinterpret_cast<const V*>(phi);
  MassAcc<T> lane[W];
  auto take = [&](const V& v) {
    const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
    for (int c = 0; c < W; ++c) {
      lane[c].add(e[c]);
      badn += isfinite(e[c]) ? 0 : 1;
    }
  };
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < nv; i += 4 * stride) {
    V v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = pv[i + u * stride];
#pragma unroll
    for (int u = 0; u < 4; ++u) take(v[u]);
  }
  for (; i < nv; i += stride) take(pv[i]);
  for (long j = nv * W + (long)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride) {
    lane[0].add(phi[j]);
    badn += isfinite(phi[j]) ? 0 : 1;
  }
  double tot = 0;
#pragma unroll
  for (int c = 0; c < W; ++c) tot += lane[c].total();
  return tot;
}

// The mass and the non-finite count of phi; the maxima start from zero.
template <class T>
__global__ void __launch_bounds__(STATS_THREADS) k_stats_mass(const InstDev<T>* __restrict__ insts, int par) {
  const InstDev<T>& I = insts[blockIdx.y];
  const int N = I.N;
  int badn = 0;
  const double mass = mass_pass<T>(I.phi[par], (long)N * N * N, badn);
  stats_finish<T>(I, mass, 0.0, 0.0, (double)badn);
}

// FP32: all diagnostics of a few small droplets in one launch, each thread's share of the mass as in
// k_stats_mass and then its sites, with the neighbours from global memory: the expressions and bits of
// k_stats_u, whose launch costs more there than its staged planes save (launch_stats).
__global__ void __launch_bounds__(STATS_THREADS) k_stats_small(const InstDev<float>* __restrict__ insts, int par) {
  const InstDev<float>& I = insts[blockIdx.y];
  const int N = I.N, n = N * N * N;
  int bad = 0;
  const double mass = mass_pass<float>(I.phi[par], n, bad);
  const float c2h = I.ph.c2h;
  float mdiv = 0.f, mu = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    Site s;
    s.init(i % N, i / N % N, i / (N * N), N);
    const float d = st_dx<float>(s.acc<float>(I.U[0]), c2h) + st_dy<float>(s.acc<float>(I.U[1]), c2h) + st_dz<float>(s.acc<float>(I.U[2]), c2h);
    mdiv = fmax(mdiv, fabs(d));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float u = I.U[a][i], q = I.P[a][i];
      mu = fmax(mu, fabs(u));
      if (!isfinite(u) || !isfinite(q)) bad += 1;
    }
  }
  stats_finish<float>(I, mass, (double)mdiv, (double)mu, (double)bad);
}

// FP32: max |D.u|, max |u| and the non-finite values of u and P, added to the partials of
// k_stats_mass (maxima and counts do not depend on the order). A CTA sweeps a 32 x 8 column tile over
// zc planes; the three components' planes (tile + 1) go through a ring of three in shared memory, so
// that each value is read once from global memory per tile instead of up to 27 times, with no
// integer divisions per site: 160^3 with the mass 272 -> 76 us, 2 x 256^3 1106 -> 416 us.
__global__ void __launch_bounds__(BX* BY) k_stats_u(const InstDev<float>* __restrict__ insts, int nchunk, int zc) {
  __shared__ float ring[3][3][SPL];
  const InstDev<float>& I = insts[blockIdx.z / nchunk];
  const int N = I.N, NN = N * N, tid = threadIdx.x;
  const int z0 = (blockIdx.z % nchunk) * zc, z1 = min(z0 + zc, N);
  const int x0 = blockIdx.x * BX, y0 = blockIdx.y * BY, lx = tid & 31, ly = tid >> 5;
  const bool on = x0 + lx < N && y0 + ly < N;
  // this thread's staged points (two at most): offset within a plane; a partial tile's wrap too
  int go[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int i = tid + k * BX * BY, r = i / SX;
    go[k] = i < SPL ? wrapi(y0 - 1 + r, N) % N * N + wrapi(x0 - 1 + i - r * SX, N) % N : -1;
  }
  // plane z's staged values are loaded a plane ahead of their use, into registers
  float v[2][3];
  auto load = [&](int z) {
    const size_t zo = (size_t)wrapi(z, N) * NN;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (go[k] >= 0) v[k][a] = __ldg(I.U[a] + zo + go[k]);
  };
  auto put = [&](int z) {
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (go[k] >= 0) ring[(z + 3) % 3][a][tid + k * BX * BY] = v[k][a];
  };
  load(z0 - 1);
  put(z0 - 1);
  load(z0);
  put(z0);
  load(z0 + 1);
  const float c2h = I.ph.c2h;
  float mdiv = 0.f, mu = 0.f;
  int bad = 0;
  for (int z = z0; z < z1; ++z) {
    __syncthreads();  // plane z - 2 has been read
    put(z + 1);
    __syncthreads();
    if (z + 1 < z1) load(z + 2);
    if (on) {
      const int c = (ly + 1) * SX + lx + 1;
      const size_t o = (size_t)z * NN + (size_t)(y0 + ly) * N + x0 + lx;
      float q[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) q[a] = __ldg(I.P[a] + o);
      AccS f[3];
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int d = 0; d < 3; ++d) f[a].p[d] = &ring[(z + 2 + d) % 3][a][c];
      const float d = st_dx<float>(f[0], c2h) + st_dy<float>(f[1], c2h) + st_dz<float>(f[2], c2h);
      mdiv = fmax(mdiv, fabs(d));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float u = f[a](0, 0, 0);
        mu = fmax(mu, fabs(u));
        if (!isfinite(u) || !isfinite(q[a])) bad += 1;
      }
    }
  }
  mdiv = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mdiv)));
  mu = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mu)));
  bad = __reduce_add_sync(0xffffffffu, bad);
  if (lx == 0)
    stats_add(I, blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * (blockIdx.z % nchunk)), __double_as_longlong((double)mdiv),
              __double_as_longlong((double)mu), bad);
}

}  // namespace

int stats_partials_per_instance(int) { return STATS_BLOCKS; }

void plain32_prepare() {
  const std::pair<const void*, size_t> k[] = {{(const void*)k_stage1, Planes<float, 4, 7>::bytes()},
                                              {(const void*)k_stage2, Planes<float, 20, 4>::bytes()},
                                              {(const void*)k_div, Planes<float, 6, 6>::bytes()},
                                              {(const void*)k_correct, Planes<float2, 1, 8>::bytes()}};
  for (const auto& f : k) {
    const cudaError_t e = cudaFuncSetAttribute(f.first, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.second);
    if (e != cudaSuccess) throw std::runtime_error(std::string("plain kernels' smem attribute: ") + cudaGetErrorString(e));
  }
}

template <>
void launch_stage1<float>(const Group<float>& g, int par, cudaStream_t st) {
  launch_planes(k_stage1, Planes<float, 4, 7>::bytes(), g, par, st, "stage1");
}
template <>
void launch_stage2<float>(const Group<float>& g, int par, cudaStream_t st) {
  launch_planes(k_stage2, Planes<float, 20, 4>::bytes(), g, par, st, "stage2");
}
template <>
void launch_div<float>(const Group<float>& g, int par, cudaStream_t st) {
  launch_planes(k_div, Planes<float, 6, 6>::bytes(), g, par, st, "div");
}
template <>
void launch_correct<float>(const Group<float>& g, int par, cudaStream_t st) {
  launch_planes(k_correct, Planes<float2, 1, 8>::bytes(), g, par, st, "correct");
}
template <>
void launch_stats_u<float>(const Group<float>& g, int, cudaStream_t st) {
  // planes per CTA: 16 (two halo planes), fewer while the grid has fewer than eight CTAs per SM
  int zc = std::min(16, g.N);
  const long long tiles = (long long)g.n * ((g.N + BX - 1) / BX) * ((g.N + BY - 1) / BY);
  while (zc > 2 && tiles * ((g.N + zc - 1) / zc) < 8 * g.sms) zc /= 2;
  int nchunk = (g.N + zc - 1) / zc;
  if ((long long)nchunk * g.n > 65535) { nchunk = 1; zc = g.N; }
  k_stats_u<<<dim3((g.N + BX - 1) / BX, (g.N + BY - 1) / BY, nchunk * g.n), BX * BY, 0, st>>>(g.d_inst, nchunk, zc);
  check_launch("stats (velocity)");
}
// FP32, all diagnostics: one launch up to 64^3 and three droplets (STATS_BLOCKS CTAs each, at most six per SM). us of
// a call with its copy to the host, two launches / one: one 8^3 20.3 / 14.5, one 32^3 21.5 / 14.8, one 64^3 24.5 /
// 24.1, 2 x 40^3 26.7 / 23.7, 3 x 24^3 31.7 / 29.2 (35.4 in some runs), 3 x 60^3 42.0 / 37.5; beyond the rule one 72^3 26.3 /
// 27.5, 4 x 16^3 34.0 / 29.2 .. 35.5, 4 x 24^3 33.8 / 35.8, 4 x 54^3 43.9 / 39.6 .. 48.2, 8 x 32^3 49.7 / 60.1, 16 x 16^3 78 / 98.
inline bool stats_in_one(const Group<float>& g) { return g.N <= 64 && (long)g.n * STATS_BLOCKS <= 6L * g.sms; }
inline bool stats_in_one(const Group<double>&) { return false; }
inline void launch_stats_small(const Group<float>& g, int par, cudaStream_t st) {
  k_stats_small<<<dim3(STATS_BLOCKS, g.n), STATS_THREADS, 0, st>>>(g.d_inst, par);
  check_launch("stats");
}
inline void launch_stats_small(const Group<double>&, int, cudaStream_t) {}

template <class T>
int launch_stats(const Group<T>& g, int par, cudaStream_t st, bool full) {
  if (full && stats_in_one(g)) {
    launch_stats_small(g, par, st);
    return STATS_BLOCKS;
  }
  k_stats_mass<T><<<dim3(STATS_BLOCKS, g.n), STATS_THREADS, 0, st>>>(g.d_inst, par);
  check_launch("stats");
  if (full) launch_stats_u<T>(g, par, st);
  return STATS_BLOCKS;
}

template int launch_stats<float>(const Group<float>&, int, cudaStream_t, bool);
template int launch_stats<double>(const Group<double>&, int, cudaStream_t, bool);

}  // namespace ttsh
