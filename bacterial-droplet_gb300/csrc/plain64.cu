// plain64.cu — the FP64 plain form of the TTSH3D step: every intermediate in a global array, the
// reference's stencils (TTSH3D.cu:3280-3343) evaluated separably on tiles of one z-plane. It is the
// library's default precision.
//
//   stage1  <- getTempVari_1 + getTempVari_2 (TTSH3D.cu:537-605) and the pointwise parts of getDtF
//   stage2  <- the rest of getDtF + getVStar + phi update of getVNew (:608-632, :471-491, :515)
//   div     <- getStream mode 0 for both fields (:664-670), packed as one complex field
//   correct <- getVNew (:494-516), pressures read from the packed complex field
#include <cmath>
#include <cstdio>
#include <stdexcept>
#include <string>

#include "common.cuh"
#include "kernels.h"
#include "tiles.h"

namespace ttsh {

namespace {

inline void check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    char buf[256];
    snprintf(buf, sizeof(buf), "%s launch failed: %s", what, cudaGetErrorString(e));
    throw std::runtime_error(buf);
  }
}

// ---- tiles ---------------------------------------------------------------------------------
// A CTA computes a tile of tx columns x ty rows of one z-plane, one site per thread. FP64 is bound
// by the FP64 pipe alone (2 lanes per SM and clock: a warp instruction occupies it for 16 clocks,
// in which the SM can issue 63 others), so the stencils are evaluated separably, each 1-D sum once
// per lattice line that needs it and handed on through shared memory, whose traffic and barriers
// are free beside it:
//   pass z (tile + 1 on every side): of the planes z-1, z, z+1, the sums s_z = [1, 4, 1],
//          c_z = [1, 0, 1] and the difference delta_z = [-1, 0, 1];
//   pass x (tile + 1 row above and below): the same along x of those;
//   pass y (the tile): the same along y, one site per thread.
// D_x = c2h/36 delta_x s_y s_z, D_y = c2h/36 s_x delta_y s_z, D_z = c2h/36 s_x s_y delta_z and
// L = cl12 (c_x c_y c_z + 8 faces - 56 centre) are the reference's 27-point and 15-point weights
// (st_dx/st_dy/st_dz/st_lap of common.cuh, TTSH3D.cu:3280-3343): the weights are integers until one
// last multiplication, where the reference rounds 16/36, 4/36 and 1/36. A gradient and a Laplacian
// of one field take about 24 operations per site of a 16 x 16 tile instead of about 90.
typedef double T;
typedef double2 C;
typedef InstDev<double> Inst;
constexpr int CTAS = 3;    // CTAs per SM that registers and shared memory leave room for

// What a thread knows of its CTA's tile. Staged points of pass z are the (tx + 2) x (ty + 2) of the
// tile and its halo (row-major), of pass x the tx x (ty + 2).
struct Tile {
  int N, NN, tx, x0, y0, px, np, nx;  // px: columns of pass z; np, nx: points of pass z and x
  int lx, ly;                         // this thread's site in the tile
  bool on;                            // ... is a site of the box
  int o;                              // its offset
  int s0;                             // this thread's first point of pass x
  int zo[3];                          // offsets of the planes z - 1, z, z + 1 (wrapped)
  bool zw[3];                         // ... lies beyond the boundary

  __device__ __forceinline__ Tile(int N_, int z, int tx_, int ty, int ntx) : N(N_), NN(N_ * N_), tx(tx_) {
    const int by = blockIdx.x / ntx, bx = blockIdx.x - by * ntx;
    x0 = bx * tx;
    y0 = by * ty;
    px = tx + 2;
    np = px * (ty + 2);
    nx = tx * (ty + 2);
    // a pass's points beyond one per thread fall on its first warps, whose schedulers are the same in
    // every CTA: in every other CTA pass x starts two warps further on
    s0 = (blockDim.x % 128 == 0 && ((blockIdx.x ^ blockIdx.z) & 1)) ? (threadIdx.x ^ 64) : threadIdx.x;
    ly = threadIdx.x / tx;
    lx = threadIdx.x - ly * tx;
    on = ly < ty && x0 + lx < N && y0 + ly < N;
    zo[0] = wrapi(z - 1, N) * NN;
    zo[1] = z * NN;
    zo[2] = wrapi(z + 1, N) * NN;
    zw[0] = z == 0;
    zw[1] = false;
    zw[2] = z == N - 1;
    o = zo[1] + (y0 + ly) * N + x0 + lx;
  }
  // f(staged index, offset within a plane, whether the point lies beyond the boundary in x or y)
  template <class F>
  __device__ __forceinline__ void pass_z(F&& f) const {
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
      const int r = i / px, gx = x0 - 1 + (i - r * px), gy = y0 - 1 + r;
      // a partial tile's points beyond the halo wrap too (their values are not used)
      f(i, wrapi(gy, N) * N + wrapi(gx, N), gx < 0 || gx >= N || gy < 0 || gy >= N);
    }
  }
  // f(index of pass x, staged index of the point's left neighbour)
  template <class F>
  __device__ __forceinline__ void pass_x(F&& f) const {
    for (int i = s0; i < nx; i += blockDim.x) {
      const int r = i / tx;
      f(i, r * px + (i - r * tx));
    }
  }
  // s_x delta_y of pass z's s_z at this thread's site, the small differences summed (1.5 operations more
  // than differencing sums of pass x, which would round at 36 times the field instead of at 6)
  __device__ __forceinline__ T diff_y_sum_x(const T* s) const {
    const T *a = s + site_z() - px, *b = s + site_z() + px;
    return fma(T(4), b[0] - a[0], (b[-1] - a[-1]) + (b[1] - a[1]));
  }
  __device__ __forceinline__ int site_z() const { return (ly + 1) * px + lx + 1; }  // staged index of the site
  __device__ __forceinline__ int site_x() const { return ly * tx + lx; }            // pass-x index of row y - 1
};

// [1, 4, 1] of three values
__device__ __forceinline__ T sum141(T a, T b, T c) { return fma(T(4), b, a + c); }

// The 1-D sums of NF fields handed from pass to pass.
template <int NF>
struct GradLap {
  T *v, *c, *s, *d;     // pass z: the value, c_z, s_z, delta_z
  T *xd, *xs, *xz, *xc; // pass x: delta_x s_z, s_x s_z, s_x delta_z, c_x c_z
  __device__ __forceinline__ GradLap(T* m, int np, int nx) {
    v = m;
    c = v + NF * np;
    s = c + NF * np;
    d = s + NF * np;
    xd = d + NF * np;
    xs = xd + NF * nx;
    xz = xs + NF * nx;
    xc = xz + NF * nx;
  }
  __device__ __forceinline__ void run(const Tile& t, const T* const* f) const {
    t.pass_z([&](int i, int o, bool) {
      T a[NF], b[NF], e[NF];
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        a[k] = __ldg(f[k] + t.zo[0] + o);
        b[k] = __ldg(f[k] + t.zo[1] + o);
        e[k] = __ldg(f[k] + t.zo[2] + o);
      }
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        const T cz = a[k] + e[k];
        v[k * t.np + i] = b[k];
        c[k * t.np + i] = cz;
        s[k * t.np + i] = T(4) * b[k] + cz;
        d[k * t.np + i] = e[k] - a[k];
      }
    });
    __syncthreads();
    t.pass_x([&](int i, int j) {
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        const T* sk = s + k * t.np + j;
        const T* dk = d + k * t.np + j;
        const T* ck = c + k * t.np + j;
        xd[k * t.nx + i] = sk[2] - sk[0];
        xs[k * t.nx + i] = sum141(sk[0], sk[1], sk[2]);
        xz[k * t.nx + i] = sum141(dk[0], dk[1], dk[2]);
        xc[k * t.nx + i] = ck[0] + ck[2];
      }
    });
    __syncthreads();
  }
  // 36/c2h D_a (a = 0, 1, 2) and L / cl12 of field k at this thread's site
  __device__ __forceinline__ void out(const Tile& t, int k, T* g, T& lap) const {
    const int j = k * t.nx + t.site_x(), i = k * t.np + t.site_z(), tx = t.tx;
    g[0] = sum141(xd[j], xd[j + tx], xd[j + 2 * tx]);
    g[1] = xs[j + 2 * tx] - xs[j];
    g[2] = sum141(xz[j], xz[j + tx], xz[j + 2 * tx]);
    const T corners = xc[j] + xc[j + 2 * tx];
    const T faces = (v[i - 1] + v[i + 1]) + (v[i - t.px] + v[i + t.px]) + c[i];
    // exactly zero for a constant field: both terms are 48 v with the rounding of 6 v
    lap = fma(T(8), faces, fma(T(-56), v[i], corners));
  }
};

// ---- stage 1: getTempVari_1, getTempVari_2 and the pointwise parts of getDtF -------------------
// Of phi, P and u (read once): mu_0, mu_b and the stress S_ab = cA phi D_a P_b - zeta phi P_a P_b,
// which stage 2 differentiates, and the rates of change that need no second derivative, which go to
// the output arrays u*, P*, phi' for stage 2 to complete. About 245 FP64 operations per site;
// forming the products on chip, as the fused FP32 form does, would repeat them on every tile's halo
// (1.27 times at 16 x 16), while the 20 words per site written and read back here take a tenth of
// the time of the arithmetic.
__global__ void __launch_bounds__(MAXT, CTAS) k_stage1(const Inst* __restrict__ insts, int par, int tx, int ty, int ntx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / N];
  const Tile t(N, blockIdx.z % N, tx, ty, ntx);
  const Phys<T>& p = I.ph;
  T* const sm = reinterpret_cast<T*>(smem_raw);
  const int o = t.o;
  // two fields at a time, so that three CTAs fit on an SM (39 KB each at 16 x 16): with four at a time and two
  // CTAs the FP64 pipe idled 18 % of the time at the barriers between the passes
  T P[3] = {0, 0, 0}, u[3] = {0, 0, 0}, w[3] = {0, 0, 0}, gp[3] = {0, 0, 0};  // w = u + lambda0 P
  T ph = 0, mu0 = 0, kap = 0, m = 0;
  // what P_b's gradient and Laplacian give (field k of G): mu_b, S_ab and dP_b/dt
  auto polarisation = [&](const GradLap<2>& G, int k, int b) {
    T g[3], lap;
    G.out(t, k, g, lap);
    // mu_b (:571-573)
    I.mu[b][o] = ph * P[b] + p.La212 * lap;
    // the stress (:587-595; the 1/28 term is an integer-division zero) and the active stress
    const T cph = p.cA * ph * p.kd, zpb = -p.zeta * ph * P[b];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      T s = cph * g[a];
      if (p.zeta != T(0)) s += zpb * P[a];
      I.sig[a * 3 + b][o] = s;
    }
    // polarisation (:623-629) without eta L mu_b; OP_b and kappa phi DP_b are integer-division zeros
    // in the reference (:579-585)
    T r = -p.kd * (w[0] * g[0] + w[1] * g[1] + w[2] * g[2]) - kap * P[b];
    if (p.A != T(0)) r -= m * gp[b];
    I.Ps[par ^ 1][b][o] = r;
  };
  {
    const GradLap<2> G(sm, t.np, t.nx);
    const T* f[2] = {I.phi[par], I.P[0]};
    G.run(t, f);
    if (t.on) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        P[b] = I.P[b][o];
        u[b] = I.U[b][o];
        w[b] = p.lambda0 * P[b] + u[b];
      }
      T lap;
      G.out(t, 0, gp, lap);
      ph = G.v[t.site_z()];
      // mu_0 (TTSH3D.cu:567), 2 aPhi (phi - 3 phi^2 + 2 phi^3) in factors
      mu0 = p.aPhi2 * (ph * ((1 - ph) * (1 - 2 * ph))) - p.kPhi12 * lap;
      I.mu0[o] = mu0;
#pragma unroll
      for (int a = 0; a < 3; ++a) gp[a] *= p.kd;  // D_a phi
      const T P2 = P[0] * P[0] + P[1] * P[1] + P[2] * P[2];
      kap = p.alpha * ph + p.beta * P2;
      if (p.A != T(0)) {  // A (|D phi|^2 |P|^2 P_b + |P| (D phi . P) D_b phi), :627-629
        const T G2 = gp[0] * gp[0] + gp[1] * gp[1] + gp[2] * gp[2];
        kap += p.A * G2 * P2;
        m = p.A * sqrt(P2) * (gp[0] * P[0] + gp[1] * P[1] + gp[2] * P[2]);
      }
      // phi (:631) without gamma L mu_0
      I.phi[par ^ 1][o] = -(u[0] * gp[0] + u[1] * gp[1] + u[2] * gp[2]);
      polarisation(G, 1, 0);
    }
    __syncthreads();  // the next fields' sums take the same shared memory
  }
  {
    const GradLap<2> G(sm, t.np, t.nx);
    const T* f[2] = {I.P[1], I.P[2]};
    G.run(t, f);
    if (t.on) {
      polarisation(G, 0, 1);
      polarisation(G, 1, 2);
    }
    __syncthreads();
  }
  // velocity (:617-621) without the stress divergence
  auto velocity = [&](const auto& G, int k, int b) {
    T g[3], lap;
    G.out(t, k, g, lap);
    I.Us[par ^ 1][b][o] = p.mu12 * lap - p.kd * (u[0] * g[0] + u[1] * g[1] + u[2] * g[2]) + mu0 * gp[b];
  };
  {
    const GradLap<2> G(sm, t.np, t.nx);
    const T* f[2] = {I.U[0], I.U[1]};
    G.run(t, f);
    if (t.on) {
      velocity(G, 0, 0);
      velocity(G, 1, 1);
    }
    __syncthreads();
  }
  const GradLap<1> G(sm, t.np, t.nx);
  const T* f[1] = {I.U[2]};
  G.run(t, f);
  if (t.on) velocity(G, 0, 2);
}

// ---- stage 2: the outer stencils of getDtF, getVStar and the phi update of getVNew -------------
// L mu_0 and L mu_b of four fields and the divergences of the three stress columns, added to stage
// 1's rates: u*, P*, phi'. About 115 FP64 operations per site.
__global__ void __launch_bounds__(MAXT, CTAS) k_stage2(const Inst* __restrict__ insts, int par, int tx, int ty, int ntx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / N];
  const Tile t(N, blockIdx.z % N, tx, ty, ntx);
  const Phys<T>& p = I.ph;
  T* const sm = reinterpret_cast<T*>(smem_raw);
  const int o = t.o, np = t.np, nx = t.nx;
  {
    // Laplacians of mu_0, mu_x, mu_y, mu_z: v, c_z; c_x c_z
    T* const v = sm;
    T* const c = v + 4 * np;
    T* const xc = c + 4 * np;
    const T* const f[4] = {I.mu0, I.mu[0], I.mu[1], I.mu[2]};
    t.pass_z([&](int i, int q, bool) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k * np + i] = f[k][t.zo[1] + q];
        c[k * np + i] = f[k][t.zo[0] + q] + f[k][t.zo[2] + q];
      }
    });
    __syncthreads();
    t.pass_x([&](int i, int j) {
#pragma unroll
      for (int k = 0; k < 4; ++k) xc[k * nx + i] = c[k * np + j] + c[k * np + j + 2];
    });
    __syncthreads();
    if (t.on) {
      T L[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = k * np + t.site_z(), j = k * nx + t.site_x();
        const T faces = (v[i - 1] + v[i + 1]) + (v[i - t.px] + v[i + t.px]) + c[i];
        L[k] = fma(T(8), faces, fma(T(-56), v[i], xc[j] + xc[j + 2 * tx]));
      }
      // phi' = phi + dt dphi/dt (:631, :515), P* = P + dt dP/dt (:623-629, :486-488)
      I.phi[par ^ 1][o] = I.phi[par][o] + p.dt * (p.gamma12 * L[0] + I.phi[par ^ 1][o]);
#pragma unroll
      for (int b = 0; b < 3; ++b) I.Ps[par ^ 1][b][o] = I.P[b][o] + p.dt * (p.eta12 * L[b + 1] + I.Ps[par ^ 1][b][o]);
    }
    __syncthreads();
  }
  // divergences D_a S_ab: s_z of S_xb and S_yb, delta_z of S_zb; delta_x s_z S_xb + s_x delta_z S_zb
  // (both take s_y) and s_x s_z S_yb (delta_y)
  T* const z = sm;            // [3 b][3 a][np]
  T* const xa = z + 9 * np;   // [3 b][nx]
  T* const xy = xa + 3 * nx;  // [3 b][nx]
  t.pass_z([&](int i, int q, bool) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const T* f = I.sig[a * 3 + b];
        const T m = f[t.zo[0] + q], n = f[t.zo[2] + q];
        z[(3 * b + a) * np + i] = a == 2 ? n - m : T(4) * f[t.zo[1] + q] + (m + n);
      }
    }
  });
  __syncthreads();
  t.pass_x([&](int i, int j) {
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const T* zx = z + (3 * b) * np + j;
      const T* zy = zx + np;
      const T* zz = zy + np;
      xa[b * nx + i] = (zx[2] - zx[0]) + sum141(zz[0], zz[1], zz[2]);
      xy[b * nx + i] = sum141(zy[0], zy[1], zy[2]);
    }
  });
  __syncthreads();
  if (!t.on) return;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const int j = b * nx + t.site_x();
    const T d = sum141(xa[j], xa[j + tx], xa[j + 2 * tx]) + (xy[j + 2 * tx] - xy[j]);
    // u* = u + dt du/dt (:617-621, :480-482)
    I.Us[par ^ 1][b][o] = I.U[b][o] + p.dt * (p.kd * d + I.Us[par ^ 1][b][o]);
  }
}

// ---- getStream mode 0 for both fields (:664-670), packed as one complex field -------------------
// The neighbours beyond the boundary come from the previous step's u*, P* (quirk Q2: the halo is
// refreshed at the start of getRHS, :369-371 and :405-407, before getVStar rewrites the interior).
// About 43 FP64 operations per site.
__global__ void __launch_bounds__(MAXT, CTAS) k_div(const Inst* __restrict__ insts, int par, int tx, int ty, int ntx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / N];
  const Tile t(N, blockIdx.z % N, tx, ty, ntx);
  const Phys<T>& p = I.ph;
  const int np = t.np, nx = t.nx;
  T* const z = reinterpret_cast<T*>(smem_raw);  // [2 fields][3 a][np]
  T* const xa = z + 6 * np;                     // [2][nx]
  const bool stale = I.stale;
  t.pass_z([&](int i, int q, bool out) {
#pragma unroll
    for (int f = 0; f < 2; ++f) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const T* cur = f == 0 ? I.Us[par ^ 1][a] : I.Ps[par ^ 1][a];
        const T* old = f == 0 ? I.Us[par][a] : I.Ps[par][a];
        auto at = [&](int k) { return (stale && (out || t.zw[k]) ? old : cur)[t.zo[k] + q]; };
        const T m = at(0), n = at(2);
        z[(3 * f + a) * np + i] = a == 2 ? n - m : T(4) * at(1) + (m + n);
      }
    }
  });
  __syncthreads();
  t.pass_x([&](int i, int j) {
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const T* zx = z + (3 * f) * np + j;
      const T* zz = zx + 2 * np;
      xa[f * nx + i] = (zx[2] - zx[0]) + sum141(zz[0], zz[1], zz[2]);
    }
  });
  __syncthreads();
  if (!t.on) return;
  T d[2];
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    const int j = f * nx + t.site_x();
    // getStream mode 0 (:666-668): the divergence over dt
    d[f] = p.kdiv * (sum141(xa[j], xa[j + tx], xa[j + 2 * tx]) + t.diff_y_sum_x(z + (3 * f + 1) * np));
  }
  I.W[t.o] = make_double2(d[0], d[1]);
}

// ---- getVNew (TTSH3D.cu:494-516): u = u* - dt D p_v, P = P* - dt D p_p ---------------------------
// About 46 FP64 operations per site.
__global__ void __launch_bounds__(MAXT, CTAS) k_correct(const Inst* __restrict__ insts, int par, int tx, int ty, int ntx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / N];
  const Tile t(N, blockIdx.z % N, tx, ty, ntx);
  const Phys<T>& p = I.ph;
  const int np = t.np, nx = t.nx;
  C* const s = reinterpret_cast<C*>(smem_raw);  // pass z, both pressures: s_z, delta_z
  C* const d = s + np;
  C* const xd = d + np;  // pass x: delta_x s_z, s_x delta_z
  C* const xz = xd + nx;
  const C* const W = I.W;
  auto sum = [](const C& a, const C& b, const C& c) {
    C r;
    r.x = sum141(a.x, b.x, c.x);
    r.y = sum141(a.y, b.y, c.y);
    return r;
  };
  auto diff = [](const C& a, const C& b) {
    C r;
    r.x = a.x - b.x;
    r.y = a.y - b.y;
    return r;
  };
  t.pass_z([&](int i, int q, bool) {
    const C m = W[t.zo[0] + q], b = W[t.zo[1] + q], n = W[t.zo[2] + q];
    s[i] = sum(m, b, n);
    d[i] = diff(n, m);
  });
  __syncthreads();
  t.pass_x([&](int i, int j) {
    xd[i] = diff(s[j + 2], s[j]);
    xz[i] = sum(d[j], d[j + 1], d[j + 2]);
  });
  __syncthreads();
  if (!t.on) return;
  const int j = t.site_x(), o = t.o;
  const C *a = s + t.site_z() - t.px, *b = s + t.site_z() + t.px;  // as diff_y_sum_x
  const C g[3] = {sum(xd[j], xd[j + tx], xd[j + 2 * tx]), sum(diff(b[-1], a[-1]), diff(b[0], a[0]), diff(b[1], a[1])),
                  sum(xz[j], xz[j + tx], xz[j + 2 * tx])};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    I.U[k][o] = I.Us[par ^ 1][k][o] - p.dt * (p.kd * g[k].x);
    I.P[k][o] = I.Ps[par ^ 1][k][o] - p.dt * (p.kd * g[k].y);
  }
}

// ---- max |D.u|, max |u| and the non-finite values of u and P ------------------------------------
// About 22 FP64 operations per site instead of 85; maxima and finiteness are taken on the bits (integers):
// 160^3 with the mass 664 -> 219 us.
__global__ void __launch_bounds__(MAXT, CTAS) k_stats_u(const Inst* __restrict__ insts, int par, int tx, int ty, int ntx) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = insts[0].N;
  const Inst& I = insts[blockIdx.z / N];
  const Tile t(N, blockIdx.z % N, tx, ty, ntx);
  T* const z = reinterpret_cast<T*>(smem_raw);  // s_z u_x, s_z u_y, delta_z u_z
  T* const xa = z + 3 * t.np;
  t.pass_z([&](int i, int q, bool) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const T m = __ldg(I.U[a] + t.zo[0] + q), n = __ldg(I.U[a] + t.zo[2] + q);
      z[a * t.np + i] = a == 2 ? n - m : sum141(m, __ldg(I.U[a] + t.zo[1] + q), n);
    }
  });
  __syncthreads();
  t.pass_x([&](int i, int j) {
    const T* zz = z + 2 * t.np + j;
    xa[i] = (z[j + 2] - z[j]) + sum141(zz[0], zz[1], zz[2]);
  });
  __syncthreads();
  constexpr long long INF = 0x7ff0000000000000ll;
  auto mag = [](T v) { return __double_as_longlong(v) & 0x7fffffffffffffffll; };
  long long mdiv = 0, mu = 0;
  int bad = 0;
  if (t.on) {
    const int j = t.site_x();
    const long long d = mag(I.ph.kd * (sum141(xa[j], xa[j + tx], xa[j + 2 * tx]) + t.diff_y_sum_x(z + t.np)));
    if (d <= INF) mdiv = d;  // a NaN is counted, not a maximum
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const long long u = mag(I.U[a][t.o]), p = mag(I.P[a][t.o]);
      if (u <= INF && u > mu) mu = u;
      if (u >= INF || p >= INF) bad += 1;
    }
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    mdiv = max(mdiv, __shfl_xor_sync(0xffffffffu, mdiv, s));
    mu = max(mu, __shfl_xor_sync(0xffffffffu, mu, s));
  }
  bad = __reduce_add_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) stats_add(I, blockIdx.x + gridDim.x * (blockIdx.z % N), mdiv, mu, bad);
}

template <class K>
void launch_tiles(K kernel, const Group<double>& g, int par, size_t (*values)(const TileDim&), cudaStream_t st, const char* what) {
  if ((long)g.N * g.n > 65535) throw std::runtime_error("too many instances of this size in one group");
  static thread_local TileDim d;
  static thread_local int last_n = 0;
  if (last_n != g.N) {
    d = pick_tile(g.N);
    last_n = g.N;
  }
  kernel<<<dim3(d.nx * d.ny, 1, g.N * g.n), d.threads(), values(d) * sizeof(T), st>>>(g.d_inst, par, d.tx, d.ty, d.nx);
  check_launch(what);
}

}  // namespace

template <>
void launch_stage1<double>(const Group<double>& g, int par, cudaStream_t st) {
  launch_tiles(k_stage1, g, par, stage1_values, st, "stage1");
}
template <>
void launch_stage2<double>(const Group<double>& g, int par, cudaStream_t st) {
  launch_tiles(k_stage2, g, par, stage2_values, st, "stage2");
}
template <>
void launch_div<double>(const Group<double>& g, int par, cudaStream_t st) {
  launch_tiles(k_div, g, par, div_values, st, "div");
}
template <>
void launch_stats_u<double>(const Group<double>& g, int par, cudaStream_t st) {
  launch_tiles(k_stats_u, g, par, stats_values, st, "stats (velocity)");
}
template <>
void launch_correct<double>(const Group<double>& g, int par, cudaStream_t st) {
  launch_tiles(k_correct, g, par, correct_values, st, "correct");
}

}  // namespace ttsh
