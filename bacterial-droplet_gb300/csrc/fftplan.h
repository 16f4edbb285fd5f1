// fftplan.h — the steps and lines per CTA of the any-size FFT, computed alike at compile time (the
// kernels built per size, fftplan_impl.cuh) and at run time (the kernel for any size, fft.cu).
#pragma once
#include <stddef.h>

namespace ttsh {
namespace fftplan {

// Radix plan of a size: factors 4, 2, 3, 5 in this order (the order a tuning starts from).
struct Radices {
  int n = 0;
  int r[16] = {};
  constexpr void add(int x) { r[n++] = x; }
};
constexpr Radices default_plan(int N) {
  Radices p;
  const int f[4] = {4, 2, 3, 5};
  for (int i = 0; i < 4; ++i)
    while (N % f[i] == 0) {
      p.add(f[i]);
      N /= f[i];
    }
  return p;
}

// The steps of a transform: FP64 a radix a[i] of dft.cuh (b[i] = 1), FP32 one or two stages a[i], b[i]
// of the radix plan.
struct Steps {
  int n = 0;
  int a[16] = {}, b[16] = {};
  constexpr void add(int x, int y) {
    a[n] = x;
    b[n++] = y;
  }
  constexpr int radix(int i) const { return a[i] * b[i]; }
};

// FP64 radices.
constexpr int kRadix[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
constexpr bool is_radix(int r) {
  for (int x : kRadix)
    if (x == r) return true;
  return false;
}
// Real operations per value of a radix-R step (the DFT of dft.cuh and its twiddles).
constexpr double step_cost(int R) {
  const double c = R == 2 ? 2 : (R == 3 || R == 4) ? 4 : R == 5 ? 7.2 : R == 6 ? 6 : R == 8 ? 6.5 : R == 9 ? 9.8 : R == 10 ? 9.2
                   : R == 12 ? 8 : R == 15 ? 11.2 : 10;
  return c + 4.0 * (R - 1) / R;
}
// Fewest steps (each boundary is a trip through shared memory), then fewest operations; larger
// radices first.
constexpr void best_steps(int N, int most, const Steps& cur, double cost, Steps& best, double& best_cost) {
  if (N == 1) {
    if (best.n == 0 || cur.n < best.n || (cur.n == best.n && cost < best_cost)) {
      best = cur;
      best_cost = cost;
    }
    return;
  }
  if (best.n && cur.n >= best.n) return;
  for (int r : kRadix)
    if (r <= most && N % r == 0) {
      Steps next = cur;
      next.add(r, 1);
      best_steps(N / r, r, next, cost + step_cost(r), best, best_cost);
    }
}

// FP32 stage pairs that a step takes in registers.
#define TTSH_STAGE_PAIRS(X) \
  X(2, 1) X(3, 1) X(4, 1) X(5, 1) X(4, 4) X(4, 2) X(4, 3) X(4, 5) X(2, 3) X(2, 5) X(3, 3) X(3, 5) X(5, 5)
constexpr bool is_pair(int r1, int r2) {
#define X(A, B) if (r1 == A && r2 == B) return true;
  TTSH_STAGE_PAIRS(X)
#undef X
  return false;
}
constexpr Steps stage_steps(const Radices& plan) {
  Steps s;
  for (int k = 0; k < plan.n; ++k) {
    if (k + 1 < plan.n && is_pair(plan.r[k], plan.r[k + 1])) {
      s.add(plan.r[k], plan.r[k + 1]);
      ++k;
    } else {
      s.add(plan.r[k], 1);
    }
  }
  return s;
}

// The steps of the default plan of size N.
template <class T>
constexpr Steps default_steps(int N) {
  if (sizeof(T) == 4) return stage_steps(default_plan(N));
  Steps best;
  double cost = 0;
  best_steps(N, 16, Steps(), 0, best, cost);
  return best;
}

// The small sizes of the register kernels in FP64 (24, 32, 48). A grid of few warps is bound by the chain
// of FP64 instructions of one thread, not by the pipe of the SM, so a step's butterflies go to as many
// threads as it has (in the register kernels the threads of the first factor's DFTs take all of the
// second's), 8 lines per CTA. The steps are the register kernels' factors in their order, and so are the
// bits. One solve (three launches), us, register kernels / these: 32^3 48.5 / 42.6, 48^3 68.4 / 59.4, 24^3
// 59.9 / 50.1; where the pipe is full they are level (8 x 48^3 206 / 208, 24 x 32^3 187 / 183).
constexpr Steps small_steps(int N) {
  const int first = N % 3 == 0 ? 12 : 8;
  Steps s;
  s.add(first, 1);
  s.add(N / first, 1);
  return s;
}
constexpr int small_lb(int N) {
  int lb = 8;
  while (N % lb != 0) --lb;
  return lb;
}

constexpr int kThreads = 256;  // most threads of a CTA
// Lines along x lie one after another in shared memory, elements spread by one in eight.
constexpr int x_pitch(int N) { return N + N / 8 + 1; }

// Lines per CTA: the divisor of N whose steps, counted in whole warps per line, cost least, among
// those that leave two CTAs' buffers on an SM (three for FP32) and whose rows along x are at least 64
// bytes where N allows. N = 100 in FP64: 25 lines (250 radix-10 butterflies in 8 warps; 4 lines, the
// largest power of two dividing 100, would fill 40 of 64 lanes).
template <class T>
constexpr int default_lb(int N) {
  const size_t csize = 2 * sizeof(T);
  const Steps st = default_steps<T>(N);
  const size_t room = (sizeof(T) == 4 ? 227 / 3 : 227 / 2) * 1024 - 1024;
  int best = 0;
  double cost = 0;
  for (int lb = 1; lb <= N && lb <= 64; ++lb) {
    if (N % lb != 0) continue;
    if (lb > 1 && 2 * (size_t)(lb * x_pitch(N)) * csize > room) break;
    double c = 0;
    for (int i = 0; i < st.n; ++i) {
      const int r = st.radix(i), warps = (lb * (N / r) + 31) / 32;
      const int rounds = (warps + kThreads / 32 - 1) / (kThreads / 32);
      // whole warps, and (a tenth of the weight) whole rounds of the CTA
      c += (sizeof(T) == 8 ? step_cost(r) : 10.0) * r * (warps + 0.1 * (rounds * (kThreads / 32) - warps));
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
// Threads of a CTA with LB lines: its steps' butterflies, at most kThreads.
constexpr int threads_for(const Steps& st, int N, int LB) {
  int most = 0;
  for (int i = 0; i < st.n; ++i)
    if (LB * (N / st.radix(i)) > most) most = LB * (N / st.radix(i));
  most = (most + 31) / 32 * 32;
  return most < kThreads ? most : kThreads;
}
// Steps of a pass (0, 1 forward x, y; 2 forward z, divide, inverse z; 3, 4 inverse y, x). FP64: the
// divide's step is the last forward and the first inverse one, and the inverse goes through the steps
// backwards; FP32: the inverse runs the plan from its start.
template <class T>
constexpr int pass_steps(int n, int pass) { return pass != 2 ? n : (sizeof(T) == 8 ? 2 * n - 1 : 2 * n); }
// CTAs of a plane's cluster: as many as split its line groups evenly, 8 (the portable most) or fewer.
constexpr int cluster_parts(int groups) {
  int p = 8;
  while (groups % p != 0) --p;
  return p;
}

}  // namespace fftplan
}  // namespace ttsh
