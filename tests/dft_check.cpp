// Host check of csrc/dft.cuh: every small DFT against the sum that defines it, FP64 and FP32.
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>

#include <cuda_runtime.h>
// the packed FP32 instructions of the device, one operation per part
static inline float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
static inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }
#include "dft.cuh"

template <class C, int R>
double error() {
  typedef decltype(C::x) T;
  std::mt19937_64 rng(R);
  std::normal_distribution<double> g;
  double num = 0, den = 0;
  for (int rep = 0; rep < 200; ++rep) {
    C v[R];
    std::complex<long double> x[R];
    for (int n = 0; n < R; ++n) {
      v[n].x = (T)g(rng);
      v[n].y = (T)g(rng);
      x[n] = {v[n].x, v[n].y};
    }
    ttsh::dft::Dft<R>::run(v);
    for (int k = 0; k < R; ++k) {
      std::complex<long double> s = 0;
      for (int n = 0; n < R; ++n) s += x[n] * std::polar(1.0L, -2 * 3.14159265358979323846264338327950288L * ((n * k) % R) / R);
      num += (double)std::norm(s - std::complex<long double>(v[k].x, v[k].y));
      den += (double)std::norm(s);
    }
  }
  return std::sqrt(num / den);
}

template <int R>
int check() {
  const double d = error<double2, R>(), f = error<float2, R>();
  std::printf("R=%d double %.2e float %.2e\n", R, d, f);
  // a few roundings per level of at most four levels
  return d < 4 * 1.2e-16 && f < 4 * 6e-8 ? 0 : 1;
}

template <int R>
int check64() {
  const double d = error<double2, R>();
  std::printf("R=%d double %.2e\n", R, d);
  return d < 5 * 1.2e-16 ? 0 : 1;
}

int main() {
  if (check64<24>() + check64<32>() + check64<40>()) return 1;
  return check<2>() + check<3>() + check<4>() + check<5>() + check<6>() + check<8>() + check<9>() + check<10>() + check<12>() +
         check<15>() + check<16>();
}
