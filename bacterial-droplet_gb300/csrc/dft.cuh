// dft.cuh — small DFTs in registers, compile-time sizes 2 .. 40, for the FFT passes.
//
// Dft<R>::run(v): v[0..R) <- sum over n of v[n] exp(-2 pi i n k / R), natural order in and out, in place.
// 2 and 4 are butterflies; 3 and 5 use the symmetry of their twiddles (the real and imaginary parts
// of exp(2 pi i k / R) are even and odd in k), 12 and 36 real operations; 6, 10, 12, 15 are
// prime-factor products (Good, 1958: the index maps below leave no twiddles between the factors), and so
// are 24 and 40; 8, 9, 16 are two radix-2/4, 3 or 4 levels with the constant twiddles written out.
#pragma once
#include <cuda_runtime.h>

namespace ttsh {
namespace dft {

template <class C>
__device__ __forceinline__ C mk(decltype(C::x) a, decltype(C::x) b) { C r; r.x = a; r.y = b; return r; }
__device__ __forceinline__ double2 add(double2 a, double2 b) { return mk<double2>(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return mk<double2>(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 axpy(double2 a, double s, double2 b) { return mk<double2>(fma(s, b.x, a.x), fma(s, b.y, a.y)); }
// FP32: one packed instruction for both parts (two IEEE operations, round to nearest)
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 axpy(float2 a, float s, float2 b) { return __ffma2_rn(make_float2(s, s), b, a); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return axpy(a, -1.f, b); }
template <class C>
__device__ __forceinline__ C mul(C a, C b) {
  return mk<C>(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
template <class C>
__device__ __forceinline__ C conj(C a) { return mk<C>(a.x, -a.y); }
template <class C>
__device__ __forceinline__ C mi(C a) { return mk<C>(a.y, -a.x); }  // -i a
template <class C>
__device__ __forceinline__ C axmi(C a, decltype(C::x) s, C b) { return axpy(a, s, mi(b)); }  // a + s (-i b)
// 1 / sqrt 2 in FP64 from above and from below. As (HI, LO) the eighth roots of unity have magnitude 1 to
// 1e-17; with the nearest value in both parts it would be 7e-17 off, the same way in every transform of
// a solve.
constexpr double R2_HI = 0.70710678118654757274, R2_LO = 0.70710678118654746172;
template <class C>
__device__ __forceinline__ C w8(C a) {  // a exp(-2 pi i / 8)
  typedef decltype(C::x) T;
  return mul(a, mk<C>(T(R2_HI), T(-R2_LO)));
}
template <class C>
__device__ __forceinline__ C w83(C a) {  // a exp(-6 pi i / 8)
  typedef decltype(C::x) T;
  return mul(a, mk<C>(T(-R2_LO), T(-R2_HI)));
}

template <int R>
struct Dft;

template <>
struct Dft<1> {
  template <class C>
  static __device__ __forceinline__ void run(C*) {}
};
template <>
struct Dft<2> {
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    const C a = v[0], b = v[1];
    v[0] = add(a, b);
    v[1] = sub(a, b);
  }
};
template <>
struct Dft<3> {
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    typedef decltype(C::x) T;
    const C p = add(v[1], v[2]), q = sub(v[1], v[2]);
    const C m = axpy(v[0], T(-0.5), p);
    v[0] = add(v[0], p);
    v[1] = axmi(m, T(0.86602540378443864676), q);
    v[2] = axmi(m, T(-0.86602540378443864676), q);
  }
};
template <>
struct Dft<4> {
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    const C a = add(v[0], v[2]), b = sub(v[0], v[2]), c = add(v[1], v[3]), d = mi(sub(v[1], v[3]));
    v[0] = add(a, c);
    v[2] = sub(a, c);
    v[1] = add(b, d);
    v[3] = sub(b, d);
  }
};
template <>
struct Dft<5> {
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    typedef decltype(C::x) T;
    constexpr T c1 = T(0.30901699437494742410), c2 = T(-0.80901699437494742410);  // cos 72, cos 144 degrees
    constexpr T s1 = T(0.95105651629515357212), s2 = T(0.58778525229247312917);   // sin
    const C p = add(v[1], v[4]), q = add(v[2], v[3]), r = sub(v[1], v[4]), s = sub(v[2], v[3]);
    const C a = axpy(axpy(v[0], c1, p), c2, q), b = axpy(axpy(v[0], c2, p), c1, q);
    v[0] = add(v[0], add(p, q));
    v[1] = axmi(axmi(a, s1, r), s2, s);
    v[4] = axmi(axmi(a, -s1, r), -s2, s);
    v[2] = axmi(axmi(b, s2, r), -s1, s);
    v[3] = axmi(axmi(b, -s2, r), s1, s);
  }
};
// R = A B, coprime: with n = B n1 + A n2 and k = k1 mod A = k2 mod B, n k = B n1 k1 + A n2 k2 mod R.
template <int A, int B>
struct DftPF {
  static constexpr int crt(int k1, int k2) {
    for (int k = 0; k < A * B; ++k)
      if (k % A == k1 && k % B == k2) return k;
    return 0;
  }
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    C u[B][A];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) u[n2][n1] = v[(B * n1 + A * n2) % (A * B)];
      Dft<A>::run(u[n2]);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      C w[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) w[n2] = u[n2][k1];
      Dft<B>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[crt(k1, k2)] = w[k2];
    }
  }
};
template <> struct Dft<6> : DftPF<3, 2> {};
template <> struct Dft<10> : DftPF<5, 2> {};
template <> struct Dft<12> : DftPF<4, 3> {};
template <> struct Dft<15> : DftPF<5, 3> {};
template <>
struct Dft<8> {
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4>::run(e);
    Dft<4>::run(o);
    o[1] = w8(o[1]);
    o[2] = mi(o[2]);
    o[3] = w83(o[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = add(e[k], o[k]);
      v[k + 4] = sub(e[k], o[k]);
    }
  }
};
template <>
struct Dft<9> {
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    typedef decltype(C::x) T;
    C u[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
#pragma unroll
      for (int m = 0; m < 3; ++m) u[r][m] = v[r + 3 * m];
      Dft<3>::run(u[r]);
    }
    const C w1 = mk<C>(T(0.76604444311897803520), T(-0.64278760968653932632));  // exp(-2 pi i / 9) and powers 2, 4
    const C w2 = mk<C>(T(0.17364817766693034885), T(-0.98480775301220805937));
    const C w4 = mk<C>(T(-0.93969262078590838405), T(-0.34202014332566873304));
    u[1][1] = mul(u[1][1], w1);
    u[1][2] = mul(u[1][2], w2);
    u[2][1] = mul(u[2][1], w2);
    u[2][2] = mul(u[2][2], w4);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      C t[3] = {u[0][k], u[1][k], u[2][k]};
      Dft<3>::run(t);
#pragma unroll
      for (int j = 0; j < 3; ++j) v[k + 3 * j] = t[j];
    }
  }
};
template <>
struct Dft<16> {
  template <class C>
  static __device__ __forceinline__ void run(C* v) {
    typedef decltype(C::x) T;
    C u[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int m = 0; m < 4; ++m) u[r][m] = v[r + 4 * m];
      Dft<4>::run(u[r]);
    }
    const C w1 = mk<C>(T(0.92387953251128675613), T(-0.38268343236508977173));  // exp(-2 pi i / 16) and power 3
    const C w3 = mk<C>(T(0.38268343236508977173), T(-0.92387953251128675613));
    u[1][1] = mul(u[1][1], w1);
    u[1][2] = w8(u[1][2]);
    u[1][3] = mul(u[1][3], w3);
    u[2][1] = w8(u[2][1]);
    u[2][2] = mi(u[2][2]);
    u[2][3] = w83(u[2][3]);
    u[3][1] = mul(u[3][1], w3);
    u[3][2] = w83(u[3][2]);
    u[3][3] = mul(u[3][3], mk<C>(-w1.x, -w1.y));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      C t[4] = {u[0][k], u[1][k], u[2][k], u[3][k]};
      Dft<4>::run(t);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[k + 4 * j] = t[j];
    }
  }
};

template <> struct Dft<24> : DftPF<8, 3> {};
template <> struct Dft<40> : DftPF<8, 5> {};
// 32 = 2 x 16 (FP64): the even and odd inputs' DFTs, the odd ones times exp(-2 pi i k / 32)
template <>
struct Dft<32> {
  static __device__ __forceinline__ void run(double2* v) {
    constexpr double c[16] = {1, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708, R2_HI,
                              0.55557023301960222474, 0.38268343236508977173, 0.19509032201612826785, 0,
                              -0.19509032201612826785, -0.38268343236508977173, -0.55557023301960222474, -R2_LO,
                              -0.83146961230254523708, -0.92387953251128675613, -0.98078528040323044913};  // cos(2 pi k / 32)
    double2 e[16], o[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      e[k] = v[2 * k];
      o[k] = v[2 * k + 1];
    }
    Dft<16>::run(e);
    Dft<16>::run(o);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      // exp(-2 pi i k / 32) = cos - i sin, sin(2 pi k / 32) = cos(2 pi (k - 8) / 32)
      const double sn = k == 4 ? R2_LO : (k == 12 ? R2_HI : c[k >= 8 ? k - 8 : 8 - k]);
      const double2 x = k == 0 ? o[0] : (k == 8 ? mi(o[8]) : mul(o[k], mk<double2>(c[k], -sn)));
      v[k] = add(e[k], x);
      v[k + 16] = sub(e[k], x);
    }
  }
};

}  // namespace dft
}  // namespace ttsh
