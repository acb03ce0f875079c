// Small DFTs in registers, FP32 or FP64, natural order in and out:
//   X[k] = sum_n v[n] W_R^(n k),  W_R = e^(-2 pi i / R)   (INV: conjugate)
// for R with the prime factors 2, 3 and 5.  A composite R = A B is split as
// n = n1 + A n2, k = k2 + B k1: B-point DFTs over n2, twiddles W_R^(n1 k2),
// A-point DFTs over n1.  Every twiddle is a compile-time constant (sine and
// cosine from their Taylor series on [0, pi/4] after exact reduction of the
// rational angle), and the trivial ones (1, -1, +-i) cost no multiplication.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>
#include <utility>

namespace rism3d {
namespace dft {

template <int N, typename F, int... I>
__device__ __forceinline__ void sfor_seq(F &&f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
// f(integral_constant<int, 0>) ... f(integral_constant<int, N - 1>)
template <int N, typename F> __device__ __forceinline__ void sfor(F &&f) {
  sfor_seq<N>(f, std::make_integer_sequence<int, N>{});
}

constexpr double kTwoPi = 6.283185307179586476925286766559;
__host__ __device__ constexpr double taylor_sin(double x) {
  double t = x, s = x;
  for (int k = 1; k < 14; ++k) { t *= -x * x / ((2 * k) * (2 * k + 1)); s += t; }
  return s;
}
__host__ __device__ constexpr double taylor_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 14; ++k) { t *= -x * x / ((2 * k - 1) * (2 * k)); s += t; }
  return s;
}
// cos and sin of 2 pi m / r, 0 <= m < r, reduced to [0, pi/4]
__host__ __device__ constexpr double cos_frac(int m, int r) {
  if (2 * m > r) m = r - m;                       // cos(2pi - x) = cos x
  if (4 * m > r) return -cos_frac(r - 2 * m, 2 * r);   // cos(pi - x), kept rational
  return 8 * m > r ? taylor_sin(kTwoPi * (r - 4 * m) / (4.0 * r)) : taylor_cos(kTwoPi * m / r);
}
__host__ __device__ constexpr double sin_frac(int m, int r) {
  if (2 * m > r) return -sin_frac(r - m, r);
  if (4 * m > r) return sin_frac(r - 2 * m, 2 * r);
  return 8 * m > r ? taylor_cos(kTwoPi * (r - 4 * m) / (4.0 * r)) : taylor_sin(kTwoPi * m / r);
}

template <typename C> __device__ __forceinline__ C add(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <typename C> __device__ __forceinline__ C sub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <typename C> __device__ __forceinline__ C cmulc(C a, C b) {
  C r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
// a * w or a * conj(w)
template <bool INV, typename C> __device__ __forceinline__ C cmulw(C a, C w) {
  if (INV) w.y = -w.y;
  return cmulc(a, w);
}
// multiply by -i (forward) or +i (inverse)
template <bool INV, typename C> __device__ __forceinline__ C mul_mi(C a) {
  C r;
  r.x = INV ? -a.y : a.y;
  r.y = INV ? a.x : -a.x;
  return r;
}
// a * W_R^M (INV: conjugate root)
template <int M, int R, bool INV, typename C> __device__ __forceinline__ C mul_root(C a) {
  constexpr int m = M % R;
  if constexpr (m == 0) {
    return a;
  } else if constexpr (2 * m == R) {
    a.x = -a.x;
    a.y = -a.y;
    return a;
  } else if constexpr (4 * m == R) {
    return mul_mi<INV>(a);
  } else if constexpr (4 * m == 3 * R) {
    return mul_mi<!INV>(a);
  } else {
    typedef decltype(a.x) T;
    constexpr double c = cos_frac(m, R), s = sin_frac(m, R);
    C w;
    w.x = (T)c;
    w.y = INV ? (T)s : (T)-s;
    return cmulc(a, w);
  }
}

template <int R> struct Split;
template <> struct Split<6> { static constexpr int A = 2; };
template <> struct Split<8> { static constexpr int A = 2; };
template <> struct Split<9> { static constexpr int A = 3; };
template <> struct Split<10> { static constexpr int A = 2; };
template <> struct Split<12> { static constexpr int A = 3; };
template <> struct Split<15> { static constexpr int A = 3; };
template <> struct Split<16> { static constexpr int A = 4; };
template <> struct Split<18> { static constexpr int A = 2; };
template <> struct Split<20> { static constexpr int A = 4; };

template <int R, bool INV, typename C> __device__ __forceinline__ void run(C (&v)[R]) {
  typedef typename std::remove_reference<decltype(v[0].x)>::type T;
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const C a = add(v[0], v[1]);
    v[1] = sub(v[0], v[1]);
    v[0] = a;
  } else if constexpr (R == 3) {
    constexpr double s = sin_frac(1, 3);
    const C t = add(v[1], v[2]), d = mul_mi<INV>(sub(v[1], v[2]));
    C m;
    m.x = v[0].x - T(0.5) * t.x;
    m.y = v[0].y - T(0.5) * t.y;
    v[0] = add(v[0], t);
    v[1].x = m.x + (T)s * d.x;
    v[1].y = m.y + (T)s * d.y;
    v[2].x = m.x - (T)s * d.x;
    v[2].y = m.y - (T)s * d.y;
  } else if constexpr (R == 4) {
    const C s02 = add(v[0], v[2]), d02 = sub(v[0], v[2]);
    const C s13 = add(v[1], v[3]), d13 = mul_mi<INV>(sub(v[1], v[3]));
    v[0] = add(s02, s13);
    v[2] = sub(s02, s13);
    v[1] = add(d02, d13);
    v[3] = sub(d02, d13);
  } else if constexpr (R == 5) {
    constexpr double c1 = cos_frac(1, 5), c2 = cos_frac(2, 5), s1 = sin_frac(1, 5),
                     s2 = sin_frac(2, 5);
    const C a = add(v[1], v[4]), b = add(v[2], v[3]);
    const C p = mul_mi<INV>(sub(v[1], v[4])), q = mul_mi<INV>(sub(v[2], v[3]));
    C m1, m2, n1, n2;
    m1.x = v[0].x + (T)c1 * a.x + (T)c2 * b.x;
    m1.y = v[0].y + (T)c1 * a.y + (T)c2 * b.y;
    m2.x = v[0].x + (T)c2 * a.x + (T)c1 * b.x;
    m2.y = v[0].y + (T)c2 * a.y + (T)c1 * b.y;
    n1.x = (T)s1 * p.x + (T)s2 * q.x;
    n1.y = (T)s1 * p.y + (T)s2 * q.y;
    n2.x = (T)s2 * p.x - (T)s1 * q.x;
    n2.y = (T)s2 * p.y - (T)s1 * q.y;
    v[0] = add(v[0], add(a, b));
    v[1] = add(m1, n1);
    v[4] = sub(m1, n1);
    v[2] = add(m2, n2);
    v[3] = sub(m2, n2);
  } else {
    constexpr int A = Split<R>::A, B = R / A;
    C u[A][B];
    sfor<A>([&](auto n1c) {
      constexpr int n1 = decltype(n1c)::value;
      C t[B];
#pragma unroll
      for (int n2 = 0; n2 < B; ++n2) t[n2] = v[n1 + A * n2];
      run<B, INV>(t);
      sfor<B>([&](auto k2c) {
        constexpr int k2 = decltype(k2c)::value;
        u[n1][k2] = mul_root<n1 * k2, R, INV>(t[k2]);
      });
    });
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) {
      C t[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) t[n1] = u[n1][k2];
      run<A, INV>(t);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) v[k2 + B * k1] = t[k1];
    }
  }
}

}  // namespace dft
}  // namespace rism3d
