// pdt_cfft.cuh -- DFTs of compile-time length in one thread's registers with compile-time roots.
//
// cfft<N, S>(x): in-place DFT of x[0..N) with sign S (-1 forward, +1 inverse, unscaled), natural order in
// and out. Unlike reg_fft (pdt_regfft.cuh), which reads its roots from a table in shared memory, every root
// is a constant expression (immediate operands): no loads, no registers held by roots.
// N = P Q is split decimation-in-time with P = 4, 2 or the smallest odd prime; primes above 5 use the
// symmetric direct DFT X[k], X[P-k] = x0 + sum_j (x_j + x_{P-j}) cos(2 pi jk/P) +- S i sum_j (x_j - x_{P-j})
// sin(2 pi jk/P).
#pragma once

#include <type_traits>

#include "pdt_device.cuh"
#include "pdt_regfft.cuh"

namespace pdt {

// cos / sin of 2 pi m / n in double precision: the Taylor series on the angle reduced to [-pi, pi]
constexpr double ct_angle(int m, int n) {
  m %= n;
  if (m < 0) m += n;
  if (2 * m > n) m -= n;
  return 2.0 * 3.14159265358979323846 * m / n;
}
constexpr double ct_series(double x, int first) {  // first = 0: cos, 1: sin
  double term = first ? x : 1.0, sum = term;
  for (int k = first + 1; k < 40; k += 2) {
    term *= -x * x / (k * (k + 1));
    sum += term;
  }
  return sum;
}
constexpr float ct_cos(int m, int n) { return (float)ct_series(ct_angle(m, n), 0); }
constexpr float ct_sin(int m, int n) { return (float)ct_series(ct_angle(m, n), 1); }

// f(integral_constant<int, B>), ..., f(integral_constant<int, E - 1>)
template <int B, int E, class F>
__host__ __device__ __forceinline__ void static_for(F&& f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    static_for<B + 1, E>(f);
  }
}

// Complex sums as packed FP32 pairs (add / fma .f32x2, round to nearest: the same values as two scalar
// operations in half the issue slots; the transforms share their issue slots with the shared-memory traffic).
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __ffma2_rn(b, c2(-1.f, -1.f), a); }
// S i (a - b)
template <int S>
__device__ __forceinline__ float2 psub_i(float2 a, float2 b) {
  return S > 0 ? c2(b.y - a.y, a.x - b.x) : c2(a.y - b.y, b.x - a.x);
}

template <int S>
__device__ __forceinline__ void cdft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 t0 = padd(a0, a2), t1 = psub(a0, a2), t2 = padd(a1, a3), t3 = psub_i<S>(a1, a3);
  a0 = padd(t0, t2);
  a2 = psub(t0, t2);
  a1 = padd(t1, t3);
  a3 = psub(t1, t3);
}

// v * exp(S 2 pi i M / N)
template <int M, int N, int S>
__device__ __forceinline__ float2 ct_rot(float2 v) {
  constexpr int m = M % N;
  if constexpr (m == 0) {
    return v;
  } else if constexpr (2 * m == N) {
    return -v;
  } else if constexpr (4 * m == N) {
    return mul_si(v, (float)S);
  } else if constexpr (4 * m == 3 * N) {
    return mul_si(v, (float)-S);
  } else {
    constexpr float c = ct_cos(m, N), s = S * ct_sin(m, N);
    return c2(v.x * c - v.y * s, v.x * s + v.y * c);
  }
}

// Symmetric direct DFT of odd prime length P; out(k, X[k]) is called for every output as soon as it is
// ready, so that a caller that stores the outputs does not hold both arrays.
template <int P, int S, class Out>
__device__ __forceinline__ void cdft_prime(const float2 (&x)[P], Out&& out) {
  constexpr int Hh = (P - 1) / 2;
  float2 t[Hh], d[Hh];
  const float2 x0 = x[0];
  float2 sum = x0;
#pragma unroll
  for (int j = 1; j <= Hh; ++j) {
    t[j - 1] = padd(x[j], x[P - j]);
    d[j - 1] = psub(x[j], x[P - j]);
    sum = padd(sum, t[j - 1]);
  }
  out(std::integral_constant<int, 0>{}, sum);
  static_for<1, Hh + 1>([&](auto K) {
    constexpr int k = decltype(K)::value;
    float2 A = x0, B = c2(0.f, 0.f);
    static_for<1, Hh + 1>([&](auto J) {
      constexpr int j = decltype(J)::value;
      constexpr float cv = ct_cos(j * k, P), sv = ct_sin(j * k, P);
      A = __ffma2_rn(c2(cv, cv), t[j - 1], A);
      B = j == 1 ? __fmul2_rn(c2(sv, sv), d[j - 1]) : __ffma2_rn(c2(sv, sv), d[j - 1], B);
    });
    out(std::integral_constant<int, k>{}, S > 0 ? c2(A.x - B.y, A.y + B.x) : c2(A.x + B.y, A.y - B.x));
    out(std::integral_constant<int, P - k>{}, S > 0 ? c2(A.x + B.y, A.y - B.x) : c2(A.x - B.y, A.y + B.x));
  });
}

template <int N, int S>
__device__ __forceinline__ void cfft(float2 (&x)[N]);

// out(k, X[k]) for every output of the DFT of x
template <int N, int S, class Out>
__device__ __forceinline__ void cfft_out(float2 (&x)[N], Out&& out) {
  if constexpr (N > 5 && ct_split(N) == N && !ct_is_base(N)) {
    cdft_prime<N, S>(x, out);
  } else {
    cfft<N, S>(x);
    static_for<0, N>([&](auto K) { out(K, x[decltype(K)::value]); });
  }
}

template <int N, int S>
__device__ __forceinline__ void cfft(float2 (&x)[N]) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2) {
    const float2 t = x[0];
    x[0] = padd(t, x[1]);
    x[1] = psub(t, x[1]);
  } else if constexpr (N == 3) {
    dft3(x, (float)S);
  } else if constexpr (N == 4) {
    cdft4<S>(x[0], x[1], x[2], x[3]);
  } else if constexpr (N == 5) {
    dft5(x, (float)S);
  } else if constexpr (N == 8) {
    float2 e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6], o0 = x[1], o1 = x[3], o2 = x[5], o3 = x[7];
    cdft4<S>(e0, e1, e2, e3);
    cdft4<S>(o0, o1, o2, o3);
    o1 = ct_rot<1, 8, S>(o1);
    o2 = ct_rot<2, 8, S>(o2);
    o3 = ct_rot<3, 8, S>(o3);
    x[0] = padd(e0, o0);
    x[4] = psub(e0, o0);
    x[1] = padd(e1, o1);
    x[5] = psub(e1, o1);
    x[2] = padd(e2, o2);
    x[6] = psub(e2, o2);
    x[3] = padd(e3, o3);
    x[7] = psub(e3, o3);
  } else if constexpr (ct_split(N) == N) {
    float2 y[N];
    cdft_prime<N, S>(x, [&](auto K, float2 v) { y[decltype(K)::value] = v; });
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = y[i];
  } else {
    constexpr int P = ct_split(N), Q = N / P;
    float2 y[P][Q];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int q = 0; q < Q; ++q) y[p][q] = x[p + P * q];
#pragma unroll
    for (int p = 0; p < P; ++p) cfft<Q, S>(y[p]);
    static_for<0, Q>([&](auto K1) {
      constexpr int k1 = decltype(K1)::value;
      float2 z[P];
      static_for<0, P>([&](auto Pp) {
        constexpr int p = decltype(Pp)::value;
        z[p] = ct_rot<p * k1, N, S>(y[p][k1]);
      });
      cfft<P, S>(z);
#pragma unroll
      for (int k2 = 0; k2 < P; ++k2) x[k1 + Q * k2] = z[k2];
    });
  }
}

}  // namespace pdt
