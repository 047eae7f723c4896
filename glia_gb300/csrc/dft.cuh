// dft.cuh — small DFTs in registers, of doubles and of 64-bit fixed-point values (fx.cuh).
//
// X[k] = sum_j v[j] exp(S 2 pi i j k / R), natural order in and out, R = 2 ... 16. Powers of two are
// radix-4 butterflies (the factors +-i and -1 are sign changes and swaps, never multiplications);
// R = A B with coprime A, B is the prime-factor mapping of Good and Thomas (no twiddles between the
// two parts); 9 = 3 x 3 has twiddles; odd primes use the symmetric sums x[j] +- x[p - j].
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace glia {

template <class C>
struct CReal;
struct fx2;  // fx.cuh: 64-bit fixed point
template <int N, int S, int E>
__host__ __device__ __forceinline__ fx2 ctw_fx(fx2 z);
template <int R, int S>
__host__ __device__ __forceinline__ void odd_dft_fx(fx2 (&v)[R]);
template <>
struct CReal<double2> {
  using type = double;
};
template <class C>
using creal_t = typename CReal<C>::type;

template <class C>
__host__ __device__ __forceinline__ C cmk(creal_t<C> x, creal_t<C> y) {
  C c;
  c.x = x;
  c.y = y;
  return c;
}
template <class C>
__host__ __device__ __forceinline__ C cadd(C a, C b) {
  return cmk<C>(a.x + b.x, a.y + b.y);
}
template <class C>
__host__ __device__ __forceinline__ C csub(C a, C b) {
  return cmk<C>(a.x - b.x, a.y - b.y);
}
template <class C>
__host__ __device__ __forceinline__ C cmul2(C a, C b) {
  return cmk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// i w a
template <class C>
__host__ __device__ __forceinline__ C cimul(creal_t<C> w, C a) {
  return cmk<C>(-w * a.y, w * a.x);
}

// cos(2 pi e / N) and sin(2 pi e / N), rounded once from 40 digits, e <= N / 2
template <int N>
__host__ __device__ constexpr double cos_half(int e) {
  static_assert(N == 3 || N == 5 || N == 7 || N == 9 || N == 11 || N == 13 || N == 16, "table");
  constexpr double t3[] = {1.0, -0.5};
  constexpr double t5[] = {1.0, 0.30901699437494745, -0.8090169943749475};
  constexpr double t7[] = {1.0, 0.6234898018587335, -0.2225209339563144, -0.9009688679024191};
  constexpr double t9[] = {1.0, 0.766044443118978, 0.17364817766693036, -0.5,
                           -0.9396926207859084};
  constexpr double t11[] = {1.0,
                            0.8412535328311812,
                            0.41541501300188644,
                            -0.14231483827328514,
                            -0.6548607339452851,
                            -0.9594929736144974};
  constexpr double t13[] = {1.0,
                            0.8854560256532099,
                            0.5680647467311558,
                            0.12053668025532305,
                            -0.3546048870425356,
                            -0.7485107481711011,
                            -0.970941817426052};
  constexpr double t16[] = {1.0,
                            0.9238795325112867,
                            0.7071067811865476,
                            0.3826834323650898,
                            0.0,
                            -0.3826834323650898,
                            -0.7071067811865476,
                            -0.9238795325112867,
                            -1.0};
  return N == 3 ? t3[e] : N == 5 ? t5[e] : N == 7 ? t7[e] : N == 9 ? t9[e]
         : N == 11 ? t11[e] : N == 13 ? t13[e] : t16[e];
}
template <int N>
__host__ __device__ constexpr double sin_half(int e) {
  constexpr double t3[] = {0.0, 0.8660254037844386};
  constexpr double t5[] = {0.0, 0.9510565162951535, 0.5877852522924731};
  constexpr double t7[] = {0.0, 0.7818314824680298, 0.9749279121818236, 0.4338837391175581};
  constexpr double t9[] = {0.0, 0.6427876096865394, 0.984807753012208, 0.8660254037844386,
                           0.3420201433256687};
  constexpr double t11[] = {0.0,
                            0.5406408174555976,
                            0.9096319953545183,
                            0.9898214418809327,
                            0.7557495743542583,
                            0.28173255684142967};
  constexpr double t13[] = {0.0,
                            0.46472317204376856,
                            0.8229838658936564,
                            0.992708874098054,
                            0.9350162426854148,
                            0.6631226582407952,
                            0.23931566428755777};
  constexpr double t16[] = {0.0,
                            0.3826834323650898,
                            0.7071067811865476,
                            0.9238795325112867,
                            1.0,
                            0.9238795325112867,
                            0.7071067811865476,
                            0.3826834323650898,
                            0.0};
  return N == 3 ? t3[e] : N == 5 ? t5[e] : N == 7 ? t7[e] : N == 9 ? t9[e]
         : N == 11 ? t11[e] : N == 13 ? t13[e] : t16[e];
}
template <int N>
__host__ __device__ constexpr double cos_n(int e) {
  e = ((e % N) + N) % N;
  return e <= N / 2 ? cos_half<N>(e) : cos_half<N>(N - e);
}
template <int N>
__host__ __device__ constexpr double sin_n(int e) {
  e = ((e % N) + N) % N;
  return e <= N / 2 ? sin_half<N>(e) : -sin_half<N>(N - e);
}

// exp(S 2 pi i E / N) z for compile-time E
template <int N, int S, int E, class C>
__host__ __device__ __forceinline__ C ctw(C z) {
  using T = creal_t<C>;
  constexpr int e = ((E % N) + N) % N;
  if constexpr (std::is_same<C, fx2>::value) {
    return ctw_fx<N, S, E>(z);
  } else if constexpr (e == 0) {
    return z;
  } else if constexpr (4 * e == N) {
    return cmk<C>(-S * z.y, S * z.x);
  } else if constexpr (2 * e == N) {
    return cmk<C>(-z.x, -z.y);
  } else if constexpr (4 * e == 3 * N) {
    return cmk<C>(S * z.y, -S * z.x);
  } else {
    constexpr T wc = (T)cos_n<N>(e), ws = (T)(S * sin_n<N>(e));
    return cmk<C>(z.x * wc - z.y * ws, z.x * ws + z.y * wc);
  }
}

template <int S, class C>
__host__ __device__ __forceinline__ void dft4(C& a0, C& a1, C& a2, C& a3) {
  const C t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = csub(a1, a3);
  a0 = cadd(t0, t2);
  a2 = csub(t0, t2);
  a1 = cmk<C>(t1.x - S * t3.y, t1.y + S * t3.x);  // t1 + S i t3
  a3 = cmk<C>(t1.x + S * t3.y, t1.y - S * t3.x);  // t1 - S i t3
}

template <int R>
__host__ __device__ constexpr int coprime_factor() {  // A of R = A B with coprime A, B (1: none)
  return R == 6 ? 3 : R == 10 ? 5 : R == 12 ? 4 : R == 14 ? 7 : R == 15 ? 5 : 1;
}
__host__ __device__ constexpr int inverse_mod(int a, int m) {
  for (int i = 1; i < m; i++)
    if (a * i % m == 1) return i;
  return 0;
}

template <int R, int S, class C>
__host__ __device__ __forceinline__ void reg_dft(C (&v)[R]) {
  using T = creal_t<C>;
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const C a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  } else if constexpr (R == 4) {
    dft4<S>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    // decimation in time: X[k] = E[k] + W^k O[k], X[k + 4] = E[k] - W^k O[k], W = w_16^2
    C e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    C o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<S>(e0, e1, e2, e3);
    dft4<S>(o0, o1, o2, o3);
    o1 = ctw<16, S, 2>(o1);
    o2 = ctw<16, S, 4>(o2);
    o3 = ctw<16, S, 6>(o3);
    v[0] = cadd(e0, o0);
    v[4] = csub(e0, o0);
    v[1] = cadd(e1, o1);
    v[5] = csub(e1, o1);
    v[2] = cadd(e2, o2);
    v[6] = csub(e2, o2);
    v[3] = cadd(e3, o3);
    v[7] = csub(e3, o3);
  } else if constexpr (R == 16) {
    // 4 x 4: j = 4 j1 + j2; DFT over j1, twiddle w_16^(j2 k1), DFT over j2; k = k1 + 4 k2
    dft4<S>(v[0], v[4], v[8], v[12]);
    dft4<S>(v[1], v[5], v[9], v[13]);
    dft4<S>(v[2], v[6], v[10], v[14]);
    dft4<S>(v[3], v[7], v[11], v[15]);
    v[5] = ctw<16, S, 1>(v[5]);
    v[6] = ctw<16, S, 2>(v[6]);
    v[7] = ctw<16, S, 3>(v[7]);
    v[9] = ctw<16, S, 2>(v[9]);
    v[10] = ctw<16, S, 4>(v[10]);
    v[11] = ctw<16, S, 6>(v[11]);
    v[13] = ctw<16, S, 3>(v[13]);
    v[14] = ctw<16, S, 6>(v[14]);
    v[15] = ctw<16, S, 9>(v[15]);
    dft4<S>(v[0], v[1], v[2], v[3]);
    dft4<S>(v[4], v[5], v[6], v[7]);
    dft4<S>(v[8], v[9], v[10], v[11]);
    dft4<S>(v[12], v[13], v[14], v[15]);
    // v[4 k1 + k2] holds X[k1 + 4 k2]: transpose to natural order
    C t[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++)
#pragma unroll
      for (int k2 = 0; k2 < 4; k2++) t[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = t[i];
  } else if constexpr (R == 9) {
    C a[3], b[3], c[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      a[j] = v[3 * j];
      b[j] = v[3 * j + 1];
      c[j] = v[3 * j + 2];
    }
    reg_dft<3, S>(a);
    reg_dft<3, S>(b);
    reg_dft<3, S>(c);
    b[1] = ctw<9, S, 1>(b[1]);
    b[2] = ctw<9, S, 2>(b[2]);
    c[1] = ctw<9, S, 2>(c[1]);
    c[2] = ctw<9, S, 4>(c[2]);
#pragma unroll
    for (int k = 0; k < 3; k++) {
      C t[3] = {a[k], b[k], c[k]};
      reg_dft<3, S>(t);
#pragma unroll
      for (int m = 0; m < 3; m++) v[k + 3 * m] = t[m];
    }
  } else if constexpr (coprime_factor<R>() > 1) {
    // j = (B j1 + A j2) mod R, k = k1 mod A = k2 mod B
    constexpr int A = coprime_factor<R>(), B = R / A;
    constexpr int ka = B * inverse_mod(B % A, A), kb = A * (B == 2 ? 1 : inverse_mod(A % B, B));
    C t[A][B];
#pragma unroll
    for (int j2 = 0; j2 < B; j2++) {
      C a[A];
#pragma unroll
      for (int j1 = 0; j1 < A; j1++) a[j1] = v[(B * j1 + A * j2) % R];
      reg_dft<A, S>(a);
#pragma unroll
      for (int k1 = 0; k1 < A; k1++) t[k1][j2] = a[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; k1++) {
      reg_dft<B, S>(t[k1]);
#pragma unroll
      for (int k2 = 0; k2 < B; k2++) v[(ka * k1 + kb * k2) % R] = t[k1][k2];
    }
  } else if constexpr (std::is_same<C, fx2>::value) {
    odd_dft_fx<R, S>(v);
  } else {
    static_assert(R == 3 || R == 5 || R == 7 || R == 11 || R == 13, "register DFT size");
    constexpr int H = R / 2;
    const C x0 = v[0];
    C p[H], m[H];
#pragma unroll
    for (int j = 0; j < H; j++) {
      p[j] = cadd(v[j + 1], v[R - 1 - j]);
      m[j] = csub(v[j + 1], v[R - 1 - j]);
    }
#pragma unroll
    for (int j = 0; j < H; j++) v[0] = cadd(v[0], p[j]);
#pragma unroll
    for (int k = 1; k <= H; k++) {
      C a = x0, b = cmk<C>(T(0), T(0));
#pragma unroll
      for (int j = 1; j <= H; j++) {
        const T c = (T)cos_n<R>(j * k), s = (T)(S * sin_n<R>(j * k));
        a.x += c * p[j - 1].x;
        a.y += c * p[j - 1].y;
        b.x += s * m[j - 1].x;
        b.y += s * m[j - 1].y;
      }
      v[k] = cmk<C>(a.x - b.y, a.y + b.x);  // a + i b
      v[R - k] = cmk<C>(a.x + b.y, a.y - b.x);
    }
  }
}

}  // namespace glia
