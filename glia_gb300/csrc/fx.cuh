// fx.cuh — DFTs of doubles in 64-bit integers.
//
// Measured on GB300, per clock and SM: FP64 add, multiply or FMA 1.7 (64 clocks per warp
// instruction in each sub-partition), 64-bit integer add 58, the upper half of a 64 x 64-bit
// product 6, conversions between FP64 and any other type 2. A DFT of R values is therefore taken
// in block fixed point: the R inputs are aligned to the largest exponent among them, with
// log2 R + 2 bits of headroom (57 bits of magnitude at R = 16, where a double has 53), and the
// butterflies run on integers. Between two DFTs of the same phase the values stay integers with an
// exponent (memory blocks, below); doubles are made only where a phase needs them: 182 -> about 80
// instructions per value and DFT, solve at 128^3 1.48 -> 1.0 ms.
//
// No precision is given up. A butterfly in FP64 rounds to 53 bits at every step, this keeps 57
// below a block's largest value. Against long double, root mean square of the error relative to the
// result: a 16-point DFT rounded to doubles 5.3e-17 (FP64 arithmetic 1.0e-16); D apply at 32^3 of
// white noise 2.2e-16 (cuFFT's FP64 transforms 5.0e-16), of a smooth field 7.9e-15 (2.5e-14); six
// steps of a simulation at 16^3 7.6e-16 (1.8e-15), at 24^3 1.7e-15 (2.2e-15). Fifty trips to the
// spectrum and back change a smooth field's amplitude by 1e-20 to 4e-18 each (1e-16 to 3e-16 with
// cuFFT): what rounding down takes away is given back (fx_transform), and a factor 1 is not a
// multiplication.
//
// A block whose largest magnitude is below 2^-952 is taken as zero; one that holds a NaN, an
// infinity or a magnitude above 2^1017 gives NaN.
#pragma once

#include "dft.cuh"

#include <cstdint>
#include <cstring>

namespace glia {

#define GLIA_HD __host__ __device__ __forceinline__

struct __align__(16) fx2 {
  int64_t x, y;
};
template <>
struct CReal<fx2> {
  using type = int64_t;
};

// a factor of magnitude at most 1 as 2^63 times its value: high word, low word >> 1
struct Fc {
  int32_t h, l;
};
GLIA_HD constexpr Fc fx_split(int64_t v) {
  return Fc{(int32_t)(v >> 32), (int32_t)((uint32_t)v >> 1)};
}
// cos and sin of 2 pi e / N times 2^63, e <= N / 2, rounded from 50 digits
template <int N>
__host__ __device__ constexpr int64_t fx_cos_half(int e) {
    constexpr int64_t t3[] = {9223372036854775807ll, -4611686018427387904ll};
    constexpr int64_t t5[] = {9223372036854775807ll, 2850178704830799621ll,
                             -7461864723258187525ll};
    constexpr int64_t t7[] = {9223372036854775807ll, 5750678403727967667ll,
                             -2052393359867478633ll, -8309971062287876938ll};
    constexpr int64_t t9[] = {9223372036854775807ll, 7065512895651570889ll,
                             1601621746143955363ll, -4611686018427387904ll,
                             -8667134641795526252ll};
    constexpr int64_t t11[] = {9223372036854775807ll, 7759194310620407470ll,
                             3831527214611262376ll, -1312622699759327971ll,
                             -6040024181505137327ll, -8849760662394592452ll};
    constexpr int64_t t13[] = {9223372036854775807ll, 8166890346874381177ll,
                             5239472500123132842ll, 1111754646082251829ll,
                             -3270652799280169514ll, -6903793103966580896ll,
                             -8955357608260403342ll};
    constexpr int64_t t16[] = {9223372036854775807ll, 8521284645587064995ll,
                             6521908912666391106ll, 3529631669043774883ll, 0ll,
                             -3529631669043774883ll, -6521908912666391106ll,
                             -8521284645587064995ll, -9223372036854775807ll};
  return N == 3 ? t3[e] : N == 5 ? t5[e] : N == 7 ? t7[e] : N == 9 ? t9[e]
         : N == 11 ? t11[e] : N == 13 ? t13[e] : t16[e];
}
template <int N>
__host__ __device__ constexpr int64_t fx_sin_half(int e) {
    constexpr int64_t t3[] = {0ll, 7987674492471257551ll};
    constexpr int64_t t5[] = {0ll, 8771948077865237882ll, 5421362059670026167ll};
    constexpr int64_t t7[] = {0ll, 7211122632928341039ll, 8992122843167040398ll,
                             4001871146622878209ll};
    constexpr int64_t t9[] = {0ll, 5928669264819548846ll, 9083248290810584424ll,
                             7987674492471257551ll, 3154579025991035578ll};
    constexpr int64_t t11[] = {0ll, 4986531397702266102ll, 8389874309781278077ll,
                             9129491408523869628ll, 6970559490963965065ll,
                             2598524186642841334ll};
    constexpr int64_t t13[] = {0ll, 4286314709906945897ll, 7590686375466191238ll,
                             9156123270093579449ll, 8624002666789673892ll,
                             6116226983022956630ll, 2207297405971185413ll};
    constexpr int64_t t16[] = {0ll, 3529631669043774883ll, 6521908912666391106ll,
                             8521284645587064995ll, 9223372036854775807ll,
                             8521284645587064995ll, 6521908912666391106ll,
                             3529631669043774883ll, 0ll};
  return N == 3 ? t3[e] : N == 5 ? t5[e] : N == 7 ? t7[e] : N == 9 ? t9[e]
         : N == 11 ? t11[e] : N == 13 ? t13[e] : t16[e];
}
template <int N>
GLIA_HD constexpr Fc fx_cos(int e) {
  e = ((e % N) + N) % N;
  return fx_split(e <= N / 2 ? fx_cos_half<N>(e) : fx_cos_half<N>(N - e));
}
template <int N, int S>
GLIA_HD constexpr Fc fx_sin(int e) {
  e = ((e % N) + N) % N;
  return fx_split(e <= N / 2 ? S * fx_sin_half<N>(e) : -S * fx_sin_half<N>(N - e));
}
// host: a factor from a long double, |c| <= 1
inline Fc fx_from(long double c) {
  const long double v = c * 9223372036854775808.0L;
  return fx_split(v >= 9223372036854775807.0L    ? INT64_MAX
                  : v <= -9223372036854775807.0L ? -INT64_MAX
                                                 : (int64_t)(v < 0 ? v - 0.5L : v + 0.5L));
}
GLIA_HD int32_t fx_mulhi(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
// a c / 2 from the three upper partial products; the + 1 (two units) takes out what their two
// floors lose on average
GLIA_HD int64_t fx_mulh(int64_t a, Fc c) {
  const int32_t ah = (int32_t)(a >> 32), al = (int32_t)((uint32_t)a >> 1);
  const int32_t t = fx_mulhi(ah, c.l) + fx_mulhi(al, c.h) + 1;
  const int64_t p = (int64_t)(((uint64_t)(uint32_t)fx_mulhi(ah, c.h) << 32) |
                              (uint32_t)((uint32_t)ah * (uint32_t)c.h));
  return p + 2 * (int64_t)t;
}
GLIA_HD int64_t fx_mul(int64_t a, Fc c) { return 2 * fx_mulh(a, c); }

// exp(S 2 pi i E / N) z for compile-time E
template <int N, int S, int E>
GLIA_HD fx2 ctw_fx(fx2 z) {
  constexpr int e = ((E % N) + N) % N;
  if constexpr (e == 0) {
    return z;
  } else if constexpr (4 * e == N) {
    return cmk<fx2>(-S * z.y, S * z.x);
  } else if constexpr (2 * e == N) {
    return cmk<fx2>(-z.x, -z.y);
  } else if constexpr (4 * e == 3 * N) {
    return cmk<fx2>(S * z.y, -S * z.x);
  } else if constexpr ((8 * e) % N == 0) {  // cos = +- sin = +- sqrt(1/2)
    constexpr int sc = cos_n<N>(e) > 0 ? 1 : -1, ss = S * (sin_n<N>(e) > 0 ? 1 : -1);
    constexpr Fc r = fx_cos<16>(2);
    return cmk<fx2>(fx_mul(sc * z.x - ss * z.y, r), fx_mul(ss * z.x + sc * z.y, r));
  } else {
    constexpr Fc c = fx_cos<N>(e), s = fx_sin<N, S>(e);
    return cmk<fx2>(2 * (fx_mulh(z.x, c) - fx_mulh(z.y, s)),
                    2 * (fx_mulh(z.x, s) + fx_mulh(z.y, c)));
  }
}

template <int R, int S>
GLIA_HD void odd_dft_fx(fx2 (&v)[R]) {
  constexpr int H = R / 2;
  const fx2 x0 = v[0];
  fx2 p[H], m[H];
#pragma unroll
  for (int j = 0; j < H; j++) {
    p[j] = cadd(v[j + 1], v[R - 1 - j]);
    m[j] = csub(v[j + 1], v[R - 1 - j]);
  }
#pragma unroll
  for (int j = 0; j < H; j++) v[0] = cadd(v[0], p[j]);
#pragma unroll
  for (int k = 1; k <= H; k++) {
    fx2 a = cmk<fx2>(0, 0), b = cmk<fx2>(0, 0);
#pragma unroll
    for (int j = 1; j <= H; j++) {
      const Fc c = fx_cos<R>(j * k), s = fx_sin<R, S>(j * k);
      a.x += fx_mulh(p[j - 1].x, c);
      a.y += fx_mulh(p[j - 1].y, c);
      b.x += fx_mulh(m[j - 1].x, s);
      b.y += fx_mulh(m[j - 1].y, s);
    }
    a = cmk<fx2>(x0.x + 2 * a.x, x0.y + 2 * a.y);
    v[k] = cmk<fx2>(a.x - 2 * b.y, a.y + 2 * b.x);  // a + i b
    v[R - k] = cmk<fx2>(a.x + 2 * b.y, a.y - 2 * b.x);
  }
}

// twiddle factor of a table: cos and sin as Fc
struct __align__(16) FxTw {
  Fc c, s;
};
// z w / 2
GLIA_HD fx2 fx_tw(fx2 z, FxTw w) {
  return cmk<fx2>(fx_mulh(z.x, w.c) - fx_mulh(z.y, w.s), fx_mulh(z.x, w.s) + fx_mulh(z.y, w.c));
}

// ---- doubles in and out of a block ---------------------------------------------------------
GLIA_HD uint32_t fx_hi(double d) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2hiint(d);
#else
  uint64_t b;
  memcpy(&b, &d, 8);
  return (uint32_t)(b >> 32);
#endif
}
GLIA_HD uint32_t fx_lo(double d) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2loint(d);
#else
  uint64_t b;
  memcpy(&b, &d, 8);
  return (uint32_t)b;
#endif
}
GLIA_HD double fx_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  memcpy(&d, &b, 8);
  return d;
#endif
}
GLIA_HD uint32_t fx_max(uint32_t a, uint32_t b) { return a > b ? a : b; }
GLIA_HD uint32_t fx_min(uint32_t a, uint32_t b) { return a < b ? a : b; }
GLIA_HD int fx_clz(uint64_t a) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
// running maximum of |re|, |im| (their high words)
GLIA_HD uint32_t fx_mag(uint32_t m, double2 z) {
  return fx_max(m, fx_max(fx_hi(z.x) & 0x7fffffffu, fx_hi(z.y) & 0x7fffffffu));
}
// d 2^(1022 - E + B) as an integer, |d| < 2^(E - 1022)
template <int B>
GLIA_HD int64_t fx_in(double d, int E) {
  static_assert(B >= 53 && B <= 62, "block bits");
  const uint32_t hi = fx_hi(d);
  const uint32_t sh = fx_min((uint32_t)(E - (int)((hi >> 20) & 0x7ff)), 63u);
  const uint64_t m =
      ((((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | fx_lo(d)) << (B - 53)) >> sh;
  const int64_t s = (int64_t)((int32_t)hi >> 31);
  return ((int64_t)m ^ s) - s;
}
// the same times w, 0 <= w < 128, for |d w| < 2^(E - 1022): E covers the exponent of d plus
// fx_wbits(w) wherever w is not zero
template <int B>
GLIA_HD int64_t fx_in_w(double d, int E, int w) {
  const uint32_t hi = fx_hi(d);
  const uint32_t sh = fx_min((uint32_t)(E - (int)((hi >> 20) & 0x7ff) - (B - 56)), 63u);
  const uint64_t m = ((((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | fx_lo(d)) *
                      (uint64_t)(uint32_t)w << 3) >> sh;
  const int64_t s = (int64_t)((int32_t)hi >> 31);
  return ((int64_t)m ^ s) - s;
}
// bits that w adds to the exponent in fx_in_w: at least B - 56, so that the shift is not negative
template <int B>
GLIA_HD int fx_wbits(int w) {
#ifdef __CUDA_ARCH__
  const int b = 32 - __clz(w);
#else
  const int b = w ? 32 - __builtin_clz((unsigned)w) : 0;
#endif
  return b > B - 56 ? b : (B > 56 ? B - 56 : 0);
}
// v 2^(E - 1022 - B + adj) as a double
GLIA_HD double fx_out(int64_t v, int field0) {  // field0 = E + 64 - B + adj
  const int64_t s = v >> 63;
  uint64_t a = (uint64_t)((v ^ s) - s);
  const int z = fx_clz(a);
  a <<= (z & 63);
  const uint64_t bits = (a >> 11) + ((a >> 10) & 1) + ((uint64_t)(uint32_t)(field0 - 1 - z) << 52);
  return a ? fx_bits(bits | ((uint64_t)s & 0x8000000000000000ull)) : 0.0;
}
enum { kFxTiny = 70, kFxHuge = 2040 };
GLIA_HD double fx_nan() { return fx_bits(0x7ff8000000000000ull); }

// log2 R rounded so that R sqrt(2) 2^(62 - fx_log2(R)) < 2^63: a result's modulus stays in range
GLIA_HD constexpr int fx_log2(int r) {
  return r <= 1 ? 0 : r <= 2 ? 1 : r <= 5 ? 2 : r <= 11 ? 3 : 4;
}

// Bits of a task's block: one more of headroom for the sums of a task (pairs, two inputs), and 58
// at most (fx_get_iw; the shift into a block drops 5 of the exponent's 6 bits, the sixth is 2^-58
// of the block's largest value).
GLIA_HD constexpr int fx_block_bits(int r) { return 61 - fx_log2(r) < 58 ? 61 - fx_log2(r) : 58; }

// results of a block: v 2^(-extra) with the block exponent E of B-bit inputs
template <int R, int B>
GLIA_HD void fx_store(const fx2 (&q)[R], double2 (&v)[R], int E, int adj) {
  if (E < kFxTiny || E > kFxHuge) {
    const double d = E > kFxHuge ? fx_nan() : 0.0;
#pragma unroll
    for (int i = 0; i < R; i++) v[i] = cmk<double2>(d, d);
    return;
  }
  const int field0 = E + 64 - B + adj;
#pragma unroll
  for (int i = 0; i < R; i++)
    v[i] = cmk<double2>(fx_out(q[i].x, field0), fx_out(q[i].y, field0));
}
template <int R>
GLIA_HD int fx_block(const double2 (&v)[R]) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < R; i++) m = fx_mag(m, v[i]);
  return (int)(m >> 20);
}

// ---- blocks in memory ----------------------------------------------------------------------
// Between tasks a complex value stays in fixed point: value = v 2^(e - 1022 - 63), |v| < 2^63, the
// exponent e (12 bits, one for all results of a task) in the low 6 bits of re (upper half) and im
// (lower half). The results of a task are shifted up together until the largest fills the word,
// so 57 bits below the block's largest value are kept. e = kFxBad marks NaN or overflow.
enum { kFxBad = 4095 };
GLIA_HD int fx_e(fx2 v) { return (((int)v.x & 63) << 6) | ((int)v.y & 63); }
GLIA_HD fx2 fx_with_e(fx2 v, int e) {
  return cmk<fx2>((v.x & ~(int64_t)63) | (e >> 6), (v.y & ~(int64_t)63) | (e & 63));
}
template <int B>
GLIA_HD int fx_shift(int E, int e) {  // right shift that brings exponent e to a block E of B bits
  return (int)fx_min((uint32_t)(E - e + 63 - B), 63u);
}
// rounds down: half a unit low on average (fx_transform makes up for it)
template <int B>
GLIA_HD fx2 fx_get(fx2 v, int E, int e) {
  const int s = fx_shift<B>(E, e);
  return cmk<fx2>(v.x >> s, v.y >> s);
}
// i w v, |w| < 128, E at least e plus the bits of w
template <int B>
GLIA_HD fx2 fx_get_iw(fx2 v, int E, int e, int w) {
  static_assert(B <= 58, "the product is shifted by 7 less");
  const int s = (int)fx_min((uint32_t)(E - e + 56 - B), 63u);
  const int64_t x = ((v.x >> 7) * w) >> s, y = ((v.y >> 7) * w) >> s;
  return cmk<fx2>(-y, x);
}
// exponent of w v (0 for w = 0), at least two above v's, so that the shift is not negative
GLIA_HD int fx_e_w(int e, int w) {
  const int a = (w < 0 ? -w : w) | 2;
#ifdef __CUDA_ARCH__
  return w == 0 ? 0 : e + 32 - __clz(a);
#else
  return w == 0 ? 0 : e + 32 - __builtin_clz((unsigned)a);
#endif
}
// results q 2^(E - 1022 - B + adj) as memory blocks
template <int R, int B>
GLIA_HD void fx_put(fx2 (&q)[R], int E, int adj) {
  uint32_t m = 1;
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int32_t a = (int32_t)(q[i].x >> 32), b = (int32_t)(q[i].y >> 32);
    m |= (uint32_t)(a ^ (a >> 31)) | (uint32_t)(b ^ (b >> 31));
  }
#ifdef __CUDA_ARCH__
  const int z = __clz(m) - 1;
#else
  const int z = __builtin_clz(m) - 1;
#endif
  const bool zero = E < kFxTiny;
  const int e = E > kFxHuge ? kFxBad : zero ? 0 : E - B + adj - z + 63;
  const int64_t keep = zero ? 0 : ~(int64_t)63;
#pragma unroll
  for (int i = 0; i < R; i++)
    q[i] = cmk<fx2>(((int64_t)((uint64_t)q[i].x << z) & keep) | (e >> 6),
                    ((int64_t)((uint64_t)q[i].y << z) & keep) | (e & 63));
}
// a + i b and (a +- conj b) / 2, (a -+ conj b) / 2i of two blocks
GLIA_HD fx2 fx_plus_i(fx2 a, fx2 b) {
  const int ea = fx_e(a), eb = fx_e(b), E = (ea > eb ? ea : eb) + 1;
  const fx2 p = fx_get<62>(a, E, ea), q = fx_get<62>(b, E, eb);
  const fx2 r = cmk<fx2>(2 * (p.x - q.y), 2 * (p.y + q.x));
  return fx_with_e(r, E > kFxHuge ? kFxBad : E);
}
GLIA_HD void fx_halves(fx2 a, fx2 b, fx2& s, fx2& d) {
  const int ea = fx_e(a), eb = fx_e(b), E = ea > eb ? ea : eb;
  const fx2 p = fx_get<62>(a, E, ea), q = fx_get<62>(b, E, eb);
  const int e = E > kFxHuge ? kFxBad : E;
  s = fx_with_e(cmk<fx2>(p.x + q.x, p.y - q.y), e);
  d = fx_with_e(cmk<fx2>(p.y + q.y, q.x - p.x), e);
}

// doubles to a block in registers, and |w| times as much
template <int B>
GLIA_HD fx2 fx_in2(double2 v, int E) {
  return cmk<fx2>(fx_in<B>(v.x, E), fx_in<B>(v.y, E));
}
template <int B>
GLIA_HD fx2 fx_in2_iw(double2 v, int E, int w) {  // i w v
  const int64_t x = fx_in_w<B>(v.x, E, w < 0 ? -w : w), y = fx_in_w<B>(v.y, E, w < 0 ? -w : w);
  return w < 0 ? cmk<fx2>(y, -x) : cmk<fx2>(-y, x);
}
template <int B>
GLIA_HD int fx_exp_w(double2 v, int w) {  // exponent bound of w v, 0 for w = 0
  const int e = (int)(fx_mag(0u, v) >> 20);
  return w == 0 ? 0 : e + fx_wbits<B>(w < 0 ? -w : w);
}

}  // namespace glia
