// Register DFTs on the host: FP64 arithmetic and 64-bit block fixed point (fx.cuh) against long
// double, root mean square over random inputs of the error relative to the result's 2-norm. One
// line per size and kind of input: R S kind fp64 fixed.
#include "../../glia_gb300/csrc/fx.cuh"

#include <cmath>
#include <complex>
#include <cstdio>
#include <random>

using namespace glia;
using ld = long double;

template <int R, int S>
void run() {
  constexpr int B = fx_block_bits(R), kRuns = 1000;
  const ld pi = 3.14159265358979323846264338327950288L;
  std::mt19937_64 gen(R);
  std::normal_distribution<double> nd;
  for (int kind = 0; kind < 4; kind++) {  // flat, decaying, spread over decades, one spike
    ld ef = 0, ex = 0;
    for (int t = 0; t < kRuns; t++) {
      double2 v[R], f[R];
      std::complex<ld> X[R];
      for (int i = 0; i < R; i++) {
        const double s = kind == 0   ? 1.0
                         : kind == 1 ? std::exp(-1.5 * i)
                         : kind == 2 ? std::exp(6.0 * nd(gen))
                                     : (i == 3 % R ? 1.0 : 1e-3);
        const double re = nd(gen), im = nd(gen);
        f[i] = v[i] = cmk<double2>(re * s, im * s);
      }
      for (int k = 0; k < R; k++) {
        X[k] = 0;
        for (int j = 0; j < R; j++) {
          const ld a = S * 2 * pi * ((j * k) % R) / R;
          X[k] += std::complex<ld>(v[j].x, v[j].y) * std::complex<ld>(cosl(a), sinl(a));
        }
      }
      reg_dft<R, S>(f);
      const int E = fx_block(v);
      fx2 q[R];
      for (int i = 0; i < R; i++) q[i] = fx_in2<B>(v[i], E);
      reg_dft<R, S>(q);
      fx_store<R, B>(q, v, E, 0);
      ld a = 0, b = 0, n = 0;
      for (int k = 0; k < R; k++) {
        a += std::norm(std::complex<ld>(f[k].x, f[k].y) - X[k]);
        b += std::norm(std::complex<ld>(v[k].x, v[k].y) - X[k]);
        n += std::norm(X[k]);
      }
      ef += a / n;
      ex += b / n;
    }
    std::printf("%d %d %d %.4e %.4e\n", R, S, kind, (double)sqrtl(ef / kRuns),
                (double)sqrtl(ex / kRuns));
  }
}

template <int R, int B>
void transform(double2 (&v)[R]) {
  const int E = fx_block(v);
  fx2 q[R];
  for (int i = 0; i < R; i++) q[i] = fx_in2<B>(v[i], E);
  reg_dft<R, 1>(q);
  fx_store<R, B>(q, v, E, 0);
}
// value of a memory block
std::complex<ld> value(fx2 v) {
  const int e = fx_e(v);
  return {ldexpl((ld)v.x, e - 1022 - 63), ldexpl((ld)v.y, e - 1022 - 63)};
}

// i w v, zeros, subnormal blocks, NaN; memory blocks: what is put is there to 2^-55 of the block's
// largest value, is got back to that and one rounding to double (2^-53; 2^-52 allowed), also times
// i w, and enters the sums of two blocks to 2^-53
int edges() {
  double2 v[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
  transform<4, 58>(v);
  for (auto& z : v)
    if (z.x != 0 || z.y != 0) return 1;
  for (int w : {0, 1, -1, 5, -64, 127}) {
    double2 a[2] = {{1.25, -3.5}, {0.0, 0.0}};
    fx2 q[2];
    int E = 0;
    for (auto& z : a) E = std::max(E, fx_exp_w<58>(z, w));
    for (int i = 0; i < 2; i++) q[i] = fx_in2_iw<58>(a[i], E, w);
    fx_store<2, 58>(q, a, E, 0);
    if (a[0].x != 3.5 * w || a[0].y != 1.25 * w || a[1].x != 0 || a[1].y != 0) return 2;
  }
  double2 n[2] = {{1.0, NAN}, {2.0, 0.0}};
  transform<2, 58>(n);
  for (auto& z : n)
    if (!std::isnan(z.x) || !std::isnan(z.y)) return 3;
  double2 t[2] = {{1e-300, 0.0}, {0.0, 1e-305}};
  transform<2, 58>(t);
  for (auto& z : t)
    if (!(std::fabs(z.x) <= 1.1e-300)) return 4;

  constexpr int R = 8, B = fx_block_bits(R);
  std::mt19937_64 gen(1);
  std::normal_distribution<double> nd;
  const ld eps = ldexpl(1, -56);
  for (int it = 0; it < 2000; it++) {
    double2 d[R];
    ld top = 0;
    const double big = std::exp(20 * nd(gen));
    for (auto& z : d) {
      z = cmk<double2>(big * nd(gen) * std::exp(3 * nd(gen)), big * nd(gen));
      top = std::max(top, std::abs(std::complex<ld>(z.x, z.y)));
    }
    fx2 q[R];
    int E = fx_block(d);
    for (int i = 0; i < R; i++) q[i] = fx_in2<B>(d[i], E);
    fx_put<R, B>(q, E, 0);
    int Em = 0;
    for (int i = 0; i < R; i++) {
      const std::complex<ld> x(d[i].x, d[i].y);
      if (std::abs(value(q[i]) - x) > 2 * eps * top) return 5;
      Em = std::max(Em, fx_e(q[i]));
    }
    for (int i = 0; i < R; i++) {  // into registers and back to doubles
      fx2 r[1] = {fx_get<B>(q[i], Em, fx_e(q[i]))};
      double2 o[1];
      fx_store<1, B>(r, o, Em, 0);
      const std::complex<ld> x(d[i].x, d[i].y);
      if (std::abs(std::complex<ld>(o[0].x, o[0].y) - x) > 16 * eps * top) return 6;
    }
    for (int w : {0, 1, -1, 2, -63, 127}) {
      int Ew = 0;
      for (int i = 0; i < R; i++) Ew = std::max(Ew, fx_e_w(fx_e(q[i]), w));
      for (int i = 0; i < R; i++) {
        fx2 r[1] = {fx_get_iw<B>(q[i], Ew, fx_e(q[i]), w)};
        double2 o[1];
        fx_store<1, B>(r, o, Ew, 0);
        const std::complex<ld> x = std::complex<ld>(d[i].x, d[i].y) * std::complex<ld>(0, w);
        if (std::abs(std::complex<ld>(o[0].x, o[0].y) - x) > 16 * eps * top * std::abs((ld)w))
          return 7;
      }
    }
    const std::complex<ld> a = value(q[0]), b = value(q[1]), i1(0, 1);
    fx2 sum, diff;
    fx_halves(q[0], q[1], sum, diff);
    if (std::abs(value(fx_plus_i(q[0], q[1])) - (a + i1 * b)) > 8 * eps * top) return 8;
    if (std::abs(value(sum) - (a + std::conj(b)) / (ld)2) > 8 * eps * top) return 9;
    if (std::abs(value(diff) - (a - std::conj(b)) / ((ld)2 * i1)) > 8 * eps * top) return 10;
  }
  fx2 z[2] = {{5, 7}, {3, 1}};
  fx_put<2, 58>(z, 0, 0);
  if (value(z[0]) != std::complex<ld>(0, 0) || fx_e(z[1]) != 0) return 11;
  fx_put<2, 58>(z, kFxBad, 0);
  if (fx_e(z[0]) != kFxBad) return 12;
  return 0;
}

int main() {
  run<4, 1>();
  run<6, 1>();
  run<8, 1>();
  run<8, -1>();
  run<9, 1>();
  run<10, -1>();
  run<12, 1>();
  run<14, 1>();
  run<15, 1>();
  run<16, 1>();
  run<16, -1>();
  run<7, 1>();
  run<11, -1>();
  run<13, 1>();
  return edges();
}
