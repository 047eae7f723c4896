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
  constexpr int B = 61 - fx_log2(R), kRuns = 1000;  // B of the kernels' tasks
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

// i w v, zeros, subnormal blocks, NaN
int edges() {
  double2 v[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
  fx_dft<4, 1, false>(v, NoTw{});
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
  fx_dft<2, 1, false>(n, NoTw{});
  for (auto& z : n)
    if (!std::isnan(z.x) || !std::isnan(z.y)) return 3;
  double2 t[2] = {{1e-300, 0.0}, {0.0, 1e-305}};
  fx_dft<2, 1, false>(t, NoTw{});
  for (auto& z : t)
    if (!(std::fabs(z.x) <= 1.1e-300)) return 4;
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
