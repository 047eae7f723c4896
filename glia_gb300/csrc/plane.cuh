// plane.cuh — a whole FP64 diffusion solve (or D apply, smoother, transform) as one persistent
// kernel.
//
// Grids whose (y, z) plane fits in shared memory. A three-dimensional transform is split by
// direction into two kinds of phase, separated by grid-wide barriers:
//  - plane phase, one work item per x plane (and gradient component): the y and z transforms of
//    the plane in shared memory. Between the inverse and the forward z transform the lines are
//    in real space, where the diffusivity multiplies, the reaction acts and fields are loaded
//    and stored.
//  - column phase, one work item per tile of T (ky, kz) columns: the x transforms, forward then
//    inverse, with the PCG vector updates between them.
// One PCG iteration is three phases:
//    columns  p = P r + b p; G_x = F_x^-1(i w_x p)/N, G_0 = F_x^-1(p)/N; sum |p|^2
//    planes   per component j: grad_j p, times k, sum k (grad_j p)^2, back -> M_j
//             (j = y: i w_y before; j = z: i w_z before and after)
//    columns  D p = i w_x F_x M_x + F_x (i w_y M_y + M_z); <p, A p> = sum p^2 + a sum k |grad p|^2
//             (the derivatives are skew-symmetric), so alpha is known here and x, r are updated
//             in the same pass; ||P r||, <P r, r>
// The scalars live in every CTA: after each barrier all CTAs add the same per-CTA partial sums in
// the same order and take the same decision.
//
// FP64 only. Arithmetic is the bound there, see fx.cuh; a barrier costs 1.0 us. As separate launches
// a solve took 7 kernels and a conditional graph node an iteration, and cuFFT's transforms ran at the
// FP64 units' rate. Measured on GB300, before -> after:
//   forward   64^3, 100 steps   151 -> 45.1 ms    gradient 128^3, 6 steps   164 -> 32.3 ms
//   adjoint  120^3, 2 steps    48.7 -> 10.5 ms    solve    256^3           53.0 -> 11.4 ms
//
// N = R1 R2 (R2 a power of two, so that a group of R2 threads is part of a warp). Inverse
// transforms read index R2 a + b (R1-point DFTs over a, twiddle w^(b k1), R2-point DFTs over b) and
// leave index k1 + R1 k2 at place k1 R2 + k2; forward transforms take that order and mirror the
// steps (R2-point DFTs over k2, twiddle, R1-point DFTs over k1), so nothing is reordered between
// them and every exchange is in place.
//
// A plane holds N / 2 packed complex per line (slot 0: the kz = 0 and kz = N/2 values, both real
// after the y transform, as re / im). Two neighbouring lines a, b of the place order form one
// complex line Z = A + i B. Column c of the first sits in slot c of the pair, column c of the
// second in slot N - c (c = 0: slot N/2), so the thread that has both lines' values at c writes
// Z[c] and Z[N - c] in their places.
#pragma once

#include "dft.cuh"
#include "fx.cuh"
#include "plane.hpp"
#include "reduce.cuh"

namespace glia {

__host__ __device__ constexpr int plane_r2(int n) { return n <= 56 ? 4 : (n < 144 ? 8 : 16); }

template <int NN>
struct PlaneGeo {
  using C = double2;
  static constexpr int N = NN, R2 = plane_r2(NN), R1 = NN / R2;
  static constexpr int NQ = N / 2, NH = N / 2 + 1;
  static constexpr int PL = N * NH;       // complex per x plane of a half spectrum
  // complex per pair of lines: one slot of padding after every R2, so that the lanes of a group
  // meet different banks when they exchange in place
  static constexpr int PS2 = N + R1;
  static __host__ __device__ constexpr int slot(int k) { return k + k / R2; }
  // planes above 200 KB: y and z in phases of their own (column blocks, lines), see k_plane
  static constexpr bool SPLIT = NQ * PS2 * 16 > 200 * 1024;
  static constexpr int TC = NQ % 16 == 0 ? 16 : 8;  // SPLIT: columns per block
  static constexpr int PLANE = SPLIT ? 0 : NQ * PS2;
  // columns per tile of a column phase: the fewest rounds of tiles over the resident CTAs that at
  // most MAXT columns allow, then the smallest multiple of 4 (a sector) that needs no more; 4 only
  // up to 32^3. Solve, fixed tiles of 16 (32 from 112^3) -> these: 32^3 108 -> 103 us, 64^3
  // 256 -> 246, 112^3 1005 -> 886, 128^3 1047 -> 992, 144^3 2070 -> 1867
  static constexpr int PB = PLANE * (int)sizeof(C);
  static constexpr int CTAS = PB > 110 * 1024 ? 152 : 304;  // resident on 152 SMs
  static constexpr int MAXT = CTAS == 304 ? 24 : 210 * 1024 / (2 * N * 16);
  static constexpr int PER = (PL + CTAS - 1) / CTAS, ROUNDS = (PER + MAXT - 1) / MAXT;
  static constexpr int T4 = ((PER + ROUNDS - 1) / ROUNDS + 3) / 4 * 4;
  static constexpr int T = SPLIT ? 8 : N > 32 && T4 < 8 ? 8 : T4;
  static constexpr int XT = (PL + T - 1) / T;
  static constexpr int TILE = N * T;
  static constexpr int RED = 4 * 512 * 8 / (int)sizeof(C);  // partial sums of a phase
  static constexpr int LINES = SPLIT ? 16 * PS2 : 0;  // one pair of lines per group of R2 lanes
  static constexpr int BUF0 = 2 * TILE > RED ? 2 * TILE : RED;
  static constexpr int BUF1 = PLANE > LINES ? PLANE : LINES, BUF = BUF0 > BUF1 ? BUF0 : BUF1;
  // + twiddles, kz' = 0 twice, wave numbers
  static constexpr int SMEM = (BUF + 3 * N + N / 2) * (int)sizeof(C);
  static constexpr int MINB = SMEM > 110 * 1024 ? 1 : 2;
  static constexpr int NT = N <= 32 ? 128 : (MINB == 2 ? 256 : 512);
  static constexpr int NW = NT / 32, GPW = 32 / R2, NG = NW * GPW;
  static constexpr int ITEMS = XT > 3 * N ? XT : 3 * N;  // most work items of a phase
  static_assert(R1 * R2 == N && N % 2 == 0, "decomposition");
  static_assert(R1 <= 16, "register DFT");
  static_assert(!SPLIT || (NG == 16 && N * TC <= BUF), "column block and lines fit the buffer");
};

// Barrier of all CTAs of a cooperative launch: cnt counts arrivals and is set back to zero by the
// last CTA that leaves the kernel. The wait is bounded by the SM clock. A launch whose wait ran out
// leaves the counters as they are until the host has read the fault and cleared both; launches until
// then return at once.
struct GridBarrier {
  unsigned* cnt;
  unsigned target;
  long long limit;
  __device__ __forceinline__ bool sync(int* fault) {
    __syncthreads();
    bool late = false;
    if (threadIdx.x == 0) {
      target += gridDim.x;
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(cnt) : "memory");
      const long long t0 = clock64();
      unsigned v;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
        if ((int)(v - target) >= 0) break;
        if (clock64() - t0 > limit) {
          late = true;
          atomicExch(fault, 2);
          break;
        }
      }
    }
    return !__syncthreads_or(late);
  }
  __device__ __forceinline__ void leave() {
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(cnt + 1, 1u) == gridDim.x - 1) {
      cnt[0] = 0;
      cnt[1] = 0;
    }
  }
};

// The DFT tasks of the phases, in registers and in block fixed point (fx.cuh). One body per radix
// for every use, called, not inlined: the integer code of a 16-point task is about 3000
// instructions, and inlined at each use it ran out of the instruction cache (measured: 5.6 stalled
// warps waiting for instructions per issue).
enum FxMode {
  FX_FWD = 1,    // forward transform (real and imaginary parts swapped around an inverse one)
  FX_IW = 2,     // inputs times i w(a), w(a) the wave number of w0 + wl a
  FX_IC = 4,     // inputs times i w0
  FX_PAIR = 8,   // results in pairs a, h -> Z[c] = a + i h, Z[N - c] = conj a + i conj h
  FX_SPLIT = 16, // inputs in pairs Z[c], Z[N - c] -> a, h
  FX_C0 = 32,    // of c = 0: re / im hold the two packed real values of each line
  FX_SUM = 64    // inputs i w0 src(a) + src2(a)
};
template <int R>
__device__ __forceinline__ void fx_swap(fx2 (&q)[R], bool swap) {
#pragma unroll
  for (int a = 0; a < R; a++)
    q[a] = cmk<fx2>(swap ? q[a].y : q[a].x, swap ? q[a].x : q[a].y);
}
// The transform of a block in registers and its twiddles (tw null: all 1); returns the power of two
// its results lack. Inputs that were
// rounded down (hx, hy = 1: re, im low by half a unit on average, -1: high) bias result 0 alone,
// the transform of a constant being R at 0.
template <int R>
__device__ __forceinline__ int fx_transform(fx2 (&q)[R], const FxTw* tw, int twl, bool fwd, int hx,
                                            int hy) {
  fx_swap(q, fwd);
  reg_dft<R, +1>(q);
  q[0].x += (fwd ? hy : hx) * R / 2;
  q[0].y += (fwd ? hx : hy) * R / 2;
  if (tw) {
    q[0] = cmk<fx2>(q[0].x >> 1, q[0].y >> 1);  // factor 1: exact, as a mean value wants it
#pragma unroll
    for (int k = 1; k < R; k++) q[k] = fx_tw(q[k], tw[k * twl]);
  }
  fx_swap(q, fwd);
  return tw ? 1 : 0;
}
// Memory blocks src[a ls] -> dst[a ld].
template <int R, int N>
__device__ __noinline__ void fx_task1(const fx2* src, const fx2* src2, int ls, fx2* dst, int ld,
                                      const FxTw* tw, int twl, int mode, int w0, int wl) {
  constexpr int B = fx_block_bits(R);
  fx2 q[R];
#pragma unroll
  for (int a = 0; a < R; a++) q[a] = src[a * ls];
  int E = 0;
  if (mode & (FX_IW | FX_IC)) {
    auto w = [&](int a) { return (mode & FX_IC) ? w0 : wavenum(w0 + wl * a, N); };
#pragma unroll
    for (int a = 0; a < R; a++) E = max(E, fx_e_w(fx_e(q[a]), w(a)));
#pragma unroll
    for (int a = 0; a < R; a++) q[a] = fx_get_iw<B>(q[a], E, fx_e(q[a]), w(a));
    if (mode & FX_SUM) {
      const int Eu = E;
      fx2 v[R];
#pragma unroll
      for (int a = 0; a < R; a++) v[a] = src2[a * ls];
#pragma unroll
      for (int a = 0; a < R; a++) E = max(E, fx_e(v[a]));
      const int sh = min(E - Eu, 63);
#pragma unroll
      for (int a = 0; a < R; a++)
        q[a] = cadd(cmk<fx2>(q[a].x >> sh, q[a].y >> sh), fx_get<B>(v[a], E, fx_e(v[a])));
    }
  } else {
#pragma unroll
    for (int a = 0; a < R; a++) E = max(E, fx_e(q[a]));
#pragma unroll
    for (int a = 0; a < R; a++) q[a] = fx_get<B>(q[a], E, fx_e(q[a]));
  }
  const int hx = (mode & FX_SUM) ? 0 : (mode & (FX_IW | FX_IC)) ? -1 : 1;
  const int adj = fx_transform(q, tw, twl, mode & FX_FWD, hx, (mode & FX_SUM) ? 2 : 1);
  fx_put<R, B>(q, E, adj);
#pragma unroll
  for (int a = 0; a < R; a++) dst[a * ld] = q[a];
}
// Memory blocks src[(a >> 1) s2 + (a & 1) s1] -> dst[(a >> 1) d2 + (a & 1) d1], with FX_PAIR or
// FX_SPLIT.
template <int R>
__device__ __noinline__ void fx_task2(const fx2* src, int s1, int s2, fx2* dst, int d1, int d2,
                                      const FxTw* tw, int mode, int c) {
  constexpr int B = fx_block_bits(R);
  fx2 q[R];
#pragma unroll
  for (int a = 0; a < R; a++) q[a] = src[(a >> 1) * s2 + (a & 1) * s1];
  int E = 0;
  if (mode & FX_IC) {
#pragma unroll
    for (int a = 0; a < R; a++) E = max(E, fx_e_w(fx_e(q[a]), c));
#pragma unroll
    for (int a = 0; a < R; a++) q[a] = fx_get_iw<B>(q[a], E, fx_e(q[a]), c);
  } else {
#pragma unroll
    for (int a = 0; a < R; a++) E = max(E, fx_e(q[a]));
#pragma unroll
    for (int a = 0; a < R; a++) q[a] = fx_get<B>(q[a], E, fx_e(q[a]));
  }
  const bool c0 = c == 0;
  if (mode & FX_SPLIT) {  // twice a and h
    // conj of an input that was multiplied by i c is minus i c times the conjugate
    const int64_t s = (mode & FX_IC) ? -1 : 0;
#pragma unroll
    for (int i = 0; i < R / 2; i++) {
      const fx2 z = q[2 * i];
      const fx2 zq = cmk<fx2>((q[2 * i + 1].x ^ s) - s, (q[2 * i + 1].y ^ s) - s);
      q[2 * i] = c0 ? cmk<fx2>(2 * z.x, 2 * zq.x) : cmk<fx2>(z.x + zq.x, z.y - zq.y);
      q[2 * i + 1] = c0 ? cmk<fx2>(2 * z.y, 2 * zq.y) : cmk<fx2>(z.y + zq.y, zq.x - z.x);
    }
    const bool ic = mode & FX_IC;  // the sums' roundings: re or im low by one
    const int adj = fx_transform(q, tw, 1, true, ic ? 0 : 2, ic || c0 ? 2 : 0);
    fx_put<R, B>(q, E, adj - 1);
  } else {
    fx_transform(q, nullptr, 0, false, (mode & FX_IC) ? -1 : 1, 1);
#pragma unroll
    for (int i = 0; i < R / 2; i++) {
      const fx2 a = q[2 * i], h = q[2 * i + 1];
      q[2 * i] = c0 ? cmk<fx2>(a.x, h.x) : cmk<fx2>(a.x - h.y, a.y + h.x);
      q[2 * i + 1] = c0 ? cmk<fx2>(a.y, h.y) : cmk<fx2>(a.x + h.y, h.x - a.y);
    }
    fx_put<R, B>(q, E, 0);
  }
#pragma unroll
  for (int a = 0; a < R; a++) dst[(a >> 1) * d2 + (a & 1) * d1] = q[a];
}
// Doubles src[a l] -> memory blocks dst[a l].
template <int R, int N>
__device__ __noinline__ void fx_enter2(const double2* src, fx2* dst, int l, const FxTw* tw,
                                       int mode, int w0, int wl) {
  constexpr int B = fx_block_bits(R);
  double2 v[R];
#pragma unroll
  for (int a = 0; a < R; a++) v[a] = src[a * l];
  fx2 q[R];
  int E = 0;
  if (mode & FX_IW) {
#pragma unroll
    for (int a = 0; a < R; a++) E = max(E, fx_exp_w<B>(v[a], wavenum(w0 + wl * a, N)));
#pragma unroll
    for (int a = 0; a < R; a++) q[a] = fx_in2_iw<B>(v[a], E, wavenum(w0 + wl * a, N));
  } else {
    E = fx_block(v);
#pragma unroll
    for (int a = 0; a < R; a++) q[a] = fx_in2<B>(v[a], E);
  }
  const int adj = fx_transform(q, tw, 1, mode & FX_FWD, 0, 0);
  fx_put<R, B>(q, E, adj);
#pragma unroll
  for (int a = 0; a < R; a++) dst[a * l] = q[a];
}
// Memory blocks src[a l] -> doubles dst[a l].
template <int R>
__device__ __noinline__ void fx_leave2(const fx2* src, double2* dst, int l, bool fwd) {
  constexpr int B = fx_block_bits(R);
  fx2 q[R];
#pragma unroll
  for (int a = 0; a < R; a++) q[a] = src[a * l];
  int E = 0;
#pragma unroll
  for (int a = 0; a < R; a++) E = max(E, fx_e(q[a]));
#pragma unroll
  for (int a = 0; a < R; a++) q[a] = fx_get<B>(q[a], E, fx_e(q[a]));
  fx_transform(q, nullptr, 0, fwd, 1, 1);
  double2 v[R];
  fx_store<R, B>(q, v, E, 0);
#pragma unroll
  for (int a = 0; a < R; a++) dst[a * l] = v[a];
}
// One row of a line pair in real space, in place: inverse transform, times the diffusivities
// ka[a ks], kb[a ks] of the two lines, forward transform and twiddles. Returns sum k z^2.
template <int R>
__device__ __noinline__ double fx_middle2(fx2* row, const double* ka, const double* kb, int ks,
                                          const FxTw* tw) {
  constexpr int B = fx_block_bits(R), G = 62 - B;
  double va[R], vb[R];
#pragma unroll
  for (int a = 0; a < R; a++) {
    va[a] = ka[a * ks];
    vb[a] = kb[a * ks];
  }
  fx2 q[R];
#pragma unroll
  for (int a = 0; a < R; a++) q[a] = row[a];
  int E = 0;
  uint32_t km = 0;
#pragma unroll
  for (int a = 0; a < R; a++) {
    E = max(E, fx_e(q[a]));
    km = fx_mag(km, cmk<double2>(va[a], vb[a]));
  }
  const int Ek = (int)(km >> 20);
#pragma unroll
  for (int a = 0; a < R; a++) q[a] = fx_get<B>(q[a], E, fx_e(q[a]));
  fx_transform(q, nullptr, 0, false, 1, 1);  // z, |q| < 2^62.5
  // k = m 2^(ek - 1085) with 63 bits of m; z m / 2^64 on the largest ek, then G more bits down
  int64_t dot = 0;
  auto times = [&](int64_t z, double k) {
    const uint32_t hi = fx_hi(k);
    const int64_t m = (int64_t)((((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | fx_lo(k)) << 10);
    const int64_t s = (int64_t)((int32_t)hi >> 31);
    const int64_t p = fx_mulh(z, fx_split((m ^ s) - s)) >>
                      fx_min((uint32_t)(Ek - (int)((hi >> 20) & 0x7ff)), 63u);
    dot += fx_mulh(p, fx_split(z)) >> 5;
    return p >> G;
  };
#pragma unroll
  for (int a = 0; a < R; a++) q[a] = cmk<fx2>(times(q[a].x, va[a]), times(q[a].y, vb[a]));
  double sum = scalbn((double)dot, 2 * E + Ek - 2996 - 2 * B);
  if (E > kFxHuge || Ek > kFxHuge) sum = fx_nan();
  if (E < kFxTiny || Ek < kFxTiny) sum = 0.0;
  E = E > kFxHuge || Ek > kFxHuge ? (int)kFxBad : max(E + Ek - 1021 + G, 0);
  const int adj = fx_transform(q, tw, 1, true, 1, 1);
  fx_put<R, B>(q, E, adj);
#pragma unroll
  for (int a = 0; a < R; a++) row[a] = q[a];
  return sum;
}

template <int NN>
__global__ void __launch_bounds__(PlaneGeo<NN>::NT, PlaneGeo<NN>::MINB)
    k_plane(const __grid_constant__ PlaneArgs A) {
  using Geo_ = PlaneGeo<NN>;
  using C = double2;
  constexpr int N = NN, R1 = Geo_::R1, R2 = Geo_::R2, NQ = Geo_::NQ, NH = Geo_::NH, PL = Geo_::PL,
                T = Geo_::T, NT = Geo_::NT, PS2 = Geo_::PS2, TILE = Geo_::TILE;
  constexpr int S = N * PL;
  auto fx = [](auto* q) {  // the same memory as fixed-point blocks
    using Q = std::conditional_t<std::is_const<std::remove_pointer_t<decltype(q)>>::value,
                                 const fx2, fx2>;
    return reinterpret_cast<Q*>(q);
  };
  extern __shared__ double2 plane_dyn[];
  C* buf = reinterpret_cast<C*>(plane_dyn);
  using Tw = FxTw;
  static_assert(sizeof(Tw) == sizeof(C), "table entry");
  Tw* twA = reinterpret_cast<Tw*>(buf + Geo_::BUF);  // [k1 R2 + b] exp(+2 pi i b k1 / N)
  C* zcol = reinterpret_cast<C*>(twA + N);           // column kz' = 0 of a plane, forward
  C* zin = zcol + N;                                 // and inverse
  double* wtab = reinterpret_cast<double*>(zin + N);  // wave numbers
  __shared__ double tot[4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (__syncthreads_or(tid == 0 && A.sc->dev_fault)) return;  // the counters are not zero
  for (int i = tid; i < N; i += NT) {
    const int k1 = i / R2, b = i - k1 * R2;
    twA[i] = reinterpret_cast<const Tw*>(A.tw)[b * k1];  // b k1 < N
    wtab[i] = (double)wavenum(i, N);
  }
  __syncthreads();
  const double invN = 1.0 / ((double)N * N * N);
  // the spectra sent to the planes keep their factor n^3
  const double a1 = A.a_cn * invN, invN2 = invN * invN;
  GridBarrier bar{A.bar, 0, A.wait};
  // PCG scalars, the same in every CTA (thread 0 updates them)
  __shared__ struct {
    double beta, beta_old, dpi, dpi_old, alpha, bcoef;
    double dp, rnorm0, ttol, pp;  // squares
    int it, iter, status, step;
  } cg;
  if (tid == 0) {
    cg.dpi = cg.dp = cg.alpha = cg.bcoef = 0.0;
    cg.it = cg.iter = cg.status = 0;
  }
  C* __restrict__ const Gp = A.G;
  C* __restrict__ const Mp = A.M;
  C* __restrict__ const xh = A.xhat;
  C* __restrict__ const rh = A.rhat;
  C* __restrict__ const ph = A.phat;
  C* __restrict__ const ch = A.chat;
  const double* __restrict__ const kf = A.k;

  // partial sums per CTA, and their totals after the next barrier (plane_steps.hpp; few FP64
  // operations: all threads' values go to shared memory and one warp adds each sum)
  auto partials = [&](const double* v, PlaneSlots s) {
    double* all = reinterpret_cast<double*>(buf);
    __syncthreads();
    for (int q = 0; q < s.count; q++) all[q * NT + tid] = v[q];
    __syncthreads();
    for (int q = warp; q < s.count; q += Geo_::NW) {
      double x = 0;
#pragma unroll
      for (int w = 0; w < Geo_::NW; w++) x += all[q * NT + 32 * w + lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) A.part[(s.first + q) * (int)gridDim.x + blockIdx.x] = x;
    }
  };
  auto totals = [&](PlaneSlots s) {
    for (int q = warp; q < s.count; q += Geo_::NW) {
      double x = 0;
      for (int b = lane; b < (int)gridDim.x; b += 32)
        x += __ldcg(&A.part[(s.first + q) * (int)gridDim.x + b]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) tot[q] = x;
    }
    __syncthreads();
  };
  // PETSc's default test (conv_test of the other engines), on the squares of the norms
  auto converged = [&](double rn) {
    if (isnan(rn) || isinf(rn)) return -9;
    if (rn <= cg.ttol) return 1;
    if (rn >= A.divtol * A.divtol * cg.rnorm0) return -4;
    return 0;
  };

  // the reaction step on two voxels as their field is read
  auto reacted = [&](C v, int64_t i0, int64_t i1) {
    const double e0 = exp(A.rho[i0] * A.dt), e1 = exp(A.rho[i1] * A.dt);
    if (A.pre == 1) {  // logistic (k_reaction_fwd)
      if (A.half) {
        A.half[i0] = v.x;
        A.half[i1] = v.y;
      }
      const double c0 = v.x * e0, c1 = v.y * e1;
      return cmk<C>(c0 / (c0 + 1.0 - v.x), c1 / (c1 + 1.0 - v.y));
    }
    // linearised at lin (k_reaction_lin)
    const double c0 = A.lin[i0], c1 = A.lin[i1];
    const double q0 = c0 * e0 + 1.0 - c0, q1 = c1 * e1 + 1.0 - c1;
    return cmk<C>(v.x * e0 / (q0 * q0), v.y * e1 / (q1 * q1));
  };

  // the twiddles of a task: none for index 0, where all are 1
  auto at_tw = [](int i, const Tw* tw) { return i ? tw : nullptr; };
  double acc[4];
  auto sums = [&](int kind) {
    switch (kind) {
      case PS_GRAD: partials(acc, plane_sums(PS_GRAD)); break;
      case PS_SETUP: partials(acc, plane_sums(PS_SETUP)); break;
      case PS_UPDATE: partials(acc, plane_sums(PS_UPDATE)); break;
      case PS_DIR: partials(acc, plane_sums(PS_DIR)); break;
      case PS_DOT: partials(acc, plane_sums(PS_DOT)); break;
      default: break;
    }
  };
  // Row k1 of a line pair in real space (places k2, z = k1 + R1 k2 of lines l0 and l1)
  auto line_middle = [&](int kind, C* row, int64_t l0, int64_t l1, int k1) {
    const Tw* tw = at_tw(k1, twA + k1 * R2);
    if (kind == PS_FWD) {
#pragma unroll 2
      for (int k2 = 0; k2 < R2; k2++) {
        const int m = k1 + R1 * k2;
        row[k2] = cmk<C>(A.in[l0 + m], A.in[l1 + m]);
        if (A.pre) row[k2] = reacted(row[k2], l0 + m, l1 + m);
      }
      fx_enter2<R2, N>(row, fx(row), 1, tw, FX_FWD, 0, 0);
    } else if (kind == PS_GRAD) {
      acc[0] += fx_middle2<R2>(fx(row), kf + l0 + k1, kf + l1 + k1, R1, tw);
    } else {
      fx_leave2<R2>(fx(row), row, 1, false);
#pragma unroll 4
      for (int k2 = 0; k2 < R2; k2++) {
        const int m = k1 + R1 * k2;
        A.out[l0 + m] = row[k2].x;
        A.out[l1 + m] = row[k2].y;
      }
    }
  };

  // slots of column c in the first and the second line of a pair
  auto even = [](int c) { return Geo_::slot(c); };
  auto odd = [](int c) { return Geo_::slot(c == 0 ? NQ : N - c); };

  int step = Geo_::SPLIT ? PS_LINE : PS_FWD;
  bool started = false;  // the solve's set-up is done
  int kind = PS_FWD;  // SPLIT: the plane phase that the current y and line phases are part of
  for (;;) {
#pragma unroll
    for (int q = 0; q < 4; q++) acc[q] = 0.0;
    if constexpr (Geo_::SPLIT) {
      if (step == PS_YINV || step == PS_YFWD) {
        // ------------------------------------------------------ SPLIT: column blocks of planes
        constexpr int TC = Geo_::TC, CB = NQ / TC;
        const int nj = kind == PS_GRAD ? 3 : 1;
        for (int item = blockIdx.x; item < nj * N * CB; item += gridDim.x) {
          const int cb = item % CB, xj = item / CB, x = xj / nj, j = xj - nj * x;
          C* const W = A.W + ((int64_t)j * N + x) * NQ * N + cb * TC;
          if (step == PS_YINV) {
            const C* G = (kind == PS_GRAD && j == 0 ? Gp : Gp + S) + x * PL + cb * TC;
            if (cb == 0)
              for (int ky = tid; ky < N; ky += NT) {
                fx(zin)[ky] = fx_plus_i(fx(G)[ky * NH], fx(G)[ky * NH + NQ]);
              }
            __syncthreads();
            for (int task = tid; task < TC * R2; task += NT) {
              const int b = task / TC, c = task - b * TC;
              const bool c0 = cb == 0 && c == 0;
              const int ld = c0 ? 1 : NH;
              fx_task1<R1, N>(fx((c0 ? zin : G + c) + b * ld), nullptr, R2 * ld,
                              fx(buf + b * TC + c), R2 * TC, at_tw(b, twA + b), R2,
                              j == 1 ? FX_IW : 0, b, R2);
            }
            __syncthreads();
            for (int task = tid; task < TC * R1; task += NT) {
              const int k1 = task / TC, c = task - k1 * TC, cc = cb * TC + c;
              fx_task2<R2>(fx(buf + k1 * R2 * TC + c), TC, 2 * TC, fx(W + k1 * (R2 / 2) * N + c),
                           (cc == 0 ? NQ : N - cc) - cc, N, nullptr,
                           FX_PAIR | (j == 2 ? FX_IC : 0), cc);
            }
          } else {
            for (int task = tid; task < TC * R1; task += NT) {
              const int k1 = task / TC, c = task - k1 * TC, cc = cb * TC + c;
              fx_task2<R2>(fx(W + k1 * (R2 / 2) * N + c), (cc == 0 ? NQ : N - cc) - cc, N,
                           fx(buf + k1 * R2 * TC + c), TC, 2 * TC, at_tw(k1, twA + k1 * R2),
                           FX_SPLIT | (j == 2 ? FX_IC : 0), cc);
            }
            __syncthreads();
            C* M = Mp + j * S + x * PL;
            for (int task = tid; task < TC * R2; task += NT) {
              const int b = task / TC, c = task - b * TC;
              const bool c0 = cb == 0 && c == 0;
              const int ld = c0 ? 1 : NH;
              fx_task1<R1, N>(fx(buf + b * TC + c), nullptr, R2 * TC,
                              fx((c0 ? zcol : M + cb * TC + c) + b * ld), R2 * ld, nullptr, 0,
                              FX_FWD, 0, 0);
            }
            __syncthreads();
            if (cb == 0)
              for (int ky = tid; ky < N; ky += NT) {
                fx_halves(fx(zcol)[ky], fx(zcol)[ky == 0 ? 0 : N - ky], fx(M)[ky * NH],
                          fx(M)[ky * NH + NQ]);
              }
          }
          __syncthreads();
        }
      } else if (step == PS_LINE) {
        // ----------------------------------------------------- SPLIT: line pairs of all planes
        const int nj = kind == PS_GRAD ? 3 : 1;
        const int g = lane / R2, t = lane % R2;
        C* const E = buf + (warp * Geo_::GPW + g) * PS2;
        C* const col = E + t;
        const int pairs = nj * N * NQ, per = gridDim.x * Geo_::NG;
        for (int base = blockIdx.x * Geo_::NG + warp * Geo_::GPW; base < pairs; base += per) {
          // pair pr of plane x, component j fastest (the three share k)
          const int id = base + g, j = id % nj, px = id / nj, x = px / NQ, pr = px - x * NQ;
          const int p0 = 2 * pr, y0 = p0 / R2 + R1 * (p0 % R2);
          const int64_t l0 = ((int64_t)x * N + y0) * N, l1 = l0 + (int64_t)R1 * N;
          C* const W = A.W + (((int64_t)j * N + x) * NQ + pr) * N + t;
          const bool on = id < pairs;
          if (kind != PS_FWD) {
            if (on)
              fx_task1<R1, N>(fx(W), nullptr, R2, fx(col), R2 + 1, at_tw(t, twA + t), R2, 0, 0, 0);
            __syncwarp();
          }
          if (on) {
            for (int k1 = t; k1 < R1; k1 += R2)
              line_middle(kind, E + k1 * (R2 + 1), l0, l1, k1);
          }
          if (kind != PS_BACK) {
            __syncwarp();
            if (on) fx_task1<R1, N>(fx(col), nullptr, R2 + 1, fx(W), R2, nullptr, 0, FX_FWD, 0, 0);
          }
          __syncwarp();
        }
        if (kind == PS_GRAD) sums(kind);
      }
    }
    if (step <= PS_BACK && !Geo_::SPLIT) {
      // ------------------------------------------------------------------------------ planes
      const int items = step == PS_GRAD ? 3 * N : N;
      for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const int x = step == PS_GRAD ? item / 3 : item;
        const int j = step == PS_GRAD ? item - 3 * x : 0;
        if (step != PS_FWD) {
          // y inverse: the kz = 0 and kz = N/2 columns as one, then rows ky = R2 a + b of column c
          const C* G = (step == PS_GRAD && j == 0 ? Gp : Gp + S) + x * PL;
          for (int ky = tid; ky < N; ky += NT) {
            fx(zin)[ky] = fx_plus_i(fx(G)[ky * NH], fx(G)[ky * NH + NQ]);
          }
          __syncthreads();
          for (int task = tid; task < NQ * R2; task += NT) {
            const int b = task / NQ, c = task - b * NQ;
            const C* src = c == 0 ? zin : G + c;
            const int ld = c == 0 ? 1 : NH;
            fx_task1<R1, N>(fx(src + b * ld), nullptr, R2 * ld,
                            fx(buf + (b >> 1) * PS2 + ((b & 1) ? odd(c) : even(c))),
                            R2 / 2 * PS2, at_tw(b, twA + b), R2, j == 1 ? FX_IW : 0, b, R2);
          }
          __syncthreads();
          for (int task = tid; task < NQ * R1; task += NT) {
            const int k1 = task / NQ, c = task - k1 * NQ;
            C* row = buf + k1 * (R2 / 2) * PS2 + even(c);
            const int od = odd(c) - even(c);
            fx_task2<R2>(fx(row), od, PS2, fx(row), od, PS2, nullptr,
                         FX_PAIR | (j == 2 ? FX_IC : 0), c);
          }
          __syncthreads();
        }
        // z lines, two at a time: R2 lanes per pair
        for (int base = warp * Geo_::GPW; base < NQ; base += Geo_::NG) {
          const int g = lane / R2, t = lane % R2, pr = base + g;
          const bool on = pr < NQ;
          C* E = buf + (on ? pr : 0) * PS2;
          const int p0 = 2 * pr, y0 = p0 / R2 + R1 * (p0 % R2), y1 = y0 + R1;
          const int64_t l0 = ((int64_t)x * N + y0) * N, l1 = ((int64_t)x * N + y1) * N;
          // thread t: index R2 a + t in place, then rows k1 = t, t + R2, ... in place, and back
          C* const col = E + t;
          if (step != PS_FWD) {
            if (on)
              fx_task1<R1, N>(fx(col), nullptr, R2 + 1, fx(col), R2 + 1, at_tw(t, twA + t), R2,
                              0, 0, 0);
            __syncwarp();
          }
          if (on) {
            for (int k1 = t; k1 < R1; k1 += R2)
              line_middle(step, E + k1 * (R2 + 1), l0, l1, k1);
          }
          if (step != PS_BACK) {
            __syncwarp();
            if (on)
              fx_task1<R1, N>(fx(col), nullptr, R2 + 1, fx(col), R2 + 1, nullptr, 0, FX_FWD, 0,
                              0);
          }
        }
        __syncthreads();
        if (step != PS_BACK) {
          // y forward: places k1 R2 + k2 of column c, split into the two lines of each pair
          for (int task = tid; task < NQ * R1; task += NT) {
            const int k1 = task / NQ, c = task - k1 * NQ;
            C* row = buf + k1 * (R2 / 2) * PS2 + even(c);
            const int od = odd(c) - even(c);
            fx_task2<R2>(fx(row), od, PS2, fx(row), od, PS2, at_tw(k1, twA + k1 * R2),
                         FX_SPLIT | (j == 2 ? FX_IC : 0), c);
          }
          __syncthreads();
          C* M = Mp + j * S + x * PL;
          for (int task = tid; task < NQ * R2; task += NT) {
            const int b = task / NQ, c = task - b * NQ;
            C* dst = c == 0 ? zcol : M + c;
            const int ld = c == 0 ? 1 : NH;
            fx_task1<R1, N>(fx(buf + (b >> 1) * PS2 + ((b & 1) ? odd(c) : even(c))), nullptr,
                            R2 / 2 * PS2, fx(dst + b * ld), R2 * ld, nullptr, 0, FX_FWD, 0, 0);
          }
          __syncthreads();
          for (int ky = tid; ky < N; ky += NT) {  // kz' = 0 into kz = 0 and kz = N/2
            fx_halves(fx(zcol)[ky], fx(zcol)[ky == 0 ? 0 : N - ky], fx(M)[ky * NH],
                      fx(M)[ky * NH + NQ]);
          }
        }
      }
      if (step == PS_GRAD) sums(step);
    } else if (step >= PS_SPEC) {
      // ----------------------------------------------------------------------------- columns
      const int nin = step == PS_SPEC || step == PS_ENTER || step == PS_SMOOTH ? 1
                      : step == PS_DIR || step == PS_LEAVE                     ? 0
                                                                               : 2;
      const int nout = step == PS_SMOOTH || step == PS_LEAVE || step == PS_APPLY ? 1
                       : step == PS_SPEC || step == PS_UPDATE || step == PS_DOT  ? 0
                                                                                 : 2;
      if (step == PS_UPDATE) {  // alpha
        totals(kPlaneAlphaSums);
        if (tid == 0) {
          if (cg.iter == 0) tot[0] = cg.pp;  // of the set-up's first direction
          cg.dpi_old = cg.dpi;
          cg.dpi = tot[0] * invN + A.a_cn * tot[1] * invN * invN;
          cg.beta_old = cg.beta;
          cg.it = cg.iter + 1;
          if (cg.dpi == 0.0 || (cg.iter > 0 && cg.dpi * cg.dpi_old <= 0.0))
            cg.status = -8;
          else if (isnan(cg.dpi) || isinf(cg.dpi))
            cg.status = -9;
          else
            cg.alpha = cg.beta / cg.dpi;
        }
        __syncthreads();
        if (cg.status != 0) {  // x and r stay as they are
          step = PS_LEAVE;
          continue;
        }
      }
      const double al = cg.alpha, alN = cg.alpha * invN, bc = cg.bcoef;
      for (int tile = blockIdx.x; tile < Geo_::XT; tile += gridDim.x) {
        // forward, first part: rows x = R2 a + b
        for (int task = tid; task < nin * T * R2; task += NT) {
          const int c = task % T, ib = task / T, i = ib >= R2, b = ib - i * R2, q = tile * T + c;
          if (q >= PL) continue;
          const C* src = Mp + i * S + q;
          // M_x, then i w_y M_y + M_z
          fx_task1<R1, N>(fx(src + b * PL), fx(src + S + b * PL), R2 * PL,
                          fx(buf + i * TILE + b * T + c), R2 * T, at_tw(b, twA + b), R2,
                          i == 1 ? FX_FWD | FX_IC | FX_SUM : FX_FWD, wavenum(q / NH, N), 0);
        }
        if (nin) __syncthreads();
        for (int task = tid; task < T * R1; task += NT) {
          const int c = task % T, k1 = task / T, q = tile * T + c;
          if (q >= PL) continue;
          const int kz = q % NH;
          const double mult = kz == 0 || kz == NQ ? 1.0 : 2.0;
          C* sl = buf + k1 * R2 * T + c;
          auto at = [&](int k2) { return (k1 + R1 * k2) * PL + q; };
          auto pm = [&](int k2) { return A.pf[at(k2)]; };
          // What a step does at one spectrum element: d = the forward x transform's result (the
          // divergence for two inputs); returns the value that is transformed back. FP64 operations
          // are what this costs: a task's sums are taken without the multiplicity, ||z||^2 and <z, r>
          // of the set-up are those of its first direction, and the spectra sent to the planes keep
          // their factor n^3 (a1 = a_cn / n^3).
          double part[4] = {0, 0, 0, 0};
          auto element = [&](int k2, C d) -> C {
            const int e = at(k2);
            switch (step) {
              case PS_SPEC:
              case PS_ENTER:
                ch[e] = d;
                return d;
              case PS_SMOOTH:
                return cmul2(d, A.mulk[e]);
              case PS_SETUP: {
                const C c0 = ch[e];
                const double P = pm(k2);
                const double br = P * (c0.x + a1 * d.x), bi = P * (c0.y + a1 * d.y);
                const C r = cmk<C>(2.0 * a1 * d.x, 2.0 * a1 * d.y);
                const C p = cmk<C>(P * r.x, P * r.y);  // the first direction
                part[0] = fma(br, br, fma(bi, bi, part[0]));
                part[1] = fma(p.x, p.x, fma(p.y, p.y, part[1]));
                part[2] = fma(p.x, r.x, fma(p.y, r.y, part[2]));
                if (A.cx) {
                  const C xv = A.cx[e];
                  part[3] = fma(xv.x, d.x, fma(xv.y, d.y, part[3]));
                }
                xh[e] = cmk<C>(c0.x * invN, c0.y * invN);
                rh[e] = r;
                ph[e] = p;
                return p;
              }
              case PS_UPDATE: {
                const C p = ph[e], xv = xh[e], rv = rh[e];
                const double P = pm(k2);
                const C r = cmk<C>(rv.x - al * (p.x - a1 * d.x), rv.y - al * (p.y - a1 * d.y));
                xh[e] = cmk<C>(xv.x + alN * p.x, xv.y + alN * p.y);
                rh[e] = r;
                const double t = P * (r.x * r.x + r.y * r.y);
                part[0] = fma(P, t, part[0]);
                part[1] += t;
                return d;
              }
              case PS_DIR: {
                const C rv = rh[e], po = ph[e];
                const double P = pm(k2);
                const C p = cmk<C>(fma(P, rv.x, bc * po.x), fma(P, rv.y, bc * po.y));
                ph[e] = p;
                part[0] = fma(p.x, p.x, fma(p.y, p.y, part[0]));
                return p;
              }
              case PS_LEAVE:
                return xh[e];
              case PS_APPLY:
                return cmk<C>(d.x * invN2, d.y * invN2);
              default: {  // PS_DOT
                const C xv = A.cx[e];
                part[0] = fma(xv.x, d.x, fma(xv.y, d.y, part[0]));
                return d;
              }
            }
          };
          const Tw* tw = at_tw(k1, twA + k1 * R2);
          if (nin) fx_leave2<R2>(fx(sl), sl, T, true);
          if (nin == 2) fx_leave2<R2>(fx(sl + TILE), sl + TILE, T, true);
#pragma unroll 2
          for (int k2 = 0; k2 < R2; k2++) {
            C d = sl[k2 * T];
            if (nin == 2) d = cadd(cimul<C>(wtab[k1 + R1 * k2], d), sl[TILE + k2 * T]);
            sl[k2 * T] = element(k2, d);
          }
#pragma unroll
          for (int q = 0; q < 4; q++) acc[q] += mult * part[q];
          if (nout == 2) fx_enter2<R2, N>(sl, fx(sl + TILE), T, tw, FX_IW, k1, R1);
          if (nout) fx_enter2<R2, N>(sl, fx(sl), T, tw, 0, 0, 0);
          continue;
        }
        __syncthreads();
        // inverse, second part: rows x = b + R2 a
        for (int task = tid; task < nout * T * R2; task += NT) {
          const int c = task % T, ib = task / T, i = ib >= R2, b = ib - i * R2, q = tile * T + c;
          if (q >= PL) continue;
          C* dst = Gp + (1 - i) * S + q;  // i = 0: G_0, i = 1: G_x
          fx_task1<R1, N>(fx(buf + i * TILE + b * T + c), nullptr, R2 * T, fx(dst + b * PL),
                          R2 * PL, nullptr, 0, 0, 0, 0);
        }
        if (nout) __syncthreads();
      }
      sums(step);
    }
    if (step == PS_SPEC || (Geo_::SPLIT ? step == PS_LINE && kind == PS_BACK : step == PS_BACK))
      break;
    if (!bar.sync(&A.sc->dev_fault)) return;

    // ---------------------------------------------------------------------- the next step
    if constexpr (Geo_::SPLIT) {  // FWD: line, y; GRAD: y, line, y; BACK: y, line
      if (step == PS_YINV) {
        step = PS_LINE;
        continue;
      }
      if (step == PS_LINE) {
        step = PS_YFWD;
        continue;
      }
      if (step == PS_YFWD) step = kind;
    }
    switch (step) {
      case PS_FWD:
        step = A.prog == PP_SPEC ? PS_SPEC : A.prog == PP_SMOOTH ? PS_SMOOTH : PS_ENTER;
        break;
      case PS_ENTER:
        step = PS_GRAD;
        break;
      case PS_GRAD:
        step = A.prog == PP_APPLY ? PS_APPLY
               : A.prog == PP_DOT ? PS_DOT
               : started          ? PS_UPDATE
                                  : PS_SETUP;
        break;
      case PS_SETUP:
        started = true;
        totals(plane_sums(PS_SETUP));
        if (tid == 0) {
          double snorm = tot[0] * invN;
          cg.dp = tot[1] * invN;
          if (snorm == 0.0) snorm = cg.dp;
          cg.rnorm0 = snorm;
          cg.ttol = fmax(A.rtol * A.rtol * snorm, A.abstol * A.abstol);
          cg.beta = tot[2] * invN;
          cg.pp = tot[1];
          cg.status = converged(cg.dp);
          if (cg.status == 0 && cg.beta == 0.0) {
            cg.status = 2;
            cg.it = 1;
          }
          if (A.cx && blockIdx.x == 0) A.sc->acc[6] += A.kdot_weight * tot[3] * invN * invN;
          cg.step = cg.status == 0 ? PS_GRAD : PS_LEAVE;
        }
        __syncthreads();
        step = cg.step;
        break;
      case PS_UPDATE:
        totals(plane_sums(PS_UPDATE));
        if (tid == 0) {
          cg.dp = tot[0] * invN;
          cg.status = converged(cg.dp);
          if (cg.status == 0) {
            const double bnew = tot[1] * invN;
            cg.beta = bnew;
            cg.bcoef = bnew / cg.beta_old;
            cg.iter++;
            if (bnew == 0.0) {
              cg.status = 2;
              cg.it = cg.iter + 1;
            } else if (cg.iter >= A.maxit) {
              cg.status = -3;
            }
          }
          cg.step = cg.status == 0 ? PS_DIR : PS_LEAVE;
        }
        __syncthreads();
        step = cg.step;
        break;
      case PS_DIR:
        step = PS_GRAD;
        break;
      case PS_DOT:
        totals(plane_sums(PS_DOT));
        if (blockIdx.x == 0 && tid == 0) A.sc->acc[6] += A.kdot_weight * tot[0] * invN * invN;
        bar.leave();
        return;
      default:  // PS_SMOOTH, PS_LEAVE, PS_APPLY
        step = PS_BACK;
    }
    if constexpr (Geo_::SPLIT) {
      if (step <= PS_BACK) {
        kind = step;
        step = PS_YINV;
      }
    }
  }
  // outcome and sweep statistics
  if (A.prog == PP_SOLVE && blockIdx.x == 0 && tid == 0) {
    DevScalars* s = A.sc;
    s->it = cg.it;
    s->iter = cg.iter;
    s->dp = sqrt(cg.dp);
    s->status = cg.status;
    s->sum_its[A.which] += cg.it;
    s->nsolves += 1;
    if (cg.it > s->max_its) s->max_its = cg.it;
    s->last_dp = s->dp;
    if (cg.status < 0 && s->err_status == 0) {
      s->err_status = cg.status;
      s->err_its = cg.it;
    }
  }
  bar.leave();
}

template <int N>
PlaneKernel plane_entry() {
  using P = PlaneGeo<N>;
  return PlaneKernel{reinterpret_cast<const void*>(&k_plane<N>), P::NT, P::SMEM, P::ITEMS,
                     P::SPLIT};
}

}  // namespace glia
