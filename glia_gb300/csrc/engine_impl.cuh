// engine_impl.cuh — host driver of the reaction–diffusion path on one GPU (one CUDA stream).
//
// Engine<R> implements, for storage type R (float: mixed path with FP64 reductions; double:
// FP64), the reference's Tumor / MatProp / DiffCoef / ReacCoef / Phi / Obs / DiffusionSolver /
// PdeOperatorsRD / DerivativeOperatorsRD state for one grid. Two diffusion-solve engines:
//  - fused (default): the PCG of DiffusionSolver::solve runs in spectral space. x, r, p, w are
//    half spectra; z = P r is never formed; the operator apply is 6 transforms
//    (1 batched C2R of the three gradient spectra, 1 batched R2C of k * grad) plus 4 fused
//    passes; the set-up reuses one D apply for both the right-hand side and r0.
//    FP64 grids with a plane kernel (plane.cuh) run all of a solve as one launch.
//  - reference-structured (GLIA_ENGINE_REFERENCE): a restatement of the reference's GPU
//    structure with our own kernels: real-space PCG, 10 transforms per D apply, one kernel per
//    PETSc vector operation and a host round trip per inner product. It is the plain baseline.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "engine.hpp"
#include "kernels.cuh"
#include "ktimer.cuh"
#include "zpass2.cuh"
#include "zpass.cuh"
#include "ownfft.cuh"
#include "plane.hpp"

#define GLIA_TIMED(slot, bytes, ...)             \
  do {                                           \
    cudaEvent_t ev_ = tm_.begin(stream_);        \
    __VA_ARGS__;                                 \
    GLIA_LAUNCH_CHECK();                         \
    tm_.end((slot), ev_, (double)(bytes), stream_); \
  } while (0)

namespace glia {

static __global__ void k_solve_config(DevScalars* s, double a_cn, double pc_c, double rtol,
                               double abstol, double divtol, int maxit, double kdot_weight) {
  s->a_cn = a_cn;
  s->pc_c = pc_c;
  s->rtol = rtol;
  s->abstol = abstol;
  s->divtol = divtol;
  s->maxit = maxit;
  s->kdot_weight = kdot_weight;
  s->status = 0;
  s->it = 0;
  s->iter = 0;
}
static __global__ void k_acc_reset(DevScalars* s) {
  for (int q = 0; q < 8; q++) s->acc[q] = 0.0;
}
static __global__ void k_keep_red0(DevScalars* s) { s->m1_keep = s->red[0]; }
static __global__ void k_solve_stats_reset(DevScalars* s) {
  s->sum_its[0] = s->sum_its[1] = s->sum_its[2] = 0;
  s->nsolves = 0;
  s->max_its = 0;
  s->err_status = 0;
  s->err_its = 0;
  s->last_dp = 0.0;
}
// End of one diffusion solve: fold its PCG outcome into the sweep statistics.
static __global__ void k_solve_finish(DevScalars* s, int which) {
  const int it = s->it;
  s->sum_its[which] += it;
  s->nsolves += 1;
  if (it > s->max_its) s->max_its = it;
  s->last_dp = s->dp;
  if (s->status < 0 && s->err_status == 0) {
    s->err_status = s->status;
    s->err_its = it;
  }
}
// Head of the PCG graph: run the loop body only if the set-up left the solve unconverged.
static __global__ void k_cond_set(DevScalars* s, cudaGraphConditionalHandle h) {
  s->guard = 0;
  cudaGraphSetConditional(h, s->status == 0 ? 1u : 0u);
}
// Tail of the loop body: continue while the PCG runs; the guard bounds the loop at maxit + 1
// body executions whatever the scalars say.
static __global__ void k_cond_step(DevScalars* s, cudaGraphConditionalHandle h) {
  s->guard += 1;
  if (s->status == 0 && s->guard > s->maxit) s->status = -3;
  cudaGraphSetConditional(h, s->status == 0 ? 1u : 0u);
}

// Status summary read back after each PCG iteration (one 32-byte copy).
struct SolveStatus {
  int status, it;
  double dp;
};

constexpr int kMaxRedBlocksPerSm = 8;

template <typename R>
class Engine final : public EngineBase {
 public:
  Engine(int n, bool refmode) : g_(n), ref_(refmode) {
    int dev = 0;
    GLIA_CUDA(cudaGetDevice(&dev));
    GLIA_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
    GLIA_CUDA(cudaStreamCreateWithFlags(&own_stream_, cudaStreamNonBlocking));
    stream_ = own_stream_;
    red_blocks_ = sms_ * 4;
    pw_blocks_ = sms_ * 8;
    N_ = g_.N;
    Ns_ = g_.Ns;
    sc_ = dalloc<DevScalars>(1);
    GLIA_CUDA(cudaMemsetAsync(sc_, 0, sizeof(DevScalars), stream_));
    GLIA_CUDA(cudaMallocHost(&hsc_, sizeof(DevScalars)));
    GLIA_CUDA(cudaMallocHost(&hst_, sizeof(SolveStatus)));
    ws_.partials = dalloc<double>((int64_t)sms_ * kMaxRedBlocksPerSm * 4);
    ws_.counter = dalloc<unsigned int>(1);
    GLIA_CUDA(cudaMemsetAsync(ws_.counter, 0, sizeof(unsigned int), stream_));
    for (R** f : {&wm_, &gm_, &csf_, &vt_, &bg_, &filter_, &kxx_, &rho_, &obs_, &c0_, &ct_, &p0_,
                  &pt_, &tmp_})
      *f = fld();
    // MatProp::setValues defaults (src/mat/MatProp.cpp:20-33): wm = 1, filter = 1
    fill(wm_, 1.0);
    fill(filter_, 1.0);
    fill(obs_, 1.0);
    filter_sum_ = (double)N_;
    chat_ = spec();
    xhat_ = spec();
    g3s_ = dalloc<R>(3 * Ns_ * 2);
    g3r_ = dalloc<R>(3 * N_);
    if (!ref_) {
      rhat_ = spec();
      phat_ = spec();
      what_ = spec();
    } else {
      for (auto& t : t_) t = fld();
      for (R** f : {&rb_, &rr_, &rz_, &rp_, &rw_, &rt2_, &kxy_, &kxz_, &kyz_, &kyy_, &kzz_})
        *f = fld();
      wh_ = spec();
      pf_ = dalloc<R>(Ns_);
    }
    make_plans();
    GLIA_CUDA(cudaStreamSynchronize(stream_));
  }

  ~Engine() override {
    cudaStreamSynchronize(stream_);
    if (cg_exec_) cudaGraphExecDestroy(cg_exec_);
    for (cufftHandle* p : {&r2c1_, &c2r1_, &r2c3_, &c2r3_, &p2d_, &r2c2d3_, &c2r2d3_})
      if (*p) cufftDestroy(*p);
    destroy_batch_plans();
    for (auto& kv : sizes_) cudaFree(kv.first);
    if (hsc_) cudaFreeHost(hsc_);
    if (hst_) cudaFreeHost(hst_);
    if (own_stream_) cudaStreamDestroy(own_stream_);
    if (cap_side_) cudaStreamDestroy(cap_side_);
  }

  // ------------------------------------------------------------------------------------------
  // configuration
  // ------------------------------------------------------------------------------------------
  void set_pointer_mode(int mode) override {
    if (mode < GLIA_PTR_HOST_F64 || mode > GLIA_PTR_DEVICE_F32)
      throw Error(GLIA_ERR_INVALID, "unknown pointer mode");
    ptr_mode_ = mode;
  }
  void set_stream(void* s) override {
    stream_ = s ? (cudaStream_t)s : own_stream_;
    for (cufftHandle p : {r2c1_, c2r1_, r2c3_, c2r3_}) GLIA_CUFFT(cufftSetStream(p, stream_));
    if (zpass_) GLIA_CUFFT(cufftSetStream(p2d_, stream_));
    if (xpass_ && !own_)
      for (cufftHandle p : {r2c2d3_, c2r2d3_}) GLIA_CUFFT(cufftSetStream(p, stream_));
  }
  void synchronize() override { GLIA_CUDA(cudaStreamSynchronize(stream_)); }
  // CTAs per SM of the bandwidth kernels (grid-stride) and of the reducing kernels. Fewer CTAs
  // let kernels of contexts on other streams run beside this one's (small grids, batches).
  void set_launch_geometry(int pw_per_sm, int red_per_sm) override {
    if (pw_per_sm < 1 || pw_per_sm > 16 || red_per_sm < 1 || red_per_sm > kMaxRedBlocksPerSm)
      throw Error(GLIA_ERR_INVALID, "launch geometry: 1 <= pointwise <= 16, 1 <= reduce <= 8");
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    pw_blocks_ = sms_ * pw_per_sm;
    red_blocks_ = sms_ * red_per_sm;
    if (cg_exec_) cudaGraphExecDestroy(cg_exec_);  // the PCG graph bakes the launch shapes in
    cg_exec_ = nullptr;
    if (graph_state_ > 0) graph_state_ = 0;
  }
  int64_t device_bytes() const override { return bytes_; }

  void set_time(double dt, int nt, int order) override {
    if (!(dt > 0) || nt < 1 || (order != 1 && order != 2))
      throw Error(GLIA_ERR_INVALID, "set_time: need dt > 0, nt >= 1, order 1 or 2");
    dt_ = dt;
    nt_ = nt;
    order_ = order;
    ctx_dt_ = dt;  // a freshly built DiffusionSolver starts from TumorParameters::dt_
    state_done_ = adjoint_done_ = false;
    release_history();
  }
  void set_pcg(double rtol, int maxit, int pc_dt_mode, double pc_dt) override {
    if (!(rtol > 0) || maxit < 1 || pc_dt_mode < 0 || pc_dt_mode > 2)
      throw Error(GLIA_ERR_INVALID, "set_pcg: bad arguments");
    rtol_ = rtol;
    maxit_ = maxit;
    pc_dt_mode_ = pc_dt_mode;
    pc_dt_fixed_ = pc_dt;
  }
  void set_history(int mode, int every, int adjoint_store) override {
    if (mode != GLIA_HISTORY_FULL && mode != GLIA_HISTORY_CHECKPOINT && mode != GLIA_HISTORY_OFF)
      throw Error(GLIA_ERR_INVALID, "set_history: unknown mode");
    if (mode == GLIA_HISTORY_CHECKPOINT && (every < 1 || ref_))
      throw Error(GLIA_ERR_INVALID,
                  "set_history: checkpointing needs every >= 1 and the fused engine");
    hist_mode_ = mode;
    every_ = every;
    adjoint_store_ = adjoint_store != 0;
    state_done_ = adjoint_done_ = false;
    release_history();
  }
  void set_opt(const glia_opt_settings& s) override {
    if (s.np < 0 || s.nk < 1 || s.nk > 3 || s.nr < 1 || s.nr > 3)
      throw Error(GLIA_ERR_INVALID, "set_opt: need np >= 0, 1 <= nk, nr <= 3");
    opt_ = s;
  }

  // ------------------------------------------------------------------------------------------
  // material properties, coefficients, preconditioner
  // ------------------------------------------------------------------------------------------
  void set_tissue(const void* wm, const void* gm, const void* csf, const void* vt) override {
    R* dst[4] = {wm_, gm_, csf_, vt_};
    const void* src[4] = {wm, gm, csf, vt};
    for (int i = 0; i < 4; i++) {
      if (src[i])
        import_field(src[i], dst[i]);
      else
        GLIA_CUDA(cudaMemsetAsync(dst[i], 0, N_ * sizeof(R), stream_));
    }
    k_matprop<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, wm_, gm_, csf_, vt_, bg_, filter_,
                                                         sc_, 0, ws_);
    GLIA_LAUNCH_CHECK();
    filter_sum_ = read_red(0);
    tissue_set_ = true;
  }
  void set_tissue_sinusoidal() override {
    k_sinusoid<R><<<red_blocks_, kThreads, 0, stream_>>>(g_, wm_, gm_, csf_, vt_, bg_, filter_,
                                                          nullptr, 0.0, sc_, 0, ws_);
    GLIA_LAUNCH_CHECK();
    filter_sum_ = (double)N_;
    tissue_set_ = true;
  }
  // DiffCoef::setValues (src/mat/DiffCoef.cpp:77-132)
  void diffcoef_set(double ks, double kgm, double kglm) {
    k_scale_ = ks;
    k_gm_wm_ = kgm;
    k_glm_wm_ = kglm;
    double dgm = ks * kgm, dwm = ks, dglm = ks * kglm;
    dgm = (dgm <= 0) ? 0.0 : dgm;
    dglm = (dglm <= 0) ? 0.0 : dglm;
    k_assemble<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, kxx_, wm_, gm_, csf_, dwm, dgm,
                                                          dglm, sc_, 0, ws_);
    GLIA_LAUNCH_CHECK();
    const double ksum = read_red(0);
    // filter sum: MatProp filter (src/mat/DiffCoef.cpp:109)
    kxx_avg_ = ksum * (1.0 / filter_sum_);
    kxx_sinusoidal_ = false;
    if (ref_) ref_copy_k();
  }
  // ReacCoef::setValues (src/mat/ReacCoef.cpp:13-38)
  void reaccoef_set(double rs, double rgm, double rglm) {
    rho_scale_ = rs;
    r_gm_wm_ = rgm;
    r_glm_wm_ = rglm;
    double dgm = rs * rgm, dwm = rs, dglm = rs * rglm;
    dgm = (dgm <= 0) ? 0.0 : dgm;
    dglm = (dglm <= 0) ? 0.0 : dglm;
    k_assemble<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, rho_, wm_, gm_, csf_, dwm, dgm,
                                                          dglm, sc_, 1, ws_);
    GLIA_LAUNCH_CHECK();
    if (plane()) {
      k_max<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, rho_, ws_.partials, 1, sc_, ws_.counter);
      GLIA_LAUNCH_CHECK();
      rho_max_ = read_red(1);
    }
  }
  void set_coefficients(double k, double kgm, double kglm, double rho, double rgm,
                        double rglm) override {
    diffcoef_set(k, kgm, kglm);
    reaccoef_set(rho, rgm, rglm);
    prec_factor();
  }
  void set_diffusivity_sinusoidal(double scale) override {
    k_scale_ = scale;
    k_sinusoid<R><<<red_blocks_, kThreads, 0, stream_>>>(g_, nullptr, nullptr, nullptr, nullptr,
                                                          nullptr, nullptr, kxx_, scale, sc_, 0,
                                                          ws_);
    GLIA_LAUNCH_CHECK();
    kxx_avg_ = read_red(0) * (1.0 / (double)N_);
    kxx_sinusoidal_ = true;
    if (ref_) ref_copy_k();
  }
  double pc_dt_now() const { return pc_dt_mode_ == GLIA_PC_DT_FIXED ? pc_dt_fixed_ : ctx_dt_; }
  // DiffusionSolver::precFactor (src/pde/DiffusionSolver.cpp:119-180): the preconditioner is the
  // pair (kbar, dt_pc) captured now; the fused path evaluates it from wave numbers on the fly.
  void prec_factor_dt(double dtpc) {
    pc_kbar_ = kxx_avg_;
    pc_dt_ = dtpc;
    if (ref_) {
      k_precfactor<R><<<pw_blocks_, kThreads, 0, stream_>>>(g_, pf_, dtpc, kxx_avg_);
      GLIA_LAUNCH_CHECK();
    }
  }
  void prec_factor() override { prec_factor_dt(pc_dt_now()); }

  // ------------------------------------------------------------------------------------------
  // diffusion solve
  // ------------------------------------------------------------------------------------------
  int diffusion_solve(void* c, double dt) override {
    if (!(dt > 0)) throw Error(GLIA_ERR_INVALID, "diffusion_solve: dt must be > 0");
    import_field(c, tmp_);
    solve(tmp_, dt, nullptr, nullptr, 0.0);
    sync_sweep();
    export_field(tmp_, c);
    return ksp_itr_;
  }

  // DiffusionSolver::solve (src/pde/DiffusionSolver.cpp:217-250). chat_slot receives F(c) (the
  // state spectrum, kept for the kappa gradient); cx/kdot_w add kdot_w * <cx, D c> to acc[6].
  // which: 0 state, 1 adjoint, 2 other (set-up, recomputation) for the iteration counters.
  // The fused engine does not wait for the solve: its outcome is folded into device counters
  // that sync_sweep() reads once per sweep.
  // pre: a reaction step taken on c first (with a plane kernel only).
  struct Pre {
    int mode = 0;  // PlaneArgs::pre
    const R* lin = nullptr;
    R* half = nullptr;
  };
  void solve(R* c, double dts, R* chat_slot, const R* cx, double kdot_w, int which = 2,
             Pre pre = {}) {
    ctx_dt_ = dts;
    if (pc_dt_mode_ == GLIA_PC_DT_MATCHED) prec_factor_dt(2.0 * dts);
    st_.total_diffusion_solves++;
    if (k_scale_ == 0) {
      ksp_itr_ = 0;
      if (chat_slot) spectrum(c, chat_slot);
      return;
    }
    if (ref_) {
      ref_solve(c, dts);
      if (which < 2) (which == 0 ? st_.diff_ksp_itr_state : st_.diff_ksp_itr_adj) += ksp_itr_;
    } else {
      fused_solve(c, dts, chat_slot ? chat_slot : chat_, cx, kdot_w, which, pre);
    }
  }

  // Arguments and launch of the grid's plane kernel (plane.cuh), all CTAs resident at once.
  static constexpr bool kPlane = std::is_same<R, double>::value;
  bool plane() const { return plane_.fn != nullptr; }
  // Whether this context's work takes the plane kernel. Rounding in tumour-free tissue grows like
  // exp(rho T) over a simulation, and its gradient feels it most: against cuFFT's transforms the
  // plane kernel moves FP64 gradients by 2e-13 of their norm at rho T = 5, 3e-11 at 10, 2e-10 at 10.5,
  // 4e-9 at 12 and 3e-8 at 14 (largest of 28 to 56 problems each, 16^3 to 96^3, 32^3 mostly; states by
  // a hundredth of that). FP64 results may move by 1e-9, so cuFFT's transforms stay beyond 10.5.
  bool plane_now() const { return plane() && rho_max_ * dt_ * nt_ <= kPlaneGrowth; }
  static double2* cx2(R* p) { return reinterpret_cast<double2*>(p); }
  static const double2* cx2(const R* p) { return reinterpret_cast<const double2*>(p); }
  PlaneArgs plane_args(int prog, const R* in, R* out, R* chat) {
    PlaneArgs a{};
    a.prog = prog;
    a.in = in;
    a.out = out;
    a.k = kxx_;
    a.chat = cx2(chat);
    a.xhat = cx2(xhat_);
    a.rhat = cx2(rhat_);
    a.phat = cx2(phat_);
    a.G = cx2(g3r_);
    a.M = cx2(g3s_);
    a.W = cx2(plane_w_);
    a.sc = sc_;
    a.part = plane_part_;
    a.bar = plane_bar_;
    a.wait = plane_wait_;
    a.tw = plane_tw_;
    a.pf = plane_pf_;
    return a;
  }
  void plane_launch(PlaneArgs& a, double bytes) {
    void* args[] = {&a};
    const int grid = std::min({plane_.items, plane_res_, red_blocks_});
    GLIA_TIMED(KS_PLANE, bytes,
               GLIA_CUDA(cudaLaunchCooperativeKernel(plane_.fn, dim3(grid), dim3(plane_.threads),
                                                     args, plane_.smem, stream_)));
  }
  // spectrum of a real field
  void spectrum(const R* in, R* out) {
    if constexpr (kPlane) {
      if (plane_now()) {
        PlaneArgs a = plane_args(PP_SPEC, in, nullptr, out);
        plane_launch(a, FB() + SB());
        st_.total_fft_execs += 1;
        return;
      }
    }
    r2c(r2c1_, in, out);
  }
  void plane_solve(R* c, double dts, R* chat, const R* cx, double kdot_w, int which, Pre pre) {
    PlaneArgs a = plane_args(PP_SOLVE, c, c, chat);
    a.which = which;
    a.pre = pre.mode;
    a.rho = rho_;
    a.lin = pre.lin;
    a.half = pre.half;
    a.dt = dt_;
    a.cx = cx2(cx);
    a.a_cn = 0.5 * dts;
    a.pc_c = 0.25 * pc_dt_ * pc_kbar_;
    if (plane_pc_ != a.pc_c) {
      k_pc_field<R><<<pw_blocks_, kThreads, 0, stream_>>>(g_, plane_pf_, a.pc_c);
      GLIA_LAUNCH_CHECK();
      plane_pc_ = a.pc_c;
    }
    a.rtol = rtol_;
    a.abstol = abstol_;
    a.divtol = divtol_;
    a.maxit = maxit_;
    a.kdot_weight = kdot_w;
    plane_launch(a, 3 * FB());  // c in and out, k
    graph_solves_ = true;
    st_.total_fft_execs += 8;  // there, the set-up's D apply, back
  }

  void fused_solve(R* c, double dts, R* chat, const R* cx, double kdot_w, int which, Pre pre) {
    if constexpr (kPlane) {
      if (plane_now()) {
        plane_solve(c, dts, chat, cx, kdot_w, which, pre);
        return;
      }
    }
    k_solve_config<<<1, 1, 0, stream_>>>(sc_, 0.5 * dts, 0.25 * pc_dt_ * pc_kbar_, rtol_, abstol_,
                                         divtol_, maxit_, kdot_w);
    GLIA_LAUNCH_CHECK();
    // set-up: chat = F c; D c; b = c + a D c; r0 = 2 a D c; x0 = c; n = 0 convergence test
    r2c(r2c1_, c, chat);
    d_front<false>(chat, nullptr);
    d_back<EPI_SETUP>(chat, cx, xhat_, rhat_, R(0));
    if (capture_) {
      capture_pcg_loop();  // the loop as a conditional node of the graph being captured
    } else if (use_graph()) {
      GLIA_CUDA(cudaGraphLaunch(cg_exec_, stream_));  // the whole PCG loop, no host round trip
      graph_solves_ = true;
    } else {
      SolveStatus s = read_status();
      while (s.status == 0) {
        cg_iteration();
        s = read_status();
      }
    }
    c2r(c2r1_, xhat_, c);  // x = F^-1 (x')
    k_solve_finish<<<1, 1, 0, stream_>>>(sc_, which);
    GLIA_LAUNCH_CHECK();
  }

  // First half of a spectral D apply, from the spectrum src (plain) or from the new PCG direction
  // p = P r + b p (CGDIR: src = r, pdir = p), up to the spectra of k grad u that d_back
  // diverges. Own transforms (default, FP32, n = 64 ... 256): k_xinv -> G in g3r_, k_yinv_bulk
  // (or k_yinv) -> packed lines in g3s_, k_zpass2 (or k_zpass; k multiplied there, in place),
  // k_yfwd -> M in g3r_. "2d": the
  // x pass writes (x, ky, kz) per component to g3s_ and cuFFT does batched 2-D (y, z)
  // transforms around k_mul_k3. Otherwise g3s_ holds the full 3-D spectra.
  template <bool CGDIR>
  void d_front(const R* src, R* pdir) {
    if (own_) {  // no cuFFT: x, y, z passes of our own, k multiplied inside the z pass
      GLIA_TIMED(KS_XINV, SB() * (CGDIR ? 5 : 3), launch_xinv<CGDIR>(src, pdir));
      GLIA_TIMED(KS_YINV, SB() * 2 + FB() * 3, launch_own(0));
      GLIA_TIMED(KS_ZFUSED, FB() * 7, launch_own(1));
      GLIA_TIMED(KS_YFWD, FB() * 3 + SB() * 2, launch_own(2));
      return;
    }
    if (xpass_) {
      GLIA_TIMED(KS_XINV, SB() * (CGDIR ? 6 : 4), launch_xinv<CGDIR>(src, pdir));
      c2r(c2r2d3_, g3s_, g3r_, 3);
      GLIA_TIMED(KS_MUL_K3, FB() * 7,
                 k_mul_k3<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, g3r_, kxx_, sc_, 0));
      r2c(r2c2d3_, g3r_, g3s_, 3);
      return;
    }
    launch_grad3<CGDIR>(src, pdir);
    apply_k_spectral();
  }
  // Second half: divergence of k grad u in spectral space and the caller's epilogue
  // (k_spec_div semantics: EPI_APPLYD out = scale D; EPI_SETUP solve set-up; EPI_CGW w = A p).
  template <int EPI>
  void d_back(const R* aux_in, const R* cx, R* out, R* aux_out, R scale) {
    const double nin = own_ ? 2 : 3;  // gradient blocks read by the divergence
    const double bytes = EPI == EPI_APPLYD ? SB() * (nin + 1)
                         : EPI == EPI_SETUP ? SB() * (nin + (cx ? 4 : 3))
                                            : SB() * (nin + 2);
    const int slot = EPI == EPI_APPLYD ? KS_DIV_APPLYD : (EPI == EPI_SETUP ? KS_DIV_SETUP : KS_DIV_CGW);
    const int blocks = EPI == EPI_APPLYD ? pw_blocks_ : red_blocks_;
    if (xpass_) {
      const int xslot = EPI == EPI_APPLYD ? KS_XFWD_APPLYD
                        : (EPI == EPI_SETUP ? KS_XFWD_SETUP : KS_XFWD_CGW);
      GLIA_TIMED(xslot, bytes, launch_xfwd<EPI>(aux_in, cx, out, aux_out, scale, blocks));
      return;
    }
    GLIA_TIMED(slot, bytes,
               k_spec_div<R, EPI><<<blocks, kThreads, 0, stream_>>>(g_, g3s_, aux_in, cx, out,
                                                                    aux_out, scale, sc_, ws_));
  }
  // x-pass and own-transform launches; kernels are instantiated per grid size (n = 64, 128, 256)
  template <int NN, bool CGDIR, bool OUT2>
  void xinv_n(const R* src, R* pdir, R* G) {
    if constexpr (std::is_same<R, float>::value) {
      constexpr int MODE = CGDIR ? 1 : 0;
      const int grid = std::min(xres_inv_, pw_blocks_);
      k_xinv<NN, MODE, OUT2><<<grid, 256, xinv_smem_bytes<NN, MODE>(), stream_>>>(
          g_, src, pdir, G, sc_, tw256_);
    }
  }
  template <bool CGDIR>
  void launch_xinv(const R* src, R* pdir) {
    const int n = g_.n;
    if (own_) {
      if (n == 256) xinv_n<256, CGDIR, true>(src, pdir, g3r_);
      else if (n == 128) xinv_n<128, CGDIR, true>(src, pdir, g3r_);
      else xinv_n<64, CGDIR, true>(src, pdir, g3r_);
    } else {
      if (n == 256) xinv_n<256, CGDIR, false>(src, pdir, g3s_);
      else if (n == 128) xinv_n<128, CGDIR, false>(src, pdir, g3s_);
      else xinv_n<64, CGDIR, false>(src, pdir, g3s_);
    }
  }
  template <int NN, int EPI, bool IN2>
  void xfwd_n(const R* G, const R* aux_in, const R* cx, R* out, R* aux_out, R scale, int blocks) {
    if constexpr (std::is_same<R, float>::value) {
      if constexpr (IN2)
        k_xfwd_own<NN, EPI><<<blocks, 256, xfwd_own_smem_bytes<NN>(), stream_>>>(
            g_, G, aux_in, cx, out, aux_out, scale, sc_, ws_, tw256_);
      else
        k_xfwd<NN, EPI><<<blocks, 256, 0, stream_>>>(g_, G, aux_in, cx, out, aux_out, scale, sc_,
                                                     ws_, tw256_);
    }
  }
  template <int EPI>
  void launch_xfwd(const R* aux_in, const R* cx, R* out, R* aux_out, R scale, int blocks) {
    const int n = g_.n;
    blocks = std::min(xres_fwd_, blocks);
    if (own_) {
      if (n == 256) xfwd_n<256, EPI, true>(g3r_, aux_in, cx, out, aux_out, scale, blocks);
      else if (n == 128) xfwd_n<128, EPI, true>(g3r_, aux_in, cx, out, aux_out, scale, blocks);
      else xfwd_n<64, EPI, true>(g3r_, aux_in, cx, out, aux_out, scale, blocks);
    } else {
      if (n == 256) xfwd_n<256, EPI, false>(g3s_, aux_in, cx, out, aux_out, scale, blocks);
      else if (n == 128) xfwd_n<128, EPI, false>(g3s_, aux_in, cx, out, aux_out, scale, blocks);
      else xfwd_n<64, EPI, false>(g3s_, aux_in, cx, out, aux_out, scale, blocks);
    }
  }
  // own y / z passes: 0 = y inverse (g3r_ -> g3s_), 1 = z pass (g3s_ in place, k), 2 = k_yfwd
  // (g3s_ -> g3r_)
  template <int NN>
  void own_n(int which) {
    if constexpr (std::is_same<R, float>::value) {
      if (which == 0 && yinv_bulk_)
        k_yinv_bulk<NN><<<std::min(own_res_[0], pw_blocks_), 256, yinv_bulk_smem_bytes<NN>(),
                          stream_>>>(g3r_, g3s_, tw256_, sc_);
      else if (which == 0)
        k_yinv<NN><<<std::min(own_res_[0], pw_blocks_), 256, yinv_smem_bytes<NN>(), stream_>>>(
            g3r_, g3s_, tw256_);
      else if (which == 1 && zpass2_)
        k_zpass2<NN><<<std::min(own_res_[1], pw_blocks_), 256, zpass2_smem_bytes<NN>(),
                       stream_>>>(g3s_, kxx_, tw256_, zrev_);
      else if (which == 1)
        k_zpass<NN><<<std::min(own_res_[1], pw_blocks_), 256, zpass_smem_bytes<NN>(), stream_>>>(
            g3s_, kxx_, tw256_);
      else if (tma_)
        k_yfwd_tma<NN><<<std::min(own_res_[2], pw_blocks_), 256, yfwd_tma_smem_bytes<NN>(),
                         stream_>>>(kmap_, g3r_, tw256_, sc_);
      else
        k_yfwd<NN><<<std::min(own_res_[2], pw_blocks_), 256, yfwd_smem_bytes<NN>(), stream_>>>(
            g3s_, g3r_, tw256_);
    }
  }
  void launch_own(int which) {
    const int n = g_.n;
    if (n == 256) own_n<256>(which);
    else if (n == 128) own_n<128>(which);
    else own_n<64>(which);
  }
  // resident CTAs of the x-pass and own-transform kernels on this device (persistent grids:
  // every CTA walks the same number of tiles to within one)
  template <int NN>
  void init_xpass_grids() {
    if constexpr (std::is_same<R, float>::value) {
      auto per_sm = [](auto kern, int smem) {
        if (smem > 48 * 1024)
          GLIA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        int b = 0;
        GLIA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, 256, smem));
        return std::max(1, std::min(b, kMaxRedBlocksPerSm));
      };
      if (own_) {
        xres_inv_ = sms_ * std::min(per_sm(k_xinv<NN, 0, true>, xinv_smem_bytes<NN, 0>()),
                                    per_sm(k_xinv<NN, 1, true>, xinv_smem_bytes<NN, 1>()));
        constexpr int fs = xfwd_own_smem_bytes<NN>();
        xres_fwd_ = sms_ * std::min({per_sm(k_xfwd_own<NN, EPI_APPLYD>, fs),
                                     per_sm(k_xfwd_own<NN, EPI_SETUP>, fs),
                                     per_sm(k_xfwd_own<NN, EPI_CGW>, fs)});
        // y-inverse rows staged by bulk copies (default) or per-thread cp.async
        // (GLIA_YINV_BULK=0)
        const char* yb = std::getenv("GLIA_YINV_BULK");
        yinv_bulk_ = !(yb && yb[0] == '0');
        own_res_[0] = sms_ * (yinv_bulk_ ? per_sm(k_yinv_bulk<NN>, yinv_bulk_smem_bytes<NN>())
                                         : per_sm(k_yinv<NN>, yinv_smem_bytes<NN>()));
        // z pass: two real lines per complex transform (k_zpass2) unless GLIA_ZPASS2=0 picks
        // the even/odd half-length version (k_zpass)
        const char* z2 = std::getenv("GLIA_ZPASS2");
        zpass2_ = !(z2 && z2[0] == '0');
        // z pass over its line blocks in descending order (default; GLIA_ZREV=0 ascending): the
        // y-inverse pass before it writes the lines in ascending order, so the z pass starts on
        // the lines still in L2, and the y-forward pass after it (ascending) starts on the lines
        // the z pass wrote last
        const char* zr = std::getenv("GLIA_ZREV");
        zrev_ = !(zr && zr[0] == '0');
        own_res_[1] = sms_ * (zpass2_ ? per_sm(k_zpass2<NN>, zpass2_smem_bytes<NN>())
                                      : per_sm(k_zpass<NN>, zpass_smem_bytes<NN>()));
        const char* te = std::getenv("GLIA_TMA");
        tma_ = te && te[0] == '1';
        own_res_[2] = sms_ * (tma_ ? per_sm(k_yfwd_tma<NN>, yfwd_tma_smem_bytes<NN>())
                                   : per_sm(k_yfwd<NN>, yfwd_smem_bytes<NN>()));
        // TMA view of the packed arrays K = [K_x, K_y, L_z]: 3 n^2 rows of n floats, tiles of
        // 2T floats x n rows (used by k_yfwd<TMA = true>, GLIA_TMA=1)
        if (tma_)
          kmap_ = make_tmap_f32_2d(g3s_, (uint64_t)NN, 3ull * NN * NN, 2 * YDecomp<NN>::T, NN);
      } else {
        xres_inv_ = sms_ * std::min(per_sm(k_xinv<NN, 0, false>, xinv_smem_bytes<NN, 0>()),
                                    per_sm(k_xinv<NN, 1, false>, xinv_smem_bytes<NN, 1>()));
        xres_fwd_ = sms_ * std::min({per_sm(k_xfwd<NN, EPI_APPLYD>, 0),
                                     per_sm(k_xfwd<NN, EPI_SETUP>, 0),
                                     per_sm(k_xfwd<NN, EPI_CGW>, 0)});
      }
    }
  }

  // one PCG iteration of the fused engine (launched directly, or captured as the loop body)
  void cg_iteration() {
    d_front<true>(rhat_, phat_);  // p = P r + b p and the spectra of k grad p
    d_back<EPI_CGW>(phat_, nullptr, what_, nullptr, R(0));  // w = A p, <p, w>, alpha
    GLIA_TIMED(KS_CG_UPDATE, SB() * 6,
               k_cg_update<R><<<red_blocks_, kThreads, 0, stream_>>>(g_, xhat_, phat_, rhat_,
                                                                     what_, sc_, ws_));
  }

  // The PCG loop as one CUDA graph: [k_cond_set] -> WHILE(cond) { iteration; k_cond_step }.
  // All buffers and scalars it touches are fixed per engine, so one instantiation serves every
  // solve. If the graph cannot be built, the host-driven loop is used instead.
  bool use_graph() {
    if (tm_.on || graph_state_ < 0) return false;
    if (graph_state_ == 0) build_cg_graph();
    return graph_state_ > 0;
  }
  void build_cg_graph() {
    cudaGraph_t g = nullptr;
    cudaStream_t cs = nullptr;
    cudaStream_t saved = stream_;
    bool capturing = false;
    try {
      GLIA_CUDA(cudaGraphCreate(&g, 0));
      cudaGraphConditionalHandle h;
      GLIA_CUDA(cudaGraphConditionalHandleCreate(&h, g, 0, 0));
      DevScalars* scp = sc_;
      void* args_set[] = {&scp, &h};
      cudaKernelNodeParams kp = {};
      kp.func = (void*)k_cond_set;
      kp.gridDim = dim3(1);
      kp.blockDim = dim3(1);
      kp.kernelParams = args_set;
      cudaGraphNode_t head;
      GLIA_CUDA(cudaGraphAddKernelNode(&head, g, nullptr, 0, &kp));
      cudaGraphNodeParams cp = {};
      cp.type = cudaGraphNodeTypeConditional;
      cp.conditional.handle = h;
      cp.conditional.type = cudaGraphCondTypeWhile;
      cp.conditional.size = 1;
      cudaGraphNode_t loop;
      GLIA_CUDA(cudaGraphAddNode(&loop, g, &head, nullptr, 1, &cp));
      cudaGraph_t body = cp.conditional.phGraph_out[0];
      GLIA_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
      for (cufftHandle p : {r2c3_, c2r3_}) GLIA_CUFFT(cufftSetStream(p, cs));
      if (zpass_) GLIA_CUFFT(cufftSetStream(p2d_, cs));
      if (xpass_ && !own_)
        for (cufftHandle p : {r2c2d3_, c2r2d3_}) GLIA_CUFFT(cufftSetStream(p, cs));
      stream_ = cs;
      GLIA_CUDA(cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0,
                                              cudaStreamCaptureModeThreadLocal));
      capturing = true;
      cg_iteration();
      k_cond_step<<<1, 1, 0, cs>>>(sc_, h);
      GLIA_LAUNCH_CHECK();
      cudaGraph_t captured = nullptr;
      capturing = false;
      GLIA_CUDA(cudaStreamEndCapture(cs, &captured));
      GLIA_CUDA(cudaGraphInstantiate(&cg_exec_, g, 0));
      graph_state_ = 1;
    } catch (const Error&) {
      if (capturing) {
        cudaGraph_t junk = nullptr;
        cudaStreamEndCapture(cs, &junk);
      }
      cudaGetLastError();
      cg_exec_ = nullptr;
      graph_state_ = -1;
    }
    stream_ = saved;
    for (cufftHandle p : {r2c3_, c2r3_}) cufftSetStream(p, stream_);
    if (zpass_) cufftSetStream(p2d_, stream_);
    if (xpass_ && !own_)
      for (cufftHandle p : {r2c2d3_, c2r2d3_}) cufftSetStream(p, stream_);
    if (cs) cudaStreamDestroy(cs);
    if (g) cudaGraphDestroy(g);
  }

  // Inside a capture of stream_: [k_cond_set] -> WHILE(cond) { iteration; k_cond_step }, the
  // same loop as the per-engine PCG graph, added as nodes of the graph being captured (its body
  // captured from a side stream into the conditional node's body graph).
  void capture_pcg_loop() {
    cudaStreamCaptureStatus cst;
    cudaGraph_t cg = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    GLIA_CUDA(cudaStreamGetCaptureInfo(stream_, &cst, nullptr, &cg, &deps, nullptr, &nd));
    if (cst != cudaStreamCaptureStatusActive)
      throw Error(GLIA_ERR_STATE, "eval_capture: the context's stream is not being captured");
    cudaGraphConditionalHandle h;
    GLIA_CUDA(cudaGraphConditionalHandleCreate(&h, cg, 0, 0));
    k_cond_set<<<1, 1, 0, stream_>>>(sc_, h);
    GLIA_LAUNCH_CHECK();
    GLIA_CUDA(cudaStreamGetCaptureInfo(stream_, &cst, nullptr, &cg, &deps, nullptr, &nd));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t loop;
    GLIA_CUDA(cudaGraphAddNode(&loop, cg, deps, nullptr, nd, &cp));
    GLIA_CUDA(cudaStreamUpdateCaptureDependencies(stream_, &loop, nullptr, 1,
                                                  cudaStreamSetCaptureDependencies));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    if (!cap_side_) GLIA_CUDA(cudaStreamCreateWithFlags(&cap_side_, cudaStreamNonBlocking));
    cudaStream_t saved = stream_;
    stream_ = cap_side_;
    set_plan_streams(cap_side_);
    bool capturing = false;
    try {
      GLIA_CUDA(cudaStreamBeginCaptureToGraph(cap_side_, body, nullptr, nullptr, 0,
                                              cudaStreamCaptureModeRelaxed));
      capturing = true;
      cg_iteration();
      k_cond_step<<<1, 1, 0, cap_side_>>>(sc_, h);
      GLIA_LAUNCH_CHECK();
      cudaGraph_t captured = nullptr;
      capturing = false;
      GLIA_CUDA(cudaStreamEndCapture(cap_side_, &captured));
    } catch (...) {
      if (capturing) {
        cudaGraph_t junk = nullptr;
        cudaStreamEndCapture(cap_side_, &junk);
      }
      stream_ = saved;
      set_plan_streams(saved);
      throw;
    }
    stream_ = saved;
    set_plan_streams(saved);
    cap_solves_ += 1;
  }
  void set_plan_streams(cudaStream_t s) {
    for (cufftHandle p : {r2c1_, c2r1_, r2c3_, c2r3_}) GLIA_CUFFT(cufftSetStream(p, s));
    if (zpass_) GLIA_CUFFT(cufftSetStream(p2d_, s));
    if (xpass_ && !own_)
      for (cufftHandle p : {r2c2d3_, c2r2d3_}) GLIA_CUFFT(cufftSetStream(p, s));
  }

  // Reads the device-side solve statistics of the sweep and reports the first failed solve.
  void sync_sweep() {
    if (ref_ || capture_) return;  // a captured evaluation reads its statistics in eval_finish
    GLIA_CUDA(cudaMemcpyAsync(hsc_, sc_, sizeof(DevScalars), cudaMemcpyDeviceToHost, stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    tm_.harvest();
    const DevScalars& h = *hsc_;
    st_.diff_ksp_itr_state += h.sum_its[0];
    st_.diff_ksp_itr_adj += h.sum_its[1];
    st_.total_pcg_iterations += h.sum_its[0] + h.sum_its[1] + h.sum_its[2];
    // transforms launched inside the PCG graph: 3 C2R + 3 R2C per iteration
    if (graph_solves_) st_.total_fft_execs += 6 * (h.sum_its[0] + h.sum_its[1] + h.sum_its[2]);
    graph_solves_ = false;
    st_.max_ksp_itr = std::max(st_.max_ksp_itr, h.max_its);
    st_.last_rnorm = h.last_dp;
    st_.last_ksp_itr = h.it;
    ksp_itr_ = h.it;
    k_solve_stats_reset<<<1, 1, 0, stream_>>>(sc_);
    GLIA_LAUNCH_CHECK();
    if (h.dev_fault) raise_device_fault();
    if (h.err_status < 0) finish_solve(SolveStatus{h.err_status, h.err_its, h.last_dp});
  }
  void selftest_bounded_wait() override {
    if constexpr (!std::is_same<R, float>::value) {
      throw Error(GLIA_ERR_INVALID, "selftest_bounded_wait: FP32 contexts only");
    } else {
      GLIA_CUDA(cudaStreamSynchronize(stream_));
      k_selftest_wait<<<1, 32, 0, stream_>>>(&sc_->dev_fault);
      GLIA_LAUNCH_CHECK();
      int f = 0;
      GLIA_CUDA(cudaMemcpyAsync(&f, &sc_->dev_fault, sizeof(int), cudaMemcpyDeviceToHost,
                                stream_));
      GLIA_CUDA(cudaStreamSynchronize(stream_));
      GLIA_CUDA(cudaMemsetAsync(&sc_->dev_fault, 0, sizeof(int), stream_));
      if (f != 1) throw Error(GLIA_ERR_CUDA, "bounded wait did not record its timeout");
      // the context must still run kernels
      k_solve_stats_reset<<<1, 1, 0, stream_>>>(sc_);
      GLIA_LAUNCH_CHECK();
      GLIA_CUDA(cudaStreamSynchronize(stream_));
    }
  }
  void selftest_wait_limit(int64_t clocks) override {
    if (!plane()) throw Error(GLIA_ERR_INVALID, "selftest_wait_limit: no plane kernel");
    plane_wait_ = clocks ? clocks : kPlaneWait;
  }
  // a kernel's bounded wait ran out (its CTA stopped early): the results are invalid
  [[noreturn]] void raise_device_fault() {
    GLIA_CUDA(cudaMemsetAsync(&sc_->dev_fault, 0, sizeof(int), stream_));
    if (plane_bar_) GLIA_CUDA(cudaMemsetAsync(plane_bar_, 0, 2 * sizeof(unsigned), stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    throw Error(GLIA_ERR_CUDA, "a device-side wait did not complete within its time limit");
  }
  void check_device_fault() {
    if (ref_) return;
    int f = 0;
    GLIA_CUDA(cudaMemcpyAsync(&f, &sc_->dev_fault, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    if (f) raise_device_fault();
  }

  template <bool CGDIR>
  void launch_grad3(const R* src, R* pdir) {
    GLIA_TIMED(CGDIR ? KS_SPEC_GRAD3_CG : KS_SPEC_GRAD3, SB() * (CGDIR ? 6 : 4),
               k_spec_grad3<R, CGDIR><<<pw_blocks_, kThreads, 0, stream_>>>(g_, src, pdir, g3s_,
                                                                            sc_));
  }
  // gradient spectra (g3s_) -> real gradient -> times k -> spectra of k * grad (g3s_).
  // FP32 with n = 64 ... 512: cuFFT does the (x, y) passes in place and k_zpass_mulk the fused
  // z pass; otherwise three-dimensional cuFFT transforms around k_mul_k3.
  void apply_k_spectral() {
    if (zpass_) {
      for (int j = 0; j < 3; j++) c2c2d(g3s_ + j * 2 * Ns_, CUFFT_INVERSE);
      const int lines = g_.n * g_.n;
      const int blocks = std::min((lines + kWarps - 1) / kWarps, sms_ * 8);
      GLIA_TIMED(KS_ZPASS, SB() * 6 + FB(), launch_zpass(blocks, lines));
      for (int j = 0; j < 3; j++) c2c2d(g3s_ + j * 2 * Ns_, CUFFT_FORWARD);
      return;
    }
    c2r(c2r3_, g3s_, g3r_, 3);
    GLIA_TIMED(KS_MUL_K3, FB() * 7,
               k_mul_k3<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, g3r_, kxx_, sc_, 0));
    r2c(r2c3_, g3r_, g3s_, 3);
  }

  void finish_solve(const SolveStatus& s) {
    ksp_itr_ = s.it;
    st_.last_ksp_itr = s.it;
    st_.max_ksp_itr = std::max(st_.max_ksp_itr, s.it);
    st_.total_pcg_iterations += s.it;
    st_.last_rnorm = s.dp;
    if (s.status < 0) {
      const char* why = s.status == -3   ? "maximum iterations"
                        : s.status == -4 ? "divergence tolerance"
                        : s.status == -8 ? "indefinite operator"
                                         : "NaN or Inf residual";
      throw Error(GLIA_ERR_NOT_CONVERGED, std::string("diffusion PCG stopped: ") + why +
                                              " after " + std::to_string(s.it) + " iterations");
    }
  }

  // ---- reference-structured path -----------------------------------------------------------
  void ref_copy_k() {  // DiffCoef keeps kyy = kzz = kxx and zero off-diagonal fields
    GLIA_CUDA(cudaMemcpyAsync(kyy_, kxx_, N_ * sizeof(R), cudaMemcpyDeviceToDevice, stream_));
    GLIA_CUDA(cudaMemcpyAsync(kzz_, kxx_, N_ * sizeof(R), cudaMemcpyDeviceToDevice, stream_));
    for (R* f : {kxy_, kxz_, kyz_}) GLIA_CUDA(cudaMemsetAsync(f, 0, N_ * sizeof(R), stream_));
  }
  void vaxpy(R* y, double a, const R* x) {
    GLIA_TIMED(KS_REF_VEC, FB() * 3, k_axpy<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, y, a, x));
  }
  void vaypx(R* y, double b, const R* x) {
    GLIA_TIMED(KS_REF_VEC, FB() * 3, k_aypx<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, y, b, x));
  }
  void vmult(R* z, const R* x, const R* y) {
    GLIA_TIMED(KS_REF_VEC, FB() * 3,
               k_pointwise_mult<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, z, x, y));
  }
  void vcopy(R* y, const R* x) {
    GLIA_TIMED(KS_COPY, FB() * 2,
               GLIA_CUDA(cudaMemcpyAsync(y, x, N_ * sizeof(R), cudaMemcpyDeviceToDevice, stream_)));
  }
  void vzero(R* y) { GLIA_CUDA(cudaMemsetAsync(y, 0, N_ * sizeof(R), stream_)); }
  double vdot(const R* x, const R* y) {  // PETSc VecDot: one reduction, scalar to the host
    GLIA_TIMED(KS_REF_DOT, FB() * 2,
               k_dot<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, x, y, sc_, 0, ws_));
    return read_red(0);
  }
  // SpectralOperators::computeGradient (src/grad/SpectralOperators.cpp:100-177)
  void ref_gradient(R* gx, R* gy, R* gz, const R* x) {
    r2c(r2c1_, x, xhat_);
    R* out[3] = {gx, gy, gz};
    for (int d = 0; d < 3; d++) {
      GLIA_TIMED(KS_REF_VEC, SB() * 2,
                 k_mult_wavenumber<R><<<pw_blocks_, kThreads, 0, stream_>>>(g_, d, xhat_, wh_));
      c2r(c2r1_, wh_, out[d]);
    }
  }
  // SpectralOperators::computeDivergence (src/grad/SpectralOperators.cpp:179-261)
  void ref_divergence(R* div, const R* dx, const R* dy, const R* dz) {
    const R* in[3] = {dx, dz, dy};
    const int dim[3] = {0, 2, 1};
    for (int q = 0; q < 3; q++) {
      r2c(r2c1_, in[q], xhat_);
      GLIA_TIMED(KS_REF_VEC, SB() * 2,
                 k_mult_wavenumber<R><<<pw_blocks_, kThreads, 0, stream_>>>(g_, dim[q], xhat_,
                                                                             wh_));
      c2r(c2r1_, wh_, q == 0 ? div : t_[7]);
      if (q) vaxpy(div, 1.0, t_[7]);
    }
  }
  // DiffCoef::applyD + applyK (src/mat/DiffCoef.cpp:206-271)
  void ref_applyD(R* dc, const R* c) {
    ref_gradient(t_[4], t_[5], t_[6], c);
    for (int i = 1; i < 4; i++) vzero(t_[i]);
    const R* K[3][3] = {{kxx_, kxy_, kxz_}, {kxy_, kyy_, kyz_}, {kxz_, kyz_, kzz_}};
    for (int row = 0; row < 3; row++)
      for (int col = 0; col < 3; col++) {
        vmult(t_[0], K[row][col], t_[4 + col]);
        vaxpy(t_[1 + row], 1.0, t_[0]);
      }
    ref_divergence(dc, t_[1], t_[2], t_[3]);
  }
  void ref_operatorA(R* y, const R* x) {  // operatorA (:97-117)
    vcopy(y, x);
    ref_applyD(rt2_, y);
    vaxpy(y, -0.5 * ctx_dt_, rt2_);
  }
  void ref_applyPC(R* y, const R* x) {  // applyPC (:182-215)
    vcopy(y, x);
    r2c(r2c1_, y, xhat_);
    GLIA_TIMED(KS_REF_VEC, SB() * 2 + Ns_ * sizeof(R),
               k_hadamard_real<R><<<pw_blocks_, kThreads, 0, stream_>>>(Ns_, xhat_, pf_));
    c2r(c2r1_, xhat_, y);
  }
  // KSPSolve_CG + KSPConvergedDefault with host scalars, as PETSc runs them
  void ref_solve(R* c, double dts) {
    vcopy(rb_, c);
    ref_applyD(rt2_, rb_);
    vaxpy(rb_, 0.5 * dts, rt2_);
    ref_operatorA(rr_, c);
    vaypx(rr_, -1.0, rb_);
    ref_applyPC(rz_, rr_);
    double dp = std::sqrt(vdot(rz_, rz_));
    ref_applyPC(rw_, rb_);
    double snorm = std::sqrt(vdot(rw_, rw_));
    if (snorm == 0) snorm = dp;
    const double rnorm0 = snorm, ttol = std::max(rtol_ * rnorm0, abstol_);
    auto conv = [&](double rn) {
      if (std::isnan(rn) || std::isinf(rn)) return -9;
      if (rn <= ttol) return 1;
      if (rn >= divtol_ * rnorm0) return -4;
      return 0;
    };
    int reason = conv(dp), its = 0;
    if (reason == 0) {
      double beta = vdot(rz_, rr_), betaold = 0, dpi = 0, dpiold = 0;
      int i = 0;
      do {
        its = i + 1;
        if (beta == 0.0) {
          reason = 2;
          break;
        }
        if (i == 0)
          vcopy(rp_, rz_);
        else
          vaypx(rp_, beta / betaold, rz_);
        dpiold = dpi;
        ref_operatorA(rw_, rp_);
        dpi = vdot(rp_, rw_);
        betaold = beta;
        if (dpi == 0.0 || (i > 0 && dpi * dpiold <= 0.0)) {
          reason = -8;
          break;
        }
        const double a = beta / dpi;
        vaxpy(c, a, rp_);
        vaxpy(rr_, -a, rw_);
        ref_applyPC(rz_, rr_);
        dp = std::sqrt(vdot(rz_, rz_));
        reason = conv(dp);
        if (reason) break;
        beta = vdot(rz_, rr_);
        i++;
      } while (i < maxit_);
      if (i >= maxit_ && reason == 0) reason = -3;
    }
    finish_solve(SolveStatus{reason < 0 ? reason : 0, its, dp});
  }

  // ------------------------------------------------------------------------------------------
  // D apply and smoother
  // ------------------------------------------------------------------------------------------
  void applyD_into(R* dc, const R* c) {
    if (ref_) {
      ref_applyD(dc, c);
      return;
    }
    if constexpr (kPlane) {
      if (plane_now()) {
        PlaneArgs a = plane_args(PP_APPLY, c, dc, chat_);
        plane_launch(a, 3 * FB());
        st_.total_fft_execs += 8;
        return;
      }
    }
    r2c(r2c1_, c, chat_);
    d_front<false>(chat_, nullptr);
    d_back<EPI_APPLYD>(nullptr, nullptr, xhat_, nullptr, (R)g_.invN);
    c2r(c2r1_, xhat_, dc);
  }
  void apply_d(const void* c, void* dc) override {
    import_field(c, tmp_);
    applyD_into(p0_, tmp_);
    check_device_fault();
    export_field(p0_, dc);
  }
  // DiffCoef::setSecondaryCoefficients (src/mat/DiffCoef.cpp:44-58): the Hessian's diffusivity
  // direction k~ = k1 wm + k2 gm + k3 csf (k2, k3 from the current ratios when nk = 1)
  void set_secondary_coefficients(double k1, double k2, double k3) override {
    if (opt_.nk == 1) {
      k2 = k_gm_wm_ * k1;
      k3 = k_glm_wm_ * k1;
    }
    if (!ksec_) ksec_ = fld();
    k_assemble_secondary<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, ksec_, wm_, gm_, csf_, k1,
                                                                   k2, k3);
    GLIA_LAUNCH_CHECK();
    ksec_set_ = true;
  }
  // DiffCoef::applyDWithSecondaryCoeffs (:273-300): out = div(k~ grad in), out may alias in. The
  // fused paths read the k field through kxx_, which points at k~ for this one apply.
  void applyD_secondary_into(R* out, const R* in) {
    if (!ksec_set_) throw Error(GLIA_ERR_STATE, "no secondary diffusion coefficients set");
    if (ref_) {
      ref_gradient(t_[4], t_[5], t_[6], in);
      vmult(t_[1], ksec_, t_[4]);
      vmult(t_[2], ksec_, t_[5]);
      vmult(t_[3], ksec_, t_[6]);
      ref_divergence(out, t_[1], t_[2], t_[3]);
      return;
    }
    struct Restore {
      R*& k;
      R* saved;
      ~Restore() { k = saved; }
    } restore{kxx_, kxx_};
    kxx_ = ksec_;
    applyD_into(out, in);
  }
  // spectrum of the normalised Weierstrass kernel for sigma, times h^3 / N
  // (SpectralOperators::weierstrassSmoother, src/grad/SpectralOperators.cpp:264-381)
  const R* smoother_kernel(double sigma) {
    if (wkern_ && wkern_sigma_ == sigma) return wkern_;
    if (!wkern_) wkern_ = spec();
    R* f = g3r_;
    k_weierstrass<R><<<red_blocks_, kThreads, 0, stream_>>>(g_, f, sigma, sc_, 0, ws_);
    GLIA_LAUNCH_CHECK();
    const double sum_f = read_red(0);
    const double h = 2.0 * M_PI / g_.n, h3 = h * h * h;
    k_scale<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, f, 1.0 / (sum_f * h3));
    GLIA_LAUNCH_CHECK();
    r2c(r2c1_, f, wkern_);
    k_scale<R><<<pw_blocks_, kThreads, 0, stream_>>>(2 * Ns_, wkern_, g_.invN * h3);
    GLIA_LAUNCH_CHECK();
    wkern_sigma_ = sigma;
    return wkern_;
  }
  // The smoother by the plane kernel: from 64^3. It is one launch, but the call then has to look for
  // a timed-out barrier, which waits for it, so small calls no longer follow each other without a
  // gap. us a call, cuFFT / plane: 16^3 56 / 55, 32^3 76 / 68, 56^3 79 / 93 (one small case among
  // others 41 / 69), 64^3 109 / 80, 96^3 242 / 130, 256^3 3693 / 1061.
  bool plane_smooth() const { return plane_now() && g_.n >= 64; }
  void smooth_into(R* out, const R* in, double sigma) {
    if (sigma == 0) {
      if (out != in) vcopy(out, in);
      return;
    }
    const R* K = smoother_kernel(sigma);
    if constexpr (kPlane) {
      if (plane_smooth()) {
        PlaneArgs a = plane_args(PP_SMOOTH, in, out, chat_);
        a.mulk = cx2(K);
        plane_launch(a, 2 * FB() + SB());
        st_.total_fft_execs += 2;
        return;
      }
    }
    r2c(r2c1_, in, chat_);
    k_spec_mul<R><<<pw_blocks_, kThreads, 0, stream_>>>(Ns_, 1, chat_, K);
    GLIA_LAUNCH_CHECK();
    c2r(c2r1_, chat_, out);
  }
  void smooth(void* out, const void* in, double sigma) override {
    import_field(in, tmp_);
    smooth_into(tmp_, tmp_, sigma);
    if (plane_smooth()) check_device_fault();
    export_field(tmp_, out);
  }

  // ------------------------------------------------------------------------------------------
  // Phi
  // ------------------------------------------------------------------------------------------
  void set_phi(const double* centers, int np, double sigma, double smoothing_factor) override {
    if (np < 1 || !(sigma > 0)) throw Error(GLIA_ERR_INVALID, "set_phi: need np >= 1, sigma > 0");
    phi_np_ = np;
    phi_sigma_ = sigma;
    centers_.assign(centers, centers + 3 * np);
    // boxes [centre - 5 sigma, centre + 5 sigma] clipped to the grid (non-periodic distances)
    const double h = 2.0 * M_PI / g_.n;
    std::vector<PhiBox> boxes(np);
    int64_t off = 0;
    for (int i = 0; i < np; i++) {
      for (int d = 0; d < 3; d++) {
        const double a = (centers[3 * i + d] - 5.0 * sigma) / h;
        const double b = (centers[3 * i + d] + 5.0 * sigma) / h;
        int l = (int)std::ceil(a - 1e-9), u = (int)std::floor(b + 1e-9);
        l = std::max(l, 0);
        u = std::min(u, g_.n - 1);
        boxes[i].lo[d] = l;
        boxes[i].ext[d] = std::max(0, u - l + 1);
      }
      boxes[i].off = off;
      off += (int64_t)boxes[i].ext[0] * boxes[i].ext[1] * boxes[i].ext[2];
    }
    phi_box_h_ = boxes;
    if (phi_store_) dfree(phi_store_);
    if (phi_boxes_) dfree(phi_boxes_);
    if (phi_centers_) dfree(phi_centers_);
    phi_store_ = dalloc<R>(std::max<int64_t>(off, 1));
    phi_store_bytes_ = (double)off * sizeof(R);
    phi_boxes_ = dalloc<PhiBox>(np);
    phi_centers_ = dalloc<double>(3 * np);
    GLIA_CUDA(cudaMemcpyAsync(phi_boxes_, boxes.data(), np * sizeof(PhiBox),
                              cudaMemcpyHostToDevice, stream_));
    GLIA_CUDA(cudaMemcpyAsync(phi_centers_, centers, 3 * np * sizeof(double),
                              cudaMemcpyHostToDevice, stream_));
    // Phi::setValues (stored mode, src/mat/Phi.cpp:96-130)
    phi_max_each_.assign(np, 0.0);
    const double sig_s = smoothing_factor * 2.0 * M_PI / g_.n;
    const int Rh = sig_s > 0 ? (int)std::ceil(9.6 * sig_s / h) : 0;
    if (2 * Rh + 1 <= g_.n) {
      phi_values_on_boxes(boxes, sigma, sig_s, Rh);
    } else {
      phi_values_full_grid(boxes, sigma, smoothing_factor);
    }
    build_phi_cells(boxes);
  }
  // The smoother's 1-D taps w(d) / sum w for offsets d = -Rh ... Rh (sigma_s = 0: no smoothing,
  // as weierstrassSmoother returns its input) and the four box passes of k_phi_box per batch of
  // boxes (two scratch buffers of at most 16 M doubles each, or one box's region).
  void phi_values_on_boxes(const std::vector<PhiBox>& boxes, double sigma, double sig_s, int Rh) {
    const int np = (int)boxes.size(), n = g_.n;
    const double h = 2.0 * M_PI / n, twopi = 2.0 * M_PI;
    std::vector<double> taps(2 * Rh + 1, 1.0);
    if (Rh > 0) {
      auto w1 = [&](int i) {
        const double a = i * h, b = i * h - twopi;
        return std::exp((-a * a) / sig_s / sig_s / 2.0) + std::exp((-b * b) / sig_s / sig_s / 2.0);
      };
      double s1 = 0.0;
      for (int i = 0; i < n; i++) s1 += w1(i);
      for (int d = -Rh; d <= Rh; d++) taps[d + Rh] = w1(((d % n) + n) % n) / s1;
    }
    double* dtaps = dalloc<double>((int64_t)taps.size());
    GLIA_CUDA(cudaMemcpyAsync(dtaps, taps.data(), taps.size() * sizeof(double),
                              cudaMemcpyHostToDevice, stream_));
    auto region = [&](const PhiBox& b) {
      return (int64_t)(b.ext[0] + 2 * Rh) * (b.ext[1] + 2 * Rh) * (b.ext[2] + 2 * Rh);
    };
    constexpr int64_t kScratch = int64_t(16) << 20;
    int64_t most = 1;
    for (const PhiBox& b : boxes) most = std::max(most, region(b));
    const int64_t cap = std::max(kScratch, most);
    double* A = dalloc<double>(cap);
    double* Bf = dalloc<double>(cap);
    int64_t* doff = dalloc<int64_t>(np);
    constexpr int xb = 16;
    double* bmax = dalloc<double>((int64_t)np * xb);
    std::vector<int64_t> off(np);
    std::vector<double> hmax((size_t)np * xb);
    for (int b0 = 0; b0 < np;) {
      int nb = 0;
      int64_t used = 0;
      while (b0 + nb < np && (nb == 0 || used + region(boxes[b0 + nb]) <= cap)) {
        off[b0 + nb] = used;
        used += region(boxes[b0 + nb]);
        nb++;
      }
      GLIA_CUDA(cudaMemcpyAsync(doff + b0, off.data() + b0, nb * sizeof(int64_t),
                                cudaMemcpyHostToDevice, stream_));
      const dim3 grid(xb, nb);
      const PhiBox* bx = phi_boxes_ + b0;
      const double* cc = phi_centers_ + 3 * b0;
      k_phi_box<R, 0><<<grid, kThreads, 0, stream_>>>(g_, nb, bx, cc, sigma, Rh, dtaps, filter_,
                                                       doff + b0, nullptr, A, phi_store_, nullptr);
      GLIA_LAUNCH_CHECK();
      k_phi_box<R, 1><<<grid, kThreads, 0, stream_>>>(g_, nb, bx, cc, sigma, Rh, dtaps, filter_,
                                                       doff + b0, A, Bf, phi_store_, nullptr);
      GLIA_LAUNCH_CHECK();
      k_phi_box<R, 2><<<grid, kThreads, 0, stream_>>>(g_, nb, bx, cc, sigma, Rh, dtaps, filter_,
                                                       doff + b0, Bf, A, phi_store_, nullptr);
      GLIA_LAUNCH_CHECK();
      k_phi_box<R, 3><<<grid, kThreads, 0, stream_>>>(g_, nb, bx, cc, sigma, Rh, dtaps, filter_,
                                                       doff + b0, A, nullptr, phi_store_,
                                                       bmax + (int64_t)b0 * xb);
      GLIA_LAUNCH_CHECK();
      b0 += nb;
    }
    GLIA_CUDA(cudaMemcpyAsync(hmax.data(), bmax, hmax.size() * sizeof(double),
                              cudaMemcpyDeviceToHost, stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    for (int b = 0; b < np; b++) {
      double m = 0.0;
      for (int q = 0; q < xb; q++) m = std::max(m, hmax[(size_t)b * xb + q]);
      phi_max_each_[b] = m;
    }
    for (void* p : {(void*)dtaps, (void*)A, (void*)Bf, (void*)doff, (void*)bmax}) dfree(p);
  }
  // The same values through full-grid transforms (a smoother wider than the grid), B functions
  // per batch: Phi::initialize on the grid, the smoother as a spectral multiplier, then
  // truncation and extraction of each box.
  void phi_values_full_grid(const std::vector<PhiBox>& boxes, double sigma,
                            double smoothing_factor) {
    const int np = (int)boxes.size();
    const int B = std::min(np, 8);
    ensure_batch_plans(B);
    R* full = dalloc<R>((int64_t)B * N_);
    R* fsp = dalloc<R>((int64_t)B * Ns_ * 2);
    GLIA_CUDA(cudaMemsetAsync(full, 0, (size_t)B * N_ * sizeof(R), stream_));
    const int xb = 8;
    double* bmax = dalloc<double>((int64_t)B * xb);
    std::vector<double> hmax((size_t)B * xb);
    const R* K = smoother_kernel(smoothing_factor * 2.0 * M_PI / g_.n);
    for (int b0 = 0; b0 < np; b0 += B) {
      const int nb = std::min(B, np - b0);
      k_phi_gauss<R><<<pw_blocks_, kThreads, 0, stream_>>>(g_, nb, phi_centers_ + 3 * b0, sigma,
                                                            filter_, full);
      GLIA_LAUNCH_CHECK();
      r2c(r2cB_, full, fsp, B);
      k_spec_mul<R><<<pw_blocks_, kThreads, 0, stream_>>>(Ns_, nb, fsp, K);
      GLIA_LAUNCH_CHECK();
      c2r(c2rB_, fsp, full, B);
      dim3 grid(xb, nb);
      k_phi_extract<R><<<grid, kThreads, 0, stream_>>>(g_, nb, full, phi_boxes_ + b0,
                                                        phi_centers_ + 3 * b0, sigma, phi_store_,
                                                        bmax);
      GLIA_LAUNCH_CHECK();
      GLIA_CUDA(cudaMemcpyAsync(hmax.data(), bmax, (size_t)nb * xb * sizeof(double),
                                cudaMemcpyDeviceToHost, stream_));
      GLIA_CUDA(cudaStreamSynchronize(stream_));
      for (int b = 0; b < nb; b++) {
        double m = 0.0;
        for (int q = 0; q < xb; q++) m = std::max(m, hmax[(size_t)b * xb + q]);
        phi_max_each_[b0 + b] = m;
      }
    }
    dfree(full);
    dfree(fsp);
    dfree(bmax);
    destroy_batch_plans();
  }
  // cell lists of the gathered apply
  void build_phi_cells(const std::vector<PhiBox>& boxes) {
    const int np = (int)boxes.size();
    const int cpd = (g_.n + 7) / 8;
    std::vector<std::vector<int>> lists((size_t)cpd * cpd * cpd);
    for (int i = 0; i < np; i++) {
      const PhiBox& bx = boxes[i];
      if (bx.ext[0] == 0 || bx.ext[1] == 0 || bx.ext[2] == 0) continue;
      int c0[3], c1[3];
      for (int d = 0; d < 3; d++) {
        c0[d] = bx.lo[d] / 8;
        c1[d] = (bx.lo[d] + bx.ext[d] - 1) / 8;
      }
      for (int a = c0[0]; a <= c1[0]; a++)
        for (int b = c0[1]; b <= c1[1]; b++)
          for (int c = c0[2]; c <= c1[2]; c++) lists[((size_t)a * cpd + b) * cpd + c].push_back(i);
    }
    std::vector<int> ptr(lists.size() + 1, 0), flat;
    for (size_t k = 0; k < lists.size(); k++) {
      ptr[k + 1] = ptr[k] + (int)lists[k].size();
      flat.insert(flat.end(), lists[k].begin(), lists[k].end());
    }
    if (cell_ptr_) dfree(cell_ptr_);
    if (cell_list_) dfree(cell_list_);
    if (phi_p_) dfree(phi_p_);
    cell_ptr_ = dalloc<int>(ptr.size());
    cell_list_ = dalloc<int>(std::max<size_t>(flat.size(), 1));
    phi_p_ = dalloc<double>(np);
    GLIA_CUDA(cudaMemcpyAsync(cell_ptr_, ptr.data(), ptr.size() * sizeof(int),
                              cudaMemcpyHostToDevice, stream_));
    if (!flat.empty())
      GLIA_CUDA(cudaMemcpyAsync(cell_list_, flat.data(), flat.size() * sizeof(int),
                                cudaMemcpyHostToDevice, stream_));
    cells_per_dim_ = cpd;
    GLIA_CUDA(cudaStreamSynchronize(stream_));
  }
  double phi_max_all() const {
    double m = 0;
    for (double v : phi_max_each_) m = std::max(m, v);
    return m;
  }
  // Phi::apply (src/mat/Phi.cpp:313-377): stored mode scales by the global max, on-the-fly mode
  // by the max over the active functions (1 when p has no non-zero).
  void phi_apply_into(R* out, const double* p) {
    if (phi_np_ < 1) throw Error(GLIA_ERR_STATE, "Phi is not set (glia_set_phi)");
    double scale;
    if (opt_.phi_store) {
      scale = 1.0 / phi_max_all();
    } else {
      double pm = 0;
      bool nnz = false;
      for (int i = 0; i < phi_np_; i++)
        if (p[i] != 0) {
          nnz = true;
          pm = std::max(pm, phi_max_each_[i]);
        }
      scale = 1.0 / (nnz ? pm : 1.0);
    }
    hphi_p_.assign(p, p + phi_np_);
    GLIA_CUDA(cudaMemcpyAsync(phi_p_, hphi_p_.data(), phi_np_ * sizeof(double),
                              cudaMemcpyHostToDevice, stream_));
    const int cells = cells_per_dim_ * cells_per_dim_ * cells_per_dim_;
    GLIA_TIMED(KS_PHI, FB() + phi_store_bytes_,
               k_phi_apply<R><<<cells, 512, 0, stream_>>>(g_, cells_per_dim_, cell_ptr_,
                                                           cell_list_, phi_boxes_, phi_store_,
                                                           phi_p_, scale, out));
    GLIA_CUDA(cudaStreamSynchronize(stream_));  // hphi_p_ may be reused by the next call
  }
  void phi_applyT_from(const R* v, double* pout) {
    if (phi_np_ < 1) throw Error(GLIA_ERR_STATE, "Phi is not set (glia_set_phi)");
    GLIA_TIMED(KS_PHI, 2.0 * phi_store_bytes_,
               k_phi_applyT<R><<<phi_np_, kThreads, 0, stream_>>>(g_, phi_boxes_, phi_store_, v,
                                                                   phi_p_));
    GLIA_CUDA(cudaMemcpyAsync(pout, phi_p_, phi_np_ * sizeof(double), cudaMemcpyDeviceToHost,
                              stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    const double s = 1.0 / phi_max_all();
    for (int i = 0; i < phi_np_; i++) pout[i] *= s;
  }
  void phi_apply(const double* p, void* c0) override {
    phi_apply_into(tmp_, p);
    export_field(tmp_, c0);
  }
  void phi_apply_transpose(const void* v, double* pout) override {
    import_field(v, tmp_);
    phi_applyT_from(tmp_, pout);
  }

  // Phi::setGaussians(Vec data) (src/mat/Phi.cpp:615-1004) for one process: the ball and the
  // lattice as the reference's loops make them (ball offsets over [(int)-r, (int)r] with
  // |o| <= r; lattice from the first to the last fmod(X, space) == 0 index by X += space on an
  // integer), counts by k_data_centers, selection count > gvf * interior in x-major order.
  void phi_data_centers(const void* data, double sigma, double thr, double gvf,
                        double spacing_factor, int max_centers, double* centers, int* np_out,
                        void* frac) override {
    const int n = g_.n;
    const double h = 2.0 * M_PI / n, r = sigma / h, space = spacing_factor * sigma / h;
    if (!(sigma > 0) || !(space >= 1.0) || !(gvf >= 0))
      throw Error(GLIA_ERR_INVALID, "phi_data_centers: sigma > 0, gaussian_vol_frac >= 0 and a "
                                    "centre spacing of at least one voxel are needed");
    std::vector<int> offs;
    const int lo = (int)(-r), hi = (int)r;
    for (int i = lo; i <= hi; i++)
      for (int j = lo; j <= hi; j++)
        for (int k = lo; k <= hi; k++)
          if (std::sqrt((double)(i * i + j * j + k * k)) <= r) {
            offs.push_back(i);
            offs.push_back(j);
            offs.push_back(k);
          }
    const int interior = (int)offs.size() / 3;
    std::vector<int> axis;
    int first = -1, last = -1;
    for (int x = 0; x < n; x++)
      if (std::fmod((double)x, space) == 0.0) {
        if (first < 0) first = x;
        last = x;
      }
    for (int x = first; first >= 0 && x <= last; x = (int)(x + space)) axis.push_back(x);
    const int nax = (int)axis.size();
    const int64_t L = (int64_t)nax * nax * nax;
    // the data in FP64 (the threshold test is exact whatever the storage type)
    double* d = stage();
    if (ptr_mode_ == GLIA_PTR_HOST_F64) {
      GLIA_CUDA(cudaMemcpyAsync(d, data, N_ * 8, cudaMemcpyHostToDevice, stream_));
    } else if (ptr_mode_ == GLIA_PTR_DEVICE_F64) {
      GLIA_CUDA(cudaMemcpyAsync(d, data, N_ * 8, cudaMemcpyDeviceToDevice, stream_));
    } else {
      k_convert<float, double><<<pw_blocks_, kThreads, 0, stream_>>>(N_, (const float*)data, d);
      GLIA_LAUNCH_CHECK();
    }
    int* dax = dalloc<int>(std::max(nax, 1));
    int* doffs = dalloc<int>(std::max<int64_t>((int64_t)offs.size(), 1));
    int* dcnt = dalloc<int>(std::max<int64_t>(L, 1));
    std::vector<int> cnt((size_t)L);
    if (L > 0) {
      GLIA_CUDA(cudaMemcpyAsync(dax, axis.data(), nax * sizeof(int), cudaMemcpyHostToDevice,
                                stream_));
      GLIA_CUDA(cudaMemcpyAsync(doffs, offs.data(), offs.size() * sizeof(int),
                                cudaMemcpyHostToDevice, stream_));
      const int blocks = (int)std::min<int64_t>((L + kThreads - 1) / kThreads, pw_blocks_);
      k_data_centers<<<blocks, kThreads, 0, stream_>>>(d, n, dax, nax, doffs, interior, thr, dcnt);
      GLIA_LAUNCH_CHECK();
      GLIA_CUDA(cudaMemcpyAsync(cnt.data(), dcnt, L * sizeof(int), cudaMemcpyDeviceToHost,
                                stream_));
    }
    if (frac) {
      fill(tmp_, 0.0);
      if (L > 0) {
        const int blocks = (int)std::min<int64_t>((L + kThreads - 1) / kThreads, pw_blocks_);
        k_data_frac<R><<<blocks, kThreads, 0, stream_>>>(dcnt, n, dax, nax, (double)interior,
                                                          tmp_);
        GLIA_LAUNCH_CHECK();
      }
      export_field(tmp_, frac);
    }
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    for (void* p : {(void*)dax, (void*)doffs, (void*)dcnt}) dfree(p);
    int count = 0;
    for (int64_t t = 0; t < L; t++) {
      if (!(cnt[(size_t)t] > gvf * interior)) continue;
      if (count < max_centers) {
        centers[3 * count] = axis[(size_t)(t / ((int64_t)nax * nax))] * h;
        centers[3 * count + 1] = axis[(size_t)((t / nax) % nax)] * h;
        centers[3 * count + 2] = axis[(size_t)(t % nax)] * h;
      }
      count++;
    }
    *np_out = count;
    if (count > max_centers)
      throw Error(GLIA_ERR_INVALID, "phi_data_centers: " + std::to_string(count) +
                                        " centres found, room for " + std::to_string(max_centers));
  }

  // ------------------------------------------------------------------------------------------
  // observation operator, initial condition
  // ------------------------------------------------------------------------------------------
  void set_obs_threshold(const void* data, double thr) override {
    import_field(data, tmp_);
    k_threshold<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, tmp_, thr, obs_);
    GLIA_LAUNCH_CHECK();
  }
  void set_obs_filter(const void* f) override { import_field(f, obs_); }
  // the observation operator at t = 0 of the two-snapshot objective (Obs::filter_0_, 1 until set)
  R* obs0() {
    if (!obs0_) {
      obs0_ = fld();
      fill(obs0_, 1.0);
    }
    return obs0_;
  }
  void set_obs_threshold0(const void* data, double thr) override {
    import_field(data, tmp_);
    k_threshold<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, tmp_, thr, obs0());
    GLIA_LAUNCH_CHECK();
  }
  void set_obs_filter0(const void* f) override { import_field(f, obs0()); }
  // Data::dt0 with TumorParameters::two_time_points_: J gains h^3/2 ||O0 c(0) - d0||^2 and the p
  // gradient h^3 Phi^T O0^T (O0 c(0) - d0); NULL ends the two-snapshot objective
  void set_data0(const void* d0) override {
    if (!d0) {
      two_tp_ = false;
      return;
    }
    if (!d0_) d0_ = fld();
    import_field(d0, d0_);
    two_tp_ = true;
  }
  void set_c0(const void* c0) override { import_field(c0, c0_); }

  // ------------------------------------------------------------------------------------------
  // time history
  // ------------------------------------------------------------------------------------------
  void release_history() {
    for (auto* v : {&c_hist_, &c_half_, &chat_hist_, &p_hist_, &ckpt_, &seg_c_, &seg_half_,
                    &seg_chat_})
      for (R*& f : *v) {
        if (f) dfree(f);
        f = nullptr;
      }
    for (auto* v : {&c_hist_, &c_half_, &chat_hist_, &p_hist_, &ckpt_, &seg_c_, &seg_half_,
                    &seg_chat_})
      v->clear();
  }
  bool full() const { return hist_mode_ == GLIA_HISTORY_FULL; }
  // which gradient terms the next adjoint sweep accumulates
  bool kappa_trick_ok() const {
    return !ref_ && opt_.nk == 1 && k_scale_ > 0 && k_gm_wm_ >= 0 && k_glm_wm_ <= 0 &&
           !kxx_sinusoidal_;
  }
  void ensure_history() {
    const bool store_half = !ref_ || adjoint_store_;
    if (hist_mode_ == GLIA_HISTORY_OFF) {
      release_history();
      return;
    }
    if (full()) {
      if ((int)c_hist_.size() != nt_ + 1) {
        release_history();
        c_hist_.resize(nt_ + 1);
        p_hist_.resize(nt_ + 1);
        for (auto& f : c_hist_) f = fld();
        for (auto& f : p_hist_) f = fld();
        // p_[nt] is read by the Hessian's kappa rows before any adjoint may have set it; the
        // reference's history vectors start at 0 (src/pde/PdeOperators.cpp:27-31)
        GLIA_CUDA(cudaMemsetAsync(p_hist_[nt_], 0, N_ * sizeof(R), stream_));
        if (store_half) {
          c_half_.resize(nt_);
          for (auto& f : c_half_) f = fld();
        }
        if (!ref_) {
          chat_hist_.resize(nt_ + 1);
          for (auto& f : chat_hist_) f = spec();
        }
      }
    } else {
      const int S = (nt_ + every_ - 1) / every_;
      if ((int)ckpt_.size() != S) {
        release_history();
        ckpt_.resize(S);
        for (auto& f : ckpt_) f = fld();
        seg_c_.resize(every_ + 1);
        seg_half_.resize(every_);
        seg_chat_.resize(every_ + 1);
        for (auto& f : seg_c_) f = fld();
        for (auto& f : seg_half_) f = fld();
        for (auto& f : seg_chat_) f = spec();
      }
    }
  }

  // One splitting step from the state in `c` (PdeOperatorsRD::solveState loop body,
  // src/pde/PdeOperators.cpp:260-300). chat_slot: spectrum of c before the step; half_out:
  // state after the first diffusion sub-step.
  void step(R* c, R* chat_slot, R* half_out, int which = 0) {
    if (order_ == 2) {
      solve(c, dt_ / 2.0, chat_slot, nullptr, 0.0, which);
      const Pre pre = react(c, 1, nullptr, half_out);
      solve(c, dt_ / 2.0, nullptr, nullptr, 0.0, which, pre);
    } else {
      solve(c, dt_, chat_slot, nullptr, 0.0, which);
      reaction(c, half_out);
    }
  }
  // The reaction step between two diffusion half steps (mode 1: logistic, storing the field in
  // half; 2: linearised at lin): a plane kernel takes it as it reads the field of the next solve,
  // otherwise it runs here.
  Pre react(R* c, int mode, const R* lin, R* half) {
    if (plane_now() && k_scale_ != 0) return Pre{mode, lin, half};
    if (mode == 1)
      reaction(c, half);
    else
      reaction_linearized(c, lin);
    return Pre{};
  }
  void reaction(R* c, R* half_out) {
    GLIA_TIMED(KS_REACTION, FB() * (half_out ? 4 : 3),
               k_reaction_fwd<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, c, rho_, (R)dt_,
                                                                        half_out));
  }

  // PdeOperatorsRD::solveState(0) (src/pde/PdeOperators.cpp:235-316)
  void solve_state_internal() {
    st_.nb_state_solves++;
    ensure_history();
    st_.diff_ksp_itr_state = 0;
    vcopy(ct_, c0_);
    const bool trick = kappa_trick_ok();
    if (hist_mode_ == GLIA_HISTORY_OFF) {  // time_history_off_: the state only
      for (int i = 0; i < nt_; i++) step(ct_, nullptr, nullptr);
      sync_sweep();
      state_done_ = false;  // nothing to linearise around or sweep back over
      adjoint_done_ = false;
      return;
    }
    if (full()) {
      vcopy(c_hist_[0], ct_);
      for (int i = 0; i < nt_; i++) {
        R* half = c_half_.empty() ? nullptr : c_half_[i];
        step(ct_, (!ref_ && trick) ? chat_hist_[i] : nullptr, half);
        vcopy(c_hist_[i + 1], ct_);
      }
      if (!ref_ && trick) spectrum(ct_, chat_hist_[nt_]);
    } else {
      // the last segment is written straight into the segment buffers, so the backward sweep
      // starts without recomputing it
      const int S = (int)ckpt_.size(), last0 = (S - 1) * every_;
      for (int i = 0; i < nt_; i++) {
        if (i % every_ == 0) vcopy(ckpt_[i / every_], ct_);
        if (i >= last0) {
          vcopy(seg_c_[i - last0], ct_);
          step(ct_, trick ? seg_chat_[i - last0] : nullptr, seg_half_[i - last0]);
        } else {
          step(ct_, nullptr, nullptr);
        }
      }
      vcopy(seg_c_[nt_ - last0], ct_);
      if (trick) spectrum(ct_, seg_chat_[nt_ - last0]);
      last_seg_resident_ = true;
      vcopy(cfin(), ct_);  // c_[nt] for the Hessian's kappa rows
    }
    sync_sweep();
    state_done_ = true;
    adjoint_done_ = false;
    trick_at_state_ = trick;
  }
  void solve_state(int linearized, const void* c0, void* c1) override {
    if (linearized < 0 || linearized > 2)
      throw Error(GLIA_ERR_INVALID, "solveState: linearized must be 0, 1 or 2");
    if (c0) import_field(c0, c0_);
    if (linearized)
      solve_state_linearized_internal(linearized);
    else
      solve_state_internal();
    if (c1) export_field(ct_, c1);
  }

  // PdeOperatorsRD::solveState(1) (src/pde/PdeOperators.cpp:235-316): the incremental forward
  // from c~0 (in c0_), the logistic step linearised at the state c_i at the start of step i
  // (reaction(1, i), :140-190: c~ *= e / (c_i e + 1 - c_i)^2). mode 2 (solveState(2)) adds the
  // diffusivity direction's sources around each step (solveIncremental, :192-233): before the
  // first diffusion half step c~ += dt/4 D~(0.5 (c_i + c_i+1) + c_i), after the second
  // c~ += dt/4 D~(0.5 (c_i + c_i+1) + c_i+1), D~ the D apply with k~. The state history of the
  // last solveState(0) is read, never written; checkpointed runs recompute each segment's states
  // from its checkpoint on the way.
  void solve_state_linearized_internal(int mode = 1) {
    if (!state_done_)
      throw Error(GLIA_ERR_STATE, "solveState(1) needs a preceding solveState(0) for its history");
    if (mode == 2 && !ksec_set_)
      throw Error(GLIA_ERR_STATE, "solveState(2) needs the secondary diffusion coefficients");
    st_.nb_state_solves++;
    st_.diff_ksp_itr_state = 0;
    vcopy(ct_, c0_);
    auto source = [&](const R* ci, const R* cj, int m) {
      if (!inc_) inc_ = fld();
      k_incr_mix<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, inc_, ci, cj, m);
      GLIA_LAUNCH_CHECK();
      applyD_secondary_into(inc_, inc_);
      vaxpy_any(ct_, (dt_ / 2.0) / 2.0, inc_);
    };
    auto lin_step = [&](const R* ci, const R* cj) {
      if (mode == 2) source(ci, cj, 1);
      if (order_ == 2) {
        solve(ct_, dt_ / 2.0, nullptr, nullptr, 0.0, 0);
        const Pre pre = react(ct_, 2, ci, nullptr);
        solve(ct_, dt_ / 2.0, nullptr, nullptr, 0.0, 0, pre);
        if (mode == 2) source(ci, cj, 2);
      } else {
        solve(ct_, dt_, nullptr, nullptr, 0.0, 0);
        reaction_linearized(ct_, ci);
      }
    };
    if (full()) {
      for (int i = 0; i < nt_; i++) lin_step(c_hist_[i], c_hist_[i + 1]);
    } else {
      const int S = (int)ckpt_.size();
      for (int s = 0; s < S; s++) {
        const int i0 = s * every_, i1 = std::min(nt_, (s + 1) * every_);
        if (!(S == 1 && last_seg_resident_)) {
          vcopy(seg_c_[0], ckpt_[s]);
          vcopy(tmp2(), ckpt_[s]);
          // recompute solves (which = 2) up to the segment's last step start, or its end when
          // the sources need c_i+1
          const int iend = mode == 2 ? i1 : i1 - 1;
          for (int i = i0; i < iend; i++) {
            step(tmp2(), nullptr, seg_half_[i - i0], 2);
            vcopy(seg_c_[i - i0 + 1], tmp2());
          }
          last_seg_resident_ = false;
        }
        for (int i = i0; i < i1; i++) lin_step(seg_c_[i - i0], seg_c_[i - i0 + 1]);
      }
    }
    sync_sweep();
  }
  void reaction_linearized(R* x, const R* c) {
    GLIA_TIMED(KS_REACTION_LIN, FB() * 4,
               k_reaction_lin<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, x, rho_, c, (R)dt_));
  }

  // adjoint step from alpha_{i+1} (in p0_) to alpha_i (PdeOperatorsRD::solveAdjoint body,
  // :392-408); cx = F(c_{i+1}) adds w_{i+1} dt <c_{i+1}, D alpha_{i+1}> for the kappa gradient.
  void adjoint_step(int i, const R* chalf, const R* cx, bool accumulate) {
    const double w = (i + 1 == nt_) ? 0.5 : 1.0;
    const R* cxx = accumulate ? cx : nullptr;
    if (order_ == 2) {
      solve(p0_, dt_ / 2.0, nullptr, cxx, w * dt_, 1);
      const Pre pre = react(p0_, 2, chalf, nullptr);
      solve(p0_, dt_ / 2.0, nullptr, nullptr, 0.0, 1, pre);
    } else {
      solve(p0_, dt_, nullptr, cxx, w * dt_, 1);
      reaction_adjoint(chalf);
    }
  }
  void reaction_adjoint(const R* chalf) { reaction_linearized(p0_, chalf); }
  // reactionAdjoint without stored half steps (src/pde/PdeOperators.cpp:331-344)
  const R* recompute_half(const R* ci) {
    vcopy(tmp_, ci);
    solve(tmp_, order_ == 2 ? dt_ / 2.0 : dt_, nullptr, nullptr, 0.0, 1);
    return tmp_;
  }
  // per-time-point gradient terms at time point i (state c_i, adjoint alpha_i in p0_)
  void grad_point(int i, const R* ci, bool explicit_kappa) {
    const double w = (i == 0 || i == nt_) ? 0.5 : 1.0;
    GLIA_TIMED(KS_GRAD_ACC, FB() * 5,
               k_grad_rho_acc<R><<<red_blocks_, kThreads, 0, stream_>>>(
                   N_, ci, p0_, wm_, gm_, csf_, w * dt_, sc_, ws_));
    if (explicit_kappa) {
      R* gc = g3r_;
      R* ga = ga3();
      if (ref_) {  // computeGradient twice, as gradDiffusion does
        ref_gradient(gc, gc + N_, gc + 2 * N_, ci);
        ref_gradient(ga, ga + N_, ga + 2 * N_, p0_);
      } else {
        grad_real(ci, gc);
        grad_real(p0_, ga);
      }
      GLIA_TIMED(KS_GRAD_ACC, FB() * 9,
                 k_grad_kappa_acc<R><<<red_blocks_, kThreads, 0, stream_>>>(
                     N_, gc, ga, wm_, gm_, csf_, w * dt_, sc_, ws_));
    }
  }
  R* ga3() {
    if (!ga3_) ga3_ = dalloc<R>(3 * N_);
    return ga3_;
  }
  void grad_real(const R* x, R* out3) {  // spectral gradient into 3 real fields
    r2c(r2c1_, x, chat_);
    launch_grad3<false>(chat_, nullptr);
    c2r(c2r3_, g3s_, out3, 3);
  }

  // PdeOperatorsRD::solveAdjoint(1) with the gradient time accumulation fused into the sweep.
  // linearized = 2 (incremental adjoint of the Hessian matvec) is the same sweep; like the
  // reference it leaves p_[nt] of the full history untouched.
  // skip_final leaves out the t = 1 term of the accumulation (the Hessian adds its own).
  void solve_adjoint_internal(bool accumulate, int linearized = 1, bool skip_final = false) {
    if (hist_mode_ == GLIA_HISTORY_OFF)
      throw Error(GLIA_ERR_STATE, "solveAdjoint: no time history (GLIA_HISTORY_OFF)");
    if (!state_done_) throw Error(GLIA_ERR_STATE, "solveAdjoint needs a preceding solveState");
    st_.nb_adjoint_solves++;
    st_.diff_ksp_itr_adj = 0;
    vcopy(p0_, pt_);
    if (!full() && linearized == 1) vcopy(pnt(), p0_);  // the reference's p_[nt]
    const bool trick = trick_at_state_ && kappa_trick_ok();
    const bool explicit_kappa = accumulate && !trick;
    kappa_used_trick_ = trick;
    if (accumulate) {
      k_acc_reset<<<1, 1, 0, stream_>>>(sc_);
      GLIA_LAUNCH_CHECK();
    }
    if (full()) {
      if (linearized == 1) vcopy(p_hist_[nt_], p0_);
      if (accumulate && !ref_ && !skip_final) grad_point(nt_, c_hist_[nt_], explicit_kappa);
      for (int i = nt_ - 1; i >= 0; i--) {
        const R* chalf = c_half_.empty() ? nullptr : c_half_[i];
        const bool kdot = accumulate && trick && !(skip_final && i + 1 == nt_);
        if (order_ == 2) {
          solve(p0_, dt_ / 2.0, nullptr, kdot ? chat_hist_[i + 1] : nullptr,
                ((i + 1 == nt_) ? 0.5 : 1.0) * dt_, 1);
          if (!chalf) chalf = recompute_half(c_hist_[i]);
          const Pre pre = react(p0_, 2, chalf, nullptr);
          solve(p0_, dt_ / 2.0, nullptr, nullptr, 0.0, 1, pre);
        } else {
          solve(p0_, dt_, nullptr, kdot ? chat_hist_[i + 1] : nullptr,
                ((i + 1 == nt_) ? 0.5 : 1.0) * dt_, 1);
          if (!chalf) chalf = recompute_half(c_hist_[i]);
          reaction_adjoint(chalf);
        }
        vcopy(p_hist_[i], p0_);
        if (accumulate && !ref_) grad_point(i, c_hist_[i], explicit_kappa);
      }
      if (accumulate && trick) kappa_dot_at(chat_hist_[0], 0.5 * dt_);
    } else {
      // checkpointed: recompute each segment forward from its checkpoint, then sweep it back
      const int S = (int)ckpt_.size();
      if (accumulate && !skip_final) grad_point(nt_, ct_, explicit_kappa);
      for (int s = S - 1; s >= 0; s--) {
        const int i0 = s * every_, i1 = std::min(nt_, (s + 1) * every_);
        // the last segment is still resident from the forward sweep (first adjoint only)
        if (s < S - 1 || !last_seg_resident_) {
          vcopy(seg_c_[0], ckpt_[s]);
          vcopy(tmp2(), ckpt_[s]);
          for (int i = i0; i < i1; i++) {
            // recompute solves are neither state nor adjoint solves (which = 2)
            step(tmp2(), trick ? seg_chat_[i - i0] : nullptr, seg_half_[i - i0], 2);
            vcopy(seg_c_[i - i0 + 1], tmp2());
          }
          if (trick) spectrum(tmp2(), seg_chat_[i1 - i0]);
        }
        for (int i = i1 - 1; i >= i0; i--) {
          adjoint_step(i, seg_half_[i - i0], trick ? seg_chat_[i - i0 + 1] : nullptr,
                       accumulate && trick && !(skip_final && i + 1 == nt_));
          if (accumulate) grad_point(i, seg_c_[i - i0], explicit_kappa);
        }
        if (s == 0 && accumulate && trick) kappa_dot_at(seg_chat_[0], 0.5 * dt_);
        last_seg_resident_ = false;  // the segment buffers now hold another segment
      }
    }
    sync_sweep();
    adjoint_done_ = true;
  }
  R* tmp2() {
    if (!tmp2_) tmp2_ = fld();
    return tmp2_;
  }
  // checkpointed runs: the reference's p_[nt] (final condition of the last linearized = 1
  // adjoint, 0 before the first) and c_[nt] (state at t = 1 of the last forward)
  R* pnt() {
    if (!pnt_) {
      pnt_ = fld();
      GLIA_CUDA(cudaMemsetAsync(pnt_, 0, N_ * sizeof(R), stream_));
    }
    return pnt_;
  }
  R* cfin() {
    if (!cfin_) cfin_ = fld();
    return cfin_;
  }
  // acc[6] += w <c_0, D alpha_0>: a D apply on alpha_0 whose spectral epilogue takes the dot
  void kappa_dot_at(const R* chat0, double w) {
    if constexpr (kPlane) {
      if (plane_now()) {
        PlaneArgs a = plane_args(PP_DOT, p0_, nullptr, xhat_);
        a.cx = cx2(chat0);
        a.kdot_weight = w;
        plane_launch(a, 2 * FB() + SB());
        st_.total_fft_execs += 7;
        return;
      }
    }
    k_solve_config<<<1, 1, 0, stream_>>>(sc_, 0.0, 0.0, rtol_, abstol_, divtol_, maxit_, w);
    GLIA_LAUNCH_CHECK();
    R* spec_a = xhat_;
    r2c(r2c1_, p0_, spec_a);
    d_front<false>(spec_a, nullptr);
    d_back<EPI_SETUP>(spec_a, chat0, rhat_, what_, R(0));
  }
  void solve_adjoint(int linearized, const void* pt, void* a0) override {
    if (linearized != 1 && linearized != 2)
      throw Error(GLIA_ERR_INVALID, "solveAdjoint: linearized must be 1 or 2");
    if (pt) import_field(pt, pt_);
    solve_adjoint_internal(false, linearized);
    if (a0) export_field(p0_, a0);
  }

  // DerivativeOperatorsRD::evaluateHessian (src/grad/DerivativeOperatorsRD.cpp:229-438), the
  // Gauss-Newton matvec of the p block (no diffusivity inversion, :398-425): c~0 = Phi p~,
  // incremental forward, p~_t = -O^T O c~(1), incremental adjoint, y = h^3 (beta Phi^T c~0 -
  // Phi^T a~0), or y = beta p~ - h^3 Phi^T a~0 with the L2b regulariser. The state history of the
  // last gradient evaluation (or solveState) is the linearisation point. Entries of y past np
  // (kappa, rho) carry beta x for L2b and 0 otherwise.
  void hessian_matvec(const double* x, int nxin, double* y) override {
    if (nxin != nx())
      throw Error(GLIA_ERR_INVALID, "x has " + std::to_string(nxin) + " entries, expected " +
                                        std::to_string(nx()) + " (np + nk + nr)");
    if (!state_done_)
      throw Error(GLIA_ERR_STATE, "evaluateHessian needs a preceding state solve or gradient");
    if (two_tp_)  // as the reference (src/grad/DerivativeOperatorsRD.cpp:234)
      throw Error(GLIA_ERR_INVALID, "evaluateHessian is not implemented for two snapshots");
    if (opt_.diffusivity_inversion) {
      hessian_diffusivity(x, y);
      return;
    }
    const int np = opt_.np;
    const double h = 2.0 * M_PI / g_.n, h3 = h * h * h;
    phi_apply_into(c0_, x);
    solve_state_linearized_internal();
    R* zero = d1_buf();
    GLIA_CUDA(cudaMemsetAsync(zero, 0, sizeof(R) * N_, stream_));
    GLIA_TIMED(KS_OBS, FB() * 4,
               k_obs_residual<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, ct_, obs_, zero, pt_,
                                                                        sc_, ws_));
    solve_adjoint_internal(false, 2);
    std::vector<double> pa(std::max(np, 1));
    phi_applyT_from(p0_, pa.data());
    const bool l2b = opt_.regularization_norm != 0;
    if (l2b) {
      for (int i = 0; i < nx(); i++) y[i] = opt_.beta * x[i] - (i < np ? h3 * pa[i] : 0.0);
    } else {
      phi_applyT_from(c0_, y);
      for (int i = 0; i < np; i++) y[i] = opt_.beta * h3 * y[i] - h3 * pa[i];
      for (int i = np; i < nx(); i++) y[i] = 0.0;
    }
  }
  // evaluateHessian with diffusivity inversion (src/grad/DerivativeOperatorsRD.cpp:244-397):
  // y = [Hpp p~ + Hpk k~; Hkp p~ + Hkk k~]. Two incremental forward / adjoint pairs around the
  // state history of the last gradient evaluation: c~0 = Phi p~ with solveState(1), then
  // c~0 = 0 with the diffusivity direction k~ (x's kappa entries) and solveState(2); each adjoint
  // starts from -O^T O c~(1). p rows: h^3 (beta Phi^T Phi p~ - Phi^T a~0) - h^3 Phi^T a~0'.
  // kappa rows: the gradDiffusion quadrature with a~ in place of the adjoint; its t = 1 term
  // takes the reference's p_[nt], which solveAdjoint(2) leaves at the final condition of the last
  // linearized = 1 adjoint. Rows past np + nk (rho) are 0 (the reference leaves them as the
  // caller's y).
  void hessian_diffusivity(const double* x, double* y) {
    const int np = opt_.np, nk = opt_.nk;
    const double h = 2.0 * M_PI / g_.n, h3 = h * h * h;
    std::fill(y, y + nx(), 0.0);
    const int npp = std::max({np, phi_np_, 1});
    std::vector<double> pa(npp), pc(npp);
    const bool trick = !ref_ && trick_at_state_ && kappa_trick_ok();
    // incremental forward (mode 1 / 2), adjoint, Phi^T a~0 into pa, kappa rows into rows
    auto pair = [&](int mode, double* rows) {
      solve_state_linearized_internal(mode);
      R* zero = d1_buf();
      GLIA_CUDA(cudaMemsetAsync(zero, 0, sizeof(R) * N_, stream_));
      GLIA_TIMED(KS_OBS, FB() * 4,
                 k_obs_residual<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, ct_, obs_, zero,
                                                                          pt_, sc_, ws_));
      double acc[8];
      if (ref_) {
        solve_adjoint_internal(false, 2);
        phi_applyT_from(p0_, pa.data());
        ref_time_integrals(acc);  // the stored p_[nt] is the reference's stale one
      } else {
        solve_adjoint_internal(true, 2, true);
        phi_applyT_from(p0_, pa.data());
        // the t = 1 term with p_[nt] and c_[nt]
        vcopy(p0_, full() ? p_hist_[nt_] : pnt());
        const R* cn = full() ? c_hist_[nt_] : cfin();
        if (trick) {
          const R* chat_n = chat_;
          if (full())
            chat_n = chat_hist_[nt_];
          else
            spectrum(cn, chat_);
          kappa_dot_at(chat_n, 0.5 * dt_);
        } else {
          grad_point(nt_, cn, true);
        }
        GLIA_CUDA(cudaMemcpyAsync(hsc_, sc_, sizeof(DevScalars), cudaMemcpyDeviceToHost, stream_));
        GLIA_CUDA(cudaStreamSynchronize(stream_));
        if (hsc_->dev_fault) raise_device_fault();
        std::memcpy(acc, hsc_->acc, sizeof(acc));
      }
      rows[0] = rows[1] = rows[2] = 0.0;
      if (trick) {
        rows[0] = -acc[6] / k_scale_ * h3;  // <wm + r gm, grad c . grad a~> = -<c, D a~>/kappa
      } else {
        rows[0] = acc[0] * h3;
        if (nk == 1) rows[0] += acc[1] * h3 * k_gm_wm_;
        if (nk > 1) rows[1] = acc[1] * h3;
        if (nk > 2) rows[2] = acc[2] * h3;
      }
    };
    double r1[3], r2[3];
    // Hpp p~ and Hkp p~
    phi_apply_into(c0_, x);
    phi_applyT_from(c0_, pc.data());
    pair(1, r1);
    for (int i = 0; i < np; i++) y[i] = (opt_.beta * pc[i] - pa[i]) * h3;
    // Hpk k~ and Hkk k~
    fill(c0_, 0.0);
    set_secondary_coefficients(x[np], nk > 1 ? x[np + 1] : 0.0, nk > 2 ? x[np + 2] : 0.0);
    pair(2, r2);
    for (int i = 0; i < np; i++) y[i] += -h3 * pa[i];
    for (int j = 0; j < std::min(nk, 3); j++) y[np + j] = r1[j] + r2[j];
  }
  void get_state(int i, void* out) override {
    if (!state_done_ || !full() || i < 0 || i > nt_)
      throw Error(GLIA_ERR_STATE, "get_state: needs a state solve with full history, 0<=i<=nt");
    export_field(c_hist_[i], out);
  }
  void get_adjoint(int i, void* out) override {
    if (!adjoint_done_ || !full() || i < 0 || i > nt_)
      throw Error(GLIA_ERR_STATE, "get_adjoint: needs an adjoint solve with full history");
    export_field(p_hist_[i], out);
  }

  // ------------------------------------------------------------------------------------------
  // derivative operators (src/grad/DerivativeOperatorsRD.cpp, DerivativeOperators.cpp)
  // ------------------------------------------------------------------------------------------
  bool update_kappa() const {
    return opt_.diffusivity_inversion || opt_.flag_reaction_inv || opt_.all_gradients;
  }
  bool update_rho() const { return opt_.flag_reaction_inv || opt_.all_gradients; }
  bool apply_phi() const { return !opt_.flag_reaction_inv || opt_.all_gradients; }
  int nx() const { return opt_.np + opt_.nk + opt_.nr; }

  // DerivativeOperators::updateReactionAndDiffusion (src/grad/DerivativeOperators.cpp:323-367)
  void update_coefficients(const double* x) {
    const int np = opt_.np, nk = opt_.nk, nr = opt_.nr;
    if (update_kappa()) {
      const double k1 = x[np] * opt_.k_scale;
      const double k2 = nk > 1 ? x[np + 1] * opt_.k_scale : 0;
      const double k3 = nk > 2 ? x[np + 2] * opt_.k_scale : 0;
      // DiffCoef::updateIsotropicCoefficients (src/mat/DiffCoef.cpp:60-75)
      diffcoef_set(k1, nk == 1 ? k_gm_wm_ : k2 / k1, nk == 1 ? k_glm_wm_ : k3 / k1);
      prec_factor();
    }
    if (update_rho()) {
      const double r1 = x[np + nk] * opt_.rho_scale;
      const double r2 = nr > 1 ? x[np + nk + 1] * opt_.rho_scale : 0;
      const double r3 = nr > 2 ? x[np + nk + 2] * opt_.rho_scale : 0;
      reaccoef_set(r1, nr == 1 ? r_gm_wm_ : r2 / r1, nr == 1 ? r_glm_wm_ : r3 / r1);
    }
  }

  void evaluate(const double* x, int nxin, const void* d1, double* J, double* dJ) override {
    if (nxin != nx())
      throw Error(GLIA_ERR_INVALID, "x has " + std::to_string(nxin) + " entries, expected " +
                                        std::to_string(nx()) + " (np + nk + nr)");
    const bool want_grad = dJ != nullptr;
    if (J) st_.nb_obj_evals++;
    if (want_grad) st_.nb_grad_evals++;
    const int np = opt_.np;
    if (want_grad) std::fill(dJ, dJ + nx(), 0.0);
    R* data = d1_buf();
    import_field(d1, data);
    update_coefficients(x);
    if (apply_phi()) phi_apply_into(c0_, x);
    // two snapshots: ||O0 c(0) - d0||^2 and r0 = -O0^T (O0 c(0) - d0)
    double m0 = 0;
    if (two_tp_) {
      if (want_grad && !r0_) r0_ = fld();
      GLIA_TIMED(KS_OBS, FB() * (want_grad ? 4 : 3),
                 k_obs_residual<R><<<red_blocks_, kThreads, 0, stream_>>>(
                     N_, c0_, obs0(), d0_, want_grad ? r0_ : nullptr, sc_, ws_));
      m0 = read_red(0);
    }
    solve_state_internal();
    const double h = 2.0 * M_PI / g_.n, h3 = h * h * h;
    GLIA_TIMED(KS_OBS, FB() * (want_grad ? 4 : 3),
               k_obs_residual<R><<<red_blocks_, kThreads, 0, stream_>>>(
                   N_, ct_, obs_, data, want_grad ? pt_ : nullptr, sc_, ws_));
    const double m1 = read_red(0);
    if (want_grad) {
      solve_adjoint_internal(true);
      if (apply_phi()) p_gradient(x, dJ, h3);
      if (two_tp_) {  // dJ_p += h^3 Phi^T O0^T (O0 c(0) - d0) (:189-196)
        std::vector<double> pr(std::max({opt_.np, phi_np_, 1}));
        phi_applyT_from(r0_, pr.data());
        for (int i = 0; i < np; i++) dJ[i] += h3 * (-pr[i]);
      }
    }
    double reg = 0;
    if (opt_.regularization_norm == 0) {
      if (opt_.beta != 0) reg = vdot_any(c0_, c0_) * 0.5 * opt_.beta * h3;
    } else {
      for (int i = 0; i < np; i++) reg += x[i] * x[i];
      reg *= 0.5 * opt_.beta;
    }
    if (J) *J = h3 * 0.5 * (m1 + m0) + reg;
    if (!want_grad) return;
    // gradDiffusion / gradReaction (src/grad/DerivativeOperators.cpp:189-321)
    double acc[8];
    if (ref_)
      ref_time_integrals(acc);
    else {
      GLIA_CUDA(cudaMemcpyAsync(hsc_, sc_, sizeof(DevScalars), cudaMemcpyDeviceToHost, stream_));
      GLIA_CUDA(cudaStreamSynchronize(stream_));
      std::memcpy(acc, hsc_->acc, sizeof(acc));
    }
    coefficient_gradient(acc, dJ, h3);
  }
  // kappa and rho blocks of the gradient from the time integrals acc (DevScalars::acc)
  void coefficient_gradient(const double* acc, double* dJ, double h3) {
    const int np = opt_.np, nk = opt_.nk, nr = opt_.nr;
    if (update_kappa()) {
      double Twm, Tgm, Tcsf;
      if (!ref_ && kappa_used_trick_) {
        // <m, grad c . grad a> = -<c, D a> / kappa with k = kappa (wm + k_gm_wm gm)
        Twm = -acc[6] / k_scale_;
        dJ[np] = Twm * h3;
      } else {
        Twm = acc[0];
        Tgm = acc[1];
        Tcsf = acc[2];
        dJ[np] = Twm * h3;
        if (nk == 1) dJ[np] += Tgm * h3 * k_gm_wm_;
        if (nk > 1) dJ[np + 1] = Tgm * h3;
        if (nk > 2) dJ[np + 2] = Tcsf * h3;
      }
    }
    if (update_rho()) {
      dJ[np + nk] = acc[3] * h3;
      if (nr == 1) dJ[np + nk] += acc[4] * h3 * r_gm_wm_;
      if (nr > 1) dJ[np + nk + 1] = acc[4] * h3;
      if (nr > 2) dJ[np + nk + 2] = acc[5] * h3;
    }
  }
  // ---- evaluation captured into a CUDA graph (glia_batch_*) -------------------------------
  // The fused engine's evaluate() with every host read moved to eval_finish: the coefficient
  // update, Phi p and the data upload run before the capture (they depend on x on the host), the
  // sweeps are captured with their PCG loops as conditional nodes, and J, the kappa / rho time
  // integrals, the Phi^T product and the solve statistics stay on the device until eval_finish.
  // One-snapshot objective, on-the-fly Phi (phi_store = 0), the reference default.
  void eval_prepare(const double* x, int nxin, const void* d1) override {
    if (ref_) throw Error(GLIA_ERR_INVALID, "graph-captured evaluations need the fused engine");
    if (two_tp_ || opt_.phi_store)
      throw Error(GLIA_ERR_INVALID,
                  "graph-captured evaluations support one snapshot and phi_store = 0");
    if (hist_mode_ == GLIA_HISTORY_OFF)
      throw Error(GLIA_ERR_STATE, "graph-captured evaluations need a time history");
    if (tm_.on) throw Error(GLIA_ERR_STATE, "disable timing before capturing an evaluation");
    if (nxin != nx())
      throw Error(GLIA_ERR_INVALID, "x has " + std::to_string(nxin) + " entries, expected " +
                                        std::to_string(nx()));
    cap_x_.assign(x, x + nxin);
    import_field(d1, d1_buf());
    update_coefficients(x);
    if (apply_phi()) phi_apply_into(c0_, x);
    const double h = 2.0 * M_PI / g_.n, h3 = h * h * h;
    cap_reg_ = 0;
    if (opt_.regularization_norm == 0) {
      if (opt_.beta != 0) cap_reg_ = vdot_any(c0_, c0_) * 0.5 * opt_.beta * h3;
    } else {
      for (int i = 0; i < opt_.np; i++) cap_reg_ += x[i] * x[i];
      cap_reg_ *= 0.5 * opt_.beta;
    }
    ensure_history();
    // buffers the sweeps allocate on first use, allocated now (never while capturing)
    if (!full()) {
      pnt();
      cfin();
      tmp2();
    }
    if (!kappa_trick_ok()) ga3();
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    cap_ready_ = true;
  }
  void eval_capture() override {
    if (!cap_ready_) throw Error(GLIA_ERR_STATE, "eval_capture needs eval_prepare first");
    const glia_stats saved = st_;  // capturing runs nothing: the counts come with eval_finish
    capture_ = true;
    cap_solves_ = 0;
    plane_pc_ = kNoField;  // the graph fills the field itself, whatever solves before a launch do
    try {
      k_solve_stats_reset<<<1, 1, 0, stream_>>>(sc_);
      GLIA_LAUNCH_CHECK();
      solve_state_internal();
      k_obs_residual<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, ct_, obs_, d1_buf(), pt_,
                                                               sc_, ws_);
      GLIA_LAUNCH_CHECK();
      k_keep_red0<<<1, 1, 0, stream_>>>(sc_);
      GLIA_LAUNCH_CHECK();
      solve_adjoint_internal(true);
      if (apply_phi()) {  // p gradient: Phi^T (alpha_0 - beta c_0), scaled in eval_finish
        if (opt_.beta != 0) vaxpy_any(p0_, -opt_.beta, c0_);
        k_phi_applyT<R><<<phi_np_, kThreads, 0, stream_>>>(g_, phi_boxes_, phi_store_, p0_,
                                                            phi_p_);
        GLIA_LAUNCH_CHECK();
      }
    } catch (...) {
      capture_ = false;
      plane_pc_ = kNoField;
      st_ = saved;
      throw;
    }
    capture_ = false;
    plane_pc_ = kNoField;  // recorded, not filled
    cap_total_solves_ = st_.total_diffusion_solves - saved.total_diffusion_solves;
    st_ = saved;
    // nothing has run yet: the history is valid only once a launch of the graph has been read
    cap_state_done_ = state_done_;
    cap_adjoint_done_ = adjoint_done_;
    state_done_ = adjoint_done_ = false;
  }
  void eval_launched() override { plane_pc_ = kNoField; }
  void eval_finish(double* J, double* dJ) override {
    if (!cap_ready_) throw Error(GLIA_ERR_STATE, "eval_finish needs a captured evaluation");
    std::vector<double> pp(std::max(phi_np_, 1));
    GLIA_CUDA(cudaMemcpyAsync(hsc_, sc_, sizeof(DevScalars), cudaMemcpyDeviceToHost, stream_));
    if (apply_phi())
      GLIA_CUDA(cudaMemcpyAsync(pp.data(), phi_p_, phi_np_ * sizeof(double),
                                cudaMemcpyDeviceToHost, stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    const DevScalars& h = *hsc_;
    st_.nb_obj_evals++;
    st_.nb_grad_evals++;
    st_.nb_state_solves++;
    st_.nb_adjoint_solves++;
    st_.diff_ksp_itr_state = h.sum_its[0];
    st_.diff_ksp_itr_adj = h.sum_its[1];
    st_.total_diffusion_solves += cap_total_solves_;
    st_.total_pcg_iterations += h.sum_its[0] + h.sum_its[1] + h.sum_its[2];
    st_.max_ksp_itr = std::max(st_.max_ksp_itr, h.max_its);
    st_.last_rnorm = h.last_dp;
    st_.last_ksp_itr = h.it;
    ksp_itr_ = h.it;
    if (h.dev_fault) raise_device_fault();
    if (h.err_status < 0) finish_solve(SolveStatus{h.err_status, h.err_its, h.last_dp});
    state_done_ = cap_state_done_;  // the launch swept the history as the capture recorded
    adjoint_done_ = cap_adjoint_done_;
    const double hh = 2.0 * M_PI / g_.n, h3 = hh * hh * hh;
    if (J) *J = h3 * 0.5 * h.m1_keep + cap_reg_;
    if (!dJ) return;
    std::fill(dJ, dJ + nx(), 0.0);
    if (apply_phi()) {  // the same products, in the same order, as p_gradient
      const double s = 1.0 / phi_max_all();
      for (int i = 0; i < opt_.np; i++) {
        const double v = pp[i] * s;
        dJ[i] = v * -h3;
      }
    }
    coefficient_gradient(h.acc, dJ, h3);
  }
  void* stream() const override { return stream_; }

  // p gradient (src/grad/DerivativeOperatorsRD.cpp:164-187)
  void p_gradient(const double* x, double* dJ, double h3) {
    const int np = opt_.np;
    std::vector<double> tmpv(std::max(np, 1));
    if (!opt_.phi_store) {
      if (opt_.beta != 0) vaxpy_any(p0_, -opt_.beta, c0_);
      phi_applyT_from(p0_, dJ);
      for (int i = 0; i < np; i++) dJ[i] *= -h3;
    } else {
      phi_applyT_from(p0_, tmpv.data());
      for (int i = 0; i < np; i++) tmpv[i] *= h3;
      if (opt_.regularization_norm == 0) {
        phi_applyT_from(c0_, dJ);
        for (int i = 0; i < np; i++) dJ[i] = dJ[i] * opt_.beta * h3 - tmpv[i];
      } else {
        for (int i = 0; i < nx(); i++) dJ[i] = x[i] * opt_.beta - (i < np ? tmpv[i] : 0.0);
      }
    }
  }
  // reference-structured gradDiffusion / gradReaction over the stored history
  void ref_time_integrals(double* acc) {
    std::fill(acc, acc + 8, 0.0);
    k_acc_reset<<<1, 1, 0, stream_>>>(sc_);
    GLIA_LAUNCH_CHECK();
    for (int i = 0; i <= nt_; i++) {
      vcopy(p0_, p_hist_[i]);
      grad_point(i, c_hist_[i], update_kappa());
    }
    GLIA_CUDA(cudaMemcpyAsync(hsc_, sc_, sizeof(DevScalars), cudaMemcpyDeviceToHost, stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    std::memcpy(acc, hsc_->acc, 8 * sizeof(double));
  }
  double vdot_any(const R* x, const R* y) {
    k_dot<R><<<red_blocks_, kThreads, 0, stream_>>>(N_, x, y, sc_, 0, ws_);
    GLIA_LAUNCH_CHECK();
    return read_red(0);
  }
  void vaxpy_any(R* y, double a, const R* x) {
    k_axpy<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, y, a, x);
    GLIA_LAUNCH_CHECK();
  }
  R* d1_buf() {
    if (!d1_) d1_ = fld();
    return d1_;
  }

  glia_stats stats() const override { return st_; }
  void set_timing(bool on) override {
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    tm_.harvest();
    tm_.reset();
    tm_.on = on;
  }
  int timing(int slot, const char** name, int64_t* launches, double* ms, double* bytes) override {
    if (slot < 0 || slot >= KS_COUNT) throw Error(GLIA_ERR_INVALID, "timing: slot out of range");
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    tm_.harvest();
    if (name) *name = kSlotNames[slot];
    if (launches) *launches = tm_.slots[slot].launches;
    if (ms) *ms = tm_.slots[slot].ms;
    if (bytes) *bytes = tm_.slots[slot].bytes;
    return KS_COUNT;
  }
  void reset_stats() override { st_ = glia_stats{}; }

 private:
  // ------------------------------------------------------------------------------------------
  // memory, transforms, transfers
  // ------------------------------------------------------------------------------------------
  template <typename T>
  T* dalloc(int64_t count) {
    void* p = nullptr;
    const size_t b = (size_t)std::max<int64_t>(count, 1) * sizeof(T);
    GLIA_CUDA(cudaMalloc(&p, b));
    sizes_[p] = b;
    bytes_ += (int64_t)b;
    return (T*)p;
  }
  void dfree(void* p) {
    auto it = sizes_.find(p);
    if (it == sizes_.end()) return;
    cudaStreamSynchronize(stream_);
    bytes_ -= (int64_t)it->second;
    sizes_.erase(it);
    cudaFree(p);
  }
  R* fld() { return dalloc<R>(N_); }
  double FB() const { return (double)N_ * sizeof(R); }         // bytes of one grid field
  double SB() const { return 2.0 * (double)Ns_ * sizeof(R); }  // bytes of one half spectrum
  R* spec() { return dalloc<R>(2 * Ns_); }
  void fill(R* f, double v) {
    k_fill<R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, f, v);
    GLIA_LAUNCH_CHECK();
  }

  cufftHandle make_plan(cufftType type, int batch, size_t* ws) {
    cufftHandle p;
    GLIA_CUFFT(cufftCreate(&p));
    GLIA_CUFFT(cufftSetAutoAllocation(p, 0));
    int dims[3] = {g_.n, g_.n, g_.n};
    const bool fwd = (type == CUFFT_R2C || type == CUFFT_D2Z);
    GLIA_CUFFT(cufftMakePlanMany(p, 3, dims, nullptr, 1, fwd ? (int)N_ : (int)Ns_, nullptr, 1,
                                 fwd ? (int)Ns_ : (int)N_, type, batch, ws));
    GLIA_CUFFT(cufftSetStream(p, stream_));
    return p;
  }
  void make_plans() {
    size_t w[5] = {0, 0, 0, 0, 0};
    r2c1_ = make_plan(CT<R>::kR2C, 1, &w[0]);
    c2r1_ = make_plan(CT<R>::kC2R, 1, &w[1]);
    r2c3_ = make_plan(CT<R>::kR2C, 3, &w[2]);
    c2r3_ = make_plan(CT<R>::kC2R, 3, &w[3]);
    const int n = g_.n;
    // Opt-in (GLIA_ZPASS=1): measured slower than the three-dimensional cuFFT path on GB300
    // because cuFFT's strided 2-D plan over (x, y) for every kz runs far below its own 3-D
    // passes; the fused path stays available for its tests and for other transform back ends.
    const char* on = std::getenv("GLIA_ZPASS");
    zpass_ = std::is_same<R, float>::value && (n == 64 || n == 128 || n == 256 || n == 512) &&
             (on && on[0] == '1') && !ref_;
    if (zpass_) {
      // 2-D C2C over (x, y) for every kz: element (x, y, kz) at (x n + y)(n/2+1) + kz
      GLIA_CUFFT(cufftCreate(&p2d_));
      GLIA_CUFFT(cufftSetAutoAllocation(p2d_, 0));
      int dims[2] = {n, n}, emb[2] = {n, n};
      GLIA_CUFFT(cufftMakePlanMany(p2d_, 2, dims, emb, g_.nh, 1, emb, g_.nh, 1, CUFFT_C2C, g_.nh,
                                   &w[4]));
      GLIA_CUFFT(cufftSetStream(p2d_, stream_));
      // twiddles W_n^j = exp(-2 pi i j / n), j < n, in double precision on the host
      std::vector<float2> tw(n);
      for (int j = 0; j < n; j++) {
        const double a = -2.0 * M_PI * (double)j / (double)n;
        tw[j] = make_float2((float)std::cos(a), (float)std::sin(a));
      }
      tw_ = dalloc<float2>(n);
      GLIA_CUDA(cudaMemcpyAsync(tw_, tw.data(), n * sizeof(float2), cudaMemcpyHostToDevice,
                                stream_));
      GLIA_CUDA(cudaStreamSynchronize(stream_));
    }
    // Transform path of the FP32 D apply at n = 64, 128, 256 (GLIA_XPASS): by default the x, y
    // and z passes are the library's own kernels (ownfft.cuh, no cuFFT inside the PCG loop);
    // "2d" keeps the x pass and lets cuFFT do batched 2-D (y, z) transforms with k multiplied in
    // between; "0" uses batched 3-D cuFFT transforms.
    const char* xenv = std::getenv("GLIA_XPASS");
    xpass_ = std::is_same<R, float>::value && (n == 64 || n == 128 || n == 256) && !zpass_ &&
             !ref_ && !(xenv && xenv[0] == '0');
    own_ = xpass_ && !(xenv && std::strcmp(xenv, "2d") == 0);
    // FP64 grids with a plane kernel (plane.hpp) run every solve as one launch; "0" and "2d" keep
    // cuFFT's transforms there.
    //
    // FP32 has none. Every solve transforms the whole field back, which leaves rounding of 6e-8 of
    // the field's maximum in tumour-free tissue, and the logistic reaction multiplies it by up to
    // exp(rho T): any change of the transforms inside a solve, even in its last bits, draws that
    // rounding anew. With float plane kernels a simulation of rho T = 10 moved by 1.5e-4 (5e-3 at
    // single voxels), its gradient by 2e-2, more than float results may move; at rho T = 14 by 7e-3
    // and 0.9. They also ran contexts side by side worse, a solve taking every SM: eight 64^3
    // gradients of 10 steps from 8 threads 18.5 -> 28.9 ms, though one alone took 9.1 -> 7.1 ms.
    if (kPlane && !ref_ && !(xenv && (xenv[0] == '0' || std::strcmp(xenv, "2d") == 0)))
      init_plane();
    size_t w2[2] = {0, 0};
    if (xpass_ && !own_) {
      int dims[2] = {n, n};
      for (int d = 0; d < 2; d++) {
        cufftHandle& p = d == 0 ? r2c2d3_ : c2r2d3_;
        GLIA_CUFFT(cufftCreate(&p));
        GLIA_CUFFT(cufftSetAutoAllocation(p, 0));
        const bool fwd = d == 0;
        GLIA_CUFFT(cufftMakePlanMany(p, 2, dims, nullptr, 1, fwd ? n * n : n * g_.nh, nullptr, 1,
                                     fwd ? n * g_.nh : n * n, fwd ? CT<R>::kR2C : CT<R>::kC2R,
                                     3 * n, &w2[d]));
        GLIA_CUFFT(cufftSetStream(p, stream_));
      }
    }
    if (xpass_) {
      std::vector<float2> tw(256);
      for (int j = 0; j < 256; j++) {
        const double a = -2.0 * M_PI * (double)j / 256.0;
        tw[j] = make_float2((float)std::cos(a), (float)std::sin(a));
      }
      tw256_ = dalloc<float2>(256);
      GLIA_CUDA(cudaMemcpy(tw256_, tw.data(), 256 * sizeof(float2), cudaMemcpyHostToDevice));
      if (n == 256)
        init_xpass_grids<256>();
      else if (n == 128)
        init_xpass_grids<128>();
      else
        init_xpass_grids<64>();
    }
    fft_ws_bytes_ = std::max({w[0], w[1], w[2], w[3], w[4], w2[0], w2[1], (size_t)16});
    fft_ws_ = dalloc<char>((int64_t)fft_ws_bytes_);
    for (cufftHandle p : {r2c1_, c2r1_, r2c3_, c2r3_}) GLIA_CUFFT(cufftSetWorkArea(p, fft_ws_));
    if (zpass_) GLIA_CUFFT(cufftSetWorkArea(p2d_, fft_ws_));
    if (xpass_ && !own_)
      for (cufftHandle p : {r2c2d3_, c2r2d3_}) GLIA_CUFFT(cufftSetWorkArea(p, fft_ws_));
  }
  void init_plane() {
    const PlaneKernel k = plane_kernel(g_.n);
    if (!k.fn) return;
    GLIA_CUDA(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
    int b = 0;
    GLIA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k.fn, k.threads, k.smem));
    if (b < 1) return;
    plane_ = k;
    plane_res_ = sms_ * b;
    plane_part_ = dalloc<double>((int64_t)kPlanePartials * plane_res_);
    plane_bar_ = dalloc<unsigned>(2);
    std::vector<int4> tw(g_.n);
    plane_twiddles(g_.n, tw.data());
    plane_tw_ = dalloc<int4>(g_.n);
    if (k.split) plane_w_ = dalloc<R>(3 * N_);
    plane_pf_ = dalloc<R>(Ns_);
    GLIA_CUDA(cudaMemsetAsync(plane_bar_, 0, 2 * sizeof(unsigned), stream_));
    GLIA_CUDA(cudaMemcpyAsync(plane_tw_, tw.data(), g_.n * sizeof(int4), cudaMemcpyHostToDevice,
                              stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
  }
  void c2c2d(R* data, int dir) {
    cudaEvent_t ev = tm_.begin(stream_);
    if constexpr (std::is_same<R, float>::value) {
      cufftComplex* d = reinterpret_cast<cufftComplex*>(data);
      GLIA_CUFFT(cufftExecC2C(p2d_, d, d, dir));
    }
    tm_.end(KS_FFT_2D, ev, 2.0 * SB(), stream_);
    st_.total_fft_execs += 1;
  }
  void launch_zpass(int blocks, int lines) {
    if constexpr (std::is_same<R, float>::value) {
      const int n = g_.n;
      float* s3 = g3s_;
      const float* k = kxx_;
      if (n == 64)
        k_zpass_mulk<1><<<blocks, kThreads, 0, stream_>>>(n, lines, s3, Ns_, k, tw_);
      else if (n == 128)
        k_zpass_mulk<2><<<blocks, kThreads, 0, stream_>>>(n, lines, s3, Ns_, k, tw_);
      else if (n == 256)
        k_zpass_mulk<4><<<blocks, kThreads, 0, stream_>>>(n, lines, s3, Ns_, k, tw_);
      else
        k_zpass_mulk<8><<<blocks, kThreads, 0, stream_>>>(n, lines, s3, Ns_, k, tw_);
    }
  }
  void ensure_batch_plans(int B) {
    destroy_batch_plans();
    size_t w[2] = {0, 0};
    r2cB_ = make_plan(CT<R>::kR2C, B, &w[0]);
    c2rB_ = make_plan(CT<R>::kC2R, B, &w[1]);
    const size_t need = std::max(w[0], w[1]);
    if (need > fft_ws_bytes_) {
      batch_ws_ = dalloc<char>((int64_t)need);
      GLIA_CUFFT(cufftSetWorkArea(r2cB_, batch_ws_));
      GLIA_CUFFT(cufftSetWorkArea(c2rB_, batch_ws_));
    } else {
      GLIA_CUFFT(cufftSetWorkArea(r2cB_, fft_ws_));
      GLIA_CUFFT(cufftSetWorkArea(c2rB_, fft_ws_));
    }
  }
  void destroy_batch_plans() {
    if (r2cB_) cufftDestroy(r2cB_);
    if (c2rB_) cufftDestroy(c2rB_);
    r2cB_ = c2rB_ = 0;
    if (batch_ws_) {
      dfree(batch_ws_);
      batch_ws_ = nullptr;
    }
  }
  int fft_slot(cufftHandle p, bool fwd) const {
    if (p == r2c3_ || p == c2r3_ || p == r2c2d3_ || p == c2r2d3_)
      return fwd ? KS_FFT_R2C3 : KS_FFT_C2R3;
    return fwd ? KS_FFT_R2C : KS_FFT_C2R;
  }
  void r2c(cufftHandle p, const R* in, R* out, int batch = 1) {
    cudaEvent_t ev = tm_.begin(stream_);
    r2c_raw(p, in, out, batch);
    tm_.end(fft_slot(p, true), ev, (double)batch * (FB() + SB()), stream_);
  }
  void c2r(cufftHandle p, R* in, R* out, int batch = 1) {
    cudaEvent_t ev = tm_.begin(stream_);
    c2r_raw(p, in, out, batch);
    tm_.end(fft_slot(p, false), ev, (double)batch * (FB() + SB()), stream_);
  }
  void r2c_raw(cufftHandle p, const R* in, R* out, int batch) {
    if constexpr (std::is_same<R, float>::value)
      GLIA_CUFFT(cufftExecR2C(p, const_cast<float*>(in), reinterpret_cast<cufftComplex*>(out)));
    else
      GLIA_CUFFT(cufftExecD2Z(p, const_cast<double*>(in),
                              reinterpret_cast<cufftDoubleComplex*>(out)));
    st_.total_fft_execs += batch;
  }
  void c2r_raw(cufftHandle p, R* in, R* out, int batch) {
    if constexpr (std::is_same<R, float>::value)
      GLIA_CUFFT(cufftExecC2R(p, reinterpret_cast<cufftComplex*>(in), out));
    else
      GLIA_CUFFT(cufftExecZ2D(p, reinterpret_cast<cufftDoubleComplex*>(in), out));
    st_.total_fft_execs += batch;
  }

  SolveStatus read_status() {
    GLIA_CUDA(cudaMemcpyAsync(&hsc_->it, &sc_->it, 3 * sizeof(int), cudaMemcpyDeviceToHost,
                              stream_));
    GLIA_CUDA(cudaMemcpyAsync(&hsc_->dp, &sc_->dp, sizeof(double), cudaMemcpyDeviceToHost,
                              stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    tm_.harvest();
    return SolveStatus{hsc_->status, hsc_->it, hsc_->dp};
  }
  double read_red(int slot) {
    GLIA_CUDA(cudaMemcpyAsync(&hsc_->red[slot], &sc_->red[slot], sizeof(double),
                              cudaMemcpyDeviceToHost, stream_));
    GLIA_CUDA(cudaStreamSynchronize(stream_));
    tm_.harvest();
    return hsc_->red[slot];
  }

  double* stage() {
    if (!stage_) stage_ = dalloc<double>(N_);
    return stage_;
  }
  // grid field in the caller's pointer mode -> device field of type R
  void import_field(const void* src, R* dst) {
    if (!src) throw Error(GLIA_ERR_INVALID, "null field pointer");
    const size_t nb = (size_t)N_;
    if (ptr_mode_ == GLIA_PTR_HOST_F64) {
      if constexpr (std::is_same<R, double>::value) {
        GLIA_CUDA(cudaMemcpyAsync(dst, src, nb * 8, cudaMemcpyHostToDevice, stream_));
      } else {
        GLIA_CUDA(cudaMemcpyAsync(stage(), src, nb * 8, cudaMemcpyHostToDevice, stream_));
        k_convert<double, R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, stage(), dst);
        GLIA_LAUNCH_CHECK();
      }
    } else if (ptr_mode_ == GLIA_PTR_DEVICE_F64) {
      if constexpr (std::is_same<R, double>::value) {
        if (src != dst)
          GLIA_CUDA(cudaMemcpyAsync(dst, src, nb * 8, cudaMemcpyDeviceToDevice, stream_));
      } else {
        k_convert<double, R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, (const double*)src, dst);
        GLIA_LAUNCH_CHECK();
      }
    } else {
      if constexpr (std::is_same<R, float>::value) {
        if (src != dst)
          GLIA_CUDA(cudaMemcpyAsync(dst, src, nb * 4, cudaMemcpyDeviceToDevice, stream_));
      } else {
        k_convert<float, R><<<pw_blocks_, kThreads, 0, stream_>>>(N_, (const float*)src, dst);
        GLIA_LAUNCH_CHECK();
      }
    }
  }
  void export_field(const R* src, void* dst) {
    if (!dst) throw Error(GLIA_ERR_INVALID, "null field pointer");
    const size_t nb = (size_t)N_;
    if (ptr_mode_ == GLIA_PTR_HOST_F64) {
      if constexpr (std::is_same<R, double>::value) {
        GLIA_CUDA(cudaMemcpyAsync(dst, src, nb * 8, cudaMemcpyDeviceToHost, stream_));
      } else {
        k_convert<R, double><<<pw_blocks_, kThreads, 0, stream_>>>(N_, src, stage());
        GLIA_LAUNCH_CHECK();
        GLIA_CUDA(cudaMemcpyAsync(dst, stage(), nb * 8, cudaMemcpyDeviceToHost, stream_));
      }
      GLIA_CUDA(cudaStreamSynchronize(stream_));
    } else if (ptr_mode_ == GLIA_PTR_DEVICE_F64) {
      if constexpr (std::is_same<R, double>::value) {
        if (src != dst)
          GLIA_CUDA(cudaMemcpyAsync(dst, src, nb * 8, cudaMemcpyDeviceToDevice, stream_));
      } else {
        k_convert<R, double><<<pw_blocks_, kThreads, 0, stream_>>>(N_, src, (double*)dst);
        GLIA_LAUNCH_CHECK();
      }
    } else {
      if constexpr (std::is_same<R, float>::value) {
        if (src != dst)
          GLIA_CUDA(cudaMemcpyAsync(dst, src, nb * 4, cudaMemcpyDeviceToDevice, stream_));
      } else {
        k_convert<R, float><<<pw_blocks_, kThreads, 0, stream_>>>(N_, src, (float*)dst);
        GLIA_LAUNCH_CHECK();
      }
    }
  }

  // ------------------------------------------------------------------------------------------
  Geo g_;
  bool ref_;
  int sms_ = 0, red_blocks_ = 0, pw_blocks_ = 0;
  int64_t N_ = 0, Ns_ = 0;
  cudaStream_t stream_ = nullptr, own_stream_ = nullptr;
  int ptr_mode_ = GLIA_PTR_HOST_F64;
  std::unordered_map<void*, size_t> sizes_;
  int64_t bytes_ = 0;
  KTimer tm_;
  int graph_state_ = 0;  // 0 not built, 1 built, -1 unavailable (host-driven loop)
  bool graph_solves_ = false;  // the current sweep ran PCG loops as graphs
  bool last_seg_resident_ = false;  // segment buffers hold the last segment of the forward
  cudaGraphExec_t cg_exec_ = nullptr;

  cufftHandle r2c1_ = 0, c2r1_ = 0, r2c3_ = 0, c2r3_ = 0, r2cB_ = 0, c2rB_ = 0, p2d_ = 0;
  bool zpass_ = false;   // fused z pass (FP32, n = 64 ... 512)
  bool xpass_ = false;   // x pass fused into the spectral kernels (FP32, n = 64 ... 256)
  cufftHandle r2c2d3_ = 0, c2r2d3_ = 0;  // batched 2-D (y, z) transforms, 3n planes
  float2* tw256_ = nullptr;
  int xres_inv_ = 0, xres_fwd_ = 0;  // resident CTAs of k_xinv / k_xfwd on this device
  int own_res_[3] = {0, 0, 0};       // ... of the y-inverse pass, the z pass, k_yfwd
  CUtensorMap kmap_{};               // TMA map of the packed line arrays (k_yfwd)
  bool tma_ = false;                 // k_yfwd stages with TMA copies (GLIA_TMA=1)
  bool zrev_ = true;                 // k_zpass2 line blocks in descending order
  bool zpass2_ = true;               // z pass with two real lines per complex transform
  bool yinv_bulk_ = true;            // y-inverse rows staged by bulk copies
  bool own_ = false;  // own y and z passes (x pass on): no cuFFT inside the D apply
  // graph-captured evaluations (eval_prepare / eval_capture / eval_finish)
  bool capture_ = false, cap_ready_ = false;
  bool cap_state_done_ = false, cap_adjoint_done_ = false;
  cudaStream_t cap_side_ = nullptr;  // captures the PCG loop bodies
  int64_t cap_solves_ = 0, cap_total_solves_ = 0;
  double cap_reg_ = 0;
  std::vector<double> cap_x_;
  // plane kernel (plane.cuh) of this grid size: resident CTAs, partial sums, barrier, twiddles
  PlaneKernel plane_{};
  R* plane_w_ = nullptr;
  int plane_res_ = 0;
  double* plane_part_ = nullptr;
  unsigned* plane_bar_ = nullptr;
  // Some 8 s: much longer than a barrier takes (1 us) or the CTAs of a launch differ (a phase, 2 ms
  // at 256^3), so that other streams' kernels or time slices of other processes, which can hold
  // some of the CTAs up, are no fault
  static constexpr long long kPlaneWait = 1LL << 34;
  long long plane_wait_ = kPlaneWait;
  int4* plane_tw_ = nullptr;
  static constexpr double kPlaneGrowth = 10.5;
  double rho_max_ = 0;
  static constexpr double kNoField = -1;
  R* plane_pf_ = nullptr;        // preconditioner field for pc_c = plane_pc_
  double plane_pc_ = kNoField;   // a launched graph fills the field for its own
  float2* tw_ = nullptr;
  char* fft_ws_ = nullptr;
  char* batch_ws_ = nullptr;
  size_t fft_ws_bytes_ = 0;

  DevScalars* sc_ = nullptr;
  DevScalars* hsc_ = nullptr;
  SolveStatus* hst_ = nullptr;
  RedWs ws_{};

  // TumorParameters / solver settings
  double dt_ = 0.5;
  int nt_ = 1, order_ = 2;
  bool adjoint_store_ = false;
  int hist_mode_ = GLIA_HISTORY_FULL, every_ = 10;
  double rtol_ = 1e-6, abstol_ = 1e-50, divtol_ = 1e4;
  int maxit_ = 5000, pc_dt_mode_ = GLIA_PC_DT_REFERENCE;
  double pc_dt_fixed_ = 0, ctx_dt_ = 0.5, pc_kbar_ = 0, pc_dt_ = 0.5;
  int ksp_itr_ = 0;
  glia_opt_settings opt_{1, 1, 1, 0, 1, 0, 1e-4, 1.0, 1.0, 0, 0};
  glia_stats st_{};

  // MatProp / DiffCoef / ReacCoef
  R *wm_ = nullptr, *gm_ = nullptr, *csf_ = nullptr, *vt_ = nullptr, *bg_ = nullptr,
    *filter_ = nullptr, *kxx_ = nullptr, *rho_ = nullptr, *obs_ = nullptr;
  bool tissue_set_ = false, kxx_sinusoidal_ = false;
  double filter_sum_ = 0, k_scale_ = 1e-2, kxx_avg_ = 0, k_gm_wm_ = 0, k_glm_wm_ = 0;
  double rho_scale_ = 0, r_gm_wm_ = 0, r_glm_wm_ = 0;

  // Tumor state and work
  R *c0_ = nullptr, *ct_ = nullptr, *p0_ = nullptr, *pt_ = nullptr, *tmp_ = nullptr,
    *tmp2_ = nullptr, *d1_ = nullptr;
  // Hessian with diffusivity inversion: k~ (DiffCoef::temp_[7]), the incremental sources' work
  // field, the reference's p_[nt] and c_[nt] of checkpointed runs
  R *ksec_ = nullptr, *inc_ = nullptr, *pnt_ = nullptr, *cfin_ = nullptr;
  bool ksec_set_ = false;
  // two-snapshot objective: O at t = 0, d0, and -O0^T (O0 c(0) - d0)
  R *obs0_ = nullptr, *d0_ = nullptr, *r0_ = nullptr;
  bool two_tp_ = false;
  R *chat_ = nullptr, *xhat_ = nullptr, *rhat_ = nullptr, *phat_ = nullptr, *what_ = nullptr;
  R *g3s_ = nullptr, *g3r_ = nullptr, *ga3_ = nullptr;
  R* wkern_ = nullptr;
  double wkern_sigma_ = -1;
  double* stage_ = nullptr;

  // reference-structured path
  R* t_[8] = {};
  R *rb_ = nullptr, *rr_ = nullptr, *rz_ = nullptr, *rp_ = nullptr, *rw_ = nullptr,
    *rt2_ = nullptr;
  R *kxy_ = nullptr, *kxz_ = nullptr, *kyz_ = nullptr, *kyy_ = nullptr, *kzz_ = nullptr;
  R *wh_ = nullptr, *pf_ = nullptr;

  // history
  std::vector<R*> c_hist_, c_half_, chat_hist_, p_hist_, ckpt_, seg_c_, seg_half_, seg_chat_;
  bool state_done_ = false, adjoint_done_ = false, trick_at_state_ = false,
       kappa_used_trick_ = false;

  // Phi
  int phi_np_ = 0, cells_per_dim_ = 0;
  double phi_sigma_ = 0;
  std::vector<double> centers_, phi_max_each_, hphi_p_;
  std::vector<PhiBox> phi_box_h_;
  R* phi_store_ = nullptr;
  double phi_store_bytes_ = 0;
  PhiBox* phi_boxes_ = nullptr;
  double* phi_centers_ = nullptr;
  double* phi_p_ = nullptr;
  int *cell_ptr_ = nullptr, *cell_list_ = nullptr;
};

}  // namespace glia
