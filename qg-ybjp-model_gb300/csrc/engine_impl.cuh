// Engine<T>: device buffers, launch sequence and CUDA-graph replay of the
// step, state conversions, routine-level drop-ins.  T = float (mixed
// precision: FP64 only in the tridiagonal solves and the diagnostics) or
// T = double (FP64 everywhere).
#pragma once
#include <cuda.h>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <cmath>
#include <algorithm>
#include "engine.h"
#include "dense_kernels.cuh"
#include "step_fx.cuh"
#include "fx_twiddles.h"

namespace qg {

#define QG_CK(call)                                                                          \
  do {                                                                                       \
    cudaError_t e_ = (call);                                                                 \
    if (e_ != cudaSuccess) {                                                                 \
      char b_[512];                                                                          \
      snprintf(b_, sizeof b_, "%s:%d: %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); \
      err = b_;                                                                              \
      return e_ == cudaErrorMemoryAllocation ? QG_ERR_NOMEM : QG_ERR_CUDA;                   \
    }                                                                                        \
  } while (0)

#define QG_LAUNCHED() QG_CK(cudaGetLastError())

#define QG_SWITCH_N(n, ...)                      \
  switch (n) {                                    \
    case 16: { constexpr int NN = 16; __VA_ARGS__; break; }    \
    case 32: { constexpr int NN = 32; __VA_ARGS__; break; }    \
    case 64: { constexpr int NN = 64; __VA_ARGS__; break; }    \
    case 128: { constexpr int NN = 128; __VA_ARGS__; break; }  \
    case 256: { constexpr int NN = 256; __VA_ARGS__; break; }  \
    case 512: { constexpr int NN = 512; __VA_ARGS__; break; }  \
    case 1024: { constexpr int NN = 1024; __VA_ARGS__; break; }\
    default: err = "unsupported n"; return QG_ERR_UNSUPPORTED; \
  }

enum { F_Q = 0, F_QO, F_BR, F_BI, F_BRO, F_BIO, F_PSI, F_AR, F_AI, F_QSTAR, F_DQ, F_NINT };

template <typename T>
class Engine : public EngineBase {
  using C = cplx<T>;

 public:
  ~Engine() override { release(); }

  int init(const qg_config& c, const HostTables& t) override {
    cfg = c;
    g.n = t.n; g.n3 = t.n3; g.K = t.K; g.KX = t.KX; g.KY = t.KY; g.KXP = t.KXP; g.kmax2 = t.kmax2;
    g.nseg = t.nseg > 0 ? t.nseg : t.n3;
    members = g.n3 / g.nseg;
    g.plane = t.plane;
    QG_CK(cudaSetDevice(cfg.device));
    // the step's stream at the highest priority, the overlapped A solves on
    // a second stream at the lowest: pending CTAs of the FP32 kernels are
    // placed first and the solves fill the room they leave
    int prio_low = 0, prio_high = 0;
    QG_CK(cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high));
    QG_CK(cudaStreamCreateWithPriority(&st, cudaStreamNonBlocking, prio_high));
    QG_CK(cudaStreamCreateWithPriority(&st2, cudaStreamNonBlocking, prio_low));
    QG_CK(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
    QG_CK(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
    QG_CK(cudaEventCreateWithFlags(&ev_diag, cudaEventDisableTiming));
    const size_t fbytes = (size_t)g.n3 * g.plane * sizeof(C);
    for (int f = 0; f < F_NINT; ++f) {
      if (f == F_DQ && !(cfg.inviscid == 0 && cfg.nuz != 0.0)) continue;
      QG_CK(cudaMalloc(&F[f], fbytes));
      QG_CK(cudaMemsetAsync(F[f], 0, fbytes, st));
    }
    if (!cfg.ybj_plus && !cfg.passive_scalar) {
      for (auto& p : sig) { QG_CK(cudaMalloc(&p, fbytes)); QG_CK(cudaMemsetAsync(p, 0, fbytes, st)); }
    }
    // tables
    // integrating factors: [members][plane]
    std::vector<T> tmp((size_t)members * g.plane);
    auto up = [&](T** d, const std::vector<double>& h) -> int {
      for (size_t i = 0; i < tmp.size(); ++i) tmp[i] = (T)h[i];
      QG_CK(cudaMalloc(d, tmp.size() * sizeof(T)));
      QG_CK(cudaMemcpy(*d, tmp.data(), tmp.size() * sizeof(T), cudaMemcpyHostToDevice));
      return QG_OK;
    };
    if (members > 1) {
      QG_CK(cudaMalloc(&mpar, t.mpar.size() * sizeof(double)));
      QG_CK(cudaMemcpy(mpar, t.mpar.data(), t.mpar.size() * sizeof(double), cudaMemcpyHostToDevice));
    }
    int rc;
    if ((rc = up(&e1, t.e1)) || (rc = up(&e2, t.e2)) || (rc = up(&e1w, t.e1w)) || (rc = up(&e2w, t.e2w))) return rc;
    {
      const std::vector<double>* om[4] = {&t.om_t1, &t.om_du, &t.om_dl, &t.om_a};
      double** dst[4] = {&om_t1, &om_du, &om_dl, &om_a};
      for (int k = 0; k < 4; ++k) {
        QG_CK(cudaMalloc(dst[k], (size_t)g.n3 * sizeof(double)));
        QG_CK(cudaMemcpy(*dst[k], om[k]->data(), (size_t)g.n3 * sizeof(double), cudaMemcpyHostToDevice));
      }
    }
    // twiddles: W_n^m in FP32, the per-pass integer tables in FP64 (fxfft.cuh)
    QG_CK(cudaMalloc(&tw, g.n * sizeof(C)));
    if (sizeof(T) == 8) {
      const std::vector<int32_t> twi = fx_twiddles(g.n);
      static_assert(sizeof(T) != 8 || sizeof(C) == 4 * sizeof(int32_t), "one table entry per complex double");
      QG_CK(cudaMemcpy(tw, twi.data(), g.n * sizeof(C), cudaMemcpyHostToDevice));
    } else {
      std::vector<C> twh(g.n);
      for (int m = 0; m < g.n; ++m) twh[m] = mk<T>((T)t.tw[2 * m], (T)t.tw[2 * m + 1]);
      QG_CK(cudaMemcpy(tw, twh.data(), g.n * sizeof(C), cudaMemcpyHostToDevice));
    }
    QG_CK(cudaMalloc(&tab_idx, g.plane * sizeof(int)));
    QG_CK(cudaMemcpy(tab_idx, t.tab_idx.data(), g.plane * sizeof(int), cudaMemcpyHostToDevice));
    // columns of the solves: every column of the rectangle (any output
    // array), and the retained ones only (the resident fields, whose other
    // entries are zeros the solves need not rewrite)
    {
      std::vector<int> all(g.plane), ret;
      for (long long m = 0; m < g.plane; ++m) {
        all[m] = (int)m;
        const int r = (int)(m / g.KXP), kx = (int)(m % g.KXP);
        if (g.mask(kx, g.ky_of_row(r))) ret.push_back((int)m);
      }
      nret = (int)ret.size();
      QG_CK(cudaMalloc(&cols_all, all.size() * sizeof(int)));
      QG_CK(cudaMemcpy(cols_all, all.data(), all.size() * sizeof(int), cudaMemcpyHostToDevice));
      QG_CK(cudaMalloc(&cols_ret, ret.size() * sizeof(int)));
      QG_CK(cudaMemcpy(cols_ret, ret.data(), ret.size() * sizeof(int), cudaMemcpyHostToDevice));
    }
    {
      std::vector<int> k2(t.ndistinct);
      for (long long m = 0; m < g.plane; ++m)
        if (t.tab_idx[m] >= 0) {
          const int kx = (int)(m % g.KXP), ky = g.ky_of_row((int)(m / g.KXP));
          k2[t.tab_idx[m]] = kx * kx + ky * ky;
        }
      om_nd = t.ndistinct;
      if (om_nd) {
        QG_CK(cudaMalloc(&om_kh2, om_nd * sizeof(int)));
        QG_CK(cudaMemcpy(om_kh2, k2.data(), om_nd * sizeof(int), cudaMemcpyHostToDevice));
      }
    }
    const size_t fb = std::max<size_t>(1, (size_t)t.ndistinct * g.nseg) * sizeof(double4);
    QG_CK(cudaMalloc(&fac_psi, fb));
    QG_CK(cudaMalloc(&fac_A, fb));
    if (t.ndistinct > 0) {
      QG_CK(cudaMemcpy(fac_psi, t.fac_psi.data(), (size_t)t.ndistinct * g.nseg * sizeof(double4), cudaMemcpyHostToDevice));
      QG_CK(cudaMemcpy(fac_A, t.fac_A.data(), (size_t)t.ndistinct * g.nseg * sizeof(double4), cudaMemcpyHostToDevice));
    }
    auto upd = [&](double** d, const std::vector<double>& h) -> int {
      QG_CK(cudaMalloc(d, h.size() * sizeof(double)));
      QG_CK(cudaMemcpy(*d, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice));
      return QG_OK;
    };
    if ((rc = upd(&du, t.du)) || (rc = upd(&cu, t.cu)) || (rc = upd(&cl, t.cl)) || (rc = upd(&r2, t.r2))) return rc;
    {
      // per-level weights of the diagnostics' vertical-difference sums:
      // w1 = 0.5/(r2 Bu dz^2) (wpe), w4 = Bu/(r2 dz^2) (pe), in FP64 and as
      // FP32 pairs (h, l) with h + l = w to ~2^-48
      std::vector<double> wv(2 * (size_t)g.nseg);
      std::vector<float2> wf(2 * (size_t)g.nseg);
      const double inv_dz2 = 1.0 / (cfg.dz * cfg.dz);
      for (int i = 0; i < g.nseg; ++i) {
        wv[i] = (0.5 / (t.r2[i] * cfg.Bu)) * inv_dz2;
        wv[g.nseg + i] = (cfg.Bu / t.r2[i]) * inv_dz2;
      }
      for (size_t i = 0; i < wv.size(); ++i) {
        const float h = (float)wv[i];
        wf[i] = make_float2(h, (float)(wv[i] - (double)h));
      }
      if ((rc = upd(&dwz, wv))) return rc;
      QG_CK(cudaMalloc(&fwz, wf.size() * sizeof(float2)));
      QG_CK(cudaMemcpy(fwz, wf.data(), wf.size() * sizeof(float2), cudaMemcpyHostToDevice));
    }
    {
      int occ = 0;
      QG_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, cfg.device));
      QG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_diag_cols<T>, kDiagThreads, 0));
      diag_slots = std::max(1, occ) * nsm;
      // partials of the largest launch (any number of whole segments)
      size_t mx = 0;
      for (int ns = 1; ns <= g.n3 / g.nseg; ++ns) mx = std::max(mx, diag_parts(ns));
      diag_part_n = mx;
    }
    QG_CK(cudaMalloc(&diag_part, diag_part_n * kNDiag * sizeof(double)));
    QG_CK(cudaMalloc(&diag_out, kNDiag * sizeof(double)));
    QG_CK(cudaMallocHost(&diag_host, kNDiag * sizeof(double)));
    QG_CK(cudaHostAlloc(&wflag_h, 3 * sizeof(int), cudaHostAllocMapped));
    wflag_h[0] = wflag_h[1] = wflag_h[2] = 0;
    QG_CK(cudaHostGetDevicePointer(&wflag, wflag_h, 0));
    nflag = wflag + 1;
    iflag = wflag + 2;
    QG_CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, cfg.device));
    // phase-A batching: by default as many levels per batch as 1.25 GB of
    // scratch planes hold (deep batches run fewer, fuller waves and longer
    // persistent row kernels; on GB300 the 512^2x256 step is fastest with
    // all 256 levels in one batch although its scratch outgrows L2)
    const size_t per_level = (size_t)kNScr * g.n * g.KXP * sizeof(C);
    int zb = cfg.levels_per_batch;
    if (zb <= 0) zb = (int)std::max<size_t>(1, (size_t)(1280u << 20) / per_level);
    zb = std::min(zb, g.n3);
    const int nb = (g.n3 + zb - 1) / zb;
    Zb = (g.n3 + nb - 1) / nb;
    lanes = std::max(1, std::min(kBatchLanes, nb));
    QG_CK(cudaMalloc(&S, (size_t)lanes * Zb * per_level));
    s_levels = lanes * Zb;
    for (int i = 1; i < kMaxLanes; ++i) {
      QG_CK(cudaStreamCreateWithPriority(&lst[i], cudaStreamNonBlocking, prio_high));
      QG_CK(cudaEventCreateWithFlags(&lev[i], cudaEventDisableTiming));
    }
    QG_CK(cudaEventCreateWithFlags(&ev_start, cudaEventDisableTiming));
    sp.delt = cfg.delt; sp.gamma = cfg.gamma; sp.Bu = cfg.Bu; sp.Ro = cfg.Ro; sp.W2F = cfg.W2F;
    sp.dz = cfg.dz; sp.nuz = cfg.nuz; sp.cdisp = 0.5 / (cfg.Bu * cfg.Ro);
    sp.adv = cfg.linear ? 0 : 1;
    sp.refr = cfg.passive_scalar ? 0 : 1;
    sp.disp = (cfg.no_dispersion || cfg.passive_scalar) ? 0 : 1;
    sp.use_dq = (cfg.inviscid == 0 && cfg.nuz != 0.0) ? 1 : 0;
    sp.euler = 0;
    sp.ybj = cfg.ybj_plus || cfg.passive_scalar ? 1 : 0;
    sp.mpar = mpar;
    need_qw = (!cfg.fixed_flow && !cfg.no_feedback);
    int r0 = set_smem_attrs();
    if (r0) return r0;
    if (cfg.solve_columns != 0 && cfg.solve_columns != 16 && cfg.solve_columns != 32 && cfg.solve_columns != 64) {
      err = "solve_columns must be 0, 16, 32 or 64";
      return QG_ERR_ARG;
    }
    solve_tc = cfg.solve_columns ? cfg.solve_columns : 32;
    // forward values of the column solves; without this scratch the solves
    // checkpoint and recompute instead (k_solve)
    if (kSolveStore && cudaMalloc(&vbuf, (size_t)6 * g.n3 * g.plane * sizeof(double)) != cudaSuccess) {
      vbuf = nullptr;
      (void)cudaGetLastError();
    }
    // per-column copies of the solve factors (coalesced reads);
    // without them the solves read the per-kh^2 tables
    if (kSolvePerColumn && vbuf) {
      if (cudaMalloc(&pcfac, (size_t)6 * g.nseg * nret * sizeof(double)) != cudaSuccess) {
        pcfac = nullptr;
        (void)cudaGetLastError();
      } else {
        k_expand_fac<<<grid_for((long long)g.nseg * nret), 256, 0, st>>>(g, tab_idx, fac_psi, fac_A, pcfac,
                                                                         cols_ret, nret);
        QG_LAUNCHED();
      }
    }
    // kept y-inverse planes of B (YBJ+ runs whose update transforms B^{n+1}
    // for q^w); without them k_col_inv transforms B again in every step
    if (kReuseB && need_qw && cfg.ybj_plus &&
        cudaMalloc(&Qp, (size_t)g.n3 * kNQ * g.n * g.KXP * sizeof(C)) != cudaSuccess) {
      Qp = nullptr;
      (void)cudaGetLastError();
    }
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  void* stream() override { return (void*)st; }

  int enqueue(int euler) override { return enqueue_step(euler ? 1 : 0); }

  int batch_levels() const override { return Zb; }
  int levels_per_member() const override { return g.nseg; }
  int member_count() const override { return members; }

  int set_batch_levels(int zb) override {
    QG_CK(cudaStreamSynchronize(st));
    for (auto& x : gexec) if (x) { cudaGraphExecDestroy(x); x = nullptr; }
    const size_t per_level = (size_t)kNScr * g.n * g.KXP * sizeof(C);
    zb = std::max(1, std::min(zb, g.n3));
    const int nb = (g.n3 + zb - 1) / zb;
    const int nz = (g.n3 + nb - 1) / nb;
    const int nl = std::max(1, std::min(want_lanes, nb));
    if (nl * nz > s_levels) {
      cudaFree(S);
      S = nullptr;
      QG_CK(dev_alloc(&S, (size_t)nl * nz * per_level));
      s_levels = nl * nz;
    }
    Zb = nz;
    lanes = nl;
    return QG_OK;
  }

  // phase-A batches in flight at once (each on its own stream and scratch)
  int batch_lanes() const override { return lanes; }
  int set_batch_lanes(int nl) override {
    if (nl < 1 || nl > kMaxLanes) { err = "batch lanes must be in [1, 8]"; return QG_ERR_ARG; }
    want_lanes = nl;
    return set_batch_levels(Zb);
  }

  int solve_columns() const override { return solve_tc; }
  int set_solve_columns(int tc) override {
    if (tc == 0) tc = 32;
    if (tc != 16 && tc != 32 && tc != 64) { err = "solve_columns must be 16, 32 or 64"; return QG_ERR_ARG; }
    QG_CK(cudaStreamSynchronize(st));
    for (auto& x : gexec) if (x) { cudaGraphExecDestroy(x); x = nullptr; }
    solve_tc = tc;
    return QG_OK;
  }

  int synchronize() override {
    QG_CK(cudaStreamSynchronize(st));
    return check_waits();
  }

  int selftest_wait() override {
    k_wait_expire<<<1, 32, 0, st>>>(wflag);
    QG_LAUNCHED();
    return synchronize();
  }

  // QG_ERR_TIMEOUT when a kernel's bounded wait expired since the last check,
  // QG_ERR_NONFINITE when a step produced a NaN or infinite q* (call after
  // the stream has drained)
  int check_waits() override {
    if (wflag_h && *(volatile int*)wflag_h) {
      *(volatile int*)wflag_h = 0;
      err = "a bounded device-side wait expired (bulk copy of the row kernels)";
      return QG_ERR_TIMEOUT;
    }
    if (wflag_h && *(volatile int*)(wflag_h + 1)) {
      *(volatile int*)(wflag_h + 1) = 0;
      err = "non-finite q* after a step: the state has blown up (time step too large?)";
      return QG_ERR_NONFINITE;
    }
    return QG_OK;
  }

  // ---- state --------------------------------------------------------------
  int set_state(int field, const double* kvar, int level0, int nlev) override {
    const int f = map_field(field);
    if (f < 0 || field == QG_CR || field == QG_CI || field == QG_QSTAR) { err = "field is read-only or unknown"; return QG_ERR_ARG; }
    if (!kvar || level0 < 0 || nlev <= 0 || level0 + nlev > g.n3) { err = "bad level range or null pointer"; return QG_ERR_ARG; }
    const size_t bytes = (size_t)nlev * g.n * (g.n / 2 + 1) * sizeof(double2);
    // pinned host or device arrays are read in place (only the retained
    // modes cross the link); others go through a device staging copy
    const double2* src = static_cast<const double2*>(device_view(kvar));
    if (!src) {
      int rc = ensure(&stage, &stage_bytes, bytes);
      if (rc) return rc;
      QG_CK(cudaMemcpyAsync(stage, kvar, bytes, cudaMemcpyDefault, st));
      src = (const double2*)stage;
    }
    *(volatile int*)(wflag_h + 2) = 0;
    if (f == F_BR || f == F_BI) q_valid = false;
    if (f == F_PSI && sizeof(T) == 4) {
      // mixed path: keep psi in FP64 until qg_init_state has built q from it
      // (init_q's vertical second difference would amplify FP32 rounding);
      // the FP32 field is rounded from that copy on the device, so the input
      // crosses the host link once
      if (!psi64) QG_CK(cudaMalloc(&psi64, (size_t)g.n3 * g.plane * sizeof(double2)));
      psi64_live.resize(g.n3, 0);
      std::fill_n(psi64_live.begin() + level0, nlev, 1);
      k_dense_to_compact<double><<<conv_grid(g.KY, nlev), 256, 0, st>>>(g, level0, src, psi64,
                                                                                        iflag);
      QG_LAUNCHED();
      k_round_compact<T><<<grid_for((long long)nlev * g.plane), 256, 0, st>>>(
          (long long)nlev * g.plane, reinterpret_cast<const cplx<double>*>(psi64) + (size_t)level0 * g.plane,
          F[f] + (size_t)level0 * g.plane);
      QG_LAUNCHED();
    } else {
      k_dense_to_compact<T><<<conv_grid(g.KY, nlev), 256, 0, st>>>(g, level0, src, F[f], iflag);
      QG_LAUNCHED();
    }
    QG_CK(cudaStreamSynchronize(st));
    if (*(volatile int*)(wflag_h + 2)) {
      *(volatile int*)(wflag_h + 2) = 0;
      err = "non-finite value (NaN or Inf) on a retained mode of the input array";
      return QG_ERR_NONFINITE;
    }
    return QG_OK;
  }

  int get_state(int field, double* kvar, int level0, int nlev) override {
    int f = map_field(field);
    if (f < 0) { err = "unknown field"; return QG_ERR_ARG; }
    if (!kvar || level0 < 0 || nlev <= 0 || level0 + nlev > g.n3) { err = "bad level range or null pointer"; return QG_ERR_ARG; }
    if (field == QG_QSTAR && !need_qw) f = F_Q;
    const int mode = (field == QG_CR || field == QG_CI) ? 1 : 0;
    const size_t bytes = (size_t)nlev * g.n * (g.n / 2 + 1) * sizeof(double2);
    double2* dst = static_cast<double2*>(const_cast<void*>(device_view(kvar)));
    if (!dst) {
      int rc = ensure(&stage, &stage_bytes, bytes);
      if (rc) return rc;
    }
    if (int rc = to_dense(F[f], dst ? dst : (double2*)stage, mode, level0, nlev)) return rc;
    if (!dst) QG_CK(cudaMemcpyAsync(kvar, stage, bytes, cudaMemcpyDefault, st));
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  // Device address through which kernels may access p: device memory as is,
  // page-locked host memory through its mapping; nullptr for anything else
  // (pageable or managed memory, an address that is not 16-byte aligned),
  // which is staged through a copy instead.
  static const void* device_view(const void* p) {
    if (reinterpret_cast<uintptr_t>(p) & 15) return nullptr;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
    if (at.type == cudaMemoryTypeDevice) return p;
    if (at.type == cudaMemoryTypeHost && at.devicePointer) return at.devicePointer;
    return nullptr;
  }

  int init_state(int apply_sumB, int q_from_psi) override {
    int rc = init_state_range(0, g.n3, apply_sumB, q_from_psi);
    if (rc) return rc;
    release_init_buffers();
    return QG_OK;
  }

  // The initialisation sequence on levels [z0, z0 + nz) (whole segments):
  // one run, or one member of a stack (whose FP64 psi copy stays until
  // release_init_buffers, so that every member's q is built from it)
  int init_state_range(int z0, int nz, int apply_sumB, int q_from_psi) override {
    if (z0 < 0 || nz <= 0 || z0 + nz > g.n3 || z0 % g.nseg || nz % g.nseg) {
      err = "initialisation range must cover whole members";
      return QG_ERR_ARG;
    }
    q_valid = false;
    if (apply_sumB) {
      k_sumB<T><<<dim3((unsigned)((g.plane + 127) / 128), 2), 128, 0, st>>>(g, F[F_BR], F[F_BI], z0, z0 + nz);
      QG_LAUNCHED();
    }
    const size_t lb = (size_t)g.plane * sizeof(C), off = (size_t)z0 * g.plane;
    if (cfg.fixed_flow) {
      // fixed flow: q = 0 for all times (main_waqg.f90:141-146)
      QG_CK(cudaMemsetAsync(F[F_Q] + off, 0, (size_t)nz * lb, st));
    } else if (q_from_psi) {
      // from the FP64 copy where the host set psi since the last
      // initialisation or step; levels it did not set join it from the
      // resident psi
      const bool copy = !psi64_live.empty() && std::count(psi64_live.begin() + z0, psi64_live.begin() + z0 + nz, 1) > 0;
      for (int a = z0, b; copy && a < z0 + nz; a = b) {
        for (b = a + 1; b < z0 + nz && psi64_live[b] == psi64_live[a]; ++b) {}
        if (psi64_live[a]) continue;
        const long long m = (long long)(b - a) * g.plane;
        k_widen_compact<T><<<grid_for(m), 256, 0, st>>>(m, F[F_PSI] + (size_t)a * g.plane, psi64 + (size_t)a * g.plane);
        QG_LAUNCHED();
      }
      const Divisor dz2(cfg.dz * cfg.dz);
      const dim3 gi((unsigned)((g.plane + 127) / 128), (g.nseg + kInitLev - 1) / kInitLev * (nz / g.nseg));
      if (copy) {
        k_init_q<T, double><<<gi, 128, 0, st>>>(g, cfg.dz, dz2, cu, cl, psi64, F[F_Q], z0);
      } else {
        k_init_q<T, T><<<gi, 128, 0, st>>>(g, cfg.dz, dz2, cu, cl, F[F_PSI], F[F_Q], z0);
      }
      QG_LAUNCHED();
    }
    QG_CK(cudaMemcpyAsync(F[F_QO] + off, F[F_Q] + off, (size_t)nz * lb, cudaMemcpyDeviceToDevice, st));
    QG_CK(cudaMemcpyAsync(F[F_BRO] + off, F[F_BR] + off, (size_t)nz * lb, cudaMemcpyDeviceToDevice, st));
    QG_CK(cudaMemcpyAsync(F[F_BIO] + off, F[F_BI] + off, (size_t)nz * lb, cudaMemcpyDeviceToDevice, st));
    if (!cfg.passive_scalar && cfg.ybj_plus) {   // regular YBJ keeps the A the host set
      int rc = solve_generic(nullptr, F[F_BR], F[F_BI], nullptr, F[F_AR], F[F_AI], 0, 1, st, z0 / g.nseg,
                             nz / g.nseg, true);
      if (rc) return rc;
    }
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  // the FP64 copy of psi that qg_set_state keeps for init_q (mixed path) is
  // used up; its memory stays for the handle's next run, or for what needs it
  // (dev_alloc)
  void release_init_buffers() override { std::fill(psi64_live.begin(), psi64_live.end(), 0); }

  // ---- the step -------------------------------------------------------------
  int step(int euler) override {
    int rc = run_step(euler ? 1 : 0);
    if (rc) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return check_waits();
  }

  int steps_async(int nsteps, int euler) override {
    for (int i = 0; i < nsteps; ++i) {
      int rc = run_step((euler && i == 0) ? 1 : 0);
      if (rc) return rc;
    }
    return QG_OK;
  }

  int diagnostics(qg_energy* out) override { return diagnostics_range(0, g.n3, out); }

  // k_diag_cols over nsegs whole segments: the levels of each segment in
  // chunks of zc, as many chunks as keep the grid within one wave of
  // resident CTAs (a second, partial wave would run at a fraction of the
  // GPU); returns the grid
  dim3 diag_grid(int nsegs, int* zc) const {
    const int cb = (nret + kDiagThreads - 1) / kDiagThreads;
    const long long per = (long long)cb * nsegs;
    const int nch0 = (int)std::max<long long>(1, std::min<long long>(g.nseg, (long long)diag_slots / per));
    *zc = (g.nseg + nch0 - 1) / nch0;
    return dim3(cb, (g.nseg + *zc - 1) / *zc, nsegs);
  }
  size_t diag_parts(int nsegs) const {
    int zc;
    const dim3 gr = diag_grid(nsegs, &zc);
    return (size_t)gr.x * gr.y * gr.z;
  }
  // the seven integrals of segments [seg0, seg0 + nsegs) into out (device)
  int launch_diag(int seg0, int nsegs, double* part, double* out, cudaStream_t s) {
    int zc;
    const dim3 grid = diag_grid(nsegs, &zc);
    const double c2 = (1.0 / 8.0) * (1.0 / (cfg.Bu * cfg.Bu)), c6 = 2.0 * (1.0 / (cfg.dz * cfg.dz));
    k_diag_cols<T><<<grid, kDiagThreads, 0, s>>>(g, seg0, zc, dwz, fwz, c2, c6, F[F_BR], F[F_BI], F[F_AR],
                                                 F[F_AI], F[F_PSI], cols_ret, nret, part);
    QG_LAUNCHED();
    k_diag_sum<<<1, 32 * kNDiag, 0, s>>>((long long)grid.x * grid.y * grid.z, nsegs * g.nseg, part, out);
    QG_LAUNCHED();
    return QG_OK;
  }

  // The integrals of the state as it stands after the work queued so far, on
  // a stream of their own: the next step's first kernels (which only read
  // the state) run beside them, and its update kernels wait for them in the
  // graph (external event wait before each k_col_update).  diagnostics_wait
  // returns the values.
  int diagnostics_async() override {
    if (!std_) {
      int prio_low = 0, prio_high = 0;
      QG_CK(cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high));
      QG_CK(cudaStreamCreateWithPriority(&std_, cudaStreamNonBlocking, prio_low));
      QG_CK(cudaEventCreateWithFlags(&ev_state, cudaEventDisableTiming));
      QG_CK(dev_alloc(&diag_part_a, diag_part_n * kNDiag * sizeof(double)));
      QG_CK(dev_alloc(&diag_out_a, kNDiag * sizeof(double)));
      QG_CK(cudaMallocHost(&diag_host_a, kNDiag * sizeof(double)));
    }
    if (diag_pending) { err = "the previous asynchronous diagnostics were not collected"; return QG_ERR_ARG; }
    QG_CK(cudaEventRecord(ev_state, st));
    QG_CK(cudaStreamWaitEvent(std_, ev_state, 0));
    if (int rc = launch_diag(0, g.n3 / g.nseg, diag_part_a, diag_out_a, std_)) return rc;
    QG_CK(cudaMemcpyAsync(diag_host_a, diag_out_a, kNDiag * sizeof(double), cudaMemcpyDeviceToHost, std_));
    QG_CK(cudaEventRecord(ev_diag, std_));
    diag_pending = true;
    return QG_OK;
  }

  int diagnostics_wait(qg_energy* out) override {
    if (!diag_pending) { err = "no asynchronous diagnostics pending"; return QG_ERR_ARG; }
    QG_CK(cudaEventSynchronize(ev_diag));
    diag_pending = false;
    out->wke = diag_host_a[0]; out->wpe = diag_host_a[1]; out->wce = diag_host_a[2];
    out->ke = diag_host_a[3]; out->pe = diag_host_a[4]; out->zeta2 = diag_host_a[5]; out->omegah2 = diag_host_a[6];
    return QG_OK;
  }

  // the integrals over levels [z0, z0 + nz): one run, or one member of a stack
  int diagnostics_range(int z0, int nz, qg_energy* out) override {
    if (z0 % g.nseg || nz % g.nseg || nz <= 0) { err = "diagnostics range is not a set of whole segments"; return QG_ERR_ARG; }
    if (int rc = launch_diag(z0 / g.nseg, nz / g.nseg, diag_part, diag_out, st)) return rc;
    QG_CK(cudaMemcpyAsync(diag_host, diag_out, kNDiag * sizeof(double), cudaMemcpyDeviceToHost, st));
    QG_CK(cudaStreamSynchronize(st));
    out->wke = diag_host[0]; out->wpe = diag_host[1]; out->wce = diag_host[2];
    out->ke = diag_host[3]; out->pe = diag_host[4]; out->zeta2 = diag_host[5]; out->omegah2 = diag_host[6];
    return QG_OK;
  }

  // ---- output path ----------------------------------------------------------
  int dump_real(int which, float* out0, float* out1, int level0, int nlev, double s1, double s2) override {
    if (level0 < 0 || nlev <= 0 || level0 + nlev > g.n3) { err = "bad level range"; return QG_ERR_ARG; }
    int rc = prep_dense(nlev, kDensePlanes);
    if (rc) return rc;
    const size_t bytes = (size_t)nlev * g.n * g.n * sizeof(float);
    const int nf = which == 0 ? 1 : 2;
    CompactIn<T> in{g, level0, {which == 0 ? F[F_PSI] : F[F_BR], F[F_BI]},
                    {which == 2 ? F[F_AR] : nullptr, which == 2 ? F[F_AI] : nullptr}, Divisor(cfg.Bu)};
    F32Out o{{nullptr, nullptr}, s1, s2};
    float* out[2] = {out0, out1};
    for (int c = 0; c < nf; ++c) {
      void* v;
      if ((rc = out_view(out[c], bytes, c, &v))) return rc;
      o.o[c] = static_cast<float*>(v);
    }
    if ((rc = d_inv(in, nlev, nf, g.K))) return rc;
    QG_SWITCH_N(g.n, {
      using DN = Dense<T, NN>;
      k_drow_c2r_f32<T, NN><<<dim3(g.n / 2 / DN::RT, nlev, nf), DN::RNT, DN::sm_row(), st>>>(iktxP(), nf, g.K, W, o, tw);
      QG_LAUNCHED();
    });
    for (int c = 0; c < nf; ++c)
      if ((rc = out_copy(out[c], o.o[c], bytes))) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  // ---- omega equation (the vertical-velocity diagnostic) ---------------------
  // right-hand side from psi (the reference's layout, or the resident field
  // when dense is null) into rhs; retained: the retained modes and zeros, else
  // every mode
  int omega_rhs_dev(const double2* dense, double2* rhs, bool retained) {
    OmegaIn<T> in{g, dense, F[F_PSI], Divisor(cfg.dz)};
    int rc = d_inv(in, g.n3, 4, g.n / 2);
    if (rc) return rc;
    const int KM = retained ? g.K : g.n / 2;
    if ((rc = d_prod(g.n3, 4, KM, 1, 1, 0, 0))) return rc;
    return d_fwd<1>(DenseOut{{rhs, nullptr, nullptr}, retained ? 2 : 0, g.kmax2, 0.0, 0.0}, g.n3, 4, 1);
  }
  // w from the dense right-hand side into w (device arrays)
  int omega_solve_dev(const double2* rhs, double2* w) {
    const int m = g.n3 - 1;
    QG_CK(cudaMemsetAsync(w, 0, dense_bytes(g.n3), st));
    if (m < 1 || om_nd == 0) return QG_OK;
    if (!om_fac) {
      double4* f = nullptr;
      QG_CK(dev_alloc(&f, (size_t)om_nd * m * sizeof(double4)));
      k_omega_fac<<<(om_nd + 127) / 128, 128, 0, st>>>(om_nd, g.n3, cfg.dz, om_kh2, om_t1, om_du, om_dl, om_a, f);
      om_fac = f;
      QG_LAUNCHED();
    }
    if (!om_scr) QG_CK(dev_alloc(&om_scr, (size_t)2 * m * nret * sizeof(double)));
    k_omega_solve<<<dim3((unsigned)((nret + 63) / 64), 2), 64, 0, st>>>(g, cfg.dz, om_du, om_fac, tab_idx, cols_ret, nret,
                                                                       rhs, om_scr, w);
    QG_LAUNCHED();
    return QG_OK;
  }
  int omega_eqn_rhs(const double* psik, double* rhs) override {
    const size_t db = dense_bytes(g.n3);
    int rc = prep_dense(g.n3, kDensePlanes);
    if (rc) return rc;
    const void* p;
    void* o;
    if ((rc = in_view(psik, db, 0, &p)) || (rc = out_view(rhs, db, 1, &o))) return rc;
    if ((rc = omega_rhs_dev((const double2*)p, (double2*)o, false)) || (rc = out_copy(rhs, o, db))) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }
  int omega_equation(const double* rhs, double* wk) override {
    const size_t db = dense_bytes(g.n3);
    int rc;
    const void* p;
    void* o;
    // (w is written while the right-hand side is read: never in place)
    if ((rc = in_view(rhs, db, 0, &p)) || (rc = out_view(wk, db, 1, &o, p))) return rc;
    if ((rc = omega_solve_dev((const double2*)p, (double2*)o)) || (rc = out_copy(wk, o, db))) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }
  int omega_from_state(double* wk) override {
    const size_t db = dense_bytes(g.n3);
    int rc = prep_dense(g.n3, kDensePlanes);
    if (rc) return rc;
    void* o;
    if ((rc = out_view(wk, db, 1, &o)) || (rc = ensure(&stg[0], &stg_bytes[0], db))) return rc;
    if ((rc = omega_rhs_dev(nullptr, (double2*)stg[0], true)) || (rc = omega_solve_dev((double2*)stg[0], (double2*)o)) ||
        (rc = out_copy(wk, o, db)))
      return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  // ---- routine-level drop-ins ---------------------------------------------
  int fft_r2c(const double* rvar, double* kvar, int nz) override {
    int rc = prep_dense(nz, 1);
    if (rc) return rc;
    const size_t rb = (size_t)nz * g.n * (g.n + 2) * sizeof(double), db = dense_bytes(nz);
    const void* r;
    void* k;
    if ((rc = in_view(rvar, rb, 0, &r)) || (rc = out_view(kvar, db, 1, &k))) return rc;
    if ((rc = d_r2c((const double*)r, g.n + 2, (double2*)k, nz)) || (rc = out_copy(kvar, k, db))) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  int fft_c2r(const double* kvar, double* rvar, int nz) override {
    int rc = prep_dense(nz, 1);
    if (rc) return rc;
    const size_t rb = (size_t)nz * g.n * (g.n + 2) * sizeof(double), db = dense_bytes(nz);
    const void* k;
    void* r;
    if ((rc = in_view(kvar, db, 0, &k)) || (rc = out_view(rvar, rb, 1, &r))) return rc;
    if ((rc = d_c2r((const double2*)k, (double*)r, g.n + 2, nz)) || (rc = out_copy(rvar, r, rb))) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  // the three nonlinear terms: inputs under their operators to (kx, y)
  // planes, rows to products, columns to outputs
  int nonlinear(std::initializer_list<const double*> ins, std::initializer_list<std::pair<int, int>> fields,
                std::initializer_list<double*> outs, int mode, int cross, int nA, int nX, int nz) {
    int rc = prep_dense(nz, kDensePlanes);
    if (rc) return rc;
    const size_t db = dense_bytes(nz);
    const void* v[kDenseFields];
    int k = 0;
    for (const double* p : ins) { if ((rc = in_view(p, db, k, &v[k]))) return rc; ++k; }
    DenseIn in{};
    in.kmax2 = g.kmax2;
    int nf = 0;
    for (const auto& f : fields) { in.p[nf] = (const double2*)v[f.first]; in.op[nf] = f.second; ++nf; }
    DenseOut o{{nullptr, nullptr, nullptr}, mode, g.kmax2, cfg.Ro, cfg.W2F};
    int no = 0;
    // (staged inputs are read before staged outputs are written)
    for (double* p : outs) { void* q; if ((rc = out_view(p, db, no, &q))) return rc; o.p[no++] = (double2*)q; }
    const int np = kDensePlanes;
    if ((rc = d_inv(in, nz, nf, g.n / 2, np)) || (rc = d_prod(nz, np, g.K, cross, 0, nA, nX))) return rc;
    if ((rc = mode == 2 ? d_fwd<1>(o, nz, np, no) : d_fwd<2>(o, nz, np, no))) return rc;
    no = 0;
    for (double* p : outs) { if ((rc = out_copy(p, o.p[no], db))) return rc; ++no; }
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  int convol_waqg(const double* uk, const double* vk, const double* qk, const double* BRk, const double* BIk,
                  double* nqk, double* nBRk, double* nBIk, int nz) override {
    return nonlinear({uk, vk, qk, BRk, BIk}, {{0, OP_ID}, {1, OP_ID}, {2, OP_ID}, {3, OP_ID}, {4, OP_ID}},
                     {nqk, nBRk, nBIk}, 1, 0, 2, 3, nz);
  }

  int refraction_waqg(const double* BRk, const double* BIk, const double* psik, double* rBRk, double* rBIk,
                      int nz) override {
    return nonlinear({BRk, BIk, psik}, {{2, OP_LAP}, {0, OP_ID}, {1, OP_ID}}, {rBRk, rBIk}, 2, 0, 1, 2, nz);
  }

  // BRy BIx - BRx BIy and BR^2 + BI^2 (derivatives.f90:973, 996)
  int compute_qw(const double* BRk, const double* BIk, double* qwk, int nz) override {
    return nonlinear({BRk, BIk}, {{0, OP_IKY}, {1, OP_IKX}, {0, OP_IKX}, {1, OP_IKY}, {0, OP_ID}, {1, OP_ID}}, {qwk}, 3, 2,
                     0, 0, nz);
  }

  int psi_solver(const double* qstar, double* psik) override {
    int rc = ensure_tmp();
    if (rc) return rc;
    if ((rc = upload_compact(qstar, tmpF[0]))) return rc;
    if ((rc = solve_generic(tmpF[0], nullptr, nullptr, tmpF[1], nullptr, nullptr, 1, 0, nullptr, 0, -1, true))) return rc;
    if ((rc = download_compact(tmpF[1], psik, 0))) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

  int A_solver(const double* bk, double* ak, double* ck) override {
    int rc = ensure_tmp();
    if (rc) return rc;
    if ((rc = upload_compact(bk, tmpF[0]))) return rc;
    if ((rc = solve_generic(nullptr, tmpF[0], nullptr, nullptr, tmpF[1], nullptr, 0, 2, nullptr, 0, -1, true))) return rc;
    if ((rc = download_compact(tmpF[1], ak, 0))) return rc;
    if (ck && (rc = download_compact(tmpF[1], ck, 1))) return rc;
    QG_CK(cudaStreamSynchronize(st));
    return QG_OK;
  }

 protected:
  qg_config cfg{};
  Geom g{};
  StepParams sp{};
  cudaStream_t st = nullptr;
  cudaStream_t st2 = nullptr;                          // the overlapped A solves
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;   // B^{n+1} ready / A solves done
  // asynchronous diagnostics: their stream, state-ready and done events,
  // their own buffers
  cudaStream_t std_ = nullptr;
  cudaEvent_t ev_state = nullptr, ev_diag = nullptr;
  double *diag_part_a = nullptr, *diag_out_a = nullptr, *diag_host_a = nullptr;
  bool diag_pending = false;
  C* F[F_NINT] = {};
  T *e1 = nullptr, *e2 = nullptr, *e1w = nullptr, *e2w = nullptr;
  C* tw = nullptr;
  int* tab_idx = nullptr;
  int* cols_all = nullptr;   // 0 .. plane-1
  int* cols_ret = nullptr;   // the retained columns (L = 1), ascending
  int nret = 0;
  double4 *fac_psi = nullptr, *fac_A = nullptr;
  double* pcfac = nullptr;   // per-column solve factors of the mixed path (k_expand_fac), or null
  double* vbuf = nullptr;    // forward values of the column solves (k_solve_st)
  int solve_tc = 32;         // columns per CTA of k_solve_st
  double *du = nullptr, *cu = nullptr, *cl = nullptr, *r2 = nullptr;
  double *diag_part = nullptr, *diag_out = nullptr, *diag_host = nullptr;
  double* dwz = nullptr;     // diagnostics' per-level weights (w1, w4), FP64
  float2* fwz = nullptr;     // the same as FP32 pairs
  int diag_slots = 1;        // resident k_diag_cols CTAs on the GPU
  size_t diag_part_n = 0;    // partials the diagnostics buffers hold
  // set by a kernel whose bounded wait expired (mapped page-locked word)
  // mapped page-locked words raised on the device: [0] a bounded wait
  // expired, [1] a step produced a non-finite q*, [2] qg_set_state's input
  // held a non-finite retained mode (wflag, nflag, iflag: device views)
  int* wflag_h = nullptr;
  int* wflag = nullptr;
  int* nflag = nullptr;
  int* iflag = nullptr;
  int nsm = 1, occ_rm = 1, occ_rq = 1;   // SMs; resident CTAs per SM of the persistent row kernels
  double *om_t1 = nullptr, *om_du = nullptr, *om_dl = nullptr, *om_a = nullptr, *om_scr = nullptr;
  double4* om_fac = nullptr;   // omega operator's factors per distinct kh2 (first use)
  int* om_kh2 = nullptr;       // the distinct kh2
  int om_nd = 0;
  C* sig[2] = {};     // regular YBJ: per-level sigma terms
  C* Qp = nullptr;             // kept y-inverse planes of B, [n3][2][n][KXP], or null
  bool q_valid = false;        // Qp holds the transforms of the current B
  int members = 1;             // ensemble members stacked in z (segments of g.nseg levels)
  double* mpar = nullptr;      // their step parameters (StepParams::mpar)
  C* S = nullptr;              // [lanes][Zb][kNScr][n][KXP] scratch planes
  int s_levels = 0;            // levels of scratch allocated
  double2* psi64 = nullptr;    // FP64 copy of psi between qg_set_state and qg_init_state
  std::vector<unsigned char> psi64_live;   // levels whose psi was set since the last initialisation or step
  int Zb = 1;
  // phase-A batches run on `lanes` streams (lane 0: st), batch b on lane
  // b % lanes with its own scratch slot; they join st before the solves
  static constexpr int kMaxLanes = 8;
  int lanes = 1, want_lanes = kBatchLanes;
  cudaStream_t lst[kMaxLanes] = {};
  cudaEvent_t lev[kMaxLanes] = {};
  cudaEvent_t ev_start = nullptr;
  bool need_qw = true;
  void* stage = nullptr; size_t stage_bytes = 0;
  // (kx, y) planes of the routine-level calls (kDensePlanes per level where
  // products are formed), and staging copies of the callers' arrays that the
  // kernels cannot use in place
  static constexpr int kDensePlanes = 6;
  C* W = nullptr;
  size_t w_planes = 0;
  void* stg[kDenseFields] = {};
  size_t stg_bytes[kDenseFields] = {};
  C* tmpF[2] = {};
  cudaGraphExec_t gexec[2] = {nullptr, nullptr};

  void release() {
    if (st) cudaStreamSynchronize(st);
    for (auto& x : gexec) if (x) { cudaGraphExecDestroy(x); x = nullptr; }
    for (auto& p : F) if (p) { cudaFree(p); p = nullptr; }
    void* ps[] = {e1, e2, e1w, e2w, tw, tab_idx, cols_all, cols_ret, fac_psi, fac_A, pcfac, vbuf, du, cu, cl, r2, diag_part, diag_out, dwz, fwz, S, stage,
                  W, psi64, om_t1, om_du, om_dl, om_a, om_scr, om_fac, om_kh2, sig[0], sig[1], mpar, Qp};
    for (void* p : ps) if (p) cudaFree(p);
    for (auto& p : stg) if (p) cudaFree(p);
    for (auto& p : tmpF) if (p) cudaFree(p);
    if (diag_host) cudaFreeHost(diag_host);
    if (wflag_h) cudaFreeHost(wflag_h);
    wflag_h = nullptr;
    wflag = nullptr;
    nflag = nullptr;
    iflag = nullptr;
    for (int i = 1; i < kMaxLanes; ++i) {
      if (lst[i]) { cudaStreamSynchronize(lst[i]); cudaStreamDestroy(lst[i]); lst[i] = nullptr; }
      if (lev[i]) { cudaEventDestroy(lev[i]); lev[i] = nullptr; }
    }
    if (ev_start) { cudaEventDestroy(ev_start); ev_start = nullptr; }
    if (std_) { cudaStreamSynchronize(std_); cudaStreamDestroy(std_); std_ = nullptr; }
    if (ev_state) { cudaEventDestroy(ev_state); ev_state = nullptr; }
    if (ev_diag) { cudaEventDestroy(ev_diag); ev_diag = nullptr; }
    if (diag_part_a) { cudaFree(diag_part_a); diag_part_a = nullptr; }
    if (diag_out_a) { cudaFree(diag_out_a); diag_out_a = nullptr; }
    if (diag_host_a) { cudaFreeHost(diag_host_a); diag_host_a = nullptr; }
    if (st2) cudaStreamSynchronize(st2);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
    ev_fork = ev_join = nullptr;
    if (st2) cudaStreamDestroy(st2);
    st2 = nullptr;
    if (st) cudaStreamDestroy(st);
    st = nullptr;
  }

  static unsigned grid_for(long long n) {
    long long b = (n + 255) / 256;
    return (unsigned)std::max<long long>(1, std::min<long long>(b, 152LL * 16));
  }

  static dim3 conv_grid(int rows, int nlev) { return dim3((rows + kConvRows - 1) / kConvRows, nlev); }
  // levels [level0, level0 + nlev) of a resident field (mode 1: their vertical
  // differences) in the reference's layout
  int to_dense(const C* f, double2* dense, int mode, int level0, int nlev) {
    const int iktx = g.n / 2 + 1;
    k_compact_to_dense<T><<<dim3((g.n * iktx + kDenseRun - 1) / kDenseRun, nlev), 256, 0, st>>>(
        g, level0, f, dense, mode, Divisor(cfg.dz), (unsigned)((0x100000000ull + iktx - 1) / iktx));
    QG_LAUNCHED();
    return QG_OK;
  }

  int map_field(int field) const {
    switch (field) {
      case QG_Q: return F_Q; case QG_QOLD: return F_QO; case QG_BR: return F_BR; case QG_BI: return F_BI;
      case QG_BROLD: return F_BRO; case QG_BIOLD: return F_BIO; case QG_PSI: return F_PSI;
      case QG_AR: case QG_CR: return F_AR;
      case QG_AI: case QG_CI: return F_AI;
      case QG_QSTAR: return F_QSTAR;
      default: return -1;
    }
  }

  // cudaMalloc of what a handle allocates after qg_create: gives the FP64 copy
  // of psi back, if it holds nothing, before it fails
  template <typename P> cudaError_t dev_alloc(P** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation || !psi64 || std::count(psi64_live.begin(), psi64_live.end(), 1)) return e;
    (void)cudaGetLastError();
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess || (e = cudaFree(psi64)) != cudaSuccess) return e;
    psi64 = nullptr;
    return cudaMalloc(p, bytes);
  }

  int ensure(void** p, size_t* have, size_t need) {
    if (*have >= need) return QG_OK;
    if (*p) { QG_CK(cudaStreamSynchronize(st)); cudaFree(*p); *p = nullptr; *have = 0; }
    QG_CK(dev_alloc(p, need));
    *have = need;
    return QG_OK;
  }

  // shared memory of the step kernels (twiddles + padded transforms)
  // column kernels on the interleaved tile (colfft.cuh): NF fields in flight
  template <int NN, int CP = 16> static constexpr size_t sm_ci(int nf) {
    return (size_t)(NN + nf * ColLay<NN, Tiles<T, NN>::CT, CP>::FS) * sizeof(C);
  }
  template <int NN> static constexpr size_t sm_rr3() { return (size_t)(NN + 3 * Tiles<T, NN>::QRT * Tiles<T, NN>::LD) * sizeof(C); }
  template <int NN> static constexpr size_t sm_rm4() { return (size_t)(NN + 4 * Tiles<T, NN>::RTM * Tiles<T, NN>::LD) * sizeof(C); }
  // the persistent row kernels add a staging copy of an item's scratch rows
  // (nf planes x rows x kxp) and its mbarrier; the attribute is set for the
  // widest rows any mask of this n can have (kxp for K = n/2)
  template <int NN> static constexpr int kxp_max() { return ((NN / 2 + 1 + 7) / 8) * 8; }
  template <int NN> static constexpr size_t sm_rm(int kxp) {
    return sm_rm4<NN>() + (Tiles<T, NN>::RPRE ? (size_t)6 * Tiles<T, NN>::RTM * kxp * sizeof(C) + 16 : 0);
  }
  template <int NN> static constexpr size_t sm_rq(int kxp) {
    return sm_rr3<NN>() + (Tiles<T, NN>::QPRE ? (size_t)4 * Tiles<T, NN>::QRT * kxp * sizeof(C) + 16 : 0);
  }

  int set_smem_attrs() {
    const int mx = cudaFuncAttributeMaxDynamicSharedMemorySize;
    QG_SWITCH_N(g.n, {
      if constexpr (kFx) {
        const int sc = (int)FxCol<NN>::smem(), sr = (int)FxQw<NN>::smem();
        QG_CK(cudaFuncSetAttribute(k_fx_col_inv<NN>, (cudaFuncAttribute)mx, sc));
        QG_CK(cudaFuncSetAttribute(k_fx_col_update<NN>, (cudaFuncAttribute)mx, sc));
        QG_CK(cudaFuncSetAttribute(k_fx_col_qw<NN>, (cudaFuncAttribute)mx, sc));
        QG_CK(cudaFuncSetAttribute(k_fx_row_main<NN>, (cudaFuncAttribute)mx, (int)FxMain<NN>::smem()));
        QG_CK(cudaFuncSetAttribute(k_fx_row_qw<NN>, (cudaFuncAttribute)mx, sr));
        QG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_rm, k_fx_row_main<NN>, FxMain<NN>::F::NT,
                                                            FxMain<NN>::smem()));
        QG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_rq, k_fx_row_qw<NN>, FxRow<NN>::NT, sr));
      } else {
        QG_CK(cudaFuncSetAttribute(k_col_inv<T, NN>, (cudaFuncAttribute)mx, (int)sm_ci<NN, Tiles<T, NN>::CIP>(Tiles<T, NN>::CINF)));
        QG_CK(cudaFuncSetAttribute(k_row_main<T, NN>, (cudaFuncAttribute)mx, (int)sm_rm<NN>(kxp_max<NN>())));
        QG_CK(cudaFuncSetAttribute(k_col_update<T, NN>, (cudaFuncAttribute)mx, (int)UpdLay<T, NN>::bytes()));
        QG_CK(cudaFuncSetAttribute(k_row_qw<T, NN>, (cudaFuncAttribute)mx, (int)sm_rq<NN>(kxp_max<NN>())));
        QG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_rm, k_row_main<T, NN>, kRowThreads, sm_rm<NN>(g.KXP)));
        QG_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_rq, k_row_qw<T, NN>, Tiles<T, NN>::QTHREADS,
                                                            sm_rq<NN>(g.KXP)));
        QG_CK(cudaFuncSetAttribute(k_col_qw<T, NN>, (cudaFuncAttribute)mx, (int)sm_ci<NN, Tiles<T, NN>::CQP>(2)));
      }
      occ_rm = std::max(occ_rm, 1);
      occ_rq = std::max(occ_rq, 1);
      // per-function attribute shared by every handle: set it for the deepest supported column
      QG_CK(cudaFuncSetAttribute(k_solve<T>, (cudaFuncAttribute)mx, (int)solve_smem(kMaxN3)));
      using DN = Dense<T, NN>;
      QG_CK(cudaFuncSetAttribute(k_dcol_inv<T, NN, DenseIn>, (cudaFuncAttribute)mx, (int)DN::sm_col()));
      QG_CK(cudaFuncSetAttribute(k_dcol_inv<T, NN, CompactIn<T>>, (cudaFuncAttribute)mx, (int)DN::sm_col()));
      QG_CK(cudaFuncSetAttribute(k_dcol_inv<T, NN, OmegaIn<T>>, (cudaFuncAttribute)mx, (int)DN::sm_col()));
      QG_CK(cudaFuncSetAttribute(k_dcol_fwd<T, NN, 1>, (cudaFuncAttribute)mx, (int)DN::sm_col(1)));
      QG_CK(cudaFuncSetAttribute(k_dcol_fwd<T, NN, 2>, (cudaFuncAttribute)mx, (int)DN::sm_col(2)));
      QG_CK(cudaFuncSetAttribute(k_drow_c2r_pad<T, NN>, (cudaFuncAttribute)mx, (int)DN::sm_row()));
      QG_CK(cudaFuncSetAttribute(k_drow_c2r_f32<T, NN>, (cudaFuncAttribute)mx, (int)DN::sm_row()));
      QG_CK(cudaFuncSetAttribute(k_drow_prod<T, NN>, (cudaFuncAttribute)mx, (int)DProd<T, NN>::smem()));
      QG_CK(cudaFuncSetAttribute(k_drow_r2c<T, NN>, (cudaFuncAttribute)mx, (int)DN::sm_row()));
    });
    return QG_OK;
  }

  StateP<T> state_ptrs() {
    StateP<T> p;
    p.q = F[F_Q]; p.qo = F[F_QO]; p.BR = F[F_BR]; p.BI = F[F_BI]; p.BRo = F[F_BRO]; p.BIo = F[F_BIO];
    p.psi = F[F_PSI]; p.AR = F[F_AR]; p.AI = F[F_AI]; p.qstar = F[F_QSTAR]; p.dq = F[F_DQ];
    p.sig1 = sig[0]; p.sig2 = sig[1];
    return p;
  }

  // Profiling: events around each launch when prof_on is set.
  bool prof_on = false;
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> prof_ev;
  int pbeg(int kind, cudaStream_t on = nullptr) {
    if (!prof_on) return QG_OK;
    cudaEvent_t a, b;
    QG_CK(cudaEventCreate(&a)); QG_CK(cudaEventCreate(&b));
    QG_CK(cudaEventRecord(a, on ? on : st));
    prof_ev.push_back({kind, {a, b}});
    return QG_OK;
  }
  int pend(cudaStream_t on = nullptr) {
    if (!prof_on) return QG_OK;
    QG_CK(cudaEventRecord(prof_ev.back().second.second, on ? on : st));
    return QG_OK;
  }

 public:
  int profile_step(int euler, double* ms, int* launches, int nclasses) override {
    for (int i = 0; i < nclasses; ++i) { ms[i] = 0.0; launches[i] = 0; }
    if (int rc = prepare()) return rc;
    prof_on = true;
    prof_ev.clear();
    int rc = enqueue_step(euler ? 1 : 0);
    prof_on = false;
    cudaError_t e = cudaStreamSynchronize(st);
    for (auto& pe : prof_ev) {
      float t = 0.f;
      if (rc == QG_OK && e == cudaSuccess && cudaEventElapsedTime(&t, pe.second.first, pe.second.second) == cudaSuccess &&
          pe.first < nclasses) {
        ms[pe.first] += t;
        launches[pe.first] += 1;
      }
      cudaEventDestroy(pe.second.first);
      cudaEventDestroy(pe.second.second);
    }
    prof_ev.clear();
    if (rc) return rc;
    QG_CK(e);
    return QG_OK;
  }

 protected:
  // FP64 steps run on the kernels of step_fx.cuh
  static constexpr bool kFx = sizeof(T) == 8;
  template <int NN> static constexpr int col_ct() {
    if constexpr (kFx) return FxCol<NN>::CT;
    else return Tiles<T, NN>::CT;
  }

  // whether a grid of n CTAs, per_sm of them resident on an SM, is at most
  // `waves` waves: k_fx_col_inv then spreads a tile's fields over several CTAs
  // (a shorter chain per CTA and more of the GPU at work) instead of looping
  // over them (one table load per tile).  us per launch, looped -> spread:
  // 64^2 x 64 22.5 -> 14.0, 128^2 x 64 36.7 -> 29.0, 256^2 x 128 (2.6 waves)
  // 144 -> 147.  (The FP32 kernels are not spread: the compiler then fuses
  // other products with additions, and the fields differ in their last bits
  // from those of larger grids.)
  bool few_ctas(long long n, int waves, int per_sm) const { return n <= (long long)waves * per_sm * nsm; }

  // k_col_inv on levels [z0, z0 + zc): mode 0 all six fields into Sb, 1 the
  // first four (BR, BI are kept in Qb), 2 BR and BI into Qb
  template <int NN>
  void launch_col_inv(int z0, int zc, const C* psi, const C* q, const C* br, const C* bi, C* Sb, C* Qb, int mode,
                      cudaStream_t on) {
    // column tiles up to kx = K (the padding columns beyond K are never read)
    const int tiles = (g.K + col_ct<NN>()) / col_ct<NN>();
    if constexpr (kFx) {
      const int f0 = mode == 2 ? 4 : 0, f1 = mode == 1 ? 4 : 6;
      const int split = few_ctas((long long)tiles * zc, 1, fx_col_ctas<NN>(kFxColCtas)) ? f1 - f0 : 1;
      k_fx_col_inv<NN><<<dim3(tiles * split, zc), FxCol<NN>::NT, FxCol<NN>::smem(), on>>>(g, z0, psi, q, br, bi, Sb, tw,
                                                                                          Qb, f0, f1, split);
      return;
    }
    if constexpr (!kFx)
      k_col_inv<T, NN><<<dim3(tiles, zc), Tiles<T, NN>::CNT, sm_ci<NN, Tiles<T, NN>::CIP>(Tiles<T, NN>::CINF), on>>>(
          g, z0, psi, q, br, bi, Sb, tw, Qb, mode);
  }

  // Enqueue one step on st (no synchronisation; graph-capturable).
  int enqueue_step(int euler) {
    StepParams s = sp;
    s.euler = euler;
    if (s.use_dq) {
      if (int rc0 = pbeg(QG_K_DISSIPATION)) return rc0;
      k_dissipation<T><<<grid_for((long long)g.n3 * g.plane), 256, 0, st>>>(g, cfg.nuz, cfg.dz,
                                                                              euler ? F[F_Q] : F[F_QO], F[F_DQ]);
      QG_LAUNCHED();
      if (int rc0 = pend()) return rc0;
    }
    StateP<T> sptr = state_ptrs();
    const int do_psi = cfg.fixed_flow ? 0 : 1;
    const int do_A = (cfg.passive_scalar || !cfg.ybj_plus) ? 0 : 1;
    // A solves beside the q^w kernels (a second stream; serialised while
    // profiling so that every launch is timed alone)
    const int nbat = (g.n3 + Zb - 1) / Zb;
    const int L = prof_on ? 1 : std::min(lanes, nbat);   // serialised while profiling
    const bool split = kSolveOverlap && need_qw && do_psi && do_A && kSolveStore && vbuf && L == 1;
    const bool overlap = split && !prof_on;
    if (L > 1) {
      QG_CK(cudaEventRecord(ev_start, st));
      for (int i = 1; i < L; ++i) QG_CK(cudaStreamWaitEvent(lst[i], ev_start, 0));
    }
    const size_t slot = (size_t)Zb * kNScr * g.n * g.KXP;
    for (int z0 = 0, b = 0; z0 < g.n3; z0 += Zb, ++b) {
      const int zc = std::min(Zb, g.n3 - z0);
      const bool last = z0 + Zb >= g.n3;
      const int lane = b % L;
      cudaStream_t bs = lane == 0 ? st : lst[lane];
      C* Sb = S + lane * slot;
      QG_SWITCH_N(g.n, {
        // column tiles up to kx = K (the padding columns beyond K are never read)
        const dim3 gc((g.K + col_ct<NN>()) / col_ct<NN>(), zc), gr(g.n / Tiles<T, NN>::QRT, zc),
            grm(g.n / Tiles<T, NN>::RTM, zc);
        if (int rc0 = pbeg(QG_K_COL_INV, bs)) return rc0;
        C* Qb = Qp ? Qp + (size_t)z0 * kNQ * g.n * g.KXP : nullptr;
        launch_col_inv<NN>(z0, zc, F[F_PSI], F[F_Q], F[F_BR], F[F_BI], Sb, Qb, Qb ? 1 : 0, bs);
        QG_LAUNCHED();
        if (int rc0 = pend(bs)) return rc0;
        if (int rc0 = pbeg(QG_K_ROW_MAIN, bs)) return rc0;
        if constexpr (kFx) {
          const int items = zc * (NN / FxMain<NN>::F::RT);
          k_fx_row_main<NN><<<std::min(items, std::max(1, nsm * occ_rm / L)), FxMain<NN>::F::NT, FxMain<NN>::smem(), bs>>>(
              g, s, Sb, tw, items, Qb);
        } else if constexpr (Tiles<T, NN>::RPRE) {
          const int items = zc * (NN / Tiles<T, NN>::RTM);
          k_row_main<T, NN><<<std::min(items, std::max(1, nsm * occ_rm / L)), kRowThreads, sm_rm<NN>(g.KXP), bs>>>(g, s, Sb, tw, items,
                                                                                                 wflag, Qb);
        } else {
          k_row_main<T, NN><<<grm, kRowThreads, sm_rm<NN>(g.KXP), bs>>>(g, s, Sb, tw, 0, wflag, Qb);
        }
        QG_LAUNCHED();
        if (int rc0 = pend(bs)) return rc0;
        {
          // asynchronous diagnostics of the previous state read B, A and psi:
          // the update waits for them (an external event node when captured)
          cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
          QG_CK(cudaStreamIsCapturing(bs, &cs));
          QG_CK(cudaStreamWaitEvent(bs, ev_diag, cs == cudaStreamCaptureStatusActive ? cudaEventWaitExternal : 0));
        }
        if (int rc0 = pbeg(QG_K_COL_UPDATE, bs)) return rc0;
        if constexpr (kFx)
          k_fx_col_update<NN><<<dim3(gc.x, gc.y, 3), FxCol<NN>::NT, FxCol<NN>::smem(), bs>>>(g, s, z0, sptr, e1, e2, e1w, e2w, Sb, tw,
                                                                           need_qw ? 1 : 0, Qb);
        else
          k_col_update<T, NN><<<gc, Tiles<T, NN>::CNT, UpdLay<T, NN>::bytes(), bs>>>(g, s, z0, sptr, e1, e2, e1w, e2w, Sb, tw,
                                                                need_qw ? 1 : 0, Qb);
        QG_LAUNCHED();
        if (int rc0 = pend(bs)) return rc0;
        if (overlap && last) {
          // B^{n+1} of every level is written: fork the A solves
          QG_CK(cudaEventRecord(ev_fork, bs));
          QG_CK(cudaStreamWaitEvent(st2, ev_fork, 0));
          if (int rc0 = solve_generic(nullptr, F[F_BR], F[F_BI], nullptr, F[F_AR], F[F_AI], 0, 1, st2, 0, -1, true))
            return rc0;
          QG_CK(cudaEventRecord(ev_join, st2));
        }
        if (need_qw) {
          if (int rc0 = pbeg(QG_K_ROW_QW, bs)) return rc0;
          if constexpr (kFx) {
            const int items = zc * (NN / FxRow<NN>::RT);
            k_fx_row_qw<NN><<<std::min(items, std::max(1, nsm * occ_rq / L)), FxRow<NN>::NT, FxQw<NN>::smem(), bs>>>(
                g, Sb, tw, items, Qb);
          } else if constexpr (Tiles<T, NN>::QPRE) {
            const int items = zc * (NN / Tiles<T, NN>::QRT);
            const int per_sm = (split && last) ? std::max(1, occ_rq - kQwReserve) : occ_rq;
            k_row_qw<T, NN><<<std::min(items, std::max(1, nsm * per_sm / L)), Tiles<T, NN>::QTHREADS, sm_rq<NN>(g.KXP), bs>>>(
                g, Sb, tw, items, wflag, Qb);
          } else {
            k_row_qw<T, NN><<<gr, Tiles<T, NN>::QTHREADS, sm_rq<NN>(g.KXP), bs>>>(g, Sb, tw, 0, wflag, Qb);
          }
          QG_LAUNCHED();
          if (int rc0 = pend(bs)) return rc0;
          if (int rc0 = pbeg(QG_K_COL_QW, bs)) return rc0;
          if constexpr (kFx)
            k_fx_col_qw<NN><<<gc, FxCol<NN>::NT, FxCol<NN>::smem(), bs>>>(g, s, z0, F[F_Q], F[F_QSTAR], Sb, tw, nflag);
          else
            k_col_qw<T, NN><<<gc, Tiles<T, NN>::CNT, sm_ci<NN, Tiles<T, NN>::CQP>(2), bs>>>(g, s, z0, F[F_Q], F[F_QSTAR], Sb, tw, nflag);
          QG_LAUNCHED();
          if (int rc0 = pend(bs)) return rc0;
        }
      });
    }
    for (int i = 1; i < L; ++i) {
      QG_CK(cudaEventRecord(lev[i], lst[i]));
      QG_CK(cudaStreamWaitEvent(st, lev[i], 0));
    }
    if (int rc0 = pbeg(QG_K_SOLVE)) return rc0;
    int rc = launch_solve(need_qw ? F[F_QSTAR] : F[F_Q], do_psi, split ? 0 : do_A);
    if (rc) return rc;
    if (overlap) {
      QG_CK(cudaStreamWaitEvent(st, ev_join, 0));
    } else if (split) {
      if (int rc0 = pend()) return rc0;
      if (int rc0 = pbeg(QG_K_SOLVE_A)) return rc0;
      if ((rc = launch_solve(nullptr, 0, 1))) return rc;
    }
    if (!cfg.ybj_plus && !cfg.passive_scalar) {
      // regular YBJ: sumB on B^{n+1}, then A from the vertical integral (main_waqg.f90:449-460)
      k_ybj_A<T><<<(unsigned)((g.plane + 127) / 128), 128, 0, st>>>(g, cfg.dz, cfg.Bu, cfg.Ro, r2, F[F_BR], F[F_BI],
                                                                    sig[0], sig[1], F[F_AR], F[F_AI]);
      QG_LAUNCHED();
    }
    return pend();
  }

  int launch_solve(C* qs, int do_psi, int do_A) {
    return solve_generic(qs, F[F_BR], F[F_BI], F[F_PSI], F[F_AR], F[F_AI], do_psi, do_A, nullptr, 0, -1, true);
  }

  // the column solves of segments [seg0, seg0 + nsegs) (nsegs < 0: all)
  // retained: the outputs are resident fields (zeros off the retained
  // modes already), so only the retained columns are solved
  int solve_generic(const C* qs, const C* br, const C* bi, C* psi, C* ar, C* ai, int do_psi, int do_A,
                    cudaStream_t on = nullptr, int seg0 = 0, int nsegs = -1, bool retained = false) {
    if (!do_psi && !do_A) return QG_OK;
    if (!on) on = st;
    if (nsegs < 0) nsegs = members - seg0;
    const int* cl = retained ? cols_ret : cols_all;
    const int ncl = retained ? nret : (int)g.plane;
    double* const pcf = retained ? pcfac : nullptr;     // the per-column factors follow the retained list
    if (kSolveStore && vbuf) {
      const int nrec = (do_psi ? 2 : 0) + (do_A == 1 ? 4 : do_A);   // recurrences per column
      // A launch of few columns spreads their recurrences over CTAs of one
      // warp, so that more SMs' FP64 pipes (2 lanes per clock) work on them,
      // and reads longer segments ahead (whatever solve_tc is).  us per solve,
      // otherwise -> so, by warps per SM: 0.9 (FP64 64^2 x 64) 42.9 -> 34.7, 3.6
      // (128^2 x 64) 45.0 -> 38.8, 4.6 (psi_solver 256^2 x 128) 123 -> 118, 13.9
      // (256^2 x 128) 147 -> 189; mixed 64^2 x 32 18.3 -> 16.3, 256^2 x 128 80 ->
      // 139
      const bool few = few_ctas((long long)((ncl + 31) / 32) * nsegs * nrec, 1, 12);
      const int zs = few ? nrec : 1;
#define QG_SOLVE_ST(TCV, PCV, SV)                                                                            \
  k_solve_st<T, TCV, PCV, SV><<<dim3((unsigned)((ncl + TCV - 1) / TCV), nsegs, zs), nrec / zs * TCV,        \
                                (size_t)g.nseg * 8, on>>>(                                                   \
      g, cfg.dz, cfg.Bu, tab_idx, fac_psi, fac_A, du, qs, br, bi, psi, ar, ai, do_psi, do_A, vbuf, pcf, seg0, cl, ncl)
      if (pcf) {
        if (few) QG_SOLVE_ST(32, true, kSegFew);
        else if (solve_tc == 16) QG_SOLVE_ST(16, true, kSegSt);
        else if (solve_tc == 64) QG_SOLVE_ST(64, true, kSegSt);
        else QG_SOLVE_ST(32, true, kSegSt);
      } else {
        if (few) QG_SOLVE_ST(32, false, kSegFew);
        else if (solve_tc == 16) QG_SOLVE_ST(16, false, kSegSt);
        else if (solve_tc == 64) QG_SOLVE_ST(64, false, kSegSt);
        else QG_SOLVE_ST(32, false, kSegSt);
      }
#undef QG_SOLVE_ST
      QG_LAUNCHED();
      return QG_OK;
    }
    k_solve<T><<<dim3((unsigned)((g.plane + kSolveTC - 1) / kSolveTC), nsegs), kSolveThreads, solve_smem(g.nseg), on>>>(g, cfg.dz, cfg.Bu, tab_idx, fac_psi, fac_A,
                                                                           du, qs, br, bi, psi, ar, ai, do_psi, do_A, seg0);
    QG_LAUNCHED();
    return QG_OK;
  }

  // Before a step (outside any stream capture): the kept B planes, when
  // they do not hold the transforms of the current B (new handle,
  // qg_set_state of BR or BI, initialisation), are computed from B.
  int prepare() override {
    release_init_buffers();     // the step replaces psi
    if (!Qp || q_valid) return QG_OK;
    for (int z0 = 0; z0 < g.n3; z0 += Zb) {
      const int zc = std::min(Zb, g.n3 - z0);
      QG_SWITCH_N(g.n, {
        launch_col_inv<NN>(z0, zc, F[F_PSI], F[F_Q], F[F_BR], F[F_BI], S, Qp + (size_t)z0 * kNQ * g.n * g.KXP, 2, st);
        QG_LAUNCHED();
      });
    }
    q_valid = true;     // every step keeps them current from here on
    return QG_OK;
  }

  int run_step(int euler) {
    if (int rc = prepare()) return rc;
    if (!cfg.use_graphs) return enqueue_step(euler);
    if (!gexec[euler]) {
      cudaGraph_t graph = nullptr;
      QG_CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
      int rc = enqueue_step(euler);
      cudaError_t e = cudaStreamEndCapture(st, &graph);
      if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
      if (e != cudaSuccess) { err = std::string("graph capture: ") + cudaGetErrorString(e); return QG_ERR_CUDA; }
      e = cudaGraphInstantiate(&gexec[euler], graph, cudaGraphInstantiateFlagUseNodePriority);
      cudaGraphDestroy(graph);
      if (e != cudaSuccess) { err = std::string("graph instantiate: ") + cudaGetErrorString(e); return QG_ERR_CUDA; }
    }
    QG_CK(cudaGraphLaunch(gexec[euler], st));
    return QG_OK;
  }

  // ---- dense drop-in plumbing ---------------------------------------------
  size_t dense_bytes(int nz) const { return (size_t)nz * g.n * (g.n / 2 + 1) * sizeof(double2); }
  int iktxP() const { return dense_kxp(g.n); }

  int prep_dense(int nz, int planes) {
    if (nz <= 0) { err = "nz must be positive"; return QG_ERR_ARG; }
    const size_t need = (size_t)nz * planes;
    if (need <= w_planes) return QG_OK;
    QG_CK(cudaStreamSynchronize(st));
    if (W) { cudaFree(W); W = nullptr; w_planes = 0; }
    QG_CK(dev_alloc(&W, need * g.n * iktxP() * sizeof(C)));
    w_planes = need;
    return QG_OK;
  }

  // Whether kernels on this device may use [p, p + bytes) in place: 16-byte
  // aligned memory of this device, inside one allocation.  Anything else goes
  // through a staging copy, whose cudaMemcpy accepts or refuses it as it does
  // any pointer.
  bool in_place(const void* p, size_t bytes) const {
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { (void)cudaGetLastError(); return false; }
    if (at.type != cudaMemoryTypeDevice || at.device != cfg.device) return false;
    using Range = CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr);
    static const Range range = []() -> Range {
      void* f = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
          q != cudaDriverEntryPointSuccess) {
        (void)cudaGetLastError();
        return nullptr;
      }
      return reinterpret_cast<Range>(f);
    }();
    CUdeviceptr base = 0;
    size_t size = 0;
    const CUdeviceptr a = reinterpret_cast<CUdeviceptr>(p);
    return range && range(&base, &size, a) == CUDA_SUCCESS && a - base + bytes <= size;
  }
  // a device view of an input (copied into staging slot `slot` if need be)
  int in_view(const void* p, size_t bytes, int slot, const void** v) {
    if (in_place(p, bytes)) { *v = p; return QG_OK; }
    if (int rc = ensure(&stg[slot], &stg_bytes[slot], bytes)) return rc;
    QG_CK(cudaMemcpyAsync(stg[slot], p, bytes, cudaMemcpyDefault, st));
    *v = stg[slot];
    return QG_OK;
  }
  // where kernels write an output: the caller's array, or staging slot `slot`
  // (also where the array overlaps `keep`, an input of the same size that is
  // read while the output is written); out_copy then brings it to the caller
  int out_view(void* p, size_t bytes, int slot, void** v, const void* keep = nullptr) {
    const char *a = (const char*)p, *k = (const char*)keep;
    if (in_place(p, bytes) && !(keep && a < k + bytes && k < a + bytes)) { *v = p; return QG_OK; }
    if (int rc = ensure(&stg[slot], &stg_bytes[slot], bytes)) return rc;
    *v = stg[slot];
    return QG_OK;
  }
  int out_copy(void* p, const void* v, size_t bytes) {
    if (v != p) QG_CK(cudaMemcpyAsync(p, v, bytes, cudaMemcpyDefault, st));
    return QG_OK;
  }

  // y-inverse transforms of nf fields of src at kx <= KM into planes 0 .. nf-1
  // (np per level)
  template <class Src> int d_inv(const Src& src, int nz, int nf, int KM, int np = 0) {
    QG_SWITCH_N(g.n, {
      using DN = Dense<T, NN>;
      k_dcol_inv<T, NN, Src><<<dim3((KM + DN::CT) / DN::CT, nz, nf), DN::CNT, DN::sm_col(), st>>>(iktxP(), np ? np : nf, src,
                                                                                               W, tw);
      QG_LAUNCHED();
    });
    return QG_OK;
  }
  int d_prod(int nz, int np, int KM, int cross, int scale, int nA, int nX) {
    QG_SWITCH_N(g.n, {
      using DN = Dense<T, NN>;
      k_drow_prod<T, NN><<<dim3(g.n / 2 / DN::RT, nz), DN::RNT, DProd<T, NN>::smem(), st>>>(iktxP(), np, KM, cross, scale, nA,
                                                                                         nX, W, tw);
      QG_LAUNCHED();
    });
    return QG_OK;
  }
  template <int NF> int d_fwd(const DenseOut& o, int nz, int np, int no) {
    QG_SWITCH_N(g.n, {
      using DN = Dense<T, NN>;
      k_dcol_fwd<T, NN, NF><<<dim3(iktxP() / DN::CT, nz, no), DN::CNT, DN::sm_col(NF), st>>>(iktxP(), np, W, o, tw);
      QG_LAUNCHED();
    });
    return QG_OK;
  }

  // c2r and r2c of nz levels; physical rows of ld doubles (n or n + 2)
  int d_c2r(const double2* spec, double* phys, int ld, int nz) {
    DenseIn in{};
    in.p[0] = spec;
    in.op[0] = OP_ID;
    if (int rc = d_inv(in, nz, 1, g.n / 2)) return rc;
    QG_SWITCH_N(g.n, {
      using DN = Dense<T, NN>;
      k_drow_c2r_pad<T, NN><<<dim3(g.n / 2 / DN::RT, nz), DN::RNT, DN::sm_row(), st>>>(iktxP(), W, phys, ld, tw);
      QG_LAUNCHED();
    });
    return QG_OK;
  }
  int d_r2c(const double* phys, int ld, double2* spec, int nz) {
    QG_SWITCH_N(g.n, {
      using DN = Dense<T, NN>;
      k_drow_r2c<T, NN><<<dim3(g.n / 2 / DN::RT, nz), DN::RNT, DN::sm_row(), st>>>(iktxP(), phys, ld, W, tw);
      QG_LAUNCHED();
    });
    return d_fwd<1>(DenseOut{{spec, nullptr, nullptr}, 0, g.kmax2, 0.0, 0.0}, nz, 1, 1);
  }

  int ensure_tmp() {
    const size_t fbytes = (size_t)g.n3 * g.plane * sizeof(C);
    for (auto& p : tmpF) if (!p) { QG_CK(dev_alloc(&p, fbytes)); QG_CK(cudaMemsetAsync(p, 0, fbytes, st)); }
    return QG_OK;
  }

  int upload_compact(const double* kvar, C* dst) {
    const void* v;
    if (int rc = in_view(kvar, dense_bytes(g.n3), 0, &v)) return rc;
    k_dense_to_compact<T><<<conv_grid(g.KY, g.n3), 256, 0, st>>>(g, 0, (const double2*)v, dst);
    QG_LAUNCHED();
    return QG_OK;
  }

  int download_compact(const C* src, double* kvar, int mode) {
    const size_t bytes = dense_bytes(g.n3);
    void* v;
    if (int rc = out_view(kvar, bytes, 0, &v)) return rc;
    if (int rc = to_dense(src, (double2*)v, mode, 0, g.n3)) return rc;
    return out_copy(kvar, v, bytes);
  }
};

}  // namespace qg
