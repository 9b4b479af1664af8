// Elementwise kernels of the adjoint (FP64, the reference's dense spectral
// layout double2 [nz][n][n/2+1] and physical layout double [nz][n][n]).
#pragma once
#include "dense_kernels.cuh"
#include "step_fx.cuh"

namespace qg {

// One term s * mult(k) * in of a spectral linear combination; s complex,
// mult: 0 -> 1, 1 -> kx, 2 -> ky, 3 -> kh^2, 4 -> per-mode table (dense [n][n/2+1]).
struct SpecTerm {
  const double2* in;
  double sr, si;
  int mult;
  const double* tab;
};

// out = mask( (acc ? out : 0) + sum_t s_t mult_t in_t )
static __global__ void k_spec_lin(int n, int kmax2, long long tot, int nt, SpecTerm t0, SpecTerm t1, SpecTerm t2,
                                  int acc, double2* out) {
  const long long plane = (long long)n * (n / 2 + 1);
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < tot; m += (long long)gridDim.x * blockDim.x) {
    int kx, ky, iky;
    dense_mode(m, n, kx, ky, iky);
    double2 o = make_double2(0.0, 0.0);
    if (dense_L(kx, ky, iky, n, kmax2)) {
      if (acc) o = out[m];
      const SpecTerm* ts[3] = {&t0, &t1, &t2};
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        if (t >= nt) break;
        const SpecTerm& T = *ts[t];
        double f = 1.0;
        if (T.mult == 1) f = (double)kx;
        else if (T.mult == 2) f = (double)ky;
        else if (T.mult == 3) f = (double)(kx * kx + ky * ky);
        else if (T.mult == 4) f = T.tab[m % plane];
        const double cr = T.sr * f, ci = T.si * f;
        const double2 v = T.in[m];
        o.x += cr * v.x - ci * v.y;
        o.y += cr * v.y + ci * v.x;
      }
    }
    out[m] = o;
  }
}

// transpose of c2r on the retained modes: out (+)= mask(2 N^2 Y), (0,0): N^2 Re Y
static __global__ void k_ct_weights(int n, int kmax2, long long tot, double N2, const double2* __restrict__ Y, int acc,
                                    double2* __restrict__ out) {
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < tot; m += (long long)gridDim.x * blockDim.x) {
    int kx, ky, iky;
    dense_mode(m, n, kx, ky, iky);
    double2 v = make_double2(0.0, 0.0);
    if (dense_L(kx, ky, iky, n, kmax2)) {
      const double2 y = Y[m];
      v = (kx == 0 && ky == 0) ? make_double2(N2 * y.x, 0.0) : make_double2(2.0 * N2 * y.x, 2.0 * N2 * y.y);
      if (acc) { const double2 o = out[m]; v.x += o.x; v.y += o.y; }
    }
    out[m] = v;
  }
}

// per-block partial sums of W (x^2 + y^2) over the objective's subvolume
// (x, y in [n/4, 3n/4), levels iz >= z0); fixed-order reduction
static __global__ void k_obj_partial(int n, int n3, int z0, const double* __restrict__ a, const double* __restrict__ b,
                                     double* __restrict__ part) {
  __shared__ double red[256];
  const long long tot = (long long)n3 * n * n;
  double acc = 0.0;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < tot; i += (long long)gridDim.x * 256) {
    const int x = (int)(i % n), y = (int)((i / n) % n), z = (int)(i / ((long long)n * n));
    if (z >= z0 && x >= n / 4 && x < 3 * n / 4 && y >= n / 4 && y < 3 * n / 4) acc += a[i] * a[i] + b[i] * b[i];
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// x *= W (the subvolume indicator)
static __global__ void k_obj_window(int n, int n3, int z0, double* __restrict__ x) {
  const long long tot = (long long)n3 * n * n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const int xx = (int)(i % n), y = (int)((i / n) % n), z = (int)(i / ((long long)n * n));
    if (!(z >= z0 && xx >= n / 4 && xx < 3 * n / 4 && y >= n / 4 && y < 3 * n / 4)) x[i] = 0.0;
  }
}


// ===========================================================================
// Fused adjoint of one step on the compact layout (FP64).
//
// Phase A' (batches of levels, scratch planes SF and SA, [zb][6][n][KXP]):
//   k_col_inv          y-inverse FFTs of u, v, zeta, q, BR, BI (the forward
//                      kernel, into SF)
//   k_adj_col_inv      adjoint tendencies lNq, lTR, lTI from the incoming
//                      adjoint state; y-inverse FFTs of l and -i ky l (SA)
//   k_adj_row          x-c2r of 14 physical fields, the transposed products,
//                      x-r2c of the 6 results (SA)
//   k_adj_col_fwd      y-forward FFTs; transposed filter / leapfrog / Euler
//                      update; right-hand sides of the symmetric solves
// Phase B: the FP64 tridiagonal solves (psi_solver, A_solver_ybj_plus) of
//   the forward step applied to (lpsi, lAR, lAI).
// Phase C' (q^w transpose):
//   k_adj_qw_col_inv   y-inverse FFTs of BR, i ky BR, BI, i ky BI, w, ky^2 w (SF)
//   k_adj_qw_row       x-c2r, transposed q^w products, x-r2c (SF)
//   k_adj_qw_col_fwd   y-forward FFTs; lq += w, lB += A-solve + q^w terms
//
// Transposes (N = n): C = c2r of the retained modes (realit included) has
// C^T y = w_k F(y) with F the unnormalised r2c, w_k = 2 and 1 at (0,0) (real
// part); (mask R)^T Y = C(Y')/(2 N^2), Y'_00 = 2 Re Y_00.
// ===========================================================================
struct AdjP {
  double dt, gam;
  double cdisp;   // disp * 0.5/(Bu Ro)
  double adv;     // 0 when linear
  double refr;    // 0 when passive_scalar
  double s;       // Ro W2F (q^w coefficient)
  int first;      // transposing the forward Euler first step
};
struct AdjIn { const double2* l[6]; };                   // (lq, lr, lBR, lBI, lcR, lcI) after the step
struct AdjOut { double2* l[6]; double2* lpsi; double2* lAR; double2* lAI; };

// transposed time update of one mode of variable w (0 q, 1 BR, 2 BI), e1, e2
// its integrating factors: the adjoint tendency, and the outputs before the
// solves and the product terms (new level, old level)
__device__ __forceinline__ void adj_update(const AdjP& p, const AdjIn& L, int w, long long m, double e1, double e2,
                                           double2& lt, double2& on, double2& oo) {
  const int fn = w == 0 ? 0 : 1 + w, fo = w == 0 ? 1 : 3 + w;      // (lq, lr), (lBR, lcR), (lBI, lcI)
  const double2 l1 = L.l[fn][m], lo = L.l[fo][m];
  if (p.first) {
    lt = cscale(l1, -p.dt * e1);
    on = cadd(lo, cscale(l1, e1));
    oo = make_double2(0.0, 0.0);
  } else {
    const double2 lp = cadd(l1, cscale(lo, p.gam));
    lt = cscale(lp, -2.0 * p.dt * e1);
    on = cscale(lo, 1.0 - 2.0 * p.gam);
    oo = cadd(cscale(lo, p.gam), cscale(lp, e2));
  }
}

// spectrum entering a c2r that applies (mask R)^T: Y/(2N^2), (0,0): Re Y/N^2
__device__ __forceinline__ double2 rt_scale(double2 v, int kx, int ky, double inv2n2) {
  return (kx == 0 && ky == 0) ? make_double2(2.0 * v.x * inv2n2, 0.0) : cscale(v, inv2n2);
}

// two half spectra get(kk, X, Y) as fx_half's
template <int N, class Get> __device__ __forceinline__ void adj_half(int j, int K, double2 (&a)[8], double2 (&b)[8], Get get) {
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    a[r] = b[r] = make_double2(0.0, 0.0);
    if (fx_zero_in<8>(r)) continue;
    const int k = j + r * (N / 8), kk = r < 4 ? k : N - k;
    if (kk <= K) get(kk, a[r], b[r]);
  }
  if (j == 0) a[0].y = b[0].y = 0.0;
}

// y-inverse transforms of one plane of a column tile: get(row, ky) is the
// value at a retained row; stored to plane f of S
template <int N, class Get>
__device__ __forceinline__ void adj_col_inverse(const FxColCtx<N>& c, const Geom& g, int kx, double2* __restrict__ dst,
                                                Get get) {
  constexpr int NB = N / 8;
  double2 d[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    d[r] = make_double2(0.0, 0.0);
    if (fx_zero_in<8>(r)) continue;
    int row; bool cj;
    col_src(g, kx, c.j + r * NB, row, cj);
    if (row < 0 || !g.mask(kx, g.ky_of_row(row))) continue;
    d[r] = get(row, g.ky_of_row(row));
    if (cj) d[r].y = -d[r].y;
  }
  fxc v[8];
  int base;
  c.template run<false>(d, v, base);
  if (kx > g.K) return;
  fx_doubles<8, true>(v, d, base);
  double2* o = dst + (long long)c.j * g.KXP + kx;
#pragma unroll
  for (int r = 0; r < 8; ++r) o[(long long)r * NB * g.KXP] = d[r];
}

// the transposed products' kernels keep one transform per thread in flight,
// as the step's (step_fx.cuh); the column kernels' independent fields are
// spread over gridDim.z CTAs where a grid would leave SMs idle
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(kFxColCtas))
k_adj_col_inv(Geom g, AdjP p, int zbase, AdjIn L, const double* __restrict__ e1t, const double* __restrict__ e2t,
              const double* __restrict__ e1wt, const double* __restrict__ e2wt, double2* __restrict__ SA,
              const double2* __restrict__ twg) {
  using F = FxCol<N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, kx = blockIdx.x * F::CT + c.c;
  const long long zoff = (long long)(zbase + zb) * g.plane;
  const double inv2n2 = 0.5 / ((double)N * (double)N);
  // l and -i ky l of the adjoint tendencies of q, BR, BI
#pragma unroll 1
  for (int f = blockIdx.z; f < 6; f += gridDim.z) {
    const int w = f >> 1;
    adj_col_inverse<N>(c, g, kx, SA + scr_off(zb, f, 0, N, g.KXP), [&](int row, int ky) {
      const long long mt = (long long)row * g.KXP + kx;
      double2 lt, on, oo;
      adj_update(p, L, w, zoff + mt, w == 0 ? e1t[mt] : e1wt[mt], w == 0 ? e2t[mt] : e2wt[mt], lt, on, oo);
      lt = rt_scale(lt, kx, ky, inv2n2);
      return (f & 1) ? cscale(cmul_mi(lt), (double)ky) : lt;
    });
  }
}

// rows: SF holds (u, v, zeta, q, BR, BI), SA the adjoint planes
// (lNq, -i ky lNq, lTR, -i ky lTR, lTI, -i ky lTI) after the y-inverse FFT;
// writes SA = (F_x lu, -i kx F_x lv - kx^2 F_x lZ, F_x lZ, F_x lQ, F_x lBR, F_x lBI).
// The physical u, v, zeta, q, BR, BI are parked in shared memory, each thread
// its own eight points; the six sums of products accumulate in registers.
template <int N> struct AdjRow {
  static constexpr size_t smem() { return FxRow<N>::smem() + (size_t)3 * FxRow<N>::RT * N * sizeof(double2); }
};
template <int N>
__global__ void __launch_bounds__(FxRow<N>::NT, fx_row_ctas<N>(2))
k_adj_row(Geom g, AdjP p, const double2* __restrict__ SF, double2* __restrict__ SA, const double2* __restrict__ twg) {
  using F = FxRow<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slots[F::SLOTS];
  FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  // point (x = j + r NB) of pair q at park[(q * 8 + r) * NT]
  double2* park = reinterpret_cast<double2*>(smem_raw) + fx_tw_count<N>() + F::RT * F::LD + threadIdx.x;
  const int zb = blockIdx.y, y = blockIdx.x * F::RT + c.rr, K = g.K, j = c.j;
  auto sf = [&](int f) { return SF + scr_off(zb, f, y, N, g.KXP); };
  auto sa = [&](int f) { return SA + scr_off(zb, f, y, N, g.KXP); };
  const double adv = p.adv, hr = 0.5 * p.refr;
  double2 luv[8], lzq[8], lbb[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) luv[r] = lzq[r] = lbb[r] = make_double2(0.0, 0.0);
  // (u, v), (zeta, q), (br, bi); (aq, aR, aI): l of q, BR, BI times (-i kx,
  // d/dy); the refraction's (lTI, -lTR)/2
#pragma unroll 1
  for (int q = 0; q < 7; ++q) {
    const double2 *A = q < 3 ? sf(2 * q) : (q < 6 ? sa(2 * (q - 3)) : sa(4));
    const double2 *B = q < 3 ? sf(2 * q + 1) : (q < 6 ? sa(2 * (q - 3) + 1) : sa(2));
    const double sb = q < 3 ? 1.0 : (q < 6 ? adv : -hr);
    double2 X[8], Y[8], o[8];
    adj_half<N>(j, K, X, Y, [&](int kk, double2& a, double2& b) {
      a = A[kk];
      b = cscale(B[kk], sb);
      if (q >= 3) a = q < 6 ? cscale(cmul_mi(a), adv * (double)kk) : cscale(a, hr);
    });
    c.inverse_d(X, Y, o);
    if (q < 3) {
#pragma unroll
      for (int r = 0; r < 8; ++r) park[(q * 8 + r) * F::NT] = o[r];
    } else if (q < 6) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const double2 uv = park[r * F::NT], x = park[((q == 3 ? 8 : 16) + r) * F::NT];
        const double f = q == 4 ? x.x : x.y;
        const double s = o[r].x * uv.x + o[r].y * uv.y;
        luv[r].x += o[r].x * f;
        luv[r].y += o[r].y * f;
        if (q == 3) lzq[r].y = s;
        else if (q == 4) lbb[r].x = s;
        else lbb[r].y = s;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const double2 bb = park[(16 + r) * F::NT];
        const double Z = park[(8 + r) * F::NT].x;
        lzq[r].x = o[r].x * bb.x + o[r].y * bb.y;
        lbb[r].x += o[r].x * Z;
        lbb[r].y += o[r].y * Z;
      }
    }
  }
  double2 lv[3];
#pragma unroll 1
  for (int f = 0; f < 3; ++f) {
    c.forward_d(luv, K, [&](int q, int k, double2 X, double2 Y) {
      if (f == 0) {
        sa(0)[k] = X;
        lv[q] = Y;
      } else if (f == 1) {
        const double kx = (double)k;
        sa(1)[k] = csub(cscale(cmul_mi(lv[q]), kx), cscale(X, kx * kx));
        sa(2)[k] = X;
        sa(3)[k] = Y;
      } else {
        sa(4)[k] = X;
        sa(5)[k] = Y;
      }
    });
#pragma unroll
    for (int r = 0; r < 8; ++r) { luv[r] = lzq[r]; lzq[r] = lbb[r]; }
  }
}

// Forward transform of plane P of a column tile times the weight of C^T (2,
// and 1 with the real part at (0,0)), at the retained rows: use(r, row, ky, m, v)
template <int N, class Use>
__device__ __forceinline__ void adj_col_plane(const FxColCtx<N>& c, const Geom& g, const double2* __restrict__ P, int kx,
                                              Use use) {
  constexpr int NB = N / 8;
  double2 d[8];
  const double2* p = P + (long long)c.j * g.KXP + kx;
#pragma unroll
  for (int r = 0; r < 8; ++r) d[r] = kx <= g.K ? p[(long long)r * NB * g.KXP] : make_double2(0.0, 0.0);
  fxc v[8];
  int base;
  c.template run<true>(d, v, base);
  if (kx > g.K) return;
  fx_doubles<8, false>(v, d, base);
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    if (fx_zero_in<8>(r)) continue;
    const int row = g.row_of_fft_index(c.j + r * NB);
    if (row < 0) continue;
    const int ky = g.ky_of_row(row);
    double2 h = make_double2(0.0, 0.0);
    if (g.mask(kx, ky)) {
      h = d[r];
      if (kx == 0 && ky == 0) h.y = 0.0;
      else h = cscale(h, 2.0);
    }
    use(r, (long long)row * g.KXP + kx, ky, h);
  }
}

template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(kFxColCtas))
k_adj_col_fwd(Geom g, AdjP p, int zbase, AdjIn L, AdjOut O, const double* __restrict__ e1t,
              const double* __restrict__ e2t, const double* __restrict__ e1wt, const double* __restrict__ e2wt,
              const double2* __restrict__ SA, const double2* __restrict__ twg) {
  using F = FxCol<N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, kx = blockIdx.x * F::CT + c.c;
  const long long zoff = (long long)(zbase + zb) * g.plane;
  // psi -> (u, v, zeta) = (-i ky, i kx, -kh^2) psi: transposes i ky, -i kx, -kh^2
  // (spread over gridDim.z = 4 CTAs: u, v, zeta; q; BR; BI)
  const int f0 = blockIdx.z ? 2 + blockIdx.z : 0, f1 = gridDim.z == 1 ? 6 : (blockIdx.z ? f0 + 1 : 3);
  double2 a[8];
#pragma unroll 1
  for (int f = f0; f < f1; ++f) {
    adj_col_plane<N>(c, g, SA + scr_off(zb, f, 0, N, g.KXP), kx, [&](int r, long long mt, int ky, double2 h) {
      const long long m = zoff + mt;
      if (f == 0) {
        a[r] = cscale(cmul_i(h), (double)ky);
      } else if (f == 1) {
        a[r] = cadd(a[r], h);
      } else if (f == 2) {
        O.lpsi[m] = csub(a[r], cscale(h, (double)ky * (double)ky));
      } else {
        const int w = f - 3;
        double2 lt = make_double2(0.0, 0.0), on = lt, oo = lt;
        if (g.mask(kx, ky)) {
          adj_update(p, L, w, m, w == 0 ? e1t[mt] : e1wt[mt], w == 0 ? e2t[mt] : e2wt[mt], lt, on, oo);
          on = cadd(on, h);
        }
        O.l[w == 0 ? 0 : 1 + w][m] = on;
        O.l[w == 0 ? 1 : 3 + w][m] = oo;
        // T_R = N_BR + c kh^2 A_I - r_BI/2, T_I = N_BI - c kh^2 A_R + r_BR/2
        const double ck = p.cdisp * (double)(kx * kx + ky * ky);
        if (w == 1) O.lAI[m] = cscale(lt, ck);
        if (w == 2) O.lAR[m] = cscale(lt, -ck);
      }
    });
  }
}

// y-inverse FFTs for the q^w transpose: BR, i ky BR, BI, i ky BI, w', ky^2 w'
// with w' = w/(2N^2) ((0,0): Re w/N^2), into SF
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(kFxColCtas))
k_adj_qw_col_inv(Geom g, int zbase, const double2* __restrict__ BR, const double2* __restrict__ BI,
                 const double2* __restrict__ w, double2* __restrict__ SF, const double2* __restrict__ twg) {
  using F = FxCol<N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, kx = blockIdx.x * F::CT + c.c;
  const long long zoff = (long long)(zbase + zb) * g.plane;
  const double inv2n2 = 0.5 / ((double)N * (double)N);
#pragma unroll 1
  for (int f = blockIdx.z; f < 6; f += gridDim.z) {
    const double2* X = f < 2 ? BR : (f < 4 ? BI : w);
    adj_col_inverse<N>(c, g, kx, SF + scr_off(zb, f, 0, N, g.KXP), [&](int row, int ky) {
      double2 x = X[zoff + (long long)row * g.KXP + kx];
      const double fky = (double)ky;
      if (f >= 4) x = rt_scale(x, kx, ky, inv2n2);
      return f == 5 ? cscale(x, fky * fky) : ((f & 1) ? cscale(cmul_i(x), fky) : x);
    });
  }
}

// rows of the q^w transpose: P1 = BRy BIx - BRx BIy, P2 = BR^2 + BI^2 with
// q^w = s R(P1) - s kh^2/4 R(P2); writes (G_R, H_R, G_I, H_I) with
// lB = w_k [F_y(G) - i ky F_y(H)], G = -i kx F_x(a) + F_x(c), H = F_x(b)
template <int N>
__global__ void __launch_bounds__(FxRow<N>::NT, fx_row_ctas<N>(kFxRowCtas))
k_adj_qw_row(Geom g, AdjP p, double2* __restrict__ SF, const double2* __restrict__ twg) {
  using F = FxRow<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slots[F::SLOTS];
  FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, y = blockIdx.x * F::RT + c.rr, K = g.K, j = c.j;
  auto sf = [&](int f) { return SF + scr_off(zb, f, y, N, g.KXP); };
  const double s = p.s;
  fxc l[8], b[8], v[8];
  int2 el, eb;
  double2 X[8], Y[8];
  {
    const double2 *W1 = sf(4), *W2 = sf(5);
    adj_half<N>(j, K, X, Y, [&](int kk, double2& x, double2& y2) {
      const double2 w1 = W1[kk], w2 = W2[kk];
      x = cscale(w1, -s);
      y2 = cscale(cadd(cscale(w1, (double)kk * (double)kk), w2), 0.25 * s);
    });
    c.inverse(X, Y, l, el);        // l.y: lP1, l.x: lP2
  }
  auto bases = [&](int e, int ex, int ey) { return make_int2(fx_prod_base(e, ex), fx_prod_base(e, ey)); };
  // (a_R, a_I) = lP1 (-BIy, BRy)
  fx_half<N>(sf(1), sf(3), j, K, X, Y);
  c.inverse(X, Y, b, eb);
#pragma unroll
  for (int r = 0; r < 8; ++r) { v[r].x = -fx_mulhi(l[r].y, b[r].x); v[r].y = fx_mulhi(l[r].y, b[r].y); }
  double2 aR[3], aI[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) aR[q] = aI[q] = make_double2(0.0, 0.0);
  c.forward(v, bases(el.y, eb.x, eb.y), K, [&](int q, int, double2 R, double2 I) { aR[q] = R; aI[q] = I; });
  // (b_R, b_I) = lP1 (BIx, -BRx)
  fx_half<N>(sf(0), sf(2), j, K, X, Y);
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const double k = (double)(r < 4 ? j + r * NB : N - (j + r * NB));
    X[r] = make_double2(-k * X[r].y, k * X[r].x);
    Y[r] = make_double2(-k * Y[r].y, k * Y[r].x);
  }
  c.inverse(X, Y, b, eb);
#pragma unroll
  for (int r = 0; r < 8; ++r) { v[r].x = fx_mulhi(l[r].y, b[r].x); v[r].y = -fx_mulhi(l[r].y, b[r].y); }
  c.forward(v, bases(el.y, eb.x, eb.y), K, [&](int, int k, double2 R, double2 I) { sf(1)[k] = R; sf(3)[k] = I; });
  // (c_R, c_I) = 2 lP2 (BR, BI)
  fx_half<N>(sf(0), sf(2), j, K, X, Y);
  c.inverse(X, Y, b, eb);
#pragma unroll
  for (int r = 0; r < 8; ++r) { v[r].x = fx_mulhi(l[r].x, b[r].y); v[r].y = fx_mulhi(l[r].x, b[r].x); }
  c.forward(v, bases(el.x + 1, eb.y, eb.x), K, [&](int q, int k, double2 R, double2 I) {
    const double kx = (double)k;
    sf(0)[k] = cadd(cscale(cmul_mi(aR[q]), kx), R);
    sf(2)[k] = cadd(cscale(cmul_mi(aI[q]), kx), I);
  });
}

// final adds: lq += w, lB += A_solver(lA) (+ q^w transpose when with_qw)
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(kFxColCtas))
k_adj_qw_col_fwd(Geom g, int zbase, double2* __restrict__ lBR, double2* __restrict__ lBI, const double2* __restrict__ SF,
                 const double2* __restrict__ twg) {
  using F = FxCol<N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, kx = blockIdx.x * F::CT + c.c;
  const long long zoff = (long long)(zbase + zb) * g.plane;
  // (spread over gridDim.z = 2 CTAs: BR; BI)
  const int f0 = 2 * blockIdx.z, f1 = gridDim.z == 1 ? 4 : f0 + 2;
  double2 a[8];
#pragma unroll 1
  for (int f = f0; f < f1; ++f) {
    double2* lB = f < 2 ? lBR : lBI;
    adj_col_plane<N>(c, g, SF + scr_off(zb, f, 0, N, g.KXP), kx, [&](int r, long long mt, int ky, double2 h) {
      if ((f & 1) == 0) { a[r] = h; return; }
      // (a(0,0) is real; ky = 0 there, so the second term vanishes)
      double2* o = lB + zoff + mt;
      *o = cadd(*o, csub(a[r], cscale(cmul_i(h), (double)ky)));
    });
  }
}

// lq += w, lB += A_solver(lA) on the compact layout (zeros off the retained modes)
static __global__ void k_adj_solved(Geom g, long long tot, double2* __restrict__ lq, double2* __restrict__ lBR,
                                    double2* __restrict__ lBI, const double2* __restrict__ w,
                                    const double2* __restrict__ lBRa, const double2* __restrict__ lBIa) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const long long mm = i % g.plane;
    const int r = (int)(mm / g.KXP), kx = (int)(mm % g.KXP);
    const bool in = g.mask(kx, g.ky_of_row(r));
    const double2 z = make_double2(0.0, 0.0);
    lq[i] = in ? cadd(lq[i], w[i]) : z;
    lBR[i] = in ? cadd(lBR[i], lBRa[i]) : z;
    lBI[i] = in ? cadd(lBI[i], lBIa[i]) : z;
  }
}

// out = mask(a + s b) on the compact layout
static __global__ void k_adj_sum(Geom g, long long tot, const double2* __restrict__ a, const double2* __restrict__ b,
                                 double s, double2* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
    const long long mm = i % g.plane;
    const int r = (int)(mm / g.KXP), kx = (int)(mm % g.KXP);
    out[i] = g.mask(kx, g.ky_of_row(r)) ? cadd(a[i], cscale(b[i], s)) : make_double2(0.0, 0.0);
  }
}

}  // namespace qg
