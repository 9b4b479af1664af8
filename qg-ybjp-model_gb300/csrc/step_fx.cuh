// The FP64 step's transform kernels on block fixed-point FFTs (fxfft.cuh):
// the same five kernels as step_kernels.cuh's FP32 ones (k_col_inv,
// k_row_main, k_col_update, k_row_qw, k_col_qw), laid out for the integer
// pipes.
//
// What bounds them: integer issue (64-bit adds at 62, 32x32->64 multiply-adds
// at 30 lanes per clock and SM) and, beside it, the FP64 pipe at 2 lanes per
// clock, so everything that can be is done on the integers: the two real rows
// of a packed transform are multiplied and split as integers, powers of two
// (1/n^2, halves) go into the exponents, and one transform at a time is in
// flight per thread to keep registers, and with them warps, available.
#pragma once
#include "step_kernels.cuh"
#include "fxctx.cuh"

namespace qg {

#ifndef QG_FX_ROW_CTAS
#define QG_FX_ROW_CTAS 4
#endif
template <int N> __host__ __device__ constexpr int fx_row_ctas(int want) {
  return imax(1, (want * 128) / FxRow<N>::NT);
}

// ===========================================================================
// Rows of convol_waqg / refraction_waqg (k_row_main's planes and results)
// ===========================================================================
template <int N>
__global__ void __launch_bounds__(FxRow<N>::NT, fx_row_ctas<N>(QG_FX_ROW_CTAS))
k_fx_row_main(Geom g, StepParams sp, double2* __restrict__ S, const double2* __restrict__ twg, int nitems,
              const double2* __restrict__ Qb) {
  using F = FxRow<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int K = g.K, j = c.j;
  constexpr int NG = N / F::RT;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int zb = it / NG, y = (it % NG) * F::RT + c.rr;
    auto plane = [&](int f) -> double2* { return S + scr_off(zb, f, y, N, g.KXP); };
    fxc zq[8], bb[8], w[8];
    int ezq, ebb, euv;
    {
      double2 d[8];
      fx_pack<N>(plane(2), plane(3), j, K, d);
      c.inverse(d, zq, ezq);
    }
    {
      double2 d[8];
      const double2* pr = Qb ? Qb + q_off(zb, 0, y, N, g.KXP) : plane(4);
      const double2* pi = Qb ? Qb + q_off(zb, 1, y, N, g.KXP) : plane(5);
      fx_pack<N>(pr, pi, j, K, d);
      c.inverse(d, bb, ebb);
    }
    // refraction: (zeta br, zeta bi); half its spectra enter planes 2 and 4
    double2 zr[3], zi[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) zr[q] = zi[q] = make_double2(0.0, 0.0);
    if (sp.refr) {
#pragma unroll
      for (int r = 0; r < 8; ++r) { w[r].x = fx_mulhi(zq[r].y, bb[r].y); w[r].y = fx_mulhi(zq[r].y, bb[r].x); }
      // (one exponent less: the halves)
      c.forward(w, ezq + ebb - 1023 + 63, K, [&](int q, int, double2 X, double2 Y) { zr[q] = X; zi[q] = Y; });
    }
    fxc uv[8];
    {
      double2 d[8];
      fx_pack<N>(plane(0), plane(1), j, K, d);
      c.inverse(d, uv, euv);
    }
    // G = i kx F(uX) (+- refraction), H = F(vX); tendency = F_y(G) + i ky F_y(H)
#pragma unroll
    for (int f = 0; f < 3; ++f) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const long long x = f == 0 ? zq[r].x : (f == 1 ? bb[r].y : bb[r].x);
        w[r].x = fx_mulhi(uv[r].y, x);
        w[r].y = fx_mulhi(uv[r].x, x);
      }
      c.forward(w, euv + (f == 0 ? ezq : ebb) - 1023 + 64, K, [&](int q, int k, double2 X, double2 Y) {
        const double kx = (double)k;
        double2 G = make_double2(0.0, 0.0), H = G;
        if (sp.adv) {
          G = make_double2(-kx * X.y, kx * X.x);
          H = Y;
        }
        if (f == 1) { G.x -= zi[q].x; G.y -= zi[q].y; }
        if (f == 2) { G.x += zr[q].x; G.y += zr[q].y; }
        plane(2 * f)[k] = G;
        plane(2 * f + 1)[k] = H;
      });
    }
    // every row reads and writes its own entries of the planes only
  }
}

// ===========================================================================
// Rows of compute_qw (k_row_qw's planes and results)
// ===========================================================================
#ifndef QG_FX_QW_CTAS
#define QG_FX_QW_CTAS 5
#endif
template <int N>
__global__ void __launch_bounds__(FxRow<N>::NT, fx_row_ctas<N>(QG_FX_QW_CTAS))
k_fx_row_qw(Geom g, double2* __restrict__ S, const double2* __restrict__ twg, int nitems, const double2* __restrict__ Qb) {
  using F = FxRow<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int K = g.K, j = c.j;
  constexpr int NG = N / F::RT;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int zb = it / NG, y = (it % NG) * F::RT + c.rr;
    auto plane = [&](int f) -> double2* { return S + scr_off(zb, f, y, N, g.KXP); };
    const double2* pr = Qb ? Qb + q_off(zb, 0, y, N, g.KXP) : plane(0);
    const double2* pi = Qb ? Qb + q_off(zb, 1, y, N, g.KXP) : plane(2);
    fxc a[8], b[8], w[8];
    int ea, eb, e1, e2;
    {
      // (BRx, BIx): i kx times the packed spectrum of (BR, BI)
      double2 d[8];
      fx_pack<N>(pr, pi, j, K, d);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const double k = (double)(j + r * NB - (r < 4 ? 0 : N));
        d[r] = make_double2(-k * d[r].y, k * d[r].x);
      }
      c.inverse(d, a, ea);
    }
    {
      double2 d[8];
      fx_pack<N>(plane(1), plane(3), j, K, d);
      c.inverse(d, b, eb);
    }
    // P1 = BRy BIx - BRx BIy (derivatives.f90:973)
#pragma unroll
    for (int r = 0; r < 8; ++r) w[r].x = fx_mulhi(b[r].y, a[r].x) - fx_mulhi(a[r].y, b[r].x);
    e1 = ea + eb - 1023 + 64;
    {
      double2 d[8];
      fx_pack<N>(pr, pi, j, K, d);
      c.inverse(d, a, ea);
    }
    // P2 = BR^2 + BI^2 (derivatives.f90:996), then both to the larger exponent
    e2 = 2 * ea - 1023 + 64;
    const int s1 = min(max(e2 - e1, 0), 63), s2 = min(max(e1 - e2, 0), 63);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      w[r].x >>= s1;
      w[r].y = (fx_mulhi(a[r].y, a[r].y) + fx_mulhi(a[r].x, a[r].x)) >> s2;
    }
    c.forward(w, max(e1, e2), K, [&](int, int k, double2 P1, double2 P2) {
      const double qk = 0.25 * (double)(k * k);
      plane(0)[k] = make_double2(P1.x - qk * P2.x, P1.y - qk * P2.y);
      plane(1)[k] = P2;
    });
  }
}

// ===========================================================================
// Columns
// ===========================================================================
#ifndef QG_FX_COL_CTAS
#define QG_FX_COL_CTAS 6
#endif
template <int N> __host__ __device__ constexpr int fx_col_ctas(int want) { return imin(32, (want * 128) / FxCol<N>::NT); }

// y-inverse transforms of the fields f in [f0, f1) of (u, v, zeta, q, BR, BI)
// into the planes f of S; BR, BI into the kept planes Qb when given
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(QG_FX_COL_CTAS))
k_fx_col_inv(Geom g, int zbase, const double2* __restrict__ psi, const double2* __restrict__ q,
             const double2* __restrict__ BR, const double2* __restrict__ BI, double2* __restrict__ S,
             const double2* __restrict__ twg, double2* __restrict__ Qb, int f0, int f1) {
  using F = FxCol<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, kx = blockIdx.x * F::CT + c.c;
  const long long zoff = (long long)(zbase + zb) * g.plane;
  for (int f = f0; f < f1; ++f) {
    const double2* X = f < 3 ? psi : (f == 3 ? q : (f == 4 ? BR : BI));
    double2 d[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      d[r] = make_double2(0.0, 0.0);
      if (fx_zero_in<8>(r)) continue;
      int row; bool cj;
      col_src(g, kx, c.j + r * NB, row, cj);
      if (row < 0) continue;
      double2 x = X[zoff + (long long)row * g.KXP + kx];
      // u = -i ky psi (derivatives.f90:1309), v = i kx psi (1310), zeta = -kh^2 psi (842)
      const int ky = g.ky_of_row(row);
      if (f == 0) x = make_double2((double)ky * x.y, -(double)ky * x.x);
      else if (f == 1) x = make_double2(-(double)kx * x.y, (double)kx * x.x);
      else if (f == 2) { const double k2 = -(double)(kx * kx + ky * ky); x = make_double2(k2 * x.x, k2 * x.y); }
      if (cj) x.y = -x.y;
      d[r] = x;
    }
    fxc v[8];
    int base;
    c.template run<false>(d, v, base);
    if (kx > g.K) continue;
    double2 o[8];
    fx_doubles<8, true>(v, o, base);
    double2* dst = (Qb && f >= 4) ? Qb + q_off(zb, f - 4, 0, N, g.KXP) : S + scr_off(zb, f, 0, N, g.KXP);
    dst += (long long)c.j * g.KXP + kx;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      dst[(long long)r * NB * g.KXP] = o[r];
  }
}

// Forward transform of scratch plane h of a column tile, scaled by 1/N^2, at
// the retained rows: out[r] at FFT index j + r NB (r = 3, 4 hold no mode)
template <int N>
__device__ __forceinline__ void fx_col_plane(const FxColCtx<N>& c, const Geom& g, const double2* __restrict__ P, int kx,
                                             double2 (&out)[8]) {
  constexpr int NB = N / 8;
  double2 d[8];
  const bool in = kx <= g.K;
  const double2* p = P + (long long)c.j * g.KXP + kx;
#pragma unroll
  for (int r = 0; r < 8; ++r) d[r] = in ? p[(long long)r * NB * g.KXP] : make_double2(0.0, 0.0);
  fxc v[8];
  int base;
  c.template run<true>(d, v, base);
  fx_doubles<8, false>(v, out, base - 2 * fx_ilog2(N));     // (out[3], out[4] are not used)
}

// y-forward transforms, time update, y-inverse transforms of B^{n+1} and
// i ky B^{n+1} (k_col_update)
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(QG_FX_COL_CTAS))
k_fx_col_update(Geom g, StepParams sp, int zbase, StateP<double> st, const double* __restrict__ e1t,
                const double* __restrict__ e2t, const double* __restrict__ e1wt, const double* __restrict__ e2wt,
                double2* __restrict__ S, const double2* __restrict__ twg, int qw_prep, double2* __restrict__ Qb) {
  using F = FxCol<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, z = zbase + zb, kx = blockIdx.x * F::CT + c.c;
  const long long zoff = (long long)z * g.plane;
  const int mem = sp.mpar ? z / g.nseg : 0;          // ensemble member of this level (stacks)
  if (sp.mpar) {
    const long long to = (long long)mem * g.plane;
    e1t += to; e2t += to; e1wt += to; e2wt += to;
  }
  const double dt = sp.mpar ? sp.mpar[4 * mem] : sp.delt;
  const double cdisp = sp.disp ? (sp.mpar ? sp.mpar[4 * mem + 1] : sp.cdisp) : 0.0;
  const double gam = sp.gamma, dt2 = 2.0 * dt;
  const bool eul = sp.euler != 0;
  for (int which = 0; which < 3; ++which) {
    double2 G[8], H[8];
    fx_col_plane<N>(c, g, S + scr_off(zb, 2 * which + 1, 0, N, g.KXP), kx, H);
    fx_col_plane<N>(c, g, S + scr_off(zb, 2 * which, 0, N, g.KXP), kx, G);
    if (kx > g.K) continue;
    double2* X = which == 0 ? st.q : (which == 1 ? st.BR : st.BI);
    double2* Xo = which == 0 ? st.qo : (which == 1 ? st.BRo : st.BIo);
    const double2* X3 = which == 0 ? st.dq : (which == 1 ? st.AI : st.AR);
    const double* t1 = which == 0 ? e1t : e1wt;
    const double* t2 = which == 0 ? e2t : e2wt;
    const bool need3 = which != 0 || sp.use_dq;
    // time update (main_waqg.f90:237-264, 362-415), one mode per output index
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (fx_zero_in<8>(r)) continue;
      const int row = g.row_of_fft_index(c.j + r * NB);
      if (row < 0) continue;
      const int ky = g.ky_of_row(row);
      const long long mt = (long long)row * g.KXP + kx, m = zoff + mt;
      const double fky = (double)ky;
      const double2 tnd = make_double2(G[r].x - fky * H[r].y, G[r].y + fky * H[r].x);   // G + i ky H
      const double2 x0 = X[m];
      const double2 xo = eul ? x0 : Xo[m];
      double2 xn = make_double2(0.0, 0.0), xf = eul ? xo : xn;
      const bool live = g.mask(kx, ky);
      if (live) {
        const double2 x3 = need3 ? X3[m] : make_double2(0.0, 0.0);
        const double e1 = t1[mt], e2 = t2[mt];
        if (which == 0) {
          if (eul) xn = cscale(cadd(csub(xo, cscale(tnd, dt)), cscale(x3, dt)), e1);
          else xn = cadd(csub(cscale(xo, e2), cscale(cscale(tnd, dt2), e1)), cscale(cscale(x3, dt2), e2));
        } else {
          // nBR - 0.5 rBI + c kh2 AI ; nBI + 0.5 rBR - c kh2 AR
          const double ck = cdisp * (double)(kx * kx + ky * ky);
          const double2 fr = which == 1 ? cadd(tnd, cscale(x3, ck)) : csub(tnd, cscale(x3, ck));
          if (eul) xn = cscale(csub(xo, cscale(fr, dt)), e1);
          else xn = csub(cscale(xo, e2), cscale(cscale(fr, dt2), e1));
        }
        // Robert-Asselin filter (main_waqg.f90:395-410)
        if (!eul) xf = cadd(x0, cscale(cadd(csub(xo, cscale(x0, 2.0)), xn), gam));
      }
      X[m] = xn;
      Xo[m] = xf;
      if (!sp.ybj && which > 0) {
        // compute_sigma (derivatives.f90:1037-1068): see k_col_update
        const int kh2 = kx * kx + ky * ky;
        double2 sv = make_double2(0.0, 0.0);
        if (kh2 > 0 && live) sv = cscale(tnd, (which == 2 ? 2.0 : -2.0) / (double)kh2);
        (which == 2 ? st.sig1 : st.sig2)[m] = sv;
      }
    }
  }
  if (!qw_prep) return;
  __syncthreads();
  // y-inverse transforms of B and i ky B at n+1 (compute_qw,
  // derivatives.f90:929-957) from this CTA's own stores: planes (BR, i ky BR,
  // BI, i ky BI) = 0..3, BR and BI to the kept planes when given
  for (int p = 0; p < 4; ++p) {
    const double2* X = (p >> 1) == 0 ? st.BR : st.BI;
    double2 d[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      d[r] = make_double2(0.0, 0.0);
      if (fx_zero_in<8>(r)) continue;
      int row; bool cj;
      col_src(g, kx, c.j + r * NB, row, cj);
      if (row < 0) continue;
      double2 x = X[zoff + (long long)row * g.KXP + kx];
      if (p & 1) { const double ky = (double)g.ky_of_row(row); x = make_double2(-ky * x.y, ky * x.x); }
      if (cj) x.y = -x.y;
      d[r] = x;
    }
    fxc v[8];
    int base;
    c.template run<false>(d, v, base);
    if (kx > g.K) continue;
    double2 o[8];
    fx_doubles<8, true>(v, o, base);
    double2* dst = (Qb && (p & 1) == 0) ? Qb + q_off(zb, p >> 1, 0, N, g.KXP) : S + scr_off(zb, p, 0, N, g.KXP);
    dst += (long long)c.j * g.KXP + kx;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      dst[(long long)r * NB * g.KXP] = o[r];
  }
}

// y-forward transforms of the q^w planes, q* = q - q^w (k_col_qw)
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(QG_FX_COL_CTAS))
k_fx_col_qw(Geom g, StepParams sp, int zbase, const double2* __restrict__ q, double2* __restrict__ qstar,
            const double2* __restrict__ S, const double2* __restrict__ twg, int* __restrict__ nflag) {
  using F = FxCol<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, z = zbase + zb, kx = blockIdx.x * F::CT + c.c;
  const long long zoff = (long long)z * g.plane;
  const int mem = sp.mpar ? z / g.nseg : 0;          // ensemble member of this level (stacks)
  const double s = sp.mpar ? sp.mpar[4 * mem + 2] * sp.mpar[4 * mem + 3] : sp.Ro * sp.W2F;
  double2 A[8], B[8];
  fx_col_plane<N>(c, g, S + scr_off(zb, 0, 0, N, g.KXP), kx, A);
  fx_col_plane<N>(c, g, S + scr_off(zb, 1, 0, N, g.KXP), kx, B);
  bool bad = false;       // a non-finite q* (the state has blown up)
  if (kx <= g.K) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (fx_zero_in<8>(r)) continue;
      const int row = g.row_of_fft_index(c.j + r * NB);
      if (row < 0) continue;
      const int ky = g.ky_of_row(row);
      const long long m = zoff + (long long)row * g.KXP + kx;
      double2 out = make_double2(0.0, 0.0);
      if (g.mask(kx, ky)) {
        const double2 R = csub(A[r], cscale(B[r], 0.25 * (double)ky * (double)ky));
        out = csub(q[m], cscale(R, s));       // q* = q - q^w (main_waqg.f90:430-439)
        bad |= !isfinite(out.x) || !isfinite(out.y);
      }
      qstar[m] = out;
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) raise_wait_flag(nflag);
}

}  // namespace qg
