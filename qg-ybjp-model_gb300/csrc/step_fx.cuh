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

// CTAs per SM (of 128 threads) that the register budgets of the row and column
// kernels target
constexpr int kFxRowCtas = 4, kFxColCtas = 7;
template <int N, int T = 128> __host__ __device__ constexpr int fx_row_ctas(int want) {
  return imin(32, imax(1, (want * 128) / FxRow<N, T>::NT));
}

// ===========================================================================
// Rows of convol_waqg / refraction_waqg (k_row_main's planes and results)
// ===========================================================================
// 256 threads, so that two CTAs' shared memory (transform buffers, and the
// physical zeta, q, BR, BI parked as integers, each thread its own eight
// points) fits an SM with one twiddle table each
constexpr int kFxMainT = 256;
template <int N> struct FxMain {
  using F = FxRow<N, kFxMainT>;
  static constexpr size_t smem() { return (size_t)(fx_tw_count<N>() + F::RT * F::LD + 2 * F::RT * N) * sizeof(double2); }
};
template <int N>
__global__ void __launch_bounds__(FxMain<N>::F::NT, fx_row_ctas<N, kFxMainT>(kFxRowCtas))
k_fx_row_main(Geom g, StepParams sp, double2* __restrict__ S, const double2* __restrict__ twg, int nitems,
              const double2* __restrict__ Qb) {
  using F = typename FxMain<N>::F;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slots[F::SLOTS];
  FxRowCtx<N, kFxMainT> c = fx_row_ctx<N, kFxMainT>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  fxc* zq = reinterpret_cast<fxc*>(smem_raw) + fx_tw_count<N>() + F::RT * F::LD + threadIdx.x;   // point r at zq[r * NT]
  fxc* bb = zq + 8 * F::NT;
  const int K = g.K, j = c.j;
  constexpr int NG = N / F::RT;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int zb = it / NG, y = (it % NG) * F::RT + c.rr;
    auto plane = [&](int f) -> double2* { return S + scr_off(zb, f, y, N, g.KXP); };
    // inverse transforms of (zeta, q), (BR, BI), parked, and (u, v); then the
    // forward transforms of (zeta br, zeta bi) (refraction) and of u and v
    // times q, br, bi.  Two copies of the transform, each in a loop: with one
    // per use the kernel's code outgrew the instruction cache, with one copy
    // for both directions the loop's selects cost as much
    fxc uv[8];
    int2 ezq = make_int2(0, 0), ebb = ezq, euv = ezq;      // (.y: zeta, BR, u; .x: q, BI, v)
#pragma unroll 1
    for (int t = 0; t < 3; ++t) {
      const double2 *X = plane(0), *Y = plane(1);
      if (t == 0) { X = plane(2); Y = plane(3); }
      else if (t == 1) { X = Qb ? Qb + q_off(zb, 0, y, N, g.KXP) : plane(4); Y = Qb ? Qb + q_off(zb, 1, y, N, g.KXP) : plane(5); }
      double2 a[8], b[8];
      fx_half<N>(X, Y, j, K, a, b);
      c.inverse(a, b, uv, euv);
      if (t < 2) {
        if (t == 0) ezq = euv;
        else ebb = euv;
        fxc* pk = t == 0 ? zq : bb;
#pragma unroll
        for (int r = 0; r < 8; ++r) pk[r * F::NT] = uv[r];
      }
    }
#pragma unroll 1
    for (int f = sp.refr ? -1 : 0; f < 3; ++f) {
      fxc w[8];
      int2 base;
      if (f < 0) {
        // (one exponent less: half of the spectra enters planes 2 and 4)
        base = make_int2(fx_prod_base(ezq.y, ebb.y) - 1, fx_prod_base(ezq.y, ebb.x) - 1);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const long long z = zq[r * F::NT].y;
          const fxc b = bb[r * F::NT];
          w[r].x = fx_mulhi(z, b.y);
          w[r].y = fx_mulhi(z, b.x);
        }
      } else {
        const int ex = f == 0 ? ezq.x : (f == 1 ? ebb.y : ebb.x);
        base = make_int2(fx_prod_base(euv.y, ex), fx_prod_base(euv.x, ex));
        const long long* px = f == 0 ? &zq->x : (f == 1 ? &bb->y : &bb->x);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const long long x = px[2 * r * F::NT];
          w[r].x = fx_mulhi(uv[r].y, x);
          w[r].y = fx_mulhi(uv[r].x, x);
        }
      }
      c.forward(w, base, K, [&](int, int k, double2 X, double2 Y) {
        // the refraction's halves wait in the planes that they go to, read
        // already (in registers they spilled: 512^2 x 256 6910 -> 6480 us)
        if (f < 0) { plane(4)[k] = X; plane(2)[k] = Y; return; }
        // G = i kx F(uX) (+- refraction), H = F(vX); tendency = F_y(G) + i ky F_y(H)
        const double kx = (double)k;
        double2 G = make_double2(0.0, 0.0), H = G;
        if (sp.adv) { G = make_double2(-kx * X.y, kx * X.x); H = Y; }
        if (f > 0 && sp.refr) {
          const double2 z = plane(2 * f)[k];
          G = f == 1 ? csub(G, z) : cadd(G, z);
        }
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
// (BRx, BIx) are parked in shared memory, each thread its own eight points: in
// registers beside two rows' spectra they spilled (us per launch, registers ->
// shared: 128^2 x 64 57 -> 53, 256^2 x 128 460 -> 432, 512^2 x 256 3730 -> 3490)
template <int N> struct FxQw {
  using F = FxRow<N>;
  static constexpr size_t smem() { return F::smem() + (size_t)F::RT * N * sizeof(fxc); }
};
// CTAs per SM that its register budget targets: three leave it 168 registers.
// us per launch, four -> three: 64^2 x 64 20.4 -> 18.3, 128^2 x 64 59 -> 53,
// 256^2 x 16 61 -> 55 (x 128 426 -> 432), 16^2 and 32^2 the same; 512^2 x 128
// 1730 -> 1750, 1024^2 x 16 1028 -> 1020 (two and four warps per row)
template <int N> __host__ __device__ constexpr int fx_qw_ctas() { return fx_row_ctas<N>(N >= 512 ? 4 : 3); }
template <int N>
__global__ void __launch_bounds__(FxRow<N>::NT, fx_qw_ctas<N>())
k_fx_row_qw(Geom g, double2* __restrict__ S, const double2* __restrict__ twg, int nitems, const double2* __restrict__ Qb) {
  using F = FxRow<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint2 slots[F::SLOTS];
  FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  fxc* park = reinterpret_cast<fxc*>(smem_raw) + fx_tw_count<N>() + F::RT * F::LD + threadIdx.x;   // point r at park[r * NT]
  const int K = g.K, j = c.j;
  constexpr int NG = N / F::RT;
  for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
    const int zb = it / NG, y = (it % NG) * F::RT + c.rr;
    auto plane = [&](int f) -> double2* { return S + scr_off(zb, f, y, N, g.KXP); };
    const double2* pr = Qb ? Qb + q_off(zb, 0, y, N, g.KXP) : plane(2);
    const double2* pi = Qb ? Qb + q_off(zb, 1, y, N, g.KXP) : plane(4);
    // inverse transforms of (BRx, BIx), (BRy, BIy), (BR, BI), then the forward
    // transform of (P1, P2), through one copy of the transform
    fxc w[8];
    long long p[8];
    int2 ea = make_int2(0, 0), base = ea;     // (.y: BRx, BRy, BR; .x: BIx, BIy, BI; then P2 and P1)
    int ep = 0;
#pragma unroll 1
    for (int t = 0; t < 4; ++t) {
      if (t < 3) {
        double2 X[8], Y[8];
        fx_half<N>(t == 1 ? plane(3) : pr, t == 1 ? plane(5) : pi, j, K, X, Y);
        if (t == 0) {
          // i kx times both
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const double k = (double)(r < 4 ? j + r * NB : N - (j + r * NB));
            X[r] = make_double2(-k * X[r].y, k * X[r].x);
            Y[r] = make_double2(-k * Y[r].y, k * Y[r].x);
          }
        }
        base = c.template ints_inverse<true>(X, Y, w);
      } else {
        fx_norm<8, 59>(w, c.template reduce<true>(fx_bits2<8>(w)), base);
      }
      c.template core<true>(w, base);
      if (t < 3) fx_norm<8, 61>(w, c.template reduce<true>(fx_bits2<8>(w)), base);
      if (t == 0) {
#pragma unroll
        for (int r = 0; r < 8; ++r) park[r * F::NT] = w[r];
        ea = base;
      } else if (t == 1) {
        // P1 = BRy BIx - BRx BIy (derivatives.f90:973)
        const FxAlign al(fx_prod_base(base.y, ea.x), fx_prod_base(ea.y, base.x));
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const fxc a = park[r * F::NT];
          p[r] = al.sub(fx_mulhi(w[r].y, a.x), fx_mulhi(a.y, w[r].x));
        }
        ep = al.e;
      } else if (t == 2) {
        // P2 = BR^2 + BI^2 (derivatives.f90:996)
        const FxAlign al(fx_prod_base(base.y, base.y), fx_prod_base(base.x, base.x));
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          w[r].y = al.add(fx_mulhi(w[r].y, w[r].y), fx_mulhi(w[r].x, w[r].x));
          w[r].x = p[r];
        }
        base = make_int2(ep, al.e);
      } else {
        c.template split<3>(w, base, K, [&](int, int k, double2 P1, double2 P2) {
          const double qk = 0.25 * (double)(k * k);
          plane(3)[k] = make_double2(P1.x - qk * P2.x, P1.y - qk * P2.y);
          plane(5)[k] = P2;
        });
      }
    }
  }
}

// ===========================================================================
// Columns
// ===========================================================================
template <int N> __host__ __device__ constexpr int fx_col_ctas(int want) { return imin(32, (want * 128) / FxCol<N>::NT); }

// y-inverse transforms of the fields f in [f0, f1) of (u, v, zeta, q, BR, BI)
// into the planes f of S; BR, BI into the kept planes Qb when given; a tile's
// fields over `split` CTAs
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(kFxColCtas))
k_fx_col_inv(Geom g, int zbase, const double2* __restrict__ psi, const double2* __restrict__ q,
             const double2* __restrict__ BR, const double2* __restrict__ BI, double2* __restrict__ S,
             const double2* __restrict__ twg, double2* __restrict__ Qb, int f0, int f1, int split) {
  using F = FxCol<N>;
  constexpr int NB = F::NB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned slots[F::SLOTS];
  const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
  const int zb = blockIdx.y, kx = (int)(blockIdx.x / split) * F::CT + c.c;
  const long long zoff = (long long)(zbase + zb) * g.plane;
#pragma unroll 1
  for (int f = f0 + (int)blockIdx.x % split; f < f1; f += split) {
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
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(kFxColCtas))
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
  // H and G of one of q, BR, BI, then the y-inverse transforms of B and i ky B
  // at n+1 (compute_qw, derivatives.f90:929-957: planes BR, i ky BR, BI,
  // i ky BI = 2..5, which this CTA alone has read, BR and BI to the kept
  // planes when given), through one copy of the transform
  double2 H[8];
  // (a CTA per variable: the chain of the ten transforms of a tile bounded
  // small grids, 65.5 -> 32.8 us at 64^2 x 64; 512^2 x 256 the same)
  const int which = blockIdx.z, nt = qw_prep && which ? 4 : 2;
#pragma unroll 1
  for (int t = 0; t < nt; ++t) {
    double2 d[8];
    fxc v[8];
    int base;
    if (t < 2) {
      const double2* p = S + scr_off(zb, 2 * which + 1 - t, 0, N, g.KXP) + (long long)c.j * g.KXP + kx;
#pragma unroll
      for (int r = 0; r < 8; ++r) d[r] = kx <= g.K ? p[(long long)r * NB * g.KXP] : make_double2(0.0, 0.0);
      base = c.template load<true>(d, v);
    } else {
      if (t == 2) __syncthreads();      // B^{n+1}: this CTA's own stores
      const double2* X = which == 1 ? st.BR : st.BI;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        d[r] = make_double2(0.0, 0.0);
        if (fx_zero_in<8>(r)) continue;
        int row; bool cj;
        col_src(g, kx, c.j + r * NB, row, cj);
        if (row < 0) continue;
        double2 x = X[zoff + (long long)row * g.KXP + kx];
        if (t & 1) { const double ky = (double)g.ky_of_row(row); x = make_double2(-ky * x.y, ky * x.x); }
        if (cj) x.y = -x.y;
        d[r] = x;
      }
      base = c.template load<false>(d, v);
    }
    c.core(v, base);
    if (kx > g.K) continue;
    if (t >= 2) {
      fx_doubles<8, true>(v, d, base);
      double2* dst = (Qb && t == 2) ? Qb + q_off(zb, which - 1, 0, N, g.KXP) : S + scr_off(zb, 2 * which + t - 2, 0, N, g.KXP);
      dst += (long long)c.j * g.KXP + kx;
#pragma unroll
      for (int r = 0; r < 8; ++r) dst[(long long)r * NB * g.KXP] = d[r];
      continue;
    }
    fx_doubles<8, false>(v, d, base - 2 * fx_ilog2(N));     // (d[3], d[4] are not used)
    if (t == 0) {
#pragma unroll
      for (int r = 0; r < 8; ++r) H[r] = d[r];
      continue;
    }
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
      const double2 tnd = make_double2(d[r].x - fky * H[r].y, d[r].y + fky * H[r].x);   // G + i ky H
      const double2 x0 = X[m];
      const double2 xo = eul ? x0 : Xo[m];
      double2 xn = make_double2(0.0, 0.0), xf = eul ? xo : xn;
      const bool live = g.mask(kx, ky);
      if (live) {
        const double2 x3 = need3 ? X3[m] : make_double2(0.0, 0.0);
        const double e1 = t1[mt], e2 = t2[mt];
        // q: tnd - dq; BR: nBR - 0.5 rBI + c kh2 AI; BI: nBI + 0.5 rBR - c kh2 AR
        const double ck = which == 0 ? 0.0 : (which == 1 ? cdisp : -cdisp) * (double)(kx * kx + ky * ky);
        const double2 fr = cadd(tnd, cscale(x3, ck));
        if (eul) {
          xn = csub(xo, cscale(fr, dt));
          if (which == 0 && sp.use_dq) xn = cadd(xn, cscale(x3, dt));
          xn = cscale(xn, e1);
        } else {
          xn = csub(cscale(xo, e2), cscale(fr, dt2 * e1));
          if (which == 0 && sp.use_dq) xn = cadd(xn, cscale(x3, dt2 * e2));
          // Robert-Asselin filter (main_waqg.f90:395-410)
          xf = cadd(x0, cscale(cadd(csub(xo, cscale(x0, 2.0)), xn), gam));
        }
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
}

// y-forward transforms of the q^w planes, q* = q - q^w (k_col_qw)
template <int N>
__global__ void __launch_bounds__(FxCol<N>::NT, fx_col_ctas<N>(kFxColCtas))
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
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    if (h == 1) {
#pragma unroll
      for (int r = 0; r < 8; ++r) A[r] = B[r];
    }
    fx_col_plane<N>(c, g, S + scr_off(zb, 3 + 2 * h, 0, N, g.KXP), kx, B);
  }
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
