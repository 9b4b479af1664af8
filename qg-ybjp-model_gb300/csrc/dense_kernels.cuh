// Kernels behind the routine-level drop-ins (fft_r2c, fft_c2r, convol_waqg,
// refraction_waqg, compute_qw): unpruned 2D transforms on the reference's
// dense half-spectrum layout, so arbitrary (also unmasked) inputs give what
// the Fortran routines give.
#pragma once
#include "step_kernels.cuh"
#include "fxctx.cuh"

namespace qg {

// dense spectral: double2 [nz][n][iktx]; W: cplx<T> [nz][n(y)][iktxP]; phys: T [nz][n][n]

// CTAs per SM (of 128 threads) that the fixed-point kernels' register budgets target
constexpr int kDenseColCtas = 6, kDenseRowCtas = 4;

// small integers (|k| < 2^24) as doubles, off the FP64 pipe
__device__ __forceinline__ double int_to64(int k) { return f32_to_f64((float)k); }

// Column tiles of CT columns, rows in pairs (one packed complex transform
// each), RT pairs per CTA with one first-pass butterfly per thread; doubles
// on the block fixed-point contexts (fxctx.cuh).
template <typename T, int N> struct Dense {
  static constexpr bool FX = sizeof(T) == 8;
  static constexpr int CT = FX ? FxCol<N>::CT : Tiles<T, N>::CT, CNT = FX ? FxCol<N>::NT : Tiles<T, N>::CNT;
  static constexpr int NB = FX ? N / 8 : N / radix_of(N);
  static constexpr int RT = FX ? imin(FxRow<N>::RT, N / 2) : imin(N / 2, imax(1, 256 / NB));
  static constexpr int RNT = FX ? FxRow<N>::NT : RT * NB;
  static constexpr int CMINB = FX ? imin(32, (kDenseColCtas * 128) / CNT) : 1;
  static constexpr int RMINB = FX ? imin(32, imax(1, (kDenseRowCtas * 128) / RNT)) : 1;
  static constexpr int LD = FX ? FxRow<N>::LD : PadLD<N>::value;
  static constexpr size_t sm_col(int nf = 1) { return FX ? FxCol<N>::smem() : (size_t)(N + nf * ColLay<N, CT>::FS) * sizeof(cplx<T>); }
  static constexpr size_t sm_row() { return FX ? FxRow<N>::smem() : (size_t)(N + RT * LD) * sizeof(cplx<T>); }
};
// row length of the (kx, y) intermediate: whole column tiles of every n
__host__ __device__ constexpr int dense_kxp(int n) { return n < 32 ? 16 : (n / 2 + 1 + 7) / 8 * 8; }
// The intermediate: plane f of level z, np planes per level
__device__ __forceinline__ long long dense_plane(int z, int np, int f, int n, int kxp) {
  return ((long long)z * np + f) * n * kxp;
}

// a flat index of the reference's layout: mode and ky row
__device__ __forceinline__ void dense_mode(long long m, int n, int& kx, int& ky, int& iky) {
  const int iktx = n / 2 + 1;
  iky = (int)((m / iktx) % n);
  kx = (int)(m % iktx);
  ky = iky < n / 2 ? iky : (iky == n / 2 ? 0 : iky - n);
}
__device__ __forceinline__ bool dense_L(int kx, int ky, int iky, int n, int kmax2) {
  return iky != n / 2 && kx * kx + ky * ky <= kmax2 && !(kx == 0 && ky < 0);
}

// ---- sources of the column transforms: the value of field f at (z, FFT index
// i, kx).  realit (fft.f90:88-107): the kx = 0 entries of negative ky are the
// conjugates of the positive ones.
// fields of the reference's layout under a spectral operator (masked by L
// unless OP_ID)
enum { OP_ID = 0, OP_LAP, OP_IKX, OP_IKY };       // a, -kh^2 a, i kx a, i ky a
constexpr int kDenseFields = 6;
struct DenseIn {
  const double2* p[kDenseFields];
  int op[kDenseFields];
  int kmax2;
  __device__ __forceinline__ bool zero(int f, int kx0) const { return op[f] != OP_ID && kx0 * kx0 > kmax2; }
  template <typename T, int N> __device__ __forceinline__ cplx<T> get(int f, long long z, int i, int kx) const {
    constexpr int IKTX = N / 2 + 1;
    const bool cj = kx == 0 && i > N / 2;
    if (kx >= IKTX) return mk<T>(0, 0);
    const int s = cj ? N - i : i;
    double2 d = make_double2(0.0, 0.0);
    if (op[f] == OP_ID) {
      d = p[f][(z * N + s) * IKTX + kx];
    } else {
      const int ky = s < N / 2 ? s : s - N;
      if (dense_L(kx, ky, s, N, kmax2)) {
        d = p[f][(z * N + s) * IKTX + kx];
        if (op[f] == OP_LAP) { const double k2 = -(double)(kx * kx + ky * ky); d = make_double2(k2 * d.x, k2 * d.y); }
        else { const double k = op[f] == OP_IKX ? (double)kx : (double)ky; d = make_double2(-k * d.y, k * d.x); }
      }
    }
    return mk<T>((T)d.x, cj ? -(T)d.y : (T)d.y);
  }
};
// resident fields (output path): a, or LA = B + 0.25 kh2 A / Bu
// (diagnostics.f90:1698-1727), left to right, where b is given
template <typename TS> struct CompactIn {
  Geom g;
  int level0;
  const cplx<TS> *a[2], *b[2];
  Divisor Bu;
  __device__ __forceinline__ bool zero(int, int) const { return false; }
  template <typename T, int N> __device__ __forceinline__ cplx<T> get(int f, long long z, int i, int kx) const {
    int row; bool cj;
    col_src(g, kx, i, row, cj);
    if (row < 0) return mk<T>(0, 0);
    const long long m = (level0 + z) * g.plane + (long long)row * g.KXP + kx;
    const cplx<TS> x = a[f][m];
    double2 d = make_double2(to64<TS>(x.x), to64<TS>(x.y));
    if (b[f]) {
      const int ky = g.ky_of_row(row);
      if (g.mask(kx, ky)) {
        const double c = 0.25 * int_to64(kx * kx + ky * ky);
        const cplx<TS> y = b[f][m];
        d = make_double2(__dadd_rn(d.x, Bu.quot(__dmul_rn(c, to64<TS>(y.x)))),
                         __dadd_rn(d.y, Bu.quot(__dmul_rn(c, to64<TS>(y.y)))));
      } else {
        d = make_double2(0.0, 0.0);
      }
    }
    return mk<T>(from64<T>(d.x), cj ? -from64<T>(d.y) : from64<T>(d.y));
  }
};
// Omega equation right-hand side, spectral part (derivatives.f90:1489-1560):
// psi_z at the unstaggered level between z and z+1 (0 at the top level),
// fields i kx psi_z, -i ky kh2 psi_avg, i ky psi_z, -i kx kh2 psi_avg with
// psi_avg = (psi(z+1) + psi(z))/2, psi at the top level itself; psi from the
// reference's layout (dense) or the resident field
template <typename TS> struct OmegaIn {
  Geom g;
  const double2* dense;
  const cplx<TS>* psi;
  Divisor dz;
  __device__ __forceinline__ bool zero(int, int kx0) const { return kx0 > g.K; }
  template <int N> __device__ __forceinline__ double2 at(long long z, int ky, int kx) const {
    if (dense) return dense[(z * N + (ky < 0 ? ky + N : ky)) * (N / 2 + 1) + kx];
    const cplx<TS> v = psi[z * g.plane + (long long)g.row_of_ky(ky) * g.KXP + kx];
    return make_double2(to64<TS>(v.x), to64<TS>(v.y));
  }
  template <typename T, int N> __device__ __forceinline__ cplx<T> get(int f, long long z, int i, int kx) const {
    const bool cj = kx == 0 && i > N / 2;
    const int s = cj ? N - i : i, ky = s < N / 2 ? s : s - N;
    if (s == N / 2 || !g.mask(kx, ky)) return mk<T>(0, 0);
    const bool top = z == g.n3 - 1;
    const double2 p0 = at<N>(z, ky, kx);
    const double k = int_to64(f == 0 || f == 3 ? kx : ky);
    double2 v = make_double2(0.0, 0.0);
    if (!(f & 1)) {
      if (!top) {
        const double2 p1 = at<N>(z + 1, ky, kx);
        const double2 rz = make_double2(dz.quot(__dsub_rn(p1.x, p0.x)), dz.quot(__dsub_rn(p1.y, p0.y)));
        v = make_double2(-k * rz.y, k * rz.x);
      }
    } else {
      const double kh2 = int_to64(kx * kx + ky * ky);
      if (!top) {
        const double2 p1 = at<N>(z + 1, ky, kx);
        const double2 sm = make_double2(p1.x + p0.x, p1.y + p0.y);
        const double c = k * kh2 * 0.5;
        v = make_double2(c * sm.y, -c * sm.x);
      } else {
        const double c = k * kh2;
        v = make_double2(c * p0.y, -c * p0.x);
      }
    }
    return mk<T>(from64<T>(v.x), cj ? -from64<T>(v.y) : from64<T>(v.y));
  }
};

// y-inverse transforms of field blockIdx.z of the source into plane
// blockIdx.z (np planes per level)
template <typename T, int N, class Src>
__global__ void __launch_bounds__(Dense<T, N>::CNT, Dense<T, N>::CMINB)
k_dcol_inv(int iktxP, int np, Src src, cplx<T>* __restrict__ W, const cplx<T>* __restrict__ twg) {
  constexpr int CT = Dense<T, N>::CT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int z = blockIdx.y, kx0 = blockIdx.x * CT, f = blockIdx.z;
  W += dense_plane(z, np, f, N, iktxP);
  if (src.zero(f, kx0)) {
    for (int e = threadIdx.x; e < N * CT; e += Dense<T, N>::CNT) W[(e / CT) * iktxP + kx0 + e % CT] = mk<T>(0, 0);
    return;
  }
  if constexpr (Dense<T, N>::FX) {
    constexpr int NB = N / 8;
    __shared__ unsigned slots[FxCol<N>::SLOTS];
    const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
    const int kx = kx0 + c.c;
    double2 d[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) d[r] = src.template get<T, N>(f, z, c.j + r * NB, kx);
    fxc v[8];
    int base;
    c.template run<false, false>(d, v, base);
    fx_doubles<8, true>(v, d, base);
#pragma unroll
    for (int r = 0; r < 8; ++r) W[(c.j + r * NB) * iktxP + kx] = d[r];
  } else {
    constexpr int NT = Dense<T, N>::CNT, R0 = radix_of(N), NB0 = N / R0, NSL = LastNS<N>::value, RL = N / NSL;
    cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
    cplx<T>* sm = tw + N;
    load_tw<T, N>(tw, twg, NT);
    auto pro = [&](int c, int j, cplx<T> (&v)[1][R0]) {
#pragma unroll
      for (int r = 0; r < R0; ++r) v[0][r] = src.template get<T, N>(f, z, j + r * NB0, kx0 + c);
    };
    auto epi = [&](int c, int j, cplx<T> (&v)[1][RL]) {
#pragma unroll
      for (int r = 0; r < RL; ++r) W[(j + r * NSL) * iktxP + kx0 + c] = v[0][r];
    };
    __syncthreads();
    col_fft<T, N, false, 1, CT, NT>(sm, tw, pro, epi);
  }
}

// Hermitian extension of two half spectra with kx in [0, n/2] (the Nyquist
// entry, like kx=0, contributes its real part only, as FFTW's c2r does);
// zeros past kx = KM.
template <typename T>
__device__ __forceinline__ cplx<T> pack_full(const cplx<T>* X, const cplx<T>* Y, int k, int n, int KM) {
  const int kk = k <= n / 2 ? k : n - k;
  if (kk > KM) return mk<T>(0, 0);
  const cplx<T> a = X[kk], b = Y[kk];
  if (k == 0 || k == n / 2) return mk<T>(a.x, b.x);
  return k < n / 2 ? mk<T>(a.x - b.y, a.y + b.x) : mk<T>(a.x + b.y, b.x - a.y);
}

// the half spectra X, Y of two rows with kx in [0, n/2] as fx_half's, zeros
// past kx = KM; real at kx = 0 and n/2
template <int N>
__device__ __forceinline__ void half_full(const double2* X, const double2* Y, int j, int KM, double2 (&a)[8], double2 (&b)[8]) {
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    a[r] = b[r] = make_double2(0.0, 0.0);
    const int k = j + r * (N / 8), kk = r < 4 ? k : N - k;
    if (kk <= KM) { a[r] = X[kk]; b[r] = Y[kk]; }
  }
  if (j == 0) a[0].y = b[0].y = a[4].y = b[4].y = 0.0;
}

// one CTA: RT pairs of rows of level z; W: the level's plane; put(y, x, value)
// stores the outputs
template <typename T, int N, class Put>
__device__ __forceinline__ void drow_c2r(int iktxP, int KM, const cplx<T>* __restrict__ W, const cplx<T>* __restrict__ twg,
                                         unsigned char* smem_raw, int p0, Put put) {
  using D = Dense<T, N>;
  if constexpr (D::FX) {
    constexpr int NB = N / 8;
    __shared__ uint2 slots[FxRow<N>::SLOTS];
    FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
    const bool live = c.rr < D::RT;
    const int y = 2 * (p0 + c.rr);
    const double2* X = W + (long long)y * iktxP;
    double2 a[8], b[8], d[8];
    half_full<N>(X, X + iktxP, c.j, live ? KM : -1, a, b);
    c.template inverse_d<false>(a, b, d);
    if (!live) return;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      put(y, c.j + r * NB, d[r].x);
      put(y + 1, c.j + r * NB, d[r].y);
    }
  } else {
    constexpr int R0 = radix_of(N), NB0 = N / R0, NSL = LastNS<N>::value, RL = N / NSL;
    cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
    cplx<T>* sm = tw + N;
    load_tw<T, N>(tw, twg, D::RNT);
    auto pro = [&](int rr, int j, cplx<T> (&v)[1][R0]) {
      const cplx<T>* X = W + (long long)2 * (p0 + rr) * iktxP;
#pragma unroll
      for (int r = 0; r < R0; ++r) v[0][r] = pack_full<T>(X, X + iktxP, j + r * NB0, N, KM);
    };
    auto epi = [&](int rr, int j, cplx<T> (&v)[1][RL]) {
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        put(2 * (p0 + rr), j + r * NSL, v[0][r].x);
        put(2 * (p0 + rr) + 1, j + r * NSL, v[0][r].y);
      }
    };
    __syncthreads();
    row_fft<T, N, false, 1, D::RT, D::RNT, D::LD>(sm, tw, pro, epi);
  }
}

// x-c2r into physical rows of ld doubles: N, or the reference's padded N + 2
// (the two padding values of a row are 0)
template <typename T, int N>
__global__ void __launch_bounds__(Dense<T, N>::RNT, Dense<T, N>::RMINB)
k_drow_c2r_pad(int iktxP, const cplx<T>* __restrict__ W, double* __restrict__ out, int ld, const cplx<T>* __restrict__ twg) {
  using D = Dense<T, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int z = blockIdx.y, p0 = blockIdx.x * D::RT;
  double* o = out + (long long)z * N * ld;
  if (ld > N)
    for (int e = threadIdx.x; e < 4 * D::RT; e += D::RNT) o[(2 * p0 + e / 2) * ld + N + e % 2] = 0.0;
  drow_c2r<T, N>(iktxP, N / 2, W + dense_plane(z, 1, 0, N, iktxP), twg, smem_raw, p0,
                 [&](int y, int x, T v) { o[y * ld + x] = (double)v; });
}

// x-c2r of plane blockIdx.z (np planes per level, kx <= KM) as a dimensional
// FP32 field [nz][N][N]: float((x * s1) * s2) (IO_ncf.f90:47-52, 139-146)
struct F32Out { float* o[2]; double s1, s2; };
template <typename T, int N>
__global__ void __launch_bounds__(Dense<T, N>::RNT, Dense<T, N>::RMINB)
k_drow_c2r_f32(int iktxP, int np, int KM, const cplx<T>* __restrict__ W, F32Out out, const cplx<T>* __restrict__ twg) {
  using D = Dense<T, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int z = blockIdx.y;
  float* o = out.o[blockIdx.z] + (long long)z * N * N;
  drow_c2r<T, N>(iktxP, KM, W + dense_plane(z, np, blockIdx.z, N, iktxP), twg, smem_raw, blockIdx.x * D::RT,
                 [&](int y, int x, T v) { o[y * N + x] = (float)((to64<T>(v) * out.s1) * out.s2); });
}

// the spectra of RT pairs of packed rows, transformed in shared memory, into
// plane rows o (FP32)
template <typename T, int N>
__device__ __forceinline__ void drow_split(const cplx<T>* sm, cplx<T>* __restrict__ o, int iktxP, int KM, int p0) {
  using D = Dense<T, N>;
  for (int e = threadIdx.x; e < D::RT * (KM + 1); e += D::RNT) {
    const int k = e % (KM + 1), rr = e / (KM + 1);
    cplx<T> x, y;
    unpack_pad<T>(sm + rr * D::LD, k, N, x, y);
    cplx<T>* q = o + (long long)2 * (p0 + rr) * iktxP + k;
    q[0] = x;
    q[iktxP] = y;
  }
}

// x-r2c of physical rows of ld doubles
template <typename T, int N>
__global__ void __launch_bounds__(Dense<T, N>::RNT, Dense<T, N>::RMINB)
k_drow_r2c(int iktxP, const double* __restrict__ phys, int ld, cplx<T>* __restrict__ W, const cplx<T>* __restrict__ twg) {
  using D = Dense<T, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int z = blockIdx.y, p0 = blockIdx.x * D::RT;
  const double* a = phys + (long long)z * N * ld;
  W += dense_plane(z, 1, 0, N, iktxP);
  if constexpr (D::FX) {
    constexpr int NB = N / 8;
    __shared__ uint2 slots[FxRow<N>::SLOTS];
    FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
    const bool live = c.rr < D::RT;
    const int y = 2 * (p0 + c.rr);
    double2 d[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const double* q = a + y * ld + c.j + r * NB;
      d[r] = live ? make_double2(q[0], q[ld]) : make_double2(0.0, 0.0);
    }
    double2* o = W + (long long)y * iktxP;
    c.template forward_d<5>(d, N / 2, [&](int, int k, double2 X, double2 Y) {
      if (!live) return;
      o[k] = X;
      o[iktxP + k] = Y;
    });
  } else {
    constexpr int R0 = radix_of(N), NB0 = N / R0, NSL = LastNS<N>::value, RL = N / NSL;
    cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
    cplx<T>* sm = tw + N;
    load_tw<T, N>(tw, twg, D::RNT);
    auto pro = [&](int rr, int j, cplx<T> (&v)[1][R0]) {
      const double* q = a + 2 * (p0 + rr) * ld + j;
#pragma unroll
      for (int r = 0; r < R0; ++r) v[0][r] = mk<T>((T)q[r * NB0], (T)q[ld + r * NB0]);
    };
    // a row's last-pass tasks write back the entries they alone have read
    auto epi = [&](int rr, int j, cplx<T> (&v)[1][RL]) {
#pragma unroll
      for (int r = 0; r < RL; ++r) sm[rr * D::LD + pad_idx(j + r * NSL)] = v[0][r];
    };
    __syncthreads();
    row_fft<T, N, true, 1, D::RT, D::RNT, D::LD>(sm, tw, pro, epi);
    __syncthreads();
    drow_split<T, N>(sm, W, iktxP, N / 2, p0);
  }
}

// Rows of the nonlinear terms, in place on np planes per level, row pairs
// packed, spectra written at kx <= KM.  The transforms of one term were 12 to
// 39 launches with every field through memory between them (products of 45
// levels at 128^2, FP64: 866 us); here each term is three launches and the
// physical fields stay in registers and shared memory.
//   cross = 0: planes a_0 .. a_{nA-1}, x_0 .. x_{nX-1} -> a_h x_k at plane k nA + h
//   cross = 1: planes a, b, c, d -> 2^scale (a b - c d) at plane 0
//   cross = 2: and e, f -> e^2 + f^2 at plane 1
template <typename T, int N> struct DProd {
  using D = Dense<T, N>;
  static constexpr size_t smem() {
    return D::FX ? FxRow<N>::smem() + (size_t)2 * 8 * D::RNT * sizeof(fxc) : D::sm_row() + (size_t)3 * D::RT * N * sizeof(cplx<T>);
  }
};
template <typename T, int N>
__global__ void __launch_bounds__(Dense<T, N>::RNT, Dense<T, N>::RMINB)
k_drow_prod(int iktxP, int np, int KM, int cross, int scale, int nA, int nX, cplx<T>* __restrict__ W,
            const cplx<T>* __restrict__ twg) {
  using D = Dense<T, N>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int z = blockIdx.y, p0 = blockIdx.x * D::RT;
  const int nt = cross == 2 ? 6 : (cross == 1 ? 4 : nA + nX);
  if constexpr (D::FX) {
    constexpr int NB = N / 8;
    __shared__ uint2 slots[FxRow<N>::SLOTS];
    FxRowCtx<N> c = fx_row_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
    fxc* park = reinterpret_cast<fxc*>(smem_raw) + fx_tw_count<N>() + FxRow<N>::RT * FxRow<N>::LD + threadIdx.x;   // [2][8][RNT]
    const bool live = c.rr < D::RT;
    const int y = 2 * (p0 + c.rr);
    auto plane = [&](int f) { return W + dense_plane(z, np, f, N, iktxP) + (long long)y * iktxP; };
    fxc x[8], p[8];
    int2 ex = make_int2(0, 0), e0 = ex, e1 = ex, ep = ex;
#pragma unroll 1
    for (int t = 0; t < nt; ++t) {
      {
        double2 a[8], b[8];
        const double2* X = plane(t);
        half_full<N>(X, X + iktxP, c.j, live ? N / 2 : -1, a, b);
        c.template inverse<false>(a, b, x, ex);
      }
      const bool keep = cross ? (t == 0 || t == 2) : t < nA;
      if (keep) {
        fxc* q = park + (cross || t == 0 ? 0 : 8 * D::RNT);
#pragma unroll
        for (int r = 0; r < 8; ++r) q[r * D::RNT] = x[r];
        if (cross || t == 0) e0 = ex; else e1 = ex;
        continue;
      }
      const int nh = cross ? 1 : nA;
#pragma unroll 1
      for (int h = 0; h < nh; ++h) {
        fxc w[8];
        const bool sq = t >= 4 && cross;
        // (w.x: the first row, whose fields are the parts y)
        const int2 ea = sq ? ex : (h ? e1 : e0);
        const int up = cross && !sq ? scale : 0;
        int2 base = make_int2(fx_prod_base(ea.y, ex.y) + up, fx_prod_base(ea.x, ex.x) + up);
        const fxc* q = park + h * 8 * D::RNT;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const fxc a = sq ? x[r] : q[r * D::RNT];
          w[r].x = fx_mulhi(a.y, x[r].y);
          w[r].y = fx_mulhi(a.x, x[r].x);
        }
        if (cross) {
          if (t == 1 || t == 4) {
            ep = base;
#pragma unroll
            for (int r = 0; r < 8; ++r) p[r] = w[r];
            continue;
          }
          // p -+ w
          const FxAlign ax(ep.x, base.x), ay(ep.y, base.y);
          base = make_int2(ax.e, ay.e);
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            w[r].x = sq ? ax.add(p[r].x, w[r].x) : ax.sub(p[r].x, w[r].x);
            w[r].y = sq ? ay.add(p[r].y, w[r].y) : ay.sub(p[r].y, w[r].y);
          }
        }
        double2* o = plane(cross ? (sq ? 1 : 0) : (t - nA) * nA + h);
        c.template forward<5>(w, base, KM, [&](int, int k, double2 X, double2 Y) {
          if (!live) return;
          o[k] = X;
          o[iktxP + k] = Y;
        });
      }
    }
  } else {
    constexpr int R0 = radix_of(N), NB0 = N / R0, NSL = LastNS<N>::value, RL = N / NSL;
    cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
    cplx<T>* sm = tw + N;
    cplx<T>* park = sm + D::RT * D::LD;        // [3][RT][N]
    constexpr int PS = D::RT * N;
    load_tw<T, N>(tw, twg, D::RNT);
    // the product of two parked fields (b < 0: a alone), rounded by itself (not fused with the first butterfly's additions)
    auto fwd = [&](int a, int b, int f) {
      auto pro = [&](int rr, int j, cplx<T> (&v)[1][R0]) {
#pragma unroll
        for (int r = 0; r < R0; ++r) {
          const int e = rr * N + j + r * NB0;
          cplx<T> u = park[a * PS + e];
          if (b >= 0) { const cplx<T> w = park[b * PS + e]; u = mk<T>(__fmul_rn(u.x, w.x), __fmul_rn(u.y, w.y)); }
          v[0][r] = u;
        }
      };
      auto epi = [&](int rr, int j, cplx<T> (&v)[1][RL]) {
#pragma unroll
        for (int r = 0; r < RL; ++r) sm[rr * D::LD + pad_idx(j + r * NSL)] = v[0][r];
      };
      __syncthreads();
      row_fft<T, N, true, 1, D::RT, D::RNT, D::LD>(sm, tw, pro, epi);
      __syncthreads();
      drow_split<T, N>(sm, W + dense_plane(z, np, f, N, iktxP), iktxP, KM, p0);
    };
#pragma unroll 1
    for (int t = 0; t < nt; ++t) {
      const cplx<T>* P = W + dense_plane(z, np, t, N, iktxP);
      auto pro = [&](int rr, int j, cplx<T> (&v)[1][R0]) {
        const cplx<T>* X = P + (long long)2 * (p0 + rr) * iktxP;
#pragma unroll
        for (int r = 0; r < R0; ++r) v[0][r] = pack_full<T>(X, X + iktxP, j + r * NB0, N, N / 2);
      };
      // cross: slots 0..2 a, b, c; then slot 0 ab - cd, e, e^2 + f^2 in turn
      const int slot = cross ? (t < 3 ? t : 0) : (t < nA ? t : nA);
      auto epi = [&](int rr, int j, cplx<T> (&v)[1][RL]) {
#pragma unroll
        for (int r = 0; r < RL; ++r) {
          const int e = rr * N + j + r * NSL;
          cplx<T> x = v[0][r];
          // (fused as the compiler fuses a b - c d and a a + b b)
          if (cross && t == 3) {
            const cplx<T> a = park[e], b = park[PS + e], q = park[2 * PS + e];
            const T m = scale ? (T)2 : (T)1;
            x = mk<T>(m * __fmaf_rn(a.x, b.x, -__fmul_rn(q.x, x.x)), m * __fmaf_rn(a.y, b.y, -__fmul_rn(q.y, x.y)));
          } else if (cross && t == 5) {
            const cplx<T> a = park[e];
            x = mk<T>(__fmaf_rn(a.x, a.x, __fmul_rn(x.x, x.x)), __fmaf_rn(a.y, a.y, __fmul_rn(x.y, x.y)));
          }
          park[slot * PS + e] = x;
        }
      };
      __syncthreads();
      row_fft<T, N, false, 1, D::RT, D::RNT, D::LD>(sm, tw, pro, epi);
      if (cross) { if (t == 3 || t == 5) fwd(0, -1, t == 3 ? 0 : 1); }
      else if (t >= nA) {
        for (int h = 0; h < nA; ++h) fwd(h, nA, (t - nA) * nA + h);
      }
    }
  }
}

// y-forward transforms into output blockIdx.z of the reference's layout,
// divided by n^2.  mode 0: plane f; 1: L ? i kx P_2f + i ky P_2f+1 : 0
// (convol_waqg); 2: L ? P_f : 0; 3: L ? (P_0 - 0.25 kh^2 P_1) s1 s2 : 0
// (compute_qw, derivatives.f90:1010-1027).  NF: planes per output.
struct DenseOut {
  double2* p[3];
  int mode, kmax2;
  double s1, s2;
};
template <typename T, int N, int NF>
__global__ void __launch_bounds__(Dense<T, N>::CNT, Dense<T, N>::CMINB)
k_dcol_fwd(int iktxP, int np, const cplx<T>* __restrict__ W, DenseOut out, const cplx<T>* __restrict__ twg) {
  constexpr int CT = Dense<T, N>::CT, IKTX = N / 2 + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int z = blockIdx.y, kx0 = blockIdx.x * CT;
  double2* o = out.p[blockIdx.z] + (long long)z * N * IKTX;
  if (out.mode && kx0 * kx0 > out.kmax2) {
    for (int e = threadIdx.x; e < N * CT; e += Dense<T, N>::CNT)
      if (kx0 + e % CT < IKTX) o[(e / CT) * IKTX + kx0 + e % CT] = make_double2(0.0, 0.0);
    return;
  }
  // the columns past the spectrum are not written by the row kernels
  const cplx<T>* P = W + dense_plane(z, np, (int)blockIdx.z * NF, N, iktxP);
  auto get = [&](int f, int y, int kx) {
    return kx < IKTX ? P[((long long)f * N + y) * iktxP + kx] : mk<T>(0, 0);
  };
  auto put = [&](int i, int kx, double2 a, double2 b) {
    double2 v = a;
    if (out.mode) {
      const int ky = i < N / 2 ? i : i - N;
      if (!dense_L(kx, ky, i, N, out.kmax2)) {
        v = make_double2(0.0, 0.0);
      } else if (out.mode == 1) {
        v = make_double2(-kx * a.y - ky * b.y, kx * a.x + ky * b.x);
      } else if (out.mode == 3) {
        const double k4 = 0.25 * (double)(kx * kx + ky * ky);
        v = make_double2((a.x - k4 * b.x) * out.s1 * out.s2, (a.y - k4 * b.y) * out.s1 * out.s2);
      }
    }
    o[i * IKTX + kx] = v;
  };
  if constexpr (Dense<T, N>::FX) {
    constexpr int NB = N / 8;
    __shared__ unsigned slots[FxCol<N>::SLOTS];
    const FxColCtx<N> c = fx_col_ctx<N>(reinterpret_cast<double2*>(smem_raw), slots, twg);
    const int kx = kx0 + c.c;
    double2 A[8], B[8];
#pragma unroll 1
    for (int f = 0; f < NF; ++f) {
      if (f) {
#pragma unroll
        for (int r = 0; r < 8; ++r) A[r] = B[r];
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) B[r] = get(f, c.j + r * NB, kx);
      fxc v[8];
      int base;
      c.template run<true, false>(B, v, base);
      fx_doubles<8, false>(v, B, base - 2 * fx_ilog2(N));     // divided by n^2
    }
    if (kx >= IKTX) return;
#pragma unroll
    for (int r = 0; r < 8; ++r) put(c.j + r * NB, kx, NF == 2 ? A[r] : B[r], B[r]);
  } else {
    constexpr int NT = Dense<T, N>::CNT, R0 = radix_of(N), NB0 = N / R0, NSL = LastNS<N>::value, RL = N / NSL;
    cplx<T>* tw = reinterpret_cast<cplx<T>*>(smem_raw);
    cplx<T>* sm = tw + N;
    load_tw<T, N>(tw, twg, NT);
    auto pro = [&](int c, int j, cplx<T> (&v)[NF][R0]) {
#pragma unroll
      for (int f = 0; f < NF; ++f)
#pragma unroll
        for (int r = 0; r < R0; ++r) v[f][r] = get(f, j + r * NB0, kx0 + c);
    };
    const double s = 1.0 / ((double)N * (double)N);
    auto epi = [&](int c, int j, cplx<T> (&v)[NF][RL]) {
      const int kx = kx0 + c;
      if (kx >= IKTX) return;
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const cplx<T> a = v[0][r], b = v[NF - 1][r];
        put(j + r * NSL, kx, make_double2((double)a.x * s, (double)a.y * s), make_double2((double)b.x * s, (double)b.y * s));
      }
    };
    __syncthreads();
    col_fft<T, N, true, NF, CT, NT>(sm, tw, pro, epi);
  }
}

// Factors of the omega equation's operator (elliptic.f90:463-567) per distinct
// kh2 (kh2[k]), n3-1 unstaggered levels: DGTSV's elimination order (no
// interchange: |d| >= 2 >= |dl|) in correctly rounded FP64 operations;
// fac[k][i] = {dl_i / d'_i, d'_i, 1/d'_i, 0}.  Built once per handle.
static __global__ void k_omega_fac(int nd, int n3, double dz, const int* __restrict__ kh2, const double* __restrict__ t1,
                                   const double* __restrict__ du, const double* __restrict__ dl,
                                   const double* __restrict__ a, double4* __restrict__ fac) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nd) return;
  const int m = n3 - 1;
  const double dzk = __dmul_rn(__dmul_rn(dz, dz), (double)kh2[k]);
  auto diag = [&](int i) { return -__dadd_rn(t1[i], __ddiv_rn(dzk, a[i])); };
  double d = diag(0);
  for (int i = 0; i < m; ++i) {
    const double f = i + 1 < m ? __ddiv_rn(dl[i], d) : 0.0;
    fac[(long long)k * m + i] = make_double4(f, d, __drcp_rn(d), 0.0);
    if (i + 1 < m) d = __dsub_rn(diag(i + 1), __dmul_rn(f, du[i]));
  }
}

// omega_equation: a thread per retained column with kh2 != 0 and part (real,
// imaginary), the right-hand sides dz^2 * rhs; w at the top level and in every
// other column is 0 (set before).  scr: [2][n3-1][ncols] forward values.  Four
// divisions per level and column bound this on the FP64 pipe; the factors
// depend on kh2 only.
constexpr int kOmegaSeg = 8;
static __global__ void k_omega_solve(Geom g, double dz, const double* __restrict__ du, const double4* __restrict__ fac,
                                     const int* __restrict__ tab_idx, const int* __restrict__ cols, int ncols,
                                     const double2* __restrict__ rhs, double* __restrict__ scr, double2* __restrict__ w) {
  const int li = blockIdx.x * blockDim.x + threadIdx.x, part = blockIdx.y;
  if (li >= ncols) return;
  const int mc = cols[li], idx = tab_idx[mc];
  if (idx < 0) return;
  const int m = g.n3 - 1, ky = g.ky_of_row(mc / g.KXP), kx = mc % g.KXP;
  const long long per = 2LL * g.n * (g.n / 2 + 1);
  const long long col = 2 * ((long long)(ky < 0 ? ky + g.n : ky) * (g.n / 2 + 1) + kx) + part;
  const double* r = reinterpret_cast<const double*>(rhs) + col;
  double* o = reinterpret_cast<double*>(w) + col;
  const double4* F = fac + (long long)idx * m;
  double* v = scr + (long long)part * m * ncols + li;
  const double dz2 = __dmul_rn(dz, dz);
  constexpr int S = kOmegaSeg;
  double x = 0.0;
  for (int j = 0; j < m; j += S) {
    double q[S], f[S];
#pragma unroll
    for (int k = 0; k < S; ++k) {
      const int i = j + k;
      q[k] = i < m ? r[i * per] : 0.0;
      f[k] = i > 0 && i < m ? F[i - 1].x : 0.0;
    }
#pragma unroll
    for (int k = 0; k < S; ++k)
      if (j + k < m) {
        const double b = __dmul_rn(dz2, q[k]);
        x = j + k > 0 ? __dsub_rn(b, __dmul_rn(f[k], x)) : b;
        v[(long long)(j + k) * ncols] = x;
      }
  }
  double xn = 0.0;
  for (int j = (m - 1) / S * S; j >= 0; j -= S) {
    double b[S], d[S], rd[S], u[S];
#pragma unroll
    for (int k = 0; k < S; ++k) {
      const int i = min(j + k, m - 1);
      const double4 fi = F[i];
      b[k] = v[(long long)i * ncols]; d[k] = fi.y; rd[k] = fi.z; u[k] = du[i];
    }
#pragma unroll
    for (int k = S - 1; k >= 0; --k) {
      const int i = j + k;
      if (i < m) {
        xn = div_by(i == m - 1 ? b[k] : __dsub_rn(b[k], __dmul_rn(u[k], xn)), d[k], rd[k]);
        o[i * per] = xn;
      }
    }
  }
}

}  // namespace qg
