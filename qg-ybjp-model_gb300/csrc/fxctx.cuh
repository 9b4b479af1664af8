// Block fixed-point transforms (fxfft.cuh) with eight values per thread in
// registers: one row of a plane per N/8 threads, or a tile of columns per CTA.
#pragma once
#include "fxfft.cuh"

namespace qg {

// inputs of index r of a first radix-8 pass of a pruned spectrum (|k| <= K <
// 3N/8): r = 3, 4 are zero for every butterfly
template <int R> __host__ __device__ constexpr bool fx_zero_in(int r) { return R == 8 && (r == 3 || r == 4); }

// doubles d[R] -> integers below 2^59 (the largest magnitude bits of the whole
// transform in mag); parts exchanged for the inverse.  Returns the base.
template <int R, bool FWD, bool PRUNED>
__device__ __forceinline__ int fx_ints(double2* d, fxc* v, unsigned mag) {
  int be = (int)(mag >> 20);
  const int base = be >= 2047 ? kFxNan : max(be, 1) - 58;
  if (be < kFxTiny) {
    be = max(be, 1) + 512;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (!(PRUNED && fx_zero_in<R>(r))) { d[r].x *= 0x1p512; d[r].y *= 0x1p512; }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (PRUNED && fx_zero_in<R>(r)) { v[r].x = v[r].y = 0; continue; }
    const long long a = fx_in1(d[r].x, be), b = fx_in1(d[r].y, be);
    v[r].x = FWD ? a : b;
    v[r].y = FWD ? b : a;
  }
  return base;
}
template <int R, bool PRUNED> __device__ __forceinline__ unsigned fx_maxp(const double2* v) {
  unsigned m = 0;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (!(PRUNED && fx_zero_in<R>(r))) m = max(m, max(fx_mag(v[r].x), fx_mag(v[r].y)));
  return m;
}

// shared placement: one pad slot every 8 elements (conflict free for 16-byte
// elements in every pass for N >= 64, checked in colfft.cuh)
__host__ __device__ __forceinline__ constexpr int fx_idx(int i) { return i + (i >> 3); }

// scale v so that its magnitudes, whose high words' bits are in o, fill TOP
// bits; base follows
template <int R, int TOP> __device__ __forceinline__ void fx_norm(fxc* v, unsigned o, int& base) {
  const int s = __clz((int)o) - (64 - TOP);
  base -= s;
  if (s >= 0) {
#pragma unroll
    for (int r = 0; r < R; ++r) { v[r].x <<= s; v[r].y <<= s; }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) { v[r].x >>= -s; v[r].y >>= -s; }
  }
}

// a b / 2^64 (|a|, |b| < 2^62)
__device__ __forceinline__ long long fx_mulhi(long long a, long long b) {
  const int al = (int)a, bl = (int)b;
  const int ah = (int)(a >> 32) + (int)((unsigned)al >> 31), bh = (int)(b >> 32) + (int)((unsigned)bl >> 31);
  long long c = (long long)ah * bl + 0x80000000LL;
  c += (long long)al * bh;
  return (long long)ah * bh + (c >> 32);
}

// ===========================================================================
// One transform per NB = N/8 threads, eight values per thread: inputs at
// j + r NB in registers, outputs at the same indices (a last pass of radix
// R < 8 runs 8/R butterflies per thread, whose outputs are those indices
// too).  at places element i in the transform's shared buffer, sync orders
// the transform's threads, red ORs a word over them (and orders them).
// At entry the threads are past their last access to the buffer; the slots
// of a thread's outputs are its own to write afterwards.  ROWS: two packed
// rows, whose spectra split() separates (fx_top).
// ===========================================================================
template <int N, int NS, bool ROWS, class P, class Sync, class Red>
__device__ __forceinline__ void fx_core_pass(fxc (&v)[8], int& base, fxc* __restrict__ buf, const int4* __restrict__ tw,
                                             int j, P at, Sync sync, Red red) {
  constexpr int R = fx_radix(N, NS), NB = N / 8, PER = 8 / R;
  constexpr bool last = NS * R == N, renorm = fx_renorm<N>();
  int s = 0;
  if constexpr (renorm) s = fx_room<fx_top<N, ROWS>(NS)>(red(fx_bits<8>(v)));    // (orders the earlier pass's stores)
  else sync();
#pragma unroll
  for (int p = 0; p < PER; ++p)
#pragma unroll
    for (int r = 0; r < R; ++r) v[p * R + r] = buf[at(j + p * NB + r * (N / R))];
  if constexpr (renorm) { fx_shl<8>(v, s); base -= s; }
  if constexpr (last) {
    fxc w[8];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      fx_butterfly<N, R, NS>(v + p * R, tw, j + p * NB);
#pragma unroll
      for (int r = 0; r < R; ++r) w[p + r * PER] = v[p * R + r];
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = w[r];
  } else {
    sync();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int jj = j + p * NB, k = jj & (NS - 1), b = (jj - k) * R + k;
      fx_butterfly<N, R, NS>(v + p * R, tw, k);
#pragma unroll
      for (int r = 0; r < R; ++r) buf[at(b + r * NS)] = v[p * R + r];
    }
    fx_core_pass<N, NS * R, ROWS>(v, base, buf, tw, j, at, sync, red);
  }
}
template <int N, bool ROWS, class P, class Sync, class Red>
__device__ __forceinline__ void fx_core(fxc (&v)[8], int& base, fxc* __restrict__ buf, const int4* __restrict__ tw, int j,
                                        P at, Sync sync, Red red) {
  fx_dft8(v);
#pragma unroll
  for (int r = 0; r < 8; ++r) buf[at(j * 8 + r)] = v[r];
  base += fx_shift_total<N>();
  fx_core_pass<N, 8, ROWS>(v, base, buf, tw, j, at, sync, red);
}

// ===========================================================================
// Rows: one row per NB threads, synchronised by the row (its warp, or a named
// barrier of its warps)
// ===========================================================================
template <int N, int T = 128> struct FxRow {
  static constexpr int NB = N / 8, LD = fx_idx(N);
  static constexpr int RT = T / NB < N ? T / NB : N;      // rows per CTA of T threads
  static constexpr int NT = RT * NB;                      // threads per CTA
  static constexpr int W = NB > 32 ? NB / 32 : 1;         // warps per row
  static constexpr int SLOTS = 3 * RT * W;
  static constexpr size_t smem() { return (size_t)(fx_tw_count<N>() + RT * LD) * sizeof(double2); }
};

template <int NB> __device__ __forceinline__ void fx_row_sync(int rr) {
  if constexpr (NB <= 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + rr), "n"(NB) : "memory");
}
// maximum or bitwise OR of m over the row's threads; orders them too
template <int NB, bool OR> __device__ __forceinline__ unsigned fx_row_reduce(unsigned m, unsigned* slots, int rr) {
  if constexpr (NB >= 32) {
    m = OR ? __reduce_or_sync(0xffffffffu, m) : __reduce_max_sync(0xffffffffu, m);
  } else {
#pragma unroll
    for (int o = 1; o < NB; o <<= 1) {
      const unsigned x = __shfl_xor_sync(0xffffffffu, m, o);
      m = OR ? (m | x) : max(m, x);
    }
  }
  if constexpr (NB <= 32) {
    __syncwarp();
  } else {
    constexpr int W = NB / 32;
    unsigned* s = slots + rr * W;
    if ((threadIdx.x & 31) == 0) s[(threadIdx.x >> 5) % W] = m;
    fx_row_sync<NB>(rr);
#pragma unroll
    for (int i = 0; i < W; ++i) m = OR ? (m | s[i]) : max(m, s[i]);
  }
  return m;
}

// The thread's view of its row: transforms of eight values per thread.
template <int N, int T = 128> struct FxRowCtx {
  static constexpr int NB = N / 8;
  fxc* buf;
  const int4* tw;
  unsigned* slots;     // three sets of [RT][W]
  int rr, j;
  int set = 0;         // reductions alternate between two sets: one follows another without a further barrier
  __device__ __forceinline__ void sync() const { fx_row_sync<NB>(rr); }
  template <bool OR> __device__ __forceinline__ unsigned reduce(unsigned m) {
    set ^= FxRow<N, T>::RT * FxRow<N, T>::W;
    return fx_row_reduce<NB, OR>(m, slots + set, rr);
  }
  __device__ __forceinline__ void core(fxc (&v)[8], int& base) const {
    fx_core<N, true>(v, base, buf, tw, j, [](int i) { return fx_idx(i); }, [&]() { sync(); },
               [&](unsigned m) { return fx_row_reduce<NB, true>(m, slots + 2 * FxRow<N, T>::RT * FxRow<N, T>::W, rr); });
  }
  // inverse transform of the packed spectrum d (PRUNED: zeros at |k| > K) into
  // integers of 61 bits: v.y the first (real) row, v.x the second
  template <bool PRUNED = true> __device__ __forceinline__ void inverse(double2 (&d)[8], fxc (&v)[8], int& base) {
    base = fx_ints<8, false, PRUNED>(d, v, reduce<false>(fx_maxp<8, PRUNED>(d)));
    core(v, base);
    fx_norm<8, 61>(v, reduce<true>(fx_bits<8>(v)), base);
  }
  // inverse transform of the packed spectrum d into doubles: o.x the first
  // row, o.y the second
  __device__ __forceinline__ void inverse_d(double2 (&d)[8], double2 (&o)[8]) {
    fxc v[8];
    int base = fx_ints<8, false, true>(d, v, reduce<false>(fx_maxp<8, true>(d)));
    core(v, base);
    fx_doubles<8, true>(v, o, base);
  }
  // forward transform of the packed rows d and its split
  template <class Put> __device__ __forceinline__ void forward_d(double2 (&d)[8], int K, Put put) {
    fxc v[8];
    int base = fx_ints<8, true, false>(d, v, reduce<false>(fx_maxp<8, false>(d)));
    core(v, base);
    split<3>(v, base, K, put);
  }
  // the spectra of the two packed rows from their transform's outputs v, at
  // k = j + q NB <= KM, q < Q: put(q, k, X, Y)
  template <int Q, class Put> __device__ __forceinline__ void split(const fxc (&v)[8], int base, int KM, Put put) const {
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (Q > 3 || !fx_zero_in<8>(r)) buf[fx_idx(j + r * NB)] = v[r];
    sync();
    fxc s[2 * Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      // X = (F[k] + conj F[N-k]) / 2, Y = (F[k] - conj F[N-k]) / (2 i): the
      // sums stay below 2^63 (each row's spectrum is at most 2^62)
      const int k = j + q * NB;
      const fxc a = v[q], b = buf[fx_idx(k == 0 ? 0 : N - k)];
      s[2 * q].x = a.x + b.x; s[2 * q].y = a.y - b.y;
      s[2 * q + 1].x = a.y + b.y; s[2 * q + 1].y = b.x - a.x;
    }
    double2 o[2 * Q];
    fx_doubles<2 * Q, false>(s, o, base - 1);
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (j + q * NB <= KM) put(q, j + q * NB, o[2 * q], o[2 * q + 1]);
  }
  // forward transform of the integers v (two packed rows) and its split
  template <int Q = 3, class Put> __device__ __forceinline__ void forward(fxc (&v)[8], int base, int K, Put put) {
    const unsigned o = reduce<true>(fx_bits<8>(v));
    fx_norm<8, 59>(v, o, base);
    core(v, base);
    split<Q>(v, base, K, put);
  }
};

template <int N, int T = 128>
__device__ __forceinline__ FxRowCtx<N, T> fx_row_ctx(double2* smem, unsigned* slots, const double2* twg) {
  using F = FxRow<N, T>;
  fx_load_tw<N>(smem, twg, F::NT);
  __syncthreads();
  FxRowCtx<N, T> c;
  c.rr = threadIdx.x / F::NB;
  c.j = threadIdx.x % F::NB;
  c.buf = reinterpret_cast<fxc*>(smem + fx_tw_count<N>()) + c.rr * F::LD;
  c.tw = reinterpret_cast<const int4*>(smem);
  c.slots = slots;
  return c;
}

// packed spectrum X + iY of two half spectra at k = j + r NB
template <int N>
__device__ __forceinline__ void fx_pack(const double2* __restrict__ X, const double2* __restrict__ Y, int j, int K,
                                        double2 (&d)[8]) {
  constexpr int NB = N / 8;
  double2 a[8], b[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    a[r] = b[r] = make_double2(0.0, 0.0);
    if (fx_zero_in<8>(r)) continue;
    const int k = j + r * NB, kk = r < 4 ? k : N - k;
    if (kk <= K) { a[r] = X[kk]; b[r] = Y[kk]; }
  }
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    if (r < 4) d[r] = make_double2(a[r].x - b[r].y, a[r].y + b[r].x);
    else d[r] = make_double2(a[r].x + b[r].y, b[r].x - a[r].y);
  }
  if (j == 0) d[0] = make_double2(a[0].x, b[0].x);     // imaginary parts at kx = 0 are ignored, as a c2r does
}

// ===========================================================================
// Columns: CT spectral columns of one level, c fastest over the threads
// ===========================================================================
template <int N> struct FxCol {
  // 128 threads for N >= 128; 16-byte elements: CT = 2 columns fill a 32-byte sector
  static constexpr int NB = N / 8, CT = N == 16 ? 16 : (N <= 128 ? 8 : (1024 / N)), NT = CT * NB, LD = fx_idx(N) * CT;
  static constexpr int W = NT > 32 ? NT / 32 : 1;
  static constexpr int SLOTS = 2 * W * CT;
  static constexpr size_t smem() { return (size_t)(fx_tw_count<N>() + LD) * sizeof(double2); }
};
template <int N> struct FxColCtx {
  using F = FxCol<N>;
  fxc* buf;
  const int4* tw;
  unsigned* slots;      // [2][W][CT]
  int c, j;
  // over the threads of the column; orders the CTA
  template <bool OR> __device__ __forceinline__ unsigned reduce(unsigned m, int set) const {
#pragma unroll
    for (int o = F::CT; o < 32; o <<= 1) {
      const unsigned x = __shfl_xor_sync(0xffffffffu, m, o);
      m = OR ? (m | x) : max(m, x);
    }
    unsigned* s = slots + set * F::W * F::CT;
    if ((threadIdx.x & 31) < F::CT) s[(threadIdx.x >> 5) * F::CT + c] = m;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < F::W; ++i) m = OR ? (m | s[i * F::CT + c]) : max(m, s[i * F::CT + c]);
    return m;
  }
  // the doubles d (index j + r NB) as integers, v.x, v.y exchanged when
  // inverse; PRUNED: zeros at |k| >= 3N/8
  template <bool FWD, bool PRUNED = !FWD> __device__ __forceinline__ int load(double2 (&d)[8], fxc (&v)[8]) const {
    return fx_ints<8, FWD, PRUNED>(d, v, reduce<false>(fx_maxp<8, PRUNED>(d), 0));
  }
  __device__ __forceinline__ void core(fxc (&v)[8], int& base) const {
    fx_core<N, false>(v, base, buf, tw, j, [&](int i) { return fx_idx(i) * F::CT + c; }, []() { __syncthreads(); },
               [&](unsigned m) { return reduce<true>(m, 1); });
  }
  template <bool FWD, bool PRUNED = !FWD> __device__ __forceinline__ void run(double2 (&d)[8], fxc (&v)[8], int& base) const {
    base = load<FWD, PRUNED>(d, v);
    core(v, base);
  }
};
template <int N> __device__ __forceinline__ FxColCtx<N> fx_col_ctx(double2* smem, unsigned* slots, const double2* twg) {
  using F = FxCol<N>;
  fx_load_tw<N>(smem, twg, F::NT);
  FxColCtx<N> c;
  c.tw = reinterpret_cast<const int4*>(smem);
  c.buf = reinterpret_cast<fxc*>(smem + fx_tw_count<N>());
  c.slots = slots;
  c.c = threadIdx.x % F::CT;
  c.j = threadIdx.x / F::CT;
  return c;
}
}  // namespace qg
