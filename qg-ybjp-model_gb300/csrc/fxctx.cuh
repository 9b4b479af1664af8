// Block fixed-point transforms (fxfft.cuh) with eight values per thread in
// registers: one row of a plane per N/8 threads, or a tile of columns per CTA.
#pragma once
#include "fxfft.cuh"

namespace qg {

// inputs of index r of a first radix-8 pass of a pruned spectrum (|k| <= K <
// 3N/8): r = 3, 4 are zero for every butterfly
template <int R> __host__ __device__ constexpr bool fx_zero_in(int r) { return R == 8 && (r == 3 || r == 4); }

// v 2^512 (exact), unless all of it is zero
template <int R, bool PRUNED> __device__ __forceinline__ void fx_raise(double2* v) {
  unsigned o = 0;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (!(PRUNED && fx_zero_in<R>(r)))
      o |= fx_mag(v[r].x) | fx_mag(v[r].y) | (unsigned)__double2loint(v[r].x) | (unsigned)__double2loint(v[r].y);
  if (!o) return;
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (!(PRUNED && fx_zero_in<R>(r))) { v[r].x *= 0x1p512; v[r].y *= 0x1p512; }
}
// doubles d[R] -> integers below 2^59 (the largest magnitude bits of the whole
// transform in mag); parts exchanged for the inverse.  Returns the base.
template <int R, bool FWD, bool PRUNED>
__device__ __forceinline__ int fx_ints(double2* d, fxc* v, unsigned mag) {
  int be;
  bool tiny;
  const int base = fx_base<59>(mag, be, tiny);
  if (tiny) fx_raise<R, PRUNED>(d);
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

// scale one part of v to TOP bits (its magnitudes' high words' bits are in o),
// to the nearest, base follows; magnitudes below 2^32 gain TOP - 32 bits
template <int R, int TOP, bool Y> __device__ __forceinline__ void fx_norm1(fxc* v, unsigned o, int& base) {
  const int s = __clz((int)o) - (64 - TOP);
  base -= s;
  if (s >= 0) {
#pragma unroll
    for (int r = 0; r < R; ++r) (Y ? v[r].y : v[r].x) <<= s;
  } else {
    const long long h = 1LL << (-s - 1);
#pragma unroll
    for (int r = 0; r < R; ++r) { long long& x = Y ? v[r].y : v[r].x; x = (x + h) >> -s; }
  }
}
template <int R, int TOP> __device__ __forceinline__ void fx_norm(fxc* v, uint2 o, int2& base) {
  fx_norm1<R, TOP, false>(v, o.x, base.x);
  fx_norm1<R, TOP, true>(v, o.y, base.y);
}
// a +- b of the bases ea, eb: integers of the larger one, e, to the nearest
struct FxAlign {
  int e, sa, sb;
  long long ha, hb;
  __device__ __forceinline__ FxAlign(int ea, int eb)
      : e(max(ea, eb)), sa(min(e - ea, 62)), sb(min(e - eb, 62)), ha((1LL << sa) >> 1), hb((1LL << sb) >> 1) {}
  __device__ __forceinline__ long long add(long long a, long long b) const { return ((a + ha) >> sa) + ((b + hb) >> sb); }
  __device__ __forceinline__ long long sub(long long a, long long b) const { return ((a + ha) >> sa) - ((b + hb) >> sb); }
};
// base of a b / 2^64
__device__ __forceinline__ int fx_prod_base(int ea, int eb) { return ea + eb - 1023 + 64; }

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
// rows, whose spectra split() separates (fx_top).  FIT: the second pass takes
// back the room that the first one's growth left, as every pass does where
// fx_renorm() holds; the word that this takes rides on the pass's barrier.
// ===========================================================================
template <int N, int NS, bool ROWS, bool FIT, class P, class Sync, class Red>
__device__ __forceinline__ void fx_core_pass(fxc (&v)[8], int& base, fxc* __restrict__ buf, const int4* __restrict__ tw,
                                             int j, P at, Sync sync, Red red) {
  constexpr int R = fx_radix(N, NS), NB = N / 8, PER = 8 / R;
  constexpr bool last = NS * R == N, renorm = fx_renorm<N>() || (FIT && NS == 8);
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
    fx_core_pass<N, NS * R, ROWS, FIT>(v, base, buf, tw, j, at, sync, red);
  }
}
template <int N, bool ROWS, bool FIT, class P, class Sync, class Red>
__device__ __forceinline__ void fx_core(fxc (&v)[8], int& base, fxc* __restrict__ buf, const int4* __restrict__ tw, int j,
                                        P at, Sync sync, Red red) {
  fx_dft8(v);
#pragma unroll
  for (int r = 0; r < 8; ++r) buf[at(j * 8 + r)] = v[r];
  base += fx_shift_total<N>();
  fx_core_pass<N, 8, ROWS, FIT>(v, base, buf, tw, j, at, sync, red);
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
  static constexpr int SLOTS = 3 * RT * W;             // (pairs)
  static constexpr size_t smem() { return (size_t)(fx_tw_count<N>() + RT * LD) * sizeof(double2); }
};

template <int NB> __device__ __forceinline__ void fx_row_sync(int rr) {
  if constexpr (NB <= 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + rr), "n"(NB) : "memory");
}
// maximum or bitwise OR of m's parts over the row's threads; orders them too
template <int NB, bool OR> __device__ __forceinline__ uint2 fx_row_reduce(uint2 m, uint2* slots, int rr) {
  if constexpr (NB >= 32) {
    m.x = OR ? __reduce_or_sync(0xffffffffu, m.x) : __reduce_max_sync(0xffffffffu, m.x);
    m.y = OR ? __reduce_or_sync(0xffffffffu, m.y) : __reduce_max_sync(0xffffffffu, m.y);
  } else {
#pragma unroll
    for (int o = 1; o < NB; o <<= 1) {
      const unsigned x = __shfl_xor_sync(0xffffffffu, m.x, o), y = __shfl_xor_sync(0xffffffffu, m.y, o);
      m.x = OR ? (m.x | x) : max(m.x, x);
      m.y = OR ? (m.y | y) : max(m.y, y);
    }
  }
  if constexpr (NB <= 32) {
    __syncwarp();
  } else {
    constexpr int W = NB / 32;
    uint2* s = slots + rr * W;
    if ((threadIdx.x & 31) == 0) s[(threadIdx.x >> 5) % W] = m;
    fx_row_sync<NB>(rr);
#pragma unroll
    for (int i = 0; i < W; ++i) {
      m.x = OR ? (m.x | s[i].x) : max(m.x, s[i].x);
      m.y = OR ? (m.y | s[i].y) : max(m.y, s[i].y);
    }
  }
  return m;
}

// The thread's view of its row pair: transforms of eight values per thread.
// Two real rows are packed as one complex row, and each has a scale of its own
// (a base per part), as two transforms would.  With one scale for both, a row
// 2^-m of its neighbour lost m of its bits, beside a uniform neighbour too,
// which a floating-point transform does not mix into it.  us per launch, one
// scale -> two: k_fx_row_main 512^2 x 256 6400 -> 6480, 256^2 x 128 725 -> 753,
// 128^2 x 64 98 -> 98; k_fx_row_qw 3260 -> 3470, 381 -> 428, 51 -> 53.
template <int N, int T = 128> struct FxRowCtx {
  static constexpr int NB = N / 8;
  fxc* buf;
  const int4* tw;
  uint2* slots;        // three sets of [RT][W]
  int rr, j;
  int set = 0;         // reductions alternate between two sets: one follows another without a further barrier
  __device__ __forceinline__ void sync() const { fx_row_sync<NB>(rr); }
  template <bool OR> __device__ __forceinline__ uint2 reduce(uint2 m) {
    set ^= FxRow<N, T>::RT * FxRow<N, T>::W;
    return fx_row_reduce<NB, OR>(m, slots + set, rr);
  }
  template <bool FIT> __device__ __forceinline__ void core(fxc (&v)[8], int2& base) const {
    int up = 0;
    fx_core<N, true, FIT>(v, up, buf, tw, j, [](int i) { return fx_idx(i); }, [&]() { sync(); }, [&](unsigned m) {
      return fx_row_reduce<NB, true>(make_uint2(m, 0u), slots + 2 * FxRow<N, T>::RT * FxRow<N, T>::W, rr).x;
    });
    base.x += up;
    base.y += up;
  }
  // integers of the packed spectrum of two rows, parts exchanged for the
  // inverse (v.y, base.y: the first row), from the half spectra a, b at
  // kk = j + r NB, or N - j - r NB for r >= 4 (PRUNED: zeros at |k| > K), real
  // at kk = 0 and N/2.  58 bits for each row, so that their sums stay below
  // 2^59 (packed as doubles, the smaller values of a row would be rounded
  // against the other row's); core<true> takes the room back.
  template <bool PRUNED> __device__ __forceinline__ int2 ints_inverse(double2 (&a)[8], double2 (&b)[8], fxc (&v)[8]) {
    const uint2 m = reduce<false>(make_uint2(fx_maxp<8, PRUNED>(a), fx_maxp<8, PRUNED>(b)));
    int ea, eb;
    bool ta, tb;
    int2 base;
    base.y = fx_base<58>(m.x, ea, ta);
    base.x = fx_base<58>(m.y, eb, tb);
    if (ta) fx_raise<8, PRUNED>(a);
    if (tb) fx_raise<8, PRUNED>(b);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (PRUNED && fx_zero_in<8>(r)) { v[r].x = v[r].y = 0; continue; }
      fxc x, y;
      x.x = fx_in1<58>(a[r].x, ea); x.y = fx_in1<58>(a[r].y, ea);
      y.x = fx_in1<58>(b[r].x, eb); y.y = fx_in1<58>(b[r].y, eb);
      if (r < 4) { v[r].y = x.x - y.y; v[r].x = x.y + y.x; }
      else { v[r].y = x.x + y.y; v[r].x = y.x - x.y; }
    }
    return base;
  }
  // inverse transform of the packed spectrum into integers of 61 bits: v.y the
  // first row, v.x the second
  template <bool PRUNED = true> __device__ __forceinline__ void inverse(double2 (&a)[8], double2 (&b)[8], fxc (&v)[8], int2& base) {
    base = ints_inverse<PRUNED>(a, b, v);
    core<true>(v, base);
    fx_norm<8, 61>(v, reduce<true>(fx_bits2<8>(v)), base);
  }
  // ... into doubles: o.x the first row, o.y the second
  template <bool PRUNED = true> __device__ __forceinline__ void inverse_d(double2 (&a)[8], double2 (&b)[8], double2 (&o)[8]) {
    fxc v[8];
    int2 base = ints_inverse<PRUNED>(a, b, v);
    core<true>(v, base);
    fx_doubles<8, true>(v, o, base);
  }
  // forward transform of the packed rows d (x the first, y the second) and its split
  template <int Q = 3, class Put> __device__ __forceinline__ void forward_d(double2 (&d)[8], int K, Put put) {
    uint2 m = make_uint2(0u, 0u);
#pragma unroll
    for (int r = 0; r < 8; ++r) { m.x = max(m.x, fx_mag(d[r].x)); m.y = max(m.y, fx_mag(d[r].y)); }
    m = reduce<false>(m);
    int ex, ey;
    bool tx, ty;
    int2 base;
    base.x = fx_base<59>(m.x, ex, tx);
    base.y = fx_base<59>(m.y, ey, ty);
    fxc v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (tx) d[r].x *= 0x1p512;
      if (ty) d[r].y *= 0x1p512;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) { v[r].x = fx_in1(d[r].x, ex); v[r].y = fx_in1(d[r].y, ey); }
    core<false>(v, base);
    split<Q>(v, base, K, put);
  }
  // the spectra of the two packed rows from their transform's outputs v, at
  // k = j + q NB <= KM, q < Q: put(q, k, X, Y)
  template <int Q, class Put> __device__ __forceinline__ void split(const fxc (&v)[8], int2 base, int KM, Put put) const {
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (Q > 3 || !fx_zero_in<8>(r)) buf[fx_idx(j + r * NB)] = v[r];
    sync();
    fxc s[2 * Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      // X = (F[k] + conj F[N-k]) / 2, Y = (F[k] - conj F[N-k]) / (2 i): the
      // sums stay below 2^63 (each row's spectrum is at most 2^62: fx_growth_ok)
      const int k = j + q * NB;
      const fxc a = v[q], b = buf[fx_idx(k == 0 ? 0 : N - k)];
      s[q].x = a.x + b.x; s[q].y = a.y - b.y;
      s[Q + q].x = a.y + b.y; s[Q + q].y = b.x - a.x;
    }
    double2 o[2 * Q];
    fx_doubles<Q, false>(s, o, base.x - 1);
    fx_doubles<Q, false>(s + Q, o + Q, base.y - 1);
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (j + q * NB <= KM) put(q, j + q * NB, o[q], o[Q + q]);
  }
  // forward transform of the integers v (two packed rows) and its split
  template <int Q = 3, class Put> __device__ __forceinline__ void forward(fxc (&v)[8], int2 base, int K, Put put) {
    fx_norm<8, 59>(v, reduce<true>(fx_bits2<8>(v)), base);
    core<false>(v, base);
    split<Q>(v, base, K, put);
  }
};

template <int N, int T = 128>
__device__ __forceinline__ FxRowCtx<N, T> fx_row_ctx(double2* smem, uint2* slots, const double2* twg) {
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

// the half spectra X, Y of two rows at kk = k (r < 4) or N - k, k = j + r NB,
// zeros past K (ints_inverse); the imaginary parts at kk = 0 are ignored, as a
// c2r does
template <int N>
__device__ __forceinline__ void fx_half(const double2* __restrict__ X, const double2* __restrict__ Y, int j, int K,
                                        double2 (&a)[8], double2 (&b)[8]) {
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    a[r] = b[r] = make_double2(0.0, 0.0);
    if (fx_zero_in<8>(r)) continue;
    const int k = j + r * (N / 8), kk = r < 4 ? k : N - k;
    if (kk <= K) { a[r] = X[kk]; b[r] = Y[kk]; }
  }
  if (j == 0) a[0].y = b[0].y = 0.0;
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
    fx_core<N, false, false>(v, base, buf, tw, j, [&](int i) { return fx_idx(i) * F::CT + c; }, []() { __syncthreads(); },
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
