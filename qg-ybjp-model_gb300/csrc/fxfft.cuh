// FP64-grade FFTs on the integer pipes: transforms of doubles carried out in
// 64-bit block fixed point.
//
// GB300 issues FP64 at 2 lanes per clock and SM; 64-bit integer additions run
// at 62 and 32x32->64 multiply-adds at 30 (measured).  A radix-8 butterfly
// with its twiddles is 82 FP64 operations (1312 SM clocks per warp) or about
// 290 integer ones (about 160 clocks), so the FP64 path transforms integers:
//
//   * Each transform finds the largest exponent among its inputs (|x| < 2^E)
//     and scales every input to an integer m = x 2^(59-E), truncated towards
//     zero (values below 2^(E-6) lose bits there, where a double keeps them;
//     against the transform's largest input that is 64 times finer than FP64's
//     own rounding).  Two real rows packed as one complex input have an
//     exponent each (FxRowCtx).
//   * A radix-R pass lets the modulus grow by at most R, so the integers stay
//     below 2^62.5 when every later pass divides its inputs by the earlier
//     pass's radix.  The division is part of the twiddle factor, w = W 2^(64-s)
//     and x w taken as the high word of the product; the untwiddled input is
//     shifted.  The passes round to nearest, or to one unit where a product's
//     low x low part is left out, at 2^-62 of the growth bound.
//   * The outputs are normalised back to doubles, rounded to nearest.
// The noise relative to the output's rms is largest for an input with a single
// nonzero value, which the divisions leave at 2^59 / 8^2 = 2^53 after the
// passes of n = 512: eight inputs of the last butterfly rounded at half a unit,
// sqrt(8/12) 2^-53 = 2^-53.3 and the earlier passes' beside it, measured
// 2^-52.7 (2^-53.9 at n = 256, 2^-55.8 at 64; white spectra 2^-57), where an
// FP64 transform is at 2^-52.1.  Longer transforms, and the inverse rows, take
// back the unused room (fx_renorm, FIT): 2^-54.3 there for such an input, up to
// 2^-52.6 for k^-4 spectra.  The tests compare with 113-bit transforms.
// A transform with a NaN or infinity among its inputs returns NaN; tiny and
// huge scales (subnormal inputs, overflowing outputs) take exact slow paths.
//
// Only the forward sign is implemented: the inverse is the forward transform
// with real and imaginary parts exchanged on the way in and out.
#pragma once
#include "fft_block.cuh"

namespace qg {

struct __align__(16) fxc { long long x, y; };

// radix of the pass with stride ns of a length-n transform: radix 8 first
// (eight values per thread throughout), then as radix_of
__host__ __device__ constexpr int fx_radix(int n, int ns) { return ns == 1 ? 8 : (n < 64 ? n / 8 : radix_of(n / ns)); }
// offset of the pass ns in the per-pass twiddle table
template <int N> __host__ __device__ constexpr int fx_tw_off(int ns) {
  int off = 0;
  for (int s = 8; s < ns; s *= fx_radix(N, s)) off += s * (fx_radix(N, s) - 1);
  return off;
}

// log2 of the factor a pass divides its inputs by: the earlier pass's radix
// (at least 4: the factor 1 of a division by 2 would not fit a signed word)
__host__ __device__ constexpr int fx_log2(int r) { return r == 8 ? 3 : (r == 4 ? 2 : 1); }
template <int N> __host__ __device__ constexpr int fx_shift(int ns) {   // pass with stride ns > 1
  int s = 1, r = 1;
  while (s < ns) { r = fx_radix(N, s); s *= r; }
  return fx_log2(r) < 2 ? 2 : fx_log2(r);
}
template <int N> __host__ __device__ constexpr int fx_shift_total() {
  int t = 0;
  for (int s = 8; s < N; s *= fx_radix(N, s)) t += fx_shift<N>(s);
  return t;
}

__host__ __device__ constexpr int fx_ilog2(int n) { int m = 0; while ((1 << m) < n) ++m; return m; }
// transforms this long take back the room that a peaked spectrum leaves
// unused below the growth bound, before each later pass: without it the
// divisions of n = 1024 would leave a single value's output at 2^51, above
// FP64's noise
template <int N> __host__ __device__ constexpr bool fx_renorm() { return N >= 1024; }

// (x + i y) * w with w = (c.hi, c.lo, s.hi, s.lo), c = c.hi 2^32 + c.lo with a
// signed low word: the high 64 bits of the products, without low x low.  The
// operands' low words are made signed too, so that every partial product is a
// signed 32x32->64 multiply-add.  |x|, |y| < 2^62.5 and |w| <= 2^62 keep the
// cross terms below 2^63.
__device__ __forceinline__ void fx_cmul(fxc& v, const int4 w) {
  const int xl = (int)v.x, yl = (int)v.y;
  const int xh = (int)(v.x >> 32) + (int)((unsigned)xl >> 31);
  const int yh = (int)(v.y >> 32) + (int)((unsigned)yl >> 31);
  const int nsh = -w.z, nsl = -w.w;
  long long cr = (long long)xh * w.y + 0x80000000LL;
  long long ci = (long long)xh * w.w + 0x80000000LL;
  cr += (long long)xl * w.x;
  ci += (long long)xl * w.z;
  cr += (long long)yh * nsl;
  ci += (long long)yh * w.y;
  cr += (long long)yl * nsh;
  ci += (long long)yl * w.x;
  long long re = (long long)xh * w.x + (cr >> 32);
  long long im = (long long)xh * w.z + (ci >> 32);
  re += (long long)yh * nsh;
  im += (long long)yh * w.x;
  v.x = re;
  v.y = im;
}

// x / sqrt(2): x + x (h - 1), h = 2^-1/2, (h - 1) 2^64 split as above
__device__ __forceinline__ long long fx_mulh(long long x) {
  constexpr long long W = -0x4AFB0CCC06219B7CLL;    // round((2^-1/2 - 1) 2^64)
  constexpr int cl = (int)W;
  constexpr int ch = (int)((W - (long long)cl) >> 32);
  const int xl = (int)x, xh = (int)(x >> 32) + (int)((unsigned)xl >> 31);
  long long c = (long long)xh * cl + 0x80000000LL;
  c += (long long)xl * ch;
  return x + ((long long)xh * ch + (c >> 32));
}

__device__ __forceinline__ fxc fx_add(fxc a, fxc b) { a.x += b.x; a.y += b.y; return a; }
__device__ __forceinline__ fxc fx_sub(fxc a, fxc b) { a.x -= b.x; a.y -= b.y; return a; }
__device__ __forceinline__ fxc fx_mul_mi(fxc a) { fxc r; r.x = a.y; r.y = -a.x; return r; }   // * -i

// (x + 2^(s-1)) >> s
__device__ __forceinline__ fxc fx_shr(fxc a, int s) {
  const long long h = 1LL << (s - 1);
  a.x = (a.x + h) >> s;
  a.y = (a.y + h) >> s;
  return a;
}

// forward DFTs of 4, 8 and R values
__device__ __forceinline__ void fx_dft4(fxc* v) {
  const fxc s02 = fx_add(v[0], v[2]), d02 = fx_sub(v[0], v[2]);
  const fxc s13 = fx_add(v[1], v[3]), t = fx_sub(v[1], v[3]);
  v[0] = fx_add(s02, s13);
  v[2] = fx_sub(s02, s13);
  // d02 +- (-i) t
  v[1].x = d02.x + t.y; v[1].y = d02.y - t.x;
  v[3].x = d02.x - t.y; v[3].y = d02.y + t.x;
}
__device__ __forceinline__ void fx_dft8(fxc* v) {
  fxc a[4], b[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) { a[n] = fx_add(v[n], v[n + 4]); b[n] = fx_sub(v[n], v[n + 4]); }
  // b[n] *= W8^n
  fxc t = b[1];
  b[1].x = fx_mulh(t.x + t.y);
  b[1].y = fx_mulh(t.y - t.x);
  b[2] = fx_mul_mi(b[2]);
  t = b[3];
  b[3].x = fx_mulh(t.y - t.x);
  b[3].y = -fx_mulh(t.x + t.y);
  fx_dft4(a);
  fx_dft4(b);
  v[0] = a[0]; v[2] = a[1]; v[4] = a[2]; v[6] = a[3];
  v[1] = b[0]; v[3] = b[1]; v[5] = b[2]; v[7] = b[3];
}
template <int R> __device__ __forceinline__ void fx_dft(fxc* v) {
  if constexpr (R == 8) fx_dft8(v);
  else if constexpr (R == 4) fx_dft4(v);
  else { const fxc t = v[0]; v[0] = fx_add(t, v[1]); v[1] = fx_sub(t, v[1]); }
}

// one later pass's butterfly: scale, twiddle, DFT; twp: the pass's table
template <int N, int R, int NS> __device__ __forceinline__ void fx_butterfly(fxc* v, const int4* __restrict__ tw, int k) {
  constexpr int s = fx_shift<N>(NS), off = fx_tw_off<N>(NS);
  v[0] = fx_shr(v[0], s);
#pragma unroll
  for (int r = 1; r < R; ++r) fx_cmul(v[r], tw[off + (r - 1) * NS + k]);
  fx_dft<R>(v);
}

// --- doubles <-> integers ---------------------------------------------------
// hi word of |x|: its maximum orders the inputs' magnitudes
__device__ __forceinline__ unsigned fx_mag(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// transforms whose largest biased exponent is below this are scaled by 2^512
// first (exact), so that subnormal inputs need no case of their own
constexpr int kFxTiny = 64;
// Exponents: an integer m stands for m 2^(base-1023).  kFxNan: a transform
// with a non-finite input (bases are sums of a few of these).
constexpr int kFxNan = 1 << 20;
// x 2^(BITS-E) truncated, be >= kFxTiny the largest biased exponent (E = be - 1022)
template <int BITS = 59> __device__ __forceinline__ long long fx_in1(double x, int be) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  const int d = min(be - ((hi >> 20) & 0x7ff), 63);
  unsigned long long m = ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32 | lo) << (BITS - 53);
  m >>= d;
  const long long s = (long long)(hi >> 31);
  return ((long long)m ^ s) - s;
}
// the base of integers of BITS bits whose largest magnitude bits are mag; be:
// the exponent that fx_in1 takes, and whether its inputs are scaled by 2^512
// first
template <int BITS> __device__ __forceinline__ int fx_base(unsigned mag, int& be, bool& tiny) {
  be = (int)(mag >> 20);
  const int base = be >= 2047 ? kFxNan : max(be, 1) - (BITS - 1);
  tiny = be < kFxTiny;
  if (tiny) be = max(be, 1) + 512;
  return base;
}
// m 2^(base-1075-...) to the nearest double: base is the biased exponent of
// the integer's bit 0, 1 <= base and base + 63 <= 2046
__device__ __forceinline__ double fx_out1(long long m, int base) {
  const long long s = m >> 63;
  const unsigned long long a = (unsigned long long)((m ^ s) - s);
  const int lz = __clzll((long long)a);
  const unsigned long long t = a << (lz & 63);
  unsigned long long r = (t >> 11) + ((t >> 10) & 1ull) + ((unsigned long long)(unsigned)(base + 62 - lz) << 52);
  r = a ? r : 0ull;
  return __longlong_as_double((long long)(r | ((unsigned long long)s & 0x8000000000000000ull)));
}
__device__ __forceinline__ bool fx_is_nan(int base) { return base > (1 << 18); }
// whether every integer's double is a normal number (or zero)
__device__ __forceinline__ bool fx_fast(int base) { return base >= 1 && base + 63 <= 2046; }
// 2^e, -1022 <= e <= 1023
__device__ __forceinline__ double fx_pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }
// o <- o 2^(base-1023) for normal o in [1, 2^63] or 0, at scales where the
// result may be subnormal, zero, infinite or NaN: three exact powers of two,
// of which only the last can round
struct FxScale {
  double a, b, c;
  __device__ __forceinline__ explicit FxScale(int base) {
    const int e = min(max(base - 1023, -2400), 2400), t = e / 3;
    a = fx_is_nan(base) ? __longlong_as_double(0x7ff8000000000000ll) : fx_pow2(t);
    b = fx_pow2(t);
    c = fx_pow2(e - 2 * t);
  }
  __device__ __forceinline__ double operator()(double o) const { return ((o * a) * b) * c; }
};
// doubles of the integers v, M complex values with parts x 2^(base.x-1023),
// y 2^(base.y-1023); SWAP exchanges the parts.  One branch for all of them: a
// rescaling per value was predicated into every conversion and made the
// kernels 25-50 % slower.
template <int M, bool SWAP> __device__ __forceinline__ void fx_doubles(const fxc* v, double2* o, int2 base) {
  const bool fast = fx_fast(base.x) && fx_fast(base.y);
  const int bx = fast ? base.x : 1023, by = fast ? base.y : 1023;
#pragma unroll
  for (int r = 0; r < M; ++r) {
    const double x = fx_out1(v[r].x, bx), y = fx_out1(v[r].y, by);
    o[r] = SWAP ? make_double2(y, x) : make_double2(x, y);
  }
  if (!fast) {
    const FxScale sx(SWAP ? base.y : base.x), sy(SWAP ? base.x : base.y);
#pragma unroll
    for (int r = 0; r < M; ++r) { o[r].x = sx(o[r].x); o[r].y = sy(o[r].y); }
  }
}
template <int M, bool SWAP> __device__ __forceinline__ void fx_doubles(const fxc* v, double2* o, int base) {
  fx_doubles<M, SWAP>(v, o, make_int2(base, base));
}
// bits set in any of the magnitudes' high words (x ^ sign): of the parts x, of
// the parts y, of both
__device__ __forceinline__ unsigned fx_hibits(long long x) { const int a = (int)(x >> 32); return (unsigned)(a ^ (a >> 31)); }
template <int R> __device__ __forceinline__ uint2 fx_bits2(const fxc* v) {
  uint2 o = make_uint2(0u, 0u);
#pragma unroll
  for (int r = 0; r < R; ++r) { o.x |= fx_hibits(v[r].x); o.y |= fx_hibits(v[r].y); }
  return o;
}
template <int R> __device__ __forceinline__ unsigned fx_bits(const fxc* v) {
  const uint2 o = fx_bits2<R>(v);
  return o.x | o.y;
}
// Growth.  A transform's inputs have components below 2^59: a modulus below
// 2^59.5, or 2^59 for each of two real rows packed as one complex input.  A
// pass of radix R lets either grow by R / 2^shift at most.  Every output has
// to stay below 2^63 in modulus; where the rows are then separated (ROWS), the
// sum of two outputs, twice one row's spectrum, has to as well.  Lengths that
// renormalise set the modulus back before each later pass, to components
// below 2^fx_top: 2^61, and 2^60 before a last pass that grows the rows by
// more than the sums leave room for (n = 1024, whose radix 8 follows a radix
// 2: there rows beside a zero or much smaller row reached 2^63.5).
// Twice the base-2 logarithms:
__host__ __device__ constexpr int fx_grow2(int r, int shift) { return 2 * (fx_log2(r) - shift); }
template <int N, bool ROWS> __host__ __device__ constexpr int fx_top(int ns) {
  return ROWS && ns * fx_radix(N, ns) == N && 2 * 61 + 1 + fx_grow2(fx_radix(N, ns), fx_shift<N>(ns)) > 2 * 62 ? 60 : 61;
}
template <int N> __host__ __device__ constexpr bool fx_growth_ok(bool fit) {
  int mod = 2 * 59 + 1 + 2 * 3, row = 2 * 59 + 2 * 3;     // after the first pass
  for (int s = 8; s < N; s *= fx_radix(N, s)) {
    if (fx_renorm<N>() || (fit && s == 8)) {      // (left shifts only)
      const int top = 2 * fx_top<N, true>(s) + 1;
      mod = mod > top ? mod : top;
      row = row > top ? row : top;
    }
    const int g = fx_grow2(fx_radix(N, s), fx_shift<N>(s));
    mod += g;
    row += g;
    if (mod >= 2 * 63 || 2 * 61 + 1 + g >= 2 * 63) return false;
  }
  return row <= 2 * 62;
}
template <int N> __host__ __device__ constexpr bool fx_growth_ok() { return fx_growth_ok<N>(false) && fx_growth_ok<N>(true); }
static_assert(fx_growth_ok<16>() && fx_growth_ok<32>() && fx_growth_ok<64>() && fx_growth_ok<128>() && fx_growth_ok<256>() &&
              fx_growth_ok<512>() && fx_growth_ok<1024>(), "the integers stay in 64 bits");
// left shift that brings components with these bits below 2^TOP
template <int TOP> __device__ __forceinline__ int fx_room(unsigned o) { return max(__clz((int)o) - (64 - TOP), 0); }
template <int R> __device__ __forceinline__ void fx_shl(fxc* v, int s) {
#pragma unroll
  for (int r = 0; r < R; ++r) { v[r].x <<= s; v[r].y <<= s; }
}
// shared copy of the per-pass integer twiddles (at most N entries; the host
// lays them out as load_tw_passes does, see fx_twiddles)
template <int N> __host__ __device__ constexpr int fx_tw_count() {
  return fx_tw_off<N>(N);
}
template <int N> __device__ __forceinline__ void fx_load_tw(double2* tw_s, const double2* __restrict__ tw_g, int nt) {
  for (int i = threadIdx.x; i < fx_tw_count<N>(); i += nt) tw_s[i] = tw_g[i];
}

}  // namespace qg
