// Host side of fxfft.cuh: the integer twiddle tables.
#pragma once
#include <cmath>
#include <cstdint>
#include <vector>
#include "fxfft.cuh"

namespace qg {

// Per-pass tables of a length-n transform, four 32-bit words per entry:
// w = W_n^{k r n/(NS R)} 2^(64-s) (s: log2 of the earlier pass's radix, at
// least 2) as cos and -sin, each split into a high and a signed low word, at
// [off(NS) + (r-1) NS + k] for the passes NS > 1.  n entries are returned
// (the tail is unused).  Angles by octant symmetry in long double (a 64-bit
// mantissa or more).
inline std::vector<int32_t> fx_twiddles(int n) {
  std::vector<int32_t> t((size_t)4 * n, 0);
  auto cs = [&](long long m, long double& c, long double& s) {   // cos, sin of 2 pi m / n
    m = ((m % n) + n) % n;
    const long long q = (8 * m) / n;                              // octant
    long long a = m - (q / 2) * (n / 4);                          // reduced to [0, n/4)
    const bool flip = 8 * a > n;                                  // above pi/4
    const long double th = 2.0L * 3.14159265358979323846264338327950288L * (long double)(flip ? n / 4 - a : a) / (long double)n;
    long double c0 = cosl(th), s0 = sinl(th);
    if (flip) { const long double x = c0; c0 = s0; s0 = x; }
    switch (q / 2) {
      case 0: c = c0; s = s0; break;
      case 1: c = -s0; s = c0; break;
      case 2: c = -c0; s = -s0; break;
      default: c = s0; s = -c0; break;
    }
  };
  int off = 0, prev = 1;
  for (int ns = 1; ns < n;) {
    const int R = fx_radix(n, ns);
    if (ns > 1) {
      const int lg = prev == 8 ? 3 : 2;
      for (int r = 1; r < R; ++r)
        for (int k = 0; k < ns; ++k) {
          long double c, s;
          cs((long long)k * r * (n / (ns * R)), c, s);
          const long double sc = ldexpl(1.0L, 64 - lg);
          const long long w[2] = {llrintl(c * sc), llrintl(-s * sc)};
          int32_t* e = &t[4 * (size_t)(off + (r - 1) * ns + k)];
          for (int j = 0; j < 2; ++j) {
            const int32_t lo = (int32_t)(uint32_t)(uint64_t)w[j];
            e[2 * j] = (int32_t)((w[j] - (long long)lo) >> 32);
            e[2 * j + 1] = lo;
          }
        }
      off += ns * (R - 1);
    }
    prev = R;
    ns *= R;
  }
  return t;
}

}  // namespace qg
