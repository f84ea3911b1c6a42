// hmp_ordered_sum.h -- FP32 sums in a fixed order, evaluated in parallel with the sequential sum's
// bits.
//
// s <- fl(s + x) one element after another is one dependent chain. While s stays inside one binade
// (|s| between 2^e and 2^(e+1), unit u = 2^(e-23)) it is a whole number S of units, and adding x
// adds a whole number of units that depends on S only through its parity:
//   x / u = k + f; f != 1/2: rint(x / u) units; f == 1/2 (a tie): the neighbour that makes the sum
//   even, k or k + 1.
// So an element is a pair of increments (S even, S odd), and runs of elements compose into such
// pairs associatively: a parallel scan gives every partial sum. The run is exact up to the first
// partial sum that leaves the binade (or an element too large to scale); that element is added as
// it stands and the scan goes on from there in its new binade.
#pragma once

#include <math.h>
#include <string.h>

#if defined(__CUDACC__)
#define HMP_HD __host__ __device__ __forceinline__
#else
#define HMP_HD inline
#endif

namespace hmp {

// Increments of a run of elements in units of the sum's last place: d0 if the sum before it is an
// even number of units, d1 if it is odd.
struct OrderedRun {
  int d0, d1;
};

// The pair of one element, r = x / u (exact: u is a power of two). False: too large, or not finite.
// Adding 1.5 * 2^23 leaves r's nearest integer, ties to even, in the low bits of the sum (additions
// only: a conversion issues at a quarter of their rate).
HMP_HD bool ordered_element(float r, OrderedRun& e) {
  constexpr float kMagic = 12582912.0f;
  if (!(fabsf(r) < 4194304.0f)) return false;
  const float t = r + kMagic;
  const float f = r - (t - kMagic);  // exact, |f| <= 1/2
  int bits;
  memcpy(&bits, &t, 4);
  e.d0 = e.d1 = bits - 0x4B400000;
  if (fabsf(f) == 0.5f) e.d1 += f > 0.f ? 1 : -1;  // d0 is the even neighbour
  return true;
}

// The increment of an element that is neither a tie nor too large, without branches; false: it is one of
// those, and d means nothing.
HMP_HD bool ordered_plain(float r, int& d) {
  constexpr float kMagic = 12582912.0f;
  const float t = r + kMagic;
  const float f = r - (t - kMagic);
  int bits;
  memcpy(&bits, &t, 4);
  d = int(unsigned(bits) - 0x4B400000u);
  return (fabsf(r) < 4194304.0f) & (fabsf(f) != 0.5f);
}

// The units a run adds to a sum of S units (unsigned arithmetic: only partial sums inside the binade
// are used, the ones past the first failure may wrap).
HMP_HD int ordered_apply(OrderedRun e, int S) { return int(unsigned(S) + unsigned((S & 1) ? e.d1 : e.d0)); }

// Run a followed by run b.
HMP_HD OrderedRun ordered_then(OrderedRun a, OrderedRun b) {
  OrderedRun c;
  c.d0 = int(unsigned(a.d0) + unsigned((a.d0 & 1) ? b.d1 : b.d0));
  c.d1 = int(unsigned(a.d1) + unsigned((a.d1 & 1) ? b.d0 : b.d1));
  return c;
}

// Partial sums strictly inside the binade: the sum before rounding was inside it too.
HMP_HD bool ordered_inside(int S) {
  const unsigned a = S < 0 ? 0u - unsigned(S) : unsigned(S);
  return a > 8388608u && a < 16777216u;
}

// Whether a sum can be scanned from (its unit and scale are normal numbers), its scale 1/u and unit u.
HMP_HD bool ordered_scale(float s, float& scale, float& unit) {
  unsigned bits;
  memcpy(&bits, &s, 4);
  const unsigned e = (bits >> 23) & 255u;  // |s| in [2^(e-127), 2^(e-126)), u = 2^(e-150)
  if (e < 24u || e > 254u) return false;
  const unsigned sb = (277u - e) << 23, ub = (e - 23u) << 23;
  memcpy(&scale, &sb, 4);
  memcpy(&unit, &ub, 4);
  return true;
}

}  // namespace hmp
