// mic_pivot.cuh -- a column's pivot: the search for the largest value over a warp's offers, and the
// pivot's reciprocal (mic_front_lu.cu).
#ifndef MIC_PIVOT_CUH
#define MIC_PIVOT_CUH

#include "mic_internal.cuh"

namespace mic {

// What a row offers as pivot of a column: |a| as an integer (all 63 bits; the images of non-negative
// doubles order as they do), its row beside it.  -1 is a NaN, -2 no row.
struct Offer {
  long long key;
  int row;
};
__device__ __forceinline__ long long pivot_key(double a) {
  const long long b = dbits(a) & 0x7fffffffffffffffLL;
  return b <= 0x7ff0000000000000LL ? b : -1;
}
__device__ __forceinline__ void take_better(Offer &o, double a, int row) {
  const long long k = pivot_key(a);
  if (k > o.key) {
    o.key = k;
    o.row = row;
  }
}
// The lane with the warp's largest key, the first of equal ones: the largest high word, then the
// largest low word of the lanes that have it.  Twice a column on the chain of a front's columns.  GB300,
// solves of 129 x 33 and 513 x 129 Stokes and of 513 x 129 temperatures: 1.96, 38.2 and 4.66 ms; with
// the second reduction behind a branch (only where lanes share the high word) 1.99, 38.2 and 4.68; high
// words alone 1.93, 38.2 and 4.63.  The leading 21 bits and the row in one integer, a single reduction,
// would take rows for equal that differ by 2^-10.
__device__ __forceinline__ int warp_best(long long key) {
  const int hi = (int)(key >> 32), top = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == top ? (unsigned)key : 0u, most = __reduce_max_sync(0xffffffffu, lo);
  return __ffs(__ballot_sync(0xffffffffu, hi == top && lo == most)) - 1;
}

// a column whose best key is 0 or less (every a zero or NaN): the largest |a| of the rows not used, the
// first of them when there is no other
__device__ inline int pivot_rare(const double *col, int stride, int rows, const int *used) {
  long long best = -2;
  int p = 0;
  for (int r = 0; r < rows; ++r) {
    if (used && used[r]) continue;
    const long long k = pivot_key(col[(int64_t)r * stride]);
    if (k > best) {
      best = k;
      p = r;
    }
  }
  return p;
}

// 1 / p by Newton's iteration of third order from an FP32 reciprocal of p's mantissa: with
// e = 1 - m r, |e| < 2^-22, r (1 + e + e^2) is 1 / m to e^3 < 2^-66, so to rounding, in three
// dependent FP64 operations (a pivot's reciprocal is on the chain of every column step).  Pivots
// whose reciprocal leaves the normal range are divided.
__device__ __forceinline__ double pivot_rcp(double p) {
  const unsigned long long b = (unsigned long long)dbits(p);
  const int ex = (int)(b >> 52) & 0x7ff;
  if (ex < 8 || ex > 2038) return p != 0.0 ? 1.0 / p : 0.0;
  const double m = __longlong_as_double((long long)((b & 0xfffffffffffffULL) | 0x3ff0000000000000ULL));
  const float f = __uint_as_float(0x3f800000u | ((unsigned)(b >> 29) & 0x7fffffu));
  const double r0 = f64_of(__frcp_rn(f));
  const double e = fma(-m, r0, 1.0);
  const double r = fma(r0, fma(e, e, e), r0);  // in (1/2, 1]
  const long long rb = dbits(r) - ((long long)(ex - 1023) << 52);
  return __longlong_as_double(rb | (long long)(b & 0x8000000000000000ULL));
}

}  // namespace mic

#endif
