// Nearest entry of a sorted 256-entry code book (the blockwise 8-bit optimizer-state codec).
//
// A binary search costs eight dependent shared-memory reads per value at addresses that differ from
// thread to thread (bank conflicts), and a coarse bracket with a scan behind it still three to six.
// Here the value's own bit pattern picks a bin so narrow that at most one boundary between two
// codes lies in it: sign, exponent (2^-24 .. 1) and the top 6 mantissa bits for the signed book
// (densest spacing 0.014 in [0.5, 1)), 7 for the unsigned one (0.007, no sign).  Two reads remain: the
// code below the bin's boundary, and the boundary itself, the largest float that still goes to the
// lower code.  Boundaries are found with the comparison that defines "nearest" (x - lo <= hi - x, ties
// to the lower code), so the result is the one a search with that comparison gives, bit for bit.
// A CTA derives the tables from the code book when it starts, so callers pass nothing new; a book
// so dense that a bin holds two boundaries is scanned forward from the bin's code.
#pragma once
#include <stdint.h>

namespace cbk {

template <bool SIGNED>
struct Book {
  static constexpr int kSub = SIGNED ? 6 : 7;                   // mantissa bits in the bin number
  static constexpr int kHalf = (24 << kSub) + 2;                // |x| < 2^-24, 24 exponents, |x| >= 1
  static constexpr int kBins = SIGNED ? 2 * kHalf : kHalf;
  float value[256];
  float bound[256];          // bound[c]: the largest float that belongs to a code <= c
  uint8_t base[kBins];       // codes whose bound lies below the bin
  int dense;                 // some bin holds two bounds

  // Bin of x, ascending with x.  |x| <= 1 is expected; anything else, NaN included, lands in a valid bin.
  static __device__ __forceinline__ int bin(float x) {
    const uint32_t b = __float_as_uint(x);
    int k = static_cast<int>((b & 0x7fffffffu) >> (23 - kSub)) - (103 << kSub);
    k = min(max(k, -1), 24 << kSub) + 1;
    if (SIGNED) return (b >> 31) ? kHalf - 1 - k : kHalf + k;
    return (b >> 31) ? 0 : k;
  }

  // All threads of a CTA of at least 256 call it; the CTA is synchronised on return.
  __device__ __forceinline__ void build(const float* __restrict__ book) {
    const int t = threadIdx.x;
    if (t < 256) value[t] = book[t];
    if (t == 0) dense = 0;
    __syncthreads();
    if (t < 255) {
      // bisection over the floats from value[t] (lower code) to value[t + 1]
      const float a = value[t], b = value[t + 1];
      int lo = ordered(a), hi = ordered(b);
      while (hi - lo > 1) {
        const int mid = lo + ((hi - lo) >> 1);
        const float x = unordered(mid);
        if (x - a <= b - x) lo = mid; else hi = mid;
      }
      bound[t] = unordered(lo);
    } else if (t == 255) {
      bound[255] = INFINITY;
    }
    __syncthreads();
    if (t < 256) {
      const int first = t == 0 ? 0 : bin(bound[t - 1]) + 1;
      const int last = t == 255 ? kBins - 1 : bin(bound[t]);
      if (t > 0 && t < 255 && last < first) dense = 1;
      for (int e = first; e <= last; ++e) base[e] = static_cast<uint8_t>(t);
    }
    __syncthreads();
  }

  __device__ __forceinline__ int nearest(float x) const {
    int c = base[bin(x)];
    if (!dense) return c + (x > bound[c] ? 1 : 0);
    while (c < 255 && x > bound[c]) ++c;
    return c;
  }

 private:
  // Order-preserving map between finite floats and ints (distance between neighbours 1).
  static __device__ __forceinline__ int ordered(float x) {
    const int b = __float_as_int(x);
    return b >= 0 ? b : static_cast<int>(0x80000000u - static_cast<uint32_t>(b));
  }
  static __device__ __forceinline__ float unordered(int o) {
    return __int_as_float(o >= 0 ? o : static_cast<int>(0x80000000u - static_cast<uint32_t>(o)));
  }
};

}  // namespace cbk
