// FP64 data in 64-bit fixed point on the integer pipe.
//
// GB300 issues one FP64 warp instruction per SM sub-partition every 64 cycles (measured: DFMA 64.1, DADD 64-76),
// a 32 x 32 + 64-bit integer multiply-add (IMAD.WIDE) every 2.1, a 64-bit add every 2-3.  The transforms and
// the block matvecs of the implicit solves are sums of products with known operators over a row or a vector
// whose largest entry is easy to find, so they run on integers: a vector is scaled by one power of two to a
// 64-bit integer each, an operator by one per row (on the host), both are split into two signed 32-bit digits
// (value = hi 2^32 + lo, lo in [-2^31, 2^31)), and a product keeps three of its four digit products in two
// 64-bit accumulators (hi hi, and hi lo + lo hi; lo lo is below the last bit kept).  The sums are exact, so
// they do not depend on their order.  Rounding to 57-60 bits below a bound on the vector replaces FP64's 53
// bits per operation: against extended precision the errors are below FP64's (transforms: the bound is the
// row's 1-norm, which no intermediate value exceeds; matvecs: 1e-18 to 1e-17 of the result's norm against
// 1.5e-16 to 1e-15 on states of the time step).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sdd {

using i64 = long long;
using u64 = unsigned long long;

__device__ __forceinline__ int fx_lo(i64 x) { return (int)x; }
__device__ __forceinline__ int fx_hi(i64 x) { return (int)(x >> 32) + (int)((unsigned)x >> 31); }
__device__ __forceinline__ i64 fx_mad(int a, int b, i64 c) { return (i64)a * b + c; }

// Host: v = hi 2^32 + lo with lo in (-2^31, 2^31) (never -2^31, so that the digits can be negated).
inline void fx_split_host(i64 v, int* hi, int* lo) {
  int l = (int)(uint32_t)(u64)v;
  if (l == INT32_MIN) {
    ++v;
    l = (int)(uint32_t)(u64)v;
  }
  *lo = l;
  *hi = (int)((v - l) >> 32);
}

// round(x 2^s), c = 1084 - s; the caller's scale keeps |x| 2^s < 2^62.  Subnormal x gives 0.
__device__ __forceinline__ i64 d2fx(double x, int c) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ffu);
  const u64 m = (((u64)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << 10;
  const int r = e ? min(c - e, 63) : 63;
  const i64 q = (i64)(((m >> r) + 1) >> 1);
  return (int)hi < 0 ? -q : q;
}

// v 2^-s as a double (rounded to nearest; below the normal range 0)
__device__ __forceinline__ double fx2d(i64 v, int s) {
  u64 a = (u64)(v < 0 ? -v : v);
  const int lz = __clzll((i64)a);
  const int e = 1086 - lz - s;                       // biased exponent
  a <<= (lz & 63);
  u64 bits = ((u64)(unsigned)(e - 1) << 52) + (a >> 11) + ((a >> 10) & 1);
  if (e >= 2047) bits = 0x7ff0000000000000ull;
  if (v == 0 || e <= 0) bits = 0;
  return __longlong_as_double((i64)(bits | ((u64)v & 0x8000000000000000ull)));
}

__device__ __forceinline__ double fx_nan() { return __longlong_as_double(0x7ff8000000000000ll); }

// |x|'s high word: its unsigned order is the order of magnitudes (to 20 mantissa bits)
__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

// -x or x by the sign bit (an FP64 negation or product would take the FP64 pipe)
__device__ __forceinline__ double neg_if(double x, bool n) {
  return __hiloint2double(__double2hiint(x) ^ (n ? (int)0x80000000 : 0), __double2loint(x));
}

// a w with w given in digits (c1, c0, s1, s0) of round(w 2^62), x -> .x c - .y s, .x s + .y c; NEG: conj(w).
// |a| components at most 2^62 in complex magnitude: no accumulator overflows.
template <bool NEG>
__device__ __forceinline__ longlong2 fx_cmul(longlong2 a, int4 w) {
  const int a0 = fx_lo(a.x), a1 = fx_hi(a.x), b0 = fx_lo(a.y), b1 = fx_hi(a.y);
  const int c1 = w.x, c0 = w.y, s1 = NEG ? -w.z : w.z, s0 = NEG ? -w.w : w.w;
  const i64 R = 1ll << 29;
  const i64 r2 = fx_mad(a1, c1, (i64)b1 * -s1);
  const i64 r1 = fx_mad(a1, c0, fx_mad(a0, c1, fx_mad(b1, -s0, fx_mad(b0, -s1, R))));
  const i64 q2 = fx_mad(a1, s1, (i64)b1 * c1);
  const i64 q1 = fx_mad(a1, s0, fx_mad(a0, s1, fx_mad(b1, c0, fx_mad(b0, c1, R))));
  longlong2 o;
  o.x = (r2 << 2) + (r1 >> 30);
  o.y = (q2 << 2) + (q1 >> 30);
  return o;
}

// x h for a real constant h = (h1 2^32 + h0) 2^-62
__device__ __forceinline__ i64 fx_rmul(i64 x, int h1, int h0) {
  const int x0 = fx_lo(x), x1 = fx_hi(x);
  return (((i64)x1 * h1) << 2) + (fx_mad(x1, h0, fx_mad(x0, h1, 1ll << 29)) >> 30);
}

// Scales of K rows by their 1-norms and their conversion in place.  Row t holds P doubles at XV + t P; mx[t]
// is the calling thread's maximum of abs_hi over its elements k = tid, tid + blockDim, ... (only those were
// written by it: no barrier is needed before the call).  Afterwards the row holds round(x 2^(60 - E[t])) as
// 64-bit integers with sum |x| < 2^E[t]: the row's transform and everything inside it stays below 2^61 (two
// rows of a pair).  E[t] = kFxBad marks a row with an infinity or NaN (left as zeros).  red: 2 K 32 words.
// Ends with a barrier.
constexpr int kFxBad = 0x7fffffff;
template <int K>
__device__ __forceinline__ void rows_to_fixed(double* XV, int P, int nrows, const unsigned (&mx)[K], unsigned* red,
                                              int* E) {
  const int tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = bd >> 5;
#pragma unroll
  for (int t = 0; t < K; ++t) {
    if (t < nrows) {
      const int ew = (int)(__reduce_max_sync(0xffffffffu, mx[t]) >> 20);
      unsigned s = 0;
      for (int k = tid; k < P; k += bd) {
        const unsigned h = abs_hi(XV[t * P + k]);
        const int e = (int)(h >> 20);
        if (e) s += (((h & 0xfffffu) | 0x100000u) >> min(ew - e, 31)) + 1;
      }
      s = __reduce_add_sync(0xffffffffu, s);
      if (lane == 0) {
        red[t * 32 + warp] = (unsigned)ew;
        red[(K + t) * 32 + warp] = s;
      }
    }
  }
  __syncthreads();
  for (int t = warp; t < K; t += nw) {                 // (a row that is not there gets a zero row's scale)
    const bool on = t < nrows && lane < nw;
    const unsigned e = on ? red[t * 32 + lane] : 0u;
    const unsigned s = on ? red[(K + t) * 32 + lane] : 0u;
    const unsigned em = __reduce_max_sync(0xffffffffu, e);
    const unsigned tot = __reduce_add_sync(0xffffffffu, s ? ((s >> 3) >> min(em - e, 31u)) + 1 : 0u);
    if (lane == 0) E[t] = em >= 0x7ffu ? kFxBad : (int)em - 1040 + (32 - __clz((int)tot));
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < K; ++t) {
    if (t < nrows) {
      const int et = E[t];
      for (int k = tid; k < P; k += bd)
        reinterpret_cast<i64*>(XV)[t * P + k] = et == kFxBad ? 0 : d2fx(XV[t * P + k], 1024 + et);
    }
  }
  __syncthreads();
}

}  // namespace sdd
