// FP64 data in 64-bit fixed point on the integer pipe.
//
// GB300 issues one FP64 warp instruction per SM sub-partition every 64 cycles (measured: DFMA 64.1, DADD 64-76),
// a 32 x 32 + 64-bit integer multiply-add every 4.5 to 5, a 64-bit add every 2.2.  The transforms and
// the block matvecs of the implicit solves are sums of products with known operators over a row or a vector
// whose largest entry is easy to find, so they run on integers: a vector is scaled by one power of two to a
// 64-bit integer each, an operator by one per row and one per column, both are split into two signed digits
// (transforms: value = hi 2^32 + lo; matvecs: see mv_digits), and a product keeps three of its four digit products in
// 64-bit accumulators (hi hi, hi lo and lo hi; lo lo is below the last bit kept).  The sums are exact, so they do not
// depend on their order.  Rounding to 59-61 bits below a bound on the vector replaces FP64's 53 bits per operation.
// Transforms: the bound is the row's 1-norm, which no intermediate value exceeds; the errors are below FP64's.
// Matvecs: operators keep 59 bits below a row's 1-norm, operands 61 below their largest entry, both after the
// columns' scales 2^cx, so a row r of a product A x is off by at most
//   2^-58 (n + 2) (sum_k |A_rk| 2^-cx_k) max_k |x_k 2^cx_k|      (n columns)
// and in the norm by less than FP64: on smooth profiles Dr's products 0.03 to 0.4 of FP64's error (N_r 8 to 65; rows
// against their own sum |A||x| 0.4 of a rounding at most, FP64 0.3 to 0.6), the solves' 1e-18 to 2e-17 of the result
// against 1e-16 to 5e-16.  What FP64 has and this has not is the relative precision of single small entries: where the operand
// falls off steeply (a layer of 1/60 of the gap), rows in its tail, whose own sum |A||x| is 1e-3 to 1e-12 of the largest,
// keep 2e-15 to 4e-13 of that sum (N_r 20 to 65) where FP64 keeps 2e-16 and the inverse itself is good to 1e-15 to
// 3e-14.
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

// The high word of |x|'s significand, 53 bits in all, from |x|'s high word h (below the normal range without the leading
// one); |x| = that 2^(e1 - 1075) with the exponent e1, the exponent field or 1.
__device__ __forceinline__ unsigned fx_mant_hi(unsigned h, int& e1) {
  e1 = max((int)(h >> 20), 1);
  return h + 0x100000u - ((unsigned)e1 << 20);
}

// round(x 2^s), c = 1084 - s; the caller's scale keeps |x| 2^s < 2^62, and s <= 1083 where x is below the normal range.
__device__ __forceinline__ i64 d2fx(double x, int c) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  int e1;
  const u64 m = (((u64)fx_mant_hi(hi & 0x7fffffffu, e1) << 32) | lo) << 10;
  const i64 q = (i64)(((m >> min((unsigned)(c - e1), 63u)) + 1) >> 1);
  return (int)hi < 0 ? -q : q;
}

// v 2^-s as a double (rounded to nearest, also below the normal range)
__device__ __forceinline__ double fx2d(i64 v, int s) {
  u64 a = (u64)(v < 0 ? -v : v);
  const int lz = __clzll((i64)a);
  const int e = 1086 - lz - s;                       // biased exponent
  a <<= (lz & 63);
  u64 bits = ((u64)(unsigned)(e - 1) << 52) + (a >> 11) + ((a >> 10) & 1);
  if (e >= 2047) bits = 0x7ff0000000000000ull;
  if (e <= 0) bits = e > -53 ? ((a >> (11 - e)) + 1) >> 1 : 0;   // in units of 2^-1074
  if (v == 0) bits = 0;
  return __longlong_as_double((i64)(bits | ((u64)v & 0x8000000000000000ull)));
}

// The same by the FP64 pipe's conversion: half the latency (66 against 107 cycles), as many cycles of issue;
// for a lone dependent value.  Below the normal range out of line: inside, either form of it made the chains of 64
// shells of 256 x 30 133 us instead of 125.
static __device__ __noinline__ double fx2d_small(i64 v, int s) { return fx2d(v, s); }
__device__ __forceinline__ double fx2d_lat(i64 v, int s) {
  const double d = __ll2double_rn(v);
  const int hi = __double2hiint(d), e = ((hi >> 20) & 0x7ff) - s;
  const double r = __hiloint2double(hi - (s << 20), __double2loint(d));
  if (v == 0) return 0.0;
  if (e <= 0) return fx2d_small(v, s);
  return e >= 2047 ? __longlong_as_double((v < 0 ? 0xfff0000000000000ll : 0x7ff0000000000000ll)) : r;
}

// n < 2^31 as a double by its bits (the conversion takes the FP64 pipe)
__device__ __forceinline__ double fx_int(unsigned n) {
  if (n == 0) return 0.0;
  const int lz = __clz((int)n);
  return __longlong_as_double((i64)(((u64)(1054 - lz) << 52) + (((u64)(n << lz) << 21) & 0xfffffffffffffull)));
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

// Scales of rows by their 1-norms and their conversion in place.  Row t holds P doubles at XV + t P, of which the
// calling thread wrote the elements k = tid, tid + blockDim, ... (no barrier is needed before the call).
// Afterwards the row holds round(x 2^(60 - E[t])) as 64-bit integers with sum |x| < 2^E[t]: the row's transform
// and everything inside it stays below 2^61 (two rows of a pair).  E is -1022 at least (2^-1082 a unit: all of a
// number below the normal range, which has no leading bit to shift up).  E[t] = kFxBad marks a row with an infinity
// or NaN (left as zeros); E of the row after an odd last one is a zero row's.  The sum is of whole numbers in units
// of the row's largest exponent, so E does not depend on how many threads share the row.  red: 2 nrows 32 words.
// Ends with a barrier.
constexpr int kFxBad = 0x7fffffff;
// (Out of line, with byte offsets into the dynamic shared memory, like the transforms' passes.)
static __device__ __noinline__ void rows_to_fixed_at(int xv, int P, int nrows, int redo, int eo) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* XV = reinterpret_cast<double*>(smem_raw + xv);
  unsigned* red = reinterpret_cast<unsigned*>(smem_raw + redo);
  int* E = reinterpret_cast<int*>(smem_raw + eo);
  const int tid = threadIdx.x, bd = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = bd >> 5;
#pragma unroll 1
  for (int t = 0; t < nrows; ++t) {
    const double* x = XV + t * P;
    unsigned m = 0;
#pragma unroll 1
    for (int k = tid; k < P; k += bd) m = max(m, abs_hi(x[k]));
    m = __reduce_max_sync(0xffffffffu, m) >> 20;
    if (lane == 0) red[t * 32 + warp] = m;
  }
  __syncthreads();
#pragma unroll 1
  for (int t = 0; t < nrows; ++t) {
    const double* x = XV + t * P;
    const int em = max((int)__reduce_max_sync(0xffffffffu, lane < nw ? red[t * 32 + lane] : 0u), 1);
    unsigned s = 0;                                    // (at most 2^18 an element)
#pragma unroll 1
    for (int k = tid; k < P; k += bd) {
      const unsigned h = abs_hi(x[k]);                 // (numbers below 2^-1042 do not count: E is -1022 at least)
      int e1;
      const unsigned m = fx_mant_hi(h, e1);
      if (h) s += (m >> min(em - e1 + 3, 31)) + 1;
    }
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) red[(nrows + t) * 32 + warp] = s;
  }
  __syncthreads();
#pragma unroll 1
  for (int t = warp; t < ((nrows + 1) & ~1); t += nw) {
    const bool on = t < nrows && lane < nw;
    const unsigned em = max(__reduce_max_sync(0xffffffffu, on ? red[t * 32 + lane] : 0u), 1u);
    const unsigned tot = __reduce_add_sync(0xffffffffu, on ? red[(nrows + t) * 32 + lane] : 0u);
    if (lane == 0) E[t] = em >= 0x7ffu ? kFxBad : max((int)em - 1040 + (32 - __clz((int)tot)), -1022);
  }
  __syncthreads();
#pragma unroll 1
  for (int t = 0; t < nrows; ++t) {
    const int et = E[t];
#pragma unroll 1
    for (int k = tid; k < P; k += bd)
      reinterpret_cast<i64*>(XV)[t * P + k] = et == kFxBad ? 0 : d2fx(XV[t * P + k], 1024 + et);
  }
  __syncthreads();
}

__device__ __forceinline__ void rows_to_fixed(double* XV, int P, int nrows, void* red, int* E) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto off = [&](const void* p) { return (int)(reinterpret_cast<const unsigned char*>(p) - smem_raw); };
  rows_to_fixed_at(off(XV), P, nrows, off(red), off(E));
}

// ---- block matvecs -------------------------------------------------------------------------------
// An nr x nr block A in global memory, padded with zeros to L x L (L = fx_ld(nr), so that the inner loops have
// no remainder) and its columns scaled to a = A 2^-cx with |a| < 1: word [col][row] = the two digits of
// round(a 2^(59 - ea)) (lo in the low half), then the L rows' exponents ea as ints, sum over a row of
// |a| < 2^ea (kFxBad: a row with an infinity or NaN), and the L columns' exponents cx.  Operands are scaled by
// 2^cx before their largest entry sets their fixed point: so the bits kept are relative to the largest product
// A_kc x_c, not to the largest x_c (the Chebyshev operators' columns differ by N^2 to N^4, and so do a state's
// derivatives against them).  Blocks start on 16 bytes.
__host__ __device__ inline int fx_ld(int nr) { return nr <= 32 ? (nr + 7) / 8 * 8 : (nr + 15) / 16 * 16; }
__host__ __device__ constexpr size_t fx_block_words(int ld) { return (size_t)(ld + 1) * ld; }
__device__ __forceinline__ const int* fx_row_exp(const i64* blk, int ld) {
  return reinterpret_cast<const int*>(blk + (size_t)ld * ld);
}
__device__ __forceinline__ const int* fx_col_exp(const i64* blk, int ld) { return fx_row_exp(blk, ld) + ld; }

// A matvec's digits (lo, hi).  Operators: 59 bits, hi 2^28 + lo with lo in [-2^27, 2^27), hi 31 bits and its sign.
// Operands: 61 bits, hi 2^32 + lo with lo in [-2^31, 2^31), |hi| <= 2^29.  So the sums of at most 64 columns stay in
// 64 bits: a row's |a| add up to 2^59 at most (its scale), hence hi hi to 2^60, hi lo to 2^31 2^31, and lo hi, whose
// operator digits have no such bound, to 64 2^27 2^29.  (27 and 27 bits of lo, 57 of both, cost the same three
// multiplies and lost what FP64 keeps: Dr's products had 1.3 times FP64's error at N_r = 30, 3.2 times at 65.)
constexpr int kMvA = 59, kMvALo = 28, kMvX = 61;
__device__ __forceinline__ int2 mv_digits(i64 a) {
  return make_int2(((int)a << (32 - kMvALo)) >> (32 - kMvALo), (int)((a + (1ll << (kMvALo - 1))) >> kMvALo));
}
__device__ __forceinline__ i64 mv_value(int2 a) { return ((i64)a.y << kMvALo) + a.x; }

// An operand's exponent (biased, after its column scale): x = 0 counts below every number, an infinity above
// (kFxInf), a NaN above that (kFxBad).
constexpr int kFxInf = kFxBad - 1;
__device__ __forceinline__ int fx_key(double x, int cx) {
  const unsigned h = abs_hi(x);
  const int e = (int)(h >> 20);
  if (e == 0x7ff) return ((h & 0xfffffu) | (unsigned)__double2loint(x)) ? kFxBad : kFxInf;
  return h | (unsigned)__double2loint(x) ? e + cx : -0x10000;   // |x| < 2^(e - 1022), also with e = 0
}
// The operand's digits, kMvX bits below the largest exponent em; with em = kFxInf its raw bits.
__device__ __forceinline__ int2 fx_digits(double x, int cx, int em) {
  const i64 X = em >= kFxInf ? __double_as_longlong(x) : d2fx(x, 1084 - 1022 - kMvX + em - cx);
  return make_int2(fx_lo(X), em >= kFxInf ? (int)(X >> 32) : fx_hi(X));
}

// A product's unit: fx_dot's integer is the product times 2^(kFxMvExp - ea - em).
constexpr int kFxMvExp = 1022 + 61;

// A value v 2^e (|v| <= 2^61), or with e = kFxBad the bits of a double.
struct FxVal {
  i64 v;
  int e;
};
__device__ __forceinline__ i64 fx_shr(i64 v, int n) { return v >> min(n, 63); }
template <bool LAT = false>
__device__ __forceinline__ double fx_val(FxVal p) {
  return p.e == kFxBad ? __longlong_as_double(p.v) : LAT ? fx2d_lat(p.v, -p.e) : fx2d(p.v, -p.e);
}

// h + p and h + p + q, summed in fixed point 59 bits below the largest and rounded once (LAT: the conversion
// with the lower latency, for the chains).
template <bool LAT = false>
__device__ __forceinline__ double fx_sum(double h, FxVal p) {
  const int eh = (int)(abs_hi(h) >> 20);
  if (p.e == kFxBad || eh == 0x7ff) return h + fx_val<LAT>(p);
  const int em = max(eh - 1081, p.e);
  const i64 v = fx_shr(p.v, em - p.e) + d2fx(h, 1084 + em);
  return LAT ? fx2d_lat(v, -em) : fx2d(v, -em);
}
template <bool LAT = false>
__device__ __forceinline__ double fx_sum(double h, FxVal p, FxVal q) {
  const int eh = (int)(abs_hi(h) >> 20);
  if (p.e == kFxBad || q.e == kFxBad || eh == 0x7ff) return (h + fx_val<LAT>(p)) + fx_val<LAT>(q);
  const int em = max(max(eh - 1081, p.e), q.e);
  const i64 v = fx_shr(p.v, em - p.e) + fx_shr(q.v, em - q.e) + d2fx(h, 1084 + em);
  return LAT ? fx2d_lat(v, -em) : fx2d(v, -em);
}

// The sums of hi hi, hi lo and lo hi (operator, operand) as one integer in units of 2^59 of the digits' units.
struct FxPart {
  i64 t2, t1, t0;
  __device__ __forceinline__ i64 value() const {
    return (t2 << 1) + (((t1 >> 4) + t0 + (1ll << (kMvALo - 2))) >> (kMvALo - 1));
  }
};
static_assert(kMvA + kMvX - 61 == 59 && 32 - kMvALo == 4, "FxPart::value");

// Row A of a block in shared memory (column stride LD words) times NC operand digits xs.
template <int NC, int LD>
__device__ __forceinline__ i64 fx_dot(const int2* A, const int2* xs) {
  const int4* x4 = reinterpret_cast<const int4*>(xs);
  i64 t2 = 0, t1 = 0, t0 = 0;
#pragma unroll
  for (int c = 0; c < NC; c += 2) {
    const int4 v = x4[c >> 1];
    const int2 a = A[c * LD], b = A[(c + 1) * LD];
    t2 = fx_mad(a.y, v.y, t2);
    t1 = fx_mad(a.y, v.x, t1);
    t0 = fx_mad(a.x, v.y, t0);
    t2 = fx_mad(b.y, v.w, t2);
    t1 = fx_mad(b.y, v.z, t1);
    t0 = fx_mad(b.x, v.w, t0);
  }
  return FxPart{t2, t1, t0}.value();
}

// The same product in FP64 over columns [c0, c1) of row r, for an operand with an infinity (em = kFxInf: raw
// doubles in xs): the infinities and NaNs that FP64 gives.
static __device__ __noinline__ double fx_dot_slow(const i64* blk, int ld, int r, const int2* xs, int c0, int c1, int em) {
  const int2* A = reinterpret_cast<const int2*>(blk) + r;
  const int ea = fx_row_exp(blk, ld)[r];
  const int* cx = fx_col_exp(blk, ld);
  double acc = 0.0;
  for (int c = c0; c < c1; ++c) {
    const int2 a = A[(size_t)c * ld], x = xs[c];
    const double av = ea == kFxBad ? fx_nan() : ldexp(__ll2double_rn(mv_value(a)), ea - kMvA + cx[c]);
    const double xv = em >= kFxInf ? __hiloint2double(x.y, x.x)
                                   : ldexp(__ll2double_rn(((i64)x.y << 32) + x.x), em - (1022 + kMvX) - cx[c]);
    acc = fma(av, xv, acc);
  }
  return acc;
}

// A vector of nr <= 32 NP elements (x[p] = element 32 p + lane) as operand digits in xs for a block with column
// exponents cx; returns its exponent em.
template <int NP>
__device__ __forceinline__ int publish_regs(const double (&x)[NP], const int (&cx)[NP], int nr, int lane, int2* xs) {
  int m = -0x10000;
#pragma unroll
  for (int p = 0; p < NP; ++p)
    if (p * 32 + lane < nr) m = max(m, fx_key(x[p], cx[p]));
  const int em = __reduce_max_sync(0xffffffffu, m);
#pragma unroll
  for (int p = 0; p < NP; ++p)
    if (p * 32 + lane < nr) xs[p * 32 + lane] = fx_digits(x[p], cx[p], em);
  __syncwarp();
  return em;
}
// Row r of a block in shared memory times an operand of one exponent.
template <int LD>
__device__ __forceinline__ FxVal block_vec(const i64* blk, int nr, int r, const int2* xs, int em) {
  const int ea = fx_row_exp(blk, LD)[r];
  FxVal p;
  p.v = fx_dot<LD, LD>(reinterpret_cast<const int2*>(blk) + r, xs);
  p.e = ea + em - kFxMvExp;
  if (em >= kFxInf || ea == kFxBad) {
    p.v = __double_as_longlong(em == kFxInf ? fx_dot_slow(blk, LD, r, xs, 0, nr, em) : fx_nan());
    p.e = kFxBad;
  }
  return p;
}

// Columns [c0, c0 + NC) of a lane's row of a block in registers (its loads all in flight at once), and their
// product with a published operand: the arithmetic of fx_dot.  LD <= 32 NP; sums of ranges add up to a row's.
template <int LD, int NP, int NC = LD>
struct FxRow {
  int2 m[NC];
  int ea, cx[NP];            // the row's exponent; the column exponents of the lane's operand elements
  __device__ __forceinline__ void load(const i64* blk, int r, int c0 = 0) {
    const int2* A = reinterpret_cast<const int2*>(blk) + r;
#pragma unroll
    for (int c = 0; c < NC; ++c) m[c] = __ldg(A + (c0 + c) * LD);
    ea = __ldg(fx_row_exp(blk, LD) + r);
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int p = 0; p < NP; ++p) cx[p] = 32 * p + lane < LD ? __ldg(fx_col_exp(blk, LD) + 32 * p + lane) : 0;
  }
  __device__ __forceinline__ FxPart part(const int2* xs) const {   // xs: from column c0 (even)
    i64 t2 = 0, t1 = 0, t0 = 0;
#pragma unroll
    for (int c = 0; c < NC; c += 2) {
      const int4 v = reinterpret_cast<const int4*>(xs)[c >> 1];
      t2 = fx_mad(m[c].y, v.y, t2);
      t1 = fx_mad(m[c].y, v.x, t1);
      t0 = fx_mad(m[c].x, v.y, t0);
      t2 = fx_mad(m[c + 1].y, v.w, t2);
      t1 = fx_mad(m[c + 1].y, v.z, t1);
      t0 = fx_mad(m[c + 1].x, v.w, t0);
    }
    return {t2, t1, t0};
  }
  __device__ __forceinline__ FxVal value(FxPart t, const i64* blk, int nr, int r, const int2* xs, int em) const {
    FxVal p;
    p.v = t.value();
    p.e = ea + em - kFxMvExp;
    if (em >= kFxInf || ea == kFxBad) {                // (after the registers of the row are done with)
      p.v = __double_as_longlong(em == kFxInf ? fx_dot_slow(blk, LD, r, xs, 0, nr, em) : fx_nan());
      p.e = kFxBad;
    }
    return p;
  }
  __device__ __forceinline__ FxVal times(const i64* blk, int nr, int r, const int2* xs, int em) const {
    return value(part(xs), blk, nr, r, xs, em);
  }
};

// ---- second derivatives --------------------------------------------------------------------------
// The second-derivative matrices take three digits of 27 bits (80 bits; sign and magnitude) on both sides: applied
// to a state that is not smooth at the walls their products' range within one row is N^4, of which the implicit
// solves then keep the small end, so two digits would lose what FP64 keeps (psi of a step at N_r = 65 and dt = 1:
// 1e-11 instead of 3e-13).  Six IMAD.WIDE a column: the digit products down to 2^-80 of the largest product.
// A block: planes of the high, middle and low digits ([col][row], L x L ints each), then the rows' and the
// columns' exponents (as in the two-digit blocks).
__host__ __device__ constexpr size_t wx_block_ints(int ld) { return (size_t)(3 * ld + 2) * ld; }

// The digits of m 2^27 >> sh, with x's sign; x = m 2^(e - 1075) in magnitude with its exponent field e.
__device__ __forceinline__ void wx_split(double x, int sh, int& d2, int& d1, int& d0) {
  const unsigned hi = (unsigned)__double2hiint(x), mask = 0x7ffffffu;
  u64 m = ((u64)(hi & 0xfffffu) << 32) | (unsigned)__double2loint(x);
  m = (hi & 0x7ff00000u) ? m | 0x10000000000000ull : m << 1;
  const unsigned a2 = (unsigned)(m >> min(27 + sh, 63)), a1 = (unsigned)(m >> min(sh, 63)) & mask;
  const unsigned a0 = (unsigned)(sh <= 27 ? m << (27 - sh) : m >> min(sh - 27, 63)) & mask;
  const int s = (int)hi >> 31;
  d2 = ((int)a2 ^ s) - s;
  d1 = ((int)a1 ^ s) - s;
  d0 = ((int)a0 ^ s) - s;
}
struct WxAcc {
  i64 s4 = 0, s3 = 0, s2 = 0;
  __device__ __forceinline__ void add(int a2, int a1, int a0, int4 x) {   // x = (high, middle, low, -)
    s4 = fx_mad(a2, x.x, s4);
    s3 = fx_mad(a1, x.x, fx_mad(a2, x.y, s3));
    s2 = fx_mad(a0, x.x, fx_mad(a1, x.y, fx_mad(a2, x.z, s2)));
  }
  // (s4 2^54 + s3 2^27 + s2) 2^e as a value of at most 61 bits
  __device__ __forceinline__ FxVal value(int e) const {
    const __int128 t = ((__int128)s4 << 54) + ((__int128)s3 << 27) + s2;
    const i64 hi = (i64)(t >> 64);
    const u64 lo = (u64)t;
    const i64 h = hi ^ (hi >> 63);
    const u64 l = lo ^ (u64)(hi >> 63);
    const int nb = h ? 128 - __clzll(h) : 64 - __clzll((i64)l);
    const int n = max(nb - 61, 0);
    FxVal p;
    p.v = n == 0 ? (i64)lo : (n < 64 ? (i64)((u64)hi << (64 - n) | lo >> n) : hi >> (n - 64));
    p.e = e + n;
    return p;
  }
};
// A product's exponent: (ea + em) - kWxExp.
constexpr int kWxExp = 1022 + 106;

// A vector as an operand for column exponents cx; returns its exponent (publish_regs); with an infinity in it the
// raw doubles.
template <int NP>
__device__ __forceinline__ int publish_wide(const double (&x)[NP], const int (&cx)[NP], int nr, int lane, int4* xs) {
  int m = -0x10000;
#pragma unroll
  for (int p = 0; p < NP; ++p)
    if (p * 32 + lane < nr) m = max(m, fx_key(x[p], cx[p]));
  const int em = __reduce_max_sync(0xffffffffu, m);
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    int4 d = make_int4(0, 0, 0, 0);
    if (em >= kFxInf) {
      d.x = __double2loint(x[p]);
      d.y = __double2hiint(x[p]);
    } else {
      wx_split(x[p], em - fx_key(x[p], cx[p]), d.x, d.y, d.z);
    }
    xs[p * 32 + lane] = d;                             // (32 NP entries: the block's padding meets zeros)
  }
  __syncwarp();
  return em;
}
// Row r of a block times an operand with an infinity (raw doubles), as FP64 gives it.
static __device__ __noinline__ double wx_dot_slow(const int* blk, int ld, int nr, int r, const int4* xs) {
  const int ea = blk[3 * ld * ld + r];
  const int* cx = blk + 3 * ld * ld + ld;
  double acc = 0.0;
  for (int c = 0; c < nr; ++c) {
    const int o = c * ld + r;
    const double a = __ll2double_rn(((i64)blk[o] << 27) + blk[ld * ld + o]);   // (its sign and zeros matter)
    acc = fma(ldexp(a, ea + cx[c] - 53), __hiloint2double(xs[c].y, xs[c].x), acc);
  }
  return acc;
}
// Row r of a block (in shared memory) times a published operand.
template <int LD>
__device__ __forceinline__ FxVal wx_dot(const int* blk, int nr, int r, const int4* xs, int em) {
  const int* A = blk + r;
  WxAcc acc;
#pragma unroll 8
  for (int c = 0; c < LD; ++c) acc.add(A[c * LD], A[(LD + c) * LD], A[(2 * LD + c) * LD], xs[c]);
  const int ea = blk[3 * LD * LD + r];
  FxVal p = acc.value(ea + em - kWxExp);
  if (em >= kFxInf || ea == kFxBad) {
    p.v = __double_as_longlong(em == kFxInf ? wx_dot_slow(blk, LD, nr, r, xs) : fx_nan());
    p.e = kFxBad;
  }
  return p;
}

// ---- asynchronous copies -------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

}  // namespace sdd
