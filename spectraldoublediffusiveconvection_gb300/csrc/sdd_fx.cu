// Row kernels of the nonlinear term, the right-hand-side assembly, the theta recurrences and the
// standalone theta transforms.
//
// k_fx_rows: one CTA per (radial row n, shell).  It forms the nine spectral rows of
// Matrix_Operators.py:631-740 (Derivatives, with J_theta_RT :437 and A2_SINE_R2 :476 evaluated as
// parity suffix sums along the row), transforms them to the 3/2-padded grid (:776-786), forms the
// products of :791-793 (NLIN_FX) or :884-887 (NLIN_DFX), and transforms four product rows back
// (:797-802).  The radial derivative Dr@(JT_psi*omega) of :791 is moved through the (theta-only) DST:
// the kernel outputs DST(JT_psi*omega) and the rhs kernel applies Dr to it in spectral space, so the
// row kernel has no cross-row dependency.
#include <cuda_runtime.h>

#include <algorithm>

#include "sdd_internal.cuh"
#include "sdd_fft.cuh"
#include "sdd_rowops.cuh"

namespace sdd {

// shared memory of k_fx_rows in units of T: RA, RB (5P complex each), W, E (P complex each), RG (9P),
// kf (P), operator rows (2 kMaxNr), reduction words (9*32 of 8 bytes), scales (32)
size_t fx_smem_bytes(int M, int P, int prec) {
  (void)M;
  const size_t es = prec == SDD_PREC_MIXED ? sizeof(float) : sizeof(double);
  return (34 * (size_t)P + 2 + 2 * kMaxNr + 32) * es + 9 * 32 * 8;
}

// DCT3 input x_k of transform t of the nine fields (see the header comment of sdd_fft.cuh); kf[k] = k.
// Fields: 0 JT_psi, 1 komega, 2 kDpsi, 3 DT, 4 DC (cosine type); 5 omega, 6 Dpsi, 7 kT, 8 kC (sine type).
template <typename T>
__device__ __forceinline__ T fx_x(int t, int k, int M, int P, const T* kf, const T* JP, const T* OM,
                                  const T* DP, const T* DTv, const T* DCv, const T* Tv, const T* Sv) {
  if (t < 5) {
    if (k >= M) return (T)0;
    switch (t) {
      case 0: return JP[k];
      case 1: return k >= 1 ? kf[k] * OM[k - 1] : (T)0;
      case 2: return k >= 1 ? kf[k] * DP[k - 1] : (T)0;
      case 3: return DTv[k];
      default: return DCv[k];
    }
  }
  const int w = P - k;  // wavenumber
  if (k == 0 || w > M - 1) return (T)0;
  switch (t) {
    case 5: return OM[w - 1];
    case 6: return DP[w - 1];
    case 7: return -(kf[w] * Tv[w]);
    default: return -(kf[w] * Sv[w]);
  }
}

// Runs body(rd) with rd(e) = element e of shell b's state as T: FP32 kernels read the caller's FP32 copy
// when there is one (the previous mixed step wrote it with the same rounding), else the FP64 state is
// converted (an FP64-pipe instruction per element).  The choice is made once, outside the loops, so the
// compiler cannot turn it into a per-element select that executes both loads and the conversion.
template <typename T, typename F>
__device__ __forceinline__ void with_x(const FxArgs& a, int b, F&& body) {
  if (sizeof(T) == 4 && a.X32) {
    const float* x = a.X32 + (size_t)b * a.x32_stride;
    body([x](size_t e) { return (T)x[e]; });
  } else {
    const double* x = a.X + (size_t)b * a.x_stride;
    body([x](size_t e) { return (T)x[e]; });
  }
}

// The linear parts of the three right-hand sides (Main.py:262-280) at one row and mode, in the three kernels that form
// them (k_fx_grid, k_rhs_lin, k_rhs), so that all give the same bits.  An FP64 instruction holds the pipe for 64 cycles
// and a dependent one waits as long: fused multiply-adds, the row's scalars multiplied once, doublings in the exponent
// and mode numbers without conversions leave 12 a mode of 22 (k_rhs_lin, 64 shells of 256 x 30: 38.9 -> 28.7 us, in a
// step 525 -> 516; mixed 315 -> 306; one shell 41.5 -> 41.1).
__device__ __forceinline__ double twice(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x), e = hi & 0x7ff00000, sgn = hi & (int)0x80000000;
  if (e == 0x7ff00000) return x;
  if (e == 0x7fe00000) return __hiloint2double(sgn | 0x7ff00000, 0);
  const int sh = (int)__funnelshift_l((unsigned)lo, (unsigned)hi, 1) & 0x7fffffff;   // (zero and below the normal range)
  return e == 0 ? __hiloint2double(sgn | sh, lo << 1) : __hiloint2double(hi + 0x100000, lo);
}
// A2_SINE: D2 psi - k1 ir2 (k2 psi_k + 2 s2), k1 = k + 1, k2 = k + 2, s2 = the parity sum from k + 2
__device__ __forceinline__ double lin_a2(double d2, double k1, double k2, double ir2, double pk, double s2) {
  return fma(-(k1 * ir2), fma(k2, pk, twice(s2)), d2);
}
// psi: A2 psi - dt Pr gr k1 (Ra T_{k+1} - Ra_s S_{k+1}); gd = dt Pr gr
__device__ __forceinline__ double lin_psi_rhs(double om, double k1, double gd, double Ra, double Ras, double t, double s) {
  return fma(-(k1 * gd), fma(Ra, t, -(Ras * s)), om);
}
// J_theta_RT: k1 psi_{k-1} + 2 s1, k = 0: s1
__device__ __forceinline__ double lin_jt(int k, double k1, double pkm, double s1) {
  return k == 0 ? s1 : fma(k1, pkm, twice(s1));
}
// T, S: r^2 f - dt dT0 J; dd = dt dT0
__device__ __forceinline__ double lin_ts_rhs(double rsq, double f, double dd, double jt) { return fma(-dd, jt, rsq * f); }

// Arithmetic shared by the fused and the split nonlinear-term kernels.  This file is compiled without
// automatic fma contraction and every multiply-add below is an explicit fma, so both kernels round
// identically.
// J_theta_RT (:437-472) and A2_SINE_R2 (:476-526) at mode k along a row: jp, and om updated from D2 psi.
template <typename T>
__device__ __forceinline__ void jp_om(int k, int M, const T* kf, const T* pv, const T* Sc, T ir4n, T& jp, T& om) {
  const T s1 = (k + 1 < M) ? Sc[k + 1] : (T)0;
  jp = (k == 0) ? s1 : fma(kf[k + 1], pv[k - 1], (T)2 * s1);
  const T s2 = (k + 2 < M) ? Sc[k + 2] : (T)0;
  om = fma(-kf[k + 1], ir4n * fma(kf[k + 2], pv[k], (T)2 * s2), om);
}
// W_k of a DCT3 pair (rows A, B with scales sa, sb): s_A V_A(k) + i s_B V_B(k), V(k) = e_k (x_k - i x_{P-k}).
template <typename T, typename C>
__device__ __forceinline__ C dct3_pack(C e, T xa, T xar, T xb, T xbr, T sa, T sb) {
  const T a1 = fma(e.x, xa, e.y * xar), a2 = fma(e.y, xa, -(e.x * xar));
  const T b1 = fma(e.x, xb, e.y * xbr), b2 = fma(e.y, xb, -(e.x * xbr));
  return cmk<C>(fma(sa, a1, -(sb * b2)), fma(sa, a2, sb * b1));
}
// y_A, y_B of a DCT2 pair from Z_k, Z_{-k} and e_k = 0.5 (cos, sin)(pi k/2P).
template <typename T, typename C>
__device__ __forceinline__ void dct2_unpack(C Zk, C Zm, C e, T& ya, T& yb) {
  ya = fma(e.x, Zk.x + Zm.x, e.y * (Zk.y - Zm.y));
  yb = fma(e.x, Zk.y + Zm.y, -(e.y * (Zk.x - Zm.x)));
}
// Grid products at point i (:791-793 for MODE 0, :884-887 for MODE 1 with base fields bs):
// pair 0 = (Q, R) (sine type), pair 1 = (NT, NS) (cosine type).
template <typename T, int MODE>
__device__ __forceinline__ void grid_products(int pair, const T* RG, const T* bs, int i, int P, T& v0, T& v1) {
  const T JT = RG[i], DPg = RG[6 * P + i];
  if (pair == 0) {
    const T kO = RG[P + i], kDP = RG[2 * P + i], O = RG[5 * P + i];
    if (MODE != 1) {
      v0 = JT * O;
      v1 = fma(kDP, O, DPg * kO);
    } else {
      const T aJT = bs[i], akO = bs[P + i], akDP = bs[2 * P + i], aO = bs[5 * P + i], aDP = bs[6 * P + i];
      v0 = fma(aJT, O, JT * aO);
      v1 = fma(akDP, O, aDP * kO) + fma(kDP, aO, DPg * akO);
    }
  } else {
    const T DTg = RG[3 * P + i], DCg = RG[4 * P + i], kT = RG[7 * P + i], kC = RG[8 * P + i];
    if (MODE != 1) {
      v0 = fma(JT, DTg, -(DPg * kT));
      v1 = fma(JT, DCg, -(DPg * kC));
    } else {
      const T aJT = bs[i], aDT = bs[3 * P + i], aDC = bs[4 * P + i], aDP = bs[6 * P + i];
      const T akT = bs[7 * P + i], akC = bs[8 * P + i];
      v0 = fma(JT, aDT, -(DPg * akT)) + fma(aJT, DTg, -(aDP * kT));
      v1 = fma(JT, aDC, -(DPg * akC)) + fma(aJT, DCg, -(aDP * kC));
    }
  }
}

// The scaling of the rows that enter a transform, their packing, and their way out, for FP32 rows (exact
// power-of-two balance of a pair, pow2_scale) and FP64 rows (64-bit fixed point, rows_to_fixed).  scl: the
// block's scale words (FP32: K scales then K inverses; FP64: K exponents as ints).
template <typename T> struct RowTr;
template <> struct RowTr<float> {
  static constexpr bool kInv = true;                   // inverse transforms with conjugated twiddles
  static __device__ __forceinline__ float sign(float v, bool n) { return n ? -v : v; }
  // W_k of a DCT3 pair (rows A = t, B = t + 1 of XV; hasb: row B is there)
  static __device__ __forceinline__ float2 pack(const float* XV, int P, int t, bool hasb, int k, const float2* Et,
                                                const float* scl) {
    const float sa = scl[t], sb = hasb ? scl[t + 1] : 0.0f;
    const float xa = XV[t * P + k], xb = hasb ? XV[(t + 1) * P + k] : 0.0f;
    if (k == 0) return cmk<float2>(sa * xa, sb * xb);
    const float xar = XV[t * P + P - k], xbr = hasb ? XV[(t + 1) * P + P - k] : 0.0f;
    return dct3_pack<float, float2>(Et[k], xa, xar, xb, xbr, sa, sb);
  }
  static __device__ __forceinline__ float2 load(const float* PR, int P, int t, int src, const float* scl) {
    return cmk<float2>(scl[t] * PR[t * P + src], scl[t + 1] * PR[(t + 1) * P + src]);
  }
  // row t + h (h = 0: A, 1: B) of a transformed pair, nrows rows in all
  static __device__ __forceinline__ float out(float2 v, int h, int t, int nrows, const float* scl) {
    return (h ? v.y : v.x) * scl[nrows + t + h];
  }
  static __device__ __forceinline__ void unpack(const float2* Z, int P, int k, int t, int nrows, const float2* Et,
                                                const float* scl, float sc, float& ya, float& yb) {
    dct2_unpack<float, float2>(Z[k], Z[(P - k) % P], Et[k], ya, yb);
    ya *= sc * scl[nrows + t];
    yb *= sc * scl[nrows + t + 1];
  }
};
template <> struct RowTr<double> {
  static constexpr bool kInv = false;                  // inverse transforms as forward ones of swapped pairs
  static __device__ __forceinline__ double sign(double v, bool n) { return neg_if(v, n); }
  static __device__ __forceinline__ longlong2 pack(const double* XV, int P, int t, bool hasb, int k, const int4* Et,
                                                   const double*) {
    const i64* A = reinterpret_cast<const i64*>(XV) + t * P;
    const i64* B = A + P;
    const i64 xa = A[k], xb = hasb ? B[k] : 0;
    if (k == 0) return make_longlong2(xb, xa);
    return dct3_pack_fx(Et[k], xa, A[P - k], xb, hasb ? B[P - k] : 0);
  }
  static __device__ __forceinline__ longlong2 load(const double* PR, int P, int t, int src, const double*) {
    const i64* A = reinterpret_cast<const i64*>(PR) + t * P;
    return make_longlong2(A[src], A[P + src]);
  }
  // a row with an infinity or NaN makes both rows of its pair NaN (they share one complex transform)
  static __device__ __forceinline__ bool bad(int t, const double* scl) {
    const int* E = reinterpret_cast<const int*>(scl);
    return E[t] == kFxBad || E[t + 1] == kFxBad;
  }
  static __device__ __forceinline__ double out(longlong2 v, int h, int t, int, const double* scl) {
    return bad(t, scl) ? fx_nan() : fx2d(h ? v.x : v.y, 60 - reinterpret_cast<const int*>(scl)[t + h]);
  }
  static __device__ __forceinline__ void unpack(const longlong2* Z, int P, int k, int t, int, const int4* Et,
                                                const double* scl, double sc, double& ya, double& yb) {
    const int* E = reinterpret_cast<const int*>(scl);
    i64 a, b;
    dct2_unpack_fx(Z[k], Z[(P - k) % P], Et[k], a, b);
    const bool n = bad(t, scl);
    ya = n ? fx_nan() : sc * fx2d(a, 60 - E[t]);
    yb = n ? fx_nan() : sc * fx2d(b, 60 - E[t + 1]);
  }
};

// f(i) for the calling thread's elements i < n of a row loop: left to the compiler to unroll in FP32, rolled up in
// FP64 (the fixed-point bodies are long: unrolled, a kernel's code outgrows the instruction cache).
template <typename T, typename F>
__device__ __forceinline__ void for_elems(int n, F&& f) {
  if constexpr (sizeof(T) == 8) {
#pragma unroll 1
    for (int i = threadIdx.x; i < n; i += blockDim.x) f(i);
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) f(i);
  }
}

// Forms NR rows (or `nrows` of them) of P elements, row(t, k), in XV and their scales.  FP32: unrolled, the maxima
// tracked as the rows are formed; FP64: rolled up (code size), rows_to_fixed reads them back.
template <typename T, int NR, typename F>
__device__ __forceinline__ void form_rows(T* XV, int P, int nrows, void* red, T* scl, F&& row) {
  const int tid = threadIdx.x, bd = blockDim.x;
  if constexpr (sizeof(T) == 4) {
    unsigned mb[NR];
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      mb[t] = 0;
      if (t < nrows)
        for (int k = tid; k < P; k += bd) {
          const T v = row(t, k);
          XV[t * P + k] = v;
          mb[t] = max(mb[t], Bits<float>::absbits(v));
        }
    }
    block_max_scales<T, NR>(mb, reinterpret_cast<unsigned*>(red), scl);
  } else {
#pragma unroll 1
    for (int t = 0; t < nrows; ++t)
#pragma unroll 1
      for (int k = tid; k < P; k += bd) XV[t * P + k] = row(t, k);
    rows_to_fixed(XV, P, nrows, red, reinterpret_cast<int*>(scl));
  }
}

// The scales of K formed rows (mx: FP32, the calling thread's maxima).
template <typename T, int K>
__device__ __forceinline__ void scale_rows(T* PR, int P, unsigned (&mx)[K], void* red, T* scl) {
  if constexpr (sizeof(T) == 4) block_max_scales<T, K>(mx, reinterpret_cast<unsigned*>(red), scl);
  else rows_to_fixed(PR, P, K, red, reinterpret_cast<int*>(scl));
}

// MODE 0: NLIN_FX (optionally storing the grid fields); 1: NLIN_DFX with base fields from the cache;
// 2: grid fields only (fills the cache).
template <typename T, int MODE>
__global__ void __launch_bounds__(kFxRowThreads) k_fx_rows(FxArgs a) {
  using C = typename Cplx<T>::type;
  using W = typename Cplx<T>::tw;
  using Tr = RowTr<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, nr = a.nr, P = a.P;
  const int n = blockIdx.x, b = blockIdx.y;
  const int tid = threadIdx.x, bd = blockDim.x;

  C* RA = reinterpret_cast<C*>(smem_raw);
  C* RB = RA + 5 * P;
  W* Wt = reinterpret_cast<W*>(RB + 5 * P);
  W* Et = Wt + P;
  T* RG = reinterpret_cast<T*>(Et + P);
  T* kf = RG + 9 * P;          // kf[k] = k, k < P + 2
  T* opr = kf + P + 2;
  T* scl = opr + 2 * kMaxNr;   // 9 scales + 9 inverse scales (inverse transforms), reused for 4+4
  void* red = scl + 32;        // 9*32 reduction words of 8 bytes
  T* pv = RG;
  T* Tv = pv + M;
  T* Sv = Tv + M;
  T* DP = Sv + M;
  T* OM = DP + M;
  T* DTv = OM + M;
  T* DCv = DTv + M;
  T* JP = DCv + M;
  T* Sc = JP + M;
  const W* wg = reinterpret_cast<const W*>(a.ops.w);
  const W* eg = reinterpret_cast<const W*>(a.ops.e);
#pragma unroll 1
  for (int i = tid; i < P; i += bd) {
    Wt[i] = wg[i];
    Et[i] = eg[i];
  }
#pragma unroll 1
  for (int i = tid; i < P + 2; i += bd) kf[i] = sizeof(T) == 8 ? (T)fx_int(i) : (T)i;
  const T* Drg = reinterpret_cast<const T*>(a.ops.Dr);
  const T* D2g = reinterpret_cast<const T*>(a.ops.D2r2);
  for (int m = tid; m < nr; m += bd) {
    opr[m] = Drg[n * nr + m];
    opr[nr + m] = D2g[n * nr + m];
  }
  const T ir4n = reinterpret_cast<const T*>(a.ops.ir4r2)[n];
  after_previous_kernel();     // (the tables and operators are the plan's)
  if (a.active && !a.active[b]) return;
  __syncthreads();

  // ---- 1. radial contractions of row n (Derivatives, :698-729) and the row values ----
  const int N = M * nr;
  // the four contractions were formed by k_fx_deriv ([op][k][n], FP64) or k_deriv_tc ([op][n][k], mixed plans
  // with tensor cores); without their scratch (and in FP32 on the CUDA cores) here
  const T* Dt = (a.deriv && (sizeof(T) == 8 || a.deriv_t))
                    ? reinterpret_cast<const T*>(a.deriv) + (size_t)b * a.deriv_stride
                    : nullptr;
  const size_t dk = a.deriv_t ? 1 : nr, d0 = a.deriv_t ? (size_t)n * M : n;
  with_x<T>(a, b, [&](auto xr) {
#pragma unroll 1
  for (int k = tid; k < M; k += bd) {
    const size_t ps = (size_t)k * nr, ts = N + (size_t)k * nr, ss = 2 * (size_t)N + (size_t)k * nr;
    const bool psi_on = !(a.sym && (k % 2 == 0));
    const bool ts_on = !(a.sym && (k % 2 == 1));
    T dp = 0, d2 = 0, dtv = 0, dcv = 0, pn = 0, tn = 0, sn = 0;
    if (psi_on) {
      if (Dt) {
        dp = Dt[d0 + k * dk];
        d2 = Dt[(size_t)N + d0 + k * dk];
      } else {
        for (int m = 0; m < nr; ++m) {
          const T x = xr(ps + m);
          dp = fma(opr[m], x, dp);
          d2 = fma(opr[nr + m], x, d2);
        }
      }
      pn = xr(ps + n);
    }
    if (ts_on) {
      if (Dt) {
        dtv = Dt[2 * (size_t)N + d0 + k * dk];
        dcv = Dt[3 * (size_t)N + d0 + k * dk];
      } else {
        for (int m = 0; m < nr; ++m) {
          dtv = fma(opr[m], xr(ts + m), dtv);
          dcv = fma(opr[m], xr(ss + m), dcv);
        }
      }
      tn = xr(ts + n);
      sn = xr(ss + n);
    }
    pv[k] = pn;
    Tv[k] = tn;
    Sv[k] = sn;
    DP[k] = dp;
    OM[k] = d2;
    DTv[k] = dtv;
    DCv[k] = dcv;
  }
  });
  __syncthreads();
  parity_suffix<T>(pv, Sc, M);
  __syncthreads();
  // J_theta_RT (:437-472) and A2_SINE_R2 (:476-526) along the row
#pragma unroll 1
  for (int k = tid; k < M; k += bd) jp_om<T>(k, M, kf, pv, Sc, ir4n, JP[k], OM[k]);
  __syncthreads();
  // ---- 2. nine inverse transforms as five paired DCT3s (:776-786) ----
  // the nine DCT3 input rows, materialised once (in RB, free until the FFT), with their maxima
  T* XV = reinterpret_cast<T*>(RB);
  form_rows<T, 9>(XV, P, 9, red, scl,
                  [&](int t, int k) { return fx_x<T>(t, k, M, P, kf, JP, OM, DP, DTv, DCv, Tv, Sv); });
  for_elems<T>(5 * P, [&](int idx) {
    const int p = idx / P;
    RA[idx] = Tr::pack(XV, P, 2 * p, p < 4, idx - p * P, Et, scl);
  });
  __syncthreads();
  C* res = fft_rows<T, Tr::kInv>(RA, RB, 5, a.st, Wt);
  for_elems<T>(9 * P, [&](int idx) {
    const int t = idx / P;
    const int i = idx - t * P;
    const int src = (i & 1) ? (P - 1 - (i >> 1)) : (i >> 1);
    const T val = Tr::out(res[(t >> 1) * P + src], t & 1, t & ~1, 9, scl);
    RG[idx] = Tr::sign(val, t >= 5 && (i & 1));
  });
  __syncthreads();

  if (MODE != 1 && a.base != nullptr) {
    T* bc = reinterpret_cast<T*>(a.base) + (size_t)b * a.base_stride + (size_t)n * 9 * P;
    for (int idx = tid; idx < 9 * P; idx += bd) bc[idx] = RG[idx];
  }
  if (MODE == 2) return;

  // ---- 3. grid products (:791-793 or :884-887); sine outputs pre-multiplied by (-1)^i ----
  T* PR = reinterpret_cast<T*>(RA);
  const T* bs = (MODE == 1) ? reinterpret_cast<const T*>(a.base) + (size_t)b * a.base_stride +
                                  (size_t)n * 9 * P
                            : nullptr;
  unsigned m4[4] = {0, 0, 0, 0};
  for_elems<T>(P, [&](int i) {
    T v[4];
    grid_products<T, MODE>(0, RG, bs, i, P, v[0], v[1]);
    grid_products<T, MODE>(1, RG, bs, i, P, v[2], v[3]);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      PR[t * P + i] = t < 2 ? Tr::sign(v[t], i & 1) : v[t];
      if constexpr (sizeof(T) == 4) m4[t] = max(m4[t], Bits<T>::absbits(v[t]));
    }
  });
  scale_rows<T, 4>(PR, P, m4, red, scl);

  // ---- 4. four forward transforms as two paired DCT2s (:797-802) ----
  for_elems<T>(2 * P, [&](int idx) {
    const int p = idx >= P ? 1 : 0;
    RB[idx] = Tr::load(PR, P, 2 * p, makhoul_src(idx - p * P, P), scl);
  });
  __syncthreads();
  C* Z = fft_rows<T, false>(RB, RA, 2, a.st, Wt);
  next_kernel_may_start();
  double* o = a.out4 + (size_t)b * a.out_stride;
  const T two_P = (T)2 / (T)P, one_P = (T)1 / (T)P;
#pragma unroll 1
  for (int idx = tid; idx < 2 * M; idx += bd) {
    const int p = idx >= M;
    const int s = idx - p * M;
    T ya = 0, yb = 0;
    bool zero = false;
    int k;
    if (p == 0) {            // sine pair: slot s <-> wavenumber s+1, read at k = P-1-s
      zero = (s == M - 1) || (a.sym && (s % 2 == 0));
      k = P - 1 - s;
    } else {
      zero = a.sym && (s % 2 == 1);
      k = s;
    }
    if (!zero) {
      Tr::unpack(Z + p * P, P, k, 2 * p, 4, Et, scl, (p == 1 && k == 0) ? one_P : two_P, ya, yb);
    }
    const size_t q0 = (size_t)(2 * p) * N + (size_t)s * nr + n;
    o[q0] = (double)ya;
    o[q0 + N] = (double)yb;
    if (sizeof(T) == 4 && p == 0 && a.q32) a.q32[(size_t)b * M * a.nr + (size_t)s * a.nr + n] = (float)ya;
  }
}

// ---- split nonlinear term: the same arithmetic over 7 CTAs per radial row ------------------------
// k_fx_rows runs a row's five paired inverse and two paired forward transforms one after the other on
// one SM, so a single shell occupies only nr SMs.  For small batches the work is split:
//   k_fx_grid (nr x 5 CTAs per shell): CTA (n, p) forms the DCT3 input rows t = 2p, 2p+1 of row n (with
//     the radial contractions those two fields need), runs their paired inverse transform and writes the
//     two grid rows to grid[shell][n][t][P] (the layout of the base-state cache);
//   k_fx_prod (nr x 2 CTAs per shell): CTA (n, p) forms product pair p on the grid of row n (p = 0: the
//     sine-type Q, R; p = 1: the cosine-type NT, NS) and runs their paired forward transform into out4.
// Per element the operations and their order are those of k_fx_rows, so the results are identical.
constexpr int kFxSplitThreads = 256;   // (up to kFxRowThreads: fx_split_threads)

// FP32 grid kernels of the fused right-hand side keep FP64 copies of the row's psi, T, S and psi's parity
// suffix sums (4 M doubles) for the linear parts, after the T-typed arrays.
__host__ __device__ inline size_t fx_grid_lin64_offset(int M, int P, int prec) {
  const size_t es = prec == SDD_PREC_MIXED ? sizeof(float) : sizeof(double);
  return (((8 * (size_t)P + P + 2 + 9 * (size_t)M + 32) * es + 2 * 32 * 8) + 15) / 16 * 16;
}
size_t fx_grid_smem_bytes(int M, int P, int prec) {
  return fx_grid_lin64_offset(M, P, prec) + (prec == SDD_PREC_MIXED ? 4 * (size_t)M * sizeof(double) : 0);
}
size_t fx_prod_smem_bytes(int P, int prec) {
  const size_t es = prec == SDD_PREC_MIXED ? sizeof(float) : sizeof(double);
  return (8 * (size_t)P + 2 * (size_t)P + 32) * es + 2 * 32 * 8;
}

// One asynchronous global -> shared copy of an element of 4, 8 or 16 bytes (the issuing thread does not
// wait for the data: a loop of such copies has all its loads in flight at once).
template <int BYTES>
__device__ __forceinline__ void cp_async_bytes(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem));
  else if constexpr (BYTES == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem));
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem));
}
template <typename E>
__device__ __forceinline__ void cp_async_elem(E* smem, const E* gmem) {
  static_assert(sizeof(E) == 4 || sizeof(E) == 8 || sizeof(E) == 16, "element size");
  cp_async_bytes<(int)sizeof(E)>(smem, gmem);
}
__device__ __forceinline__ void cp_async_all_done() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_all;\n" ::: "memory");
}

// The pending correction of modes k0 .. k0 + kn - 1 (see FixArgs) on xd (the modes' FP64 psi, T, S rows, in
// shared memory, still in flight).  s_c = d_{c-1} + part_{c,0} + ... in index order
// (per chain f vectors of 2 nr, nr, nr doubles); then xd += G_jj s_c in the arithmetic
// of k_mode_mv (the same bits).  Four tasks of NP^2 warps (32 rows and the columns, or half of them) per mode:
// psi's two operand halves, T, S; 8 warps take two modes at once, 16 warps one.  The corrected rows are written
// back to the state (and its FP32 copy).  sc: 4 nr doubles a mode.
constexpr int deriv_warps(int ld) { return ld <= 32 ? 8 : 16; }

__device__ __forceinline__ double carried_term(const FixArgs& x, int b, int par, int c, int e, int nr) {
  const int f = e < 2 * nr ? 0 : (e < 3 * nr ? 1 : 2), i = e - (f == 0 ? 0 : (f + 1) * nr);
  const size_t chain = (size_t)(f * 2 + par);
  const double* d = x.dbuf + (size_t)b * x.d_stride + (chain * x.nch + (c - 1)) * x.ldd;
  const double* row = x.pbuf + (size_t)b * x.p_stride + (chain * x.np + (size_t)(c - 1) * (c - 2) / 2) * x.ldd;
  const int nt = c - 1;
  double v = __ldcg(d + i);
  for (int u0 = 0; u0 < nt; u0 += 8) {                 // eight loads in flight
    double tv[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) tv[k] = u0 + k < nt ? __ldcg(row + (size_t)(u0 + k) * x.ldd + i) : 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (u0 + k < nt) v += tv[k];
  }
  return v;
}

// A warp's task and its rows of G.
template <int LD>
struct FixRow {
  static constexpr int NP = (LD + 31) / 32, NC = LD / NP, kMw = 4 * NP * NP, kG = deriv_warps(LD) / kMw;
  FxRow<LD, NP, NC> G;
  int task, sl, h;
  static __device__ __forceinline__ int chunk_of(const FxArgs& a, int k) { return ((a.M - 1 - k) >> 1) / a.fix.kc; }
  static __device__ __forceinline__ bool on(const FxArgs& a, int k, bool psi) {
    return chunk_of(a, k) >= 1 && (!a.sym || ((a.M - 1 - k) & 1) == (psi ? 0 : 1));
  }
  __device__ __forceinline__ bool mine(const FxArgs& a, int k0, int kn, int m) const {   // uniform over the warp
    return m < kn && on(a, k0 + m, task < 2);
  }
  __device__ __forceinline__ const i64* block(const FxArgs& a, int k) const {
    constexpr int bw = (int)fx_block_words(LD);
    const size_t jj = a.M - 1 - k;
    return task < 2 ? a.fix.GA4 + (jj * 2 + task) * bw : (task == 2 ? a.fix.GT : a.fix.GS) + jj * bw;
  }
  __device__ __forceinline__ int row(int nr) const { return min(sl * 32 + (int)(threadIdx.x & 31), nr - 1); }
  __device__ __forceinline__ void load(const FxArgs& a, int k0, int kn, int m) {
    if (mine(a, k0, kn, m)) G.load(block(a, k0 + m), row(a.nr), h * NC);
  }
  __device__ __forceinline__ void first(const FxArgs& a, int k0, int kn) {
    const int warp = threadIdx.x >> 5;
    task = warp % kMw / (NP * NP);
    sl = warp / NP % NP;
    h = warp % NP;
    load(a, k0, kn, warp / kMw);
  }
};

template <int LD>
__device__ void apply_pending_fix(const FxArgs& a, int b, int k0, int kn, double* xd, double* sc, FixRow<LD>& fx) {
  constexpr int NP = FixRow<LD>::NP, NC = FixRow<LD>::NC, kMw = FixRow<LD>::kMw, kG = FixRow<LD>::kG;
  __shared__ __align__(16) int2 s_x[deriv_warps(LD)][32 * NP];
  __shared__ i64 s_v[kG][4][32 * NP];
  __shared__ int s_e[kG][4][32 * NP];
  __shared__ FxPart s_p[NP > 1 ? 8 : 1][32];           // the second column half's sums, per task and row slab
  const FixArgs& x = a.fix;
  const int M = a.M, nr = a.nr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto chunk_of = [&](int k) { return fx.chunk_of(a, k); };
  auto on = [&](int k, bool psi) { return fx.on(a, k, psi); };
  auto mine = [&](int m) { return fx.mine(a, k0, kn, m); };
  const int task = fx.task, sl = fx.sl, h = fx.h;
  const int r = sl * 32 + lane, rr = fx.row(nr);
  FxRow<LD, NP, NC>& G = fx.G;
  int m = warp / kMw;
  for (int q = threadIdx.x; q < kn * 4 * nr; q += blockDim.x) {
    const int mm = q / (4 * nr), e = q - mm * 4 * nr;
    if (on(k0 + mm, e < 2 * nr)) sc[q] = carried_term(x, b, (M - 1 - k0 - mm) & 1, chunk_of(k0 + mm), e, nr);
  }
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll 1
  for (int g = 0; g < kn; g += kG, m += kG) {
    const int mg = m - g;
    FxPart t;
    int em;
    const bool act = mine(m);
    if (act) {
      double xv[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) xv[p] = 32 * p + lane < nr ? sc[(m * 4 + task) * nr + 32 * p + lane] : 0.0;
      em = publish_regs<NP>(xv, G.cx, nr, lane, s_x[warp]);
      t = G.part(s_x[warp] + h * NC);
      if (NP > 1 && h == 1) s_p[task * NP + sl][lane] = t;
    }
    if (NP > 1) __syncthreads();
    if (act && h == 0) {
      if (NP > 1) {
        const FxPart u = s_p[task * NP + sl][lane];
        t.t2 += u.t2;
        t.t1 += u.t1;
        t.t0 += u.t0;
      }
      const FxVal p = G.value(t, fx.block(a, k0 + m), nr, rr, s_x[warp], em);
      s_v[mg][task][r] = p.v;
      s_e[mg][task][r] = p.e;
    }
    fx.load(a, k0, kn, m + kG);
    __syncthreads();
    const int gn = min(kG, kn - g);
    for (int q = threadIdx.x; q < gn * 3 * nr; q += blockDim.x) {
      const int mm = q / (3 * nr), e = q - mm * 3 * nr, f = e / nr, i = e - f * nr, k = k0 + g + mm;
      if (!on(k, f == 0)) continue;
      double* xp = xd + (size_t)(g + mm) * 3 * nr + e;
      const FxVal p{s_v[mm][f == 0 ? 0 : f + 1][i], s_e[mm][f == 0 ? 0 : f + 1][i]}, u{s_v[mm][1][i], s_e[mm][1][i]};
      const double v = f == 0 ? fx_sum(*xp, p, u) : fx_sum(*xp, p);
      *xp = v;
      const size_t o = (size_t)f * M * nr + (size_t)k * nr + i;
      x.X[(size_t)b * a.x_stride + o] = v;
      if (x.X32) x.X32[(size_t)b * a.x32_stride + o] = (float)v;
    }
    __syncthreads();
  }
}

// Shared memory of k_fx_deriv: the fixed-point operators (FP64: D2r2, Dr and with the fused right-hand side
// A2_SINE's D2; FP32: the latter alone), the modes' FP64 rows (3 nr each), with a pending correction the carried
// states (4 nr); FP32 contractions on the CUDA cores: Dr, D2r2 and the modes' rows in FP32.
template <typename T>
__host__ __device__ inline size_t deriv_op_bytes(int ld, bool d2s) {
  return (sizeof(T) == 8 ? wx_block_ints(ld) * sizeof(int) + fx_block_words(ld) * sizeof(i64) : 0) +
         (d2s ? wx_block_ints(ld) * sizeof(int) : 0);
}
template <typename T>
static size_t fx_deriv_smem_bytes(int nr, bool d2s, bool fix, int km, bool f32) {
  return deriv_op_bytes<T>(fx_ld(nr), d2s) + (size_t)km * (fix ? 7 : 3) * nr * sizeof(double) +
         (f32 ? (2 * (size_t)nr * nr + (size_t)km * 3 * nr) * sizeof(float) : 0);
}

// Radial contractions (Derivatives, Matrix_Operators.py:698-729) of km modes of one shell per CTA: Dr psi_k,
// D2r2 psi_k, Dr T_k, Dr S_k for every radial row n, and with the fused right-hand side A2_SINE's D2 psi in
// FP64 as a fifth block (per shell: 4 M nr T, [op][k][n], then M nr doubles).  FP64 contractions run in fixed
// point (sdd_fixed.cuh), a warp per operator, 32 rows and mode, the operators in shared memory; FP32 ones
// (contract: not already on the tensor cores) as sequential FP32 chains in the order of the fused kernel's.  Inside sdd_step a pending chain correction is applied to the rows first.
// Dr takes two digits here (0.03 to 0.4 of FP64's error in the norm, sdd_fixed.cuh): its products with psi, T and S go
// into pointwise products, which no operator differentiates again on the way to the result (the h kernel's Dr Q and D2
// psi meet the implicit solves, which cancel their large parts, and take three).
// Bound: 64 shells of 256 x 30, the integer pipe (a D2 product is about 1500 warp cycles, a Dr product 800): 79 us,
// 146 us with every operator in three digits.  One shell, the L2 round trips of the rows, the correction's blocks
// and the operators: 14 us; 540 x 65: 37 us (64 us with the operators' rows in registers, loaded for every mode).
template <typename T, int LD>
__global__ void __launch_bounds__(32 * deriv_warps(LD), LD <= 32 ? 2 : 1)
    k_fx_deriv(FxArgs a, T* deriv, size_t deriv_stride, int km, int contract) {
  constexpr int NP = (LD + 31) / 32, kW = deriv_warps(LD);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int4 s_x[kW][32 * NP];
  const int M = a.M, nr = a.nr;
  const int k0 = blockIdx.x * km, kn = min(km, M - k0), b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t N = (size_t)M * nr;
  const bool d2s = a.fuse_rhs;
  int* opw = reinterpret_cast<int*>(smem_raw);         // the wide blocks, then Dr
  i64* opd = reinterpret_cast<i64*>(opw + ((sizeof(T) == 8) + d2s) * wx_block_ints(LD));
  double* xd = reinterpret_cast<double*>(smem_raw + deriv_op_bytes<T>(LD, d2s));   // [mode][field][nr]
  double* sc = xd + (size_t)km * 3 * nr;
  // FP32 on the CUDA cores: the operators and rows in FP32, behind the doubles
  float* ops = reinterpret_cast<float*>(xd + (size_t)km * (a.fix.on ? 7 : 3) * nr);
  constexpr int wq = (int)wx_block_ints(LD) / 4, dq = (int)fx_block_words(LD) / 2;
  if (sizeof(T) == 8) {
    for (int e = threadIdx.x; e < wq; e += blockDim.x) cp_async16(opw + 4 * e, a.ops.wx[0] + 4 * e);
    for (int e = threadIdx.x; e < dq; e += blockDim.x) cp_async16(opd + 2 * e, a.ops.fxDr + 2 * e);
  }
  if (d2s) {
    int* dst = opw + (sizeof(T) == 8 ? 4 * wq : 0);
    for (int e = threadIdx.x; e < wq; e += blockDim.x) cp_async16(dst + 4 * e, a.ops.wx[1] + 4 * e);
  }
  if (contract) {
    const float* Drg = reinterpret_cast<const float*>(a.ops.Dr);
    const float* D2g = reinterpret_cast<const float*>(a.ops.D2r2);
    for (int e = threadIdx.x; e < nr * nr; e += blockDim.x) {
      cp_async_elem(ops + e, Drg + e);
      cp_async_elem(ops + nr * nr + e, D2g + e);
    }
  }
  cp_async_commit();
  FixRow<LD> fix;
  if (a.fix.on) fix.first(a, k0, kn);
  after_previous_kernel();                             // (the operators and the correction's blocks are the plan's)
  if (a.active && !a.active[b]) {
    cp_async_wait<0>();
    return;
  }
  const double* Xs = (a.fix.on ? a.fix.X : a.X) + (size_t)b * a.x_stride;
  for (int q = threadIdx.x; q < kn * 3 * nr; q += blockDim.x) {
    const int m = q / (3 * nr), e = q - m * 3 * nr, f = e / nr;
    cp_async_elem(xd + q, Xs + f * N + (size_t)(k0 + m) * nr + (e - f * nr));
  }
  cp_async_commit();
  T* D = deriv + (size_t)b * deriv_stride;
  double* D5 = reinterpret_cast<double*>(D) + 4 * N * sizeof(T) / 8;
  if (a.fix.on) apply_pending_fix<LD>(a, b, k0, kn, xd, sc, fix);
  cp_async_wait<0>();
  __syncthreads();
  // the fixed-point contractions, as items (operator, row slab, mode): D2 first, whose products cost twice Dr's
  // (FP64: D2r2 psi, A2_SINE's D2 psi where it is asked for, then Dr psi, Dr T, Dr S; FP32: A2_SINE's D2 psi)
  next_kernel_may_start();
  const int nd2 = (sizeof(T) == 8) + d2s, nit = (nd2 + (sizeof(T) == 8 ? 3 : 0)) * NP * kn;
#pragma unroll 1
  for (int it = warp; it < nit; it += kW) {
    const int oi = it / (NP * kn), m = it / NP % kn;
    const int r = (it % NP) * 32 + lane, rr = min(r, nr - 1);
    const size_t o = (size_t)(k0 + m) * nr + r;
    const int f = oi < nd2 ? 0 : oi - nd2;
    const double* xr = xd + (m * 3 + f) * nr;
    const int* ce = oi < nd2 ? opw + oi * (4 * wq) + 3 * LD * LD + LD : fx_col_exp(opd, LD);
    double x[NP];
    int cx[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      x[p] = 32 * p + lane < nr ? xr[32 * p + lane] : 0.0;
      cx[p] = 32 * p + lane < nr ? ce[32 * p + lane] : 0;
    }
    if (oi < nd2) {
      const int em = publish_wide<NP>(x, cx, nr, lane, s_x[warp]);
      const double v = fx_val(wx_dot<LD>(opw + oi * (4 * wq), nr, rr, s_x[warp], em));
      if (r < nr) {
        if (sizeof(T) == 4 || oi == 1) D5[o] = v;
        else D[N + o] = (T)v;
      }
    } else {
      int2* xs = reinterpret_cast<int2*>(s_x[warp]);
      const int em = publish_regs<NP>(x, cx, nr, lane, xs);
      const double v = fx_val(block_vec<LD>(opd, nr, rr, xs, em));
      if (r < nr) D[(f == 0 ? 0 : f + 1) * N + o] = (T)v;   // Dr of psi, T, S: blocks 0, 2, 3
    }
    __syncwarp();                                      // the digits are read before the next item's replace them
  }
  if (contract) {
    float* xv = ops + 2 * nr * nr;
    if (a.X32 && !a.fix.on) {                          // the caller's FP32 copy (the same values)
      for (int q = threadIdx.x; q < kn * 3 * nr; q += blockDim.x) {
        const int m = q / (3 * nr), e = q - m * 3 * nr, f = e / nr;
        xv[q] = a.X32[(size_t)b * a.x32_stride + f * N + (size_t)(k0 + m) * nr + (e - f * nr)];
      }
    } else {
      for (int q = threadIdx.x; q < kn * 3 * nr; q += blockDim.x) xv[q] = (float)xd[q];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < kn * 4 * nr; q += blockDim.x) {
      const int m = q / (4 * nr), e = q - m * 4 * nr, o = e / nr, n = e - o * nr;
      const float* row = ops + (o == 1 ? nr * nr : 0) + (size_t)n * nr;
      const float* x = xv + m * 3 * nr + (o < 2 ? 0 : (o - 1) * nr);
      float acc = 0.0f;
      for (int c = 0; c < nr; ++c) acc = fmaf(row[c], x[c], acc);
      D[o * N + (size_t)(k0 + m) * nr + n] = (T)acc;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kFxRowThreads) k_fx_grid(FxArgs a, T* grid, size_t grid_stride) {
  using C = typename Cplx<T>::type;
  using W = typename Cplx<T>::tw;
  using Tr = RowTr<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, nr = a.nr, P = a.P;
  const int n = blockIdx.x, pr = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x, bd = blockDim.x;
  const int ta = 2 * pr, tb = 2 * pr + 1;      // tb = 9 (absent) for the last pair

  C* RA = reinterpret_cast<C*>(smem_raw);
  C* RB = RA + P;
  W* Wt = reinterpret_cast<W*>(RB + P);
  W* Et = Wt + P;
  T* kf = reinterpret_cast<T*>(Et + P);   // kf[k] = k, k < P + 2
  T* pv = kf + P + 2;
  T* Tv = pv + M;
  T* Sv = Tv + M;
  T* DP = Sv + M;
  T* OM = DP + M;
  T* DTv = OM + M;
  T* DCv = DTv + M;
  T* JP = DCv + M;
  T* Sc = JP + M;
  T* scl = Sc + M;
  void* red = scl + 32;
  const W* wg = reinterpret_cast<const W*>(a.ops.w);
  const W* eg = reinterpret_cast<const W*>(a.ops.e);
#pragma unroll 1
  for (int i = tid; i < P; i += bd) {               // asynchronous: in flight while the row loads
    cp_async_elem(Wt + i, wg + i);
    cp_async_elem(Et + i, eg + i);
  }
#pragma unroll 1
  for (int i = tid; i < P + 2; i += bd) kf[i] = sizeof(T) == 8 ? (T)fx_int(i) : (T)i;
  const T ir4n = reinterpret_cast<const T*>(a.ops.ir4r2)[n];
  // (no barrier: the row loads below do not read the tables; the one after them covers both)
  after_previous_kernel();                          // (the tables are the plan's)
  if (a.active && !a.active[b]) {
    cp_async_all_done();
    return;
  }

  // which row quantities the pair's two fields need (fields: 0 JT_psi, 1 komega, 2 kDpsi, 3 DT, 4 DC,
  // 5 omega, 6 Dpsi, 7 kT, 8 kC)
  const bool need_psi = pr == 0 || pr == 2;            // pv (JT_psi, omega's A2 term) and D2 psi (omega)
  // The linear parts of the fused right-hand sides.  FP64 kernels split them over three pairs: pair 2 the T
  // and S parts, and psi's part by modes between pair 0 (k < M/2) and pair 4, whose one field leaves it the
  // least work (it forms psi's parity sums for that alone): so no pair carries all of psi's part beside its
  // own rows.  FP32 kernels form all three in pair 0 from FP64 copies of the row.
  const bool lin = a.fuse_rhs && (pr == 0 || (sizeof(T) == 8 && (pr == 2 || pr == 4)));
  const bool lin_psi = lin && (pr == 0 || pr == 4);
  const bool lin_ts = lin && (pr == 2 || sizeof(T) == 4);
  const int kp0 = (sizeof(T) == 8 && pr == 4) ? M / 2 : 0;   // psi's part: modes [kp0, kp1) of this pair
  const int kp1 = (sizeof(T) == 8 && pr == 0) ? M / 2 : M;
  double* pv64 = nullptr;
  if (sizeof(T) == 4 && lin)
    pv64 = reinterpret_cast<double*>(smem_raw + fx_grid_lin64_offset(M, P, SDD_PREC_MIXED));
  const int N = M * nr;
  const double* Xs = a.X + (size_t)b * a.x_stride;
  const T* Dv = reinterpret_cast<const T*>(a.deriv) + (size_t)b * a.deriv_stride;   // k_fx_deriv
  // the psi part's FP64 D2 psi (k_fx_deriv's fifth block) for this thread's first mode, loaded with the row
  const double* D2p = reinterpret_cast<const double*>(Dv) + (size_t)4 * M * nr * sizeof(T) / 8;
  double d2s0 = 0.0;
  if (lin_psi && tid >= kp0 && tid < kp1 && !(a.sym && (tid % 2 == 0))) d2s0 = D2p[(size_t)tid * nr + n];
  // the linear parts' per-row scalars, also loaded with the row (read after the parity sums)
  double lRa = 0.0, lRas = 0.0, lir2 = 0.0, lrsq = 0.0, ldT0 = 0.0, lgr = 0.0;
  if (lin) {
    lRa = a.rl.Ra[b];
    lRas = a.rl.Ra_s[b];
    lir2 = a.rl.ir2s[n];
    lrsq = a.rl.rsq[n];
    ldT0 = a.rl.dT0[n];
    lgr = a.rl.gr[n];
  }
  with_x<T>(a, b, [&](auto xr) {
  for (int k = tid; k < M; k += bd) {
    const bool psi_on = !(a.sym && (k % 2 == 0));
    const bool ts_on = !(a.sym && (k % 2 == 1));
    T dp = 0, d2 = 0, dtv = 0, dcv = 0, pn = 0, tn = 0, sn = 0;
    // k_fx_deriv writes [op][k][n]; k_deriv_tc (deriv_t) the transposed [op][n][k]
    const size_t o0 = a.deriv_t ? (size_t)n * M + k : (size_t)k * nr + n;
    const size_t ob = (size_t)M * nr;
    if (psi_on) {
      dp = Dv[o0];
      d2 = Dv[ob + o0];
      pn = xr((size_t)k * nr + n);
    }
    if (ts_on) {
      dtv = Dv[2 * ob + o0];
      dcv = Dv[3 * ob + o0];
      tn = xr(N + (size_t)k * nr + n);
      sn = xr(2 * (size_t)N + (size_t)k * nr + n);
    }
    pv[k] = pn;
    Tv[k] = tn;
    Sv[k] = sn;
    DP[k] = dp;
    OM[k] = d2;
    DTv[k] = dtv;
    DCv[k] = dcv;
    if (pv64) {
      pv64[k] = psi_on ? Xs[(size_t)k * nr + n] : 0.0;
      pv64[2 * M + k] = ts_on ? Xs[N + (size_t)k * nr + n] : 0.0;
      pv64[3 * M + k] = ts_on ? Xs[2 * N + (size_t)k * nr + n] : 0.0;
    }
  }
  });
  cp_async_all_done();
  __syncthreads();
  if (need_psi || lin_psi) {
    parity_suffix<T>(pv, Sc, M);                       // (ends with a barrier)
    if (pv64) parity_suffix<double>(pv64, pv64 + M, M);
    // one loop: the linear parts of the right-hand sides at row n (k_rhs's expressions, Main.py:262-280, in
    // FP64) and J_theta_RT / A2_SINE_R2 of the row, independent per k
    const double* pvd = pv64 ? pv64 : reinterpret_cast<const double*>(pv);
    const double* Scd = pv64 ? pv64 + M : reinterpret_cast<const double*>(Sc);
    const double* Tvd = pv64 ? pv64 + 2 * M : reinterpret_cast<const double*>(Tv);
    const double* Svd = pv64 ? pv64 + 3 * M : reinterpret_cast<const double*>(Sv);
    const RhsArgs& r = a.rl;
    const double gd = r.dt * r.Pr * lgr, dd = r.dt * ldT0;
    double* R = lin ? r.rhs + (size_t)b * r.rhs_stride : nullptr;
#pragma unroll 1
    for (int k = tid; k < M; k += bd) {
      if (need_psi) jp_om<T>(k, M, kf, pv, Sc, ir4n, JP[k], OM[k]);
      if (lin) {
        double k1, k2;                                 // (conversions would take the FP64 pipe)
        if constexpr (sizeof(T) == 8) {
          k1 = kf[k + 1];
          k2 = kf[k + 2];
        } else {
          k1 = fx_int(k + 1);
          k2 = fx_int(k + 2);
        }
        const size_t o = (size_t)k * nr + n;
        if (lin_psi && k >= kp0 && k < kp1) {
          const double s2 = (k + 2 < M) ? Scd[k + 2] : 0.0;
          const bool psi_on = !(a.sym && (k % 2 == 0));
          const double d2s = k == tid ? d2s0 : (psi_on ? D2p[(size_t)k * nr + n] : 0.0);
          const double om = lin_a2(d2s, k1, k2, lir2, pvd[k], s2);
          R[o] = k < M - 1 ? lin_psi_rhs(om, k1, gd, lRa, lRas, Tvd[k + 1], Svd[k + 1]) : om;
        }
        if (lin_ts) {
          const double jt = lin_jt(k, k1, k > 0 ? pvd[k - 1] : 0.0, (k + 1 < M) ? Scd[k + 1] : 0.0);
          R[N + o] = lin_ts_rhs(lrsq, Tvd[k], dd, jt);
          R[2 * N + o] = lin_ts_rhs(lrsq, Svd[k], dd, jt);
        }
      }
    }
    __syncthreads();
  }
  // the pair's two DCT3 input rows (in RB, free until the FFT) and their scales
  const int nt = (tb < 9) ? 2 : 1;
  T* XV = reinterpret_cast<T*>(RB);
  form_rows<T, 2>(XV, P, nt, red, scl,
                  [&](int u, int k) { return fx_x<T>(ta + u, k, M, P, kf, JP, OM, DP, DTv, DCv, Tv, Sv); });
  for_elems<T>(P, [&](int k) { RA[k] = Tr::pack(XV, P, 0, nt > 1, k, Et, scl); });
  __syncthreads();
  C* res = fft_rows<T, Tr::kInv, false>(RA, RB, 1, a.st, Wt);
  next_kernel_may_start();
  T* g = grid + (size_t)b * grid_stride + (size_t)n * 9 * P;
  for_elems<T>(nt * P, [&](int idx) {
    const int u = idx >= P ? 1 : 0;
    const int i = idx - u * P;
    const int t = ta + u;
    const int src = (i & 1) ? (P - 1 - (i >> 1)) : (i >> 1);
    const T val = Tr::out(res[src], u, 0, 2, scl);
    g[(size_t)t * P + i] = Tr::sign(val, t >= 5 && (i & 1));
  });
}

template <typename T, int MODE>
__global__ void __launch_bounds__(kFxRowThreads) k_fx_prod(FxArgs a, const T* grid, size_t grid_stride) {
  using C = typename Cplx<T>::type;
  using W = typename Cplx<T>::tw;
  using Tr = RowTr<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, nr = a.nr, P = a.P;
  const int n = blockIdx.x, p = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x, bd = blockDim.x;
  C* RA = reinterpret_cast<C*>(smem_raw);
  C* RB = RA + P;
  W* Wt = reinterpret_cast<W*>(RB + P);
  W* Et = Wt + P;
  T* PR = reinterpret_cast<T*>(Et + P);
  T* scl = PR + 2 * P;
  void* red = scl + 32;
  const W* wg = reinterpret_cast<const W*>(a.ops.w);
  const W* eg = reinterpret_cast<const W*>(a.ops.e);
#pragma unroll 1
  for (int i = tid; i < P; i += bd) {               // asynchronous: in flight while the products load
    cp_async_elem(Wt + i, wg + i);
    cp_async_elem(Et + i, eg + i);
  }
  after_previous_kernel();                          // (the tables are the plan's)
  if (a.active && !a.active[b]) {
    cp_async_all_done();
    return;
  }
  const T* RG = grid + (size_t)b * grid_stride + (size_t)n * 9 * P;
  const T* bs = (MODE == 1) ? reinterpret_cast<const T*>(a.base) + (size_t)b * a.base_stride + (size_t)n * 9 * P
                            : nullptr;
  unsigned m2[2] = {0, 0};
#pragma unroll 2
  for (int i = tid; i < P; i += bd) {               // (unrolled: both iterations' grid loads in flight)
    T v[2];
    grid_products<T, MODE>(p, RG, bs, i, P, v[0], v[1]);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      PR[t * P + i] = p == 0 ? Tr::sign(v[t], i & 1) : v[t];
      if constexpr (sizeof(T) == 4) m2[t] = max(m2[t], Bits<T>::absbits(v[t]));
    }
  }
  scale_rows<T, 2>(PR, P, m2, red, scl);
  for_elems<T>(P, [&](int nn) { RB[nn] = Tr::load(PR, P, 0, makhoul_src(nn, P), scl); });
  cp_async_all_done();
  __syncthreads();
  C* Z = fft_rows<T, false, false>(RB, RA, 1, a.st, Wt);
  next_kernel_may_start();
  const int N = M * nr;
  double* o = a.out4 + (size_t)b * a.out_stride;
  const T two_P = (T)2 / (T)P, one_P = (T)1 / (T)P;
#pragma unroll 1
  for (int s = tid; s < M; s += bd) {
    T ya = 0, yb = 0;
    bool zero;
    int k;
    if (p == 0) {            // sine pair: slot s <-> wavenumber s+1, read at k = P-1-s
      zero = (s == M - 1) || (a.sym && (s % 2 == 0));
      k = P - 1 - s;
    } else {
      zero = a.sym && (s % 2 == 1);
      k = s;
    }
    if (!zero) {
      Tr::unpack(Z, P, k, 0, 2, Et, scl, (p == 1 && k == 0) ? one_P : two_P, ya, yb);
    }
    const size_t q0 = (size_t)(2 * p) * N + (size_t)s * nr + n;
    o[q0] = (double)ya;
    o[q0 + N] = (double)yb;
    if (sizeof(T) == 4 && p == 0 && a.q32) a.q32[(size_t)b * M * a.nr + (size_t)s * a.nr + n] = (float)ya;
  }
}

// ---- right-hand sides of the three implicit solves (Main.py:262-280) ---------------------------
// Linear steps, and (cnab2) the second-order step with the nonlinear term's outputs and the history; other steps form
// theirs in k_fx_grid or k_rhs_lin and the h kernel.
__global__ void __launch_bounds__(kFxThreads) k_rhs(RhsArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, nr = a.nr;
  const int n = blockIdx.x, b = blockIdx.y;
  const int tid = threadIdx.x, bd = blockDim.x;
  double* sm = reinterpret_cast<double*>(smem_raw);
  double* pv = sm;
  double* Sc = pv + M;
  double* D2p = Sc + M;
  double* DrQ = D2p + M;
  double* Tv = DrQ + M;
  double* Sv = Tv + M;
  double* opr = Sv + M;  // Dr row n, D2s row n
  // kd[k] = k: the mode numbers as doubles, read instead of converted (a conversion is an FP64-pipe
  // instruction on this GPU); the same exact values, so the same bits
  double* kd = opr + 2 * nr;
  for (int m = tid; m < nr; m += bd) {
    opr[m] = a.Dr[n * nr + m];
    opr[nr + m] = a.D2s[n * nr + m];
  }
  for (int k = tid; k < M + 3; k += bd) kd[k] = fx_int(k);
  after_previous_kernel();     // (the operators are the plan's)
  if (a.active && !a.active[b]) return;
  __syncthreads();
  const int N = M * nr;
  const double* Xs = a.X + (size_t)b * a.x_stride;
  const double* O4 = a.linear ? nullptr : a.out4 + (size_t)b * a.out_stride;
  for (int k = tid; k < M; k += bd) {
    const bool psi_on = !(a.sym && (k % 2 == 0));
    const bool ts_on = !(a.sym && (k % 2 == 1));
    const double* ps = Xs + (size_t)k * nr;
    double d2 = 0, pn = 0, q = 0;
    if (psi_on) {
      for (int m = 0; m < nr; ++m) d2 = fma(opr[nr + m], ps[m], d2);
      pn = ps[n];
    }
    if (O4 && a.q32) {         // FP32 nonlinear term: Dr Q in FP32 (the h kernel's order of sums)
      const float* qs = a.q32 + (size_t)b * M * nr + (size_t)k * nr;
      const float* drn = a.Dr32 + (size_t)n * nr;
      float d = 0.0f;
      for (int m = 0; m < nr; ++m) d = fmaf(__ldg(drn + m), qs[m], d);
      q = (double)d;
    } else if (O4) {
      const double* qs = O4 + (size_t)k * nr;
      for (int m = 0; m < nr; ++m) q = fma(opr[m], qs[m], q);
    }
    pv[k] = pn;
    D2p[k] = d2;
    DrQ[k] = q;
    Tv[k] = ts_on ? Xs[N + (size_t)k * nr + n] : 0.0;
    Sv[k] = ts_on ? Xs[2 * N + (size_t)k * nr + n] : 0.0;
  }
  __syncthreads();
  parity_suffix<double>(pv, Sc, M);
  next_kernel_may_start();
  __syncthreads();
  const double dt = a.dt, dtPr = a.dt * a.Pr;
  const double Ra = a.Ra[b], Ras = a.Ra_s[b];
  const double ir2 = a.ir2s[n], rsq = a.rsq[n], dT0 = a.dT0[n], gr = a.gr[n];
  double* R = a.rhs + (size_t)b * a.rhs_stride;
  const double gd = dtPr * gr, dd = dt * dT0;
  for (int k = tid; k < M; k += bd) {
    const double k1 = kd[k + 1], k2 = kd[k + 2];
    const double JP = lin_jt(k, k1, k > 0 ? pv[k - 1] : 0.0, (k + 1 < M) ? Sc[k + 1] : 0.0);    // J_theta_RT
    const double Om = lin_a2(D2p[k], k1, k2, ir2, pv[k], (k + 2 < M) ? Sc[k + 2] : 0.0);          // A2_SINE
    const size_t o = (size_t)k * nr + n;
    if (a.cnab2) {
      const double grv = (k < M - 1) ? (-k1 * gr) * (Ra * Tv[k + 1] - Ras * Sv[k + 1]) : 0.0;
      const double psiT0 = dT0 * JP;                                            // DT0_theta
      // explicit terms per unit time at this step, and the Adams-Bashforth 2 extrapolation
      const double ep = -(DrQ[k] - O4[N + o]) + a.Pr * grv;
      const double et = -O4[2 * N + o] - psiT0;
      const double es = -O4[3 * N + o] - psiT0;
      double* H = a.hist + (size_t)b * a.rhs_stride;
      double xp = ep, xt = et, xs = es;
      if (a.hist_valid) {
        xp = fma(1.5, ep, -0.5 * H[o]);
        xt = fma(1.5, et, -0.5 * H[N + o]);
        xs = fma(1.5, es, -0.5 * H[2 * N + o]);
      }
      H[o] = ep;
      H[N + o] = et;
      H[2 * N + o] = es;
      R[o] = fma(dt, xp, 2.0 * Om);
      R[N + o] = fma(dt, xt, 2.0 * (rsq * Tv[k]));
      R[2 * N + o] = fma(dt, xs, 2.0 * (rsq * Sv[k]));
      continue;
    }
    R[o] = k < M - 1 ? lin_psi_rhs(Om, k1, gd, Ra, Ras, Tv[k + 1], Sv[k + 1]) : Om;
    R[N + o] = lin_ts_rhs(rsq, Tv[k], dd, JP);
    R[2 * N + o] = lin_ts_rhs(rsq, Sv[k], dd, JP);
  }
}

// The linear parts alone (fuse_rhs with the fused row kernel; k_fx_grid forms the same expressions in the split
// path), with A2_SINE's D2 psi formed by k_fx_deriv.  One CTA per (row, shell).  Bound by the FP64 pipe (about 16
// operations an element, of them 12 in the loop) and its column-strided loads: 29 us at 64 shells of 256 x 30, 76 us as
// k_rhs with D2 psi.
__global__ void __launch_bounds__(kFxThreads) k_rhs_lin(RhsArgs a, const double* d2psi, size_t d2_stride) {
  after_previous_kernel();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, nr = a.nr;
  const int n = blockIdx.x, b = blockIdx.y;
  if (a.active && !a.active[b]) return;
  const int tid = threadIdx.x, bd = blockDim.x;
  double* pv = reinterpret_cast<double*>(smem_raw);
  double* Sc = pv + M;
  double* D2p = Sc + M;
  double* Tv = D2p + M;
  double* Sv = Tv + M;
  const size_t N = (size_t)M * nr;
  const double* Xs = a.X + (size_t)b * a.x_stride;
  const double* d2 = d2psi + (size_t)b * d2_stride;
  for (int k = tid; k < M; k += bd) {
    const bool psi_on = !(a.sym && (k % 2 == 0));
    const bool ts_on = !(a.sym && (k % 2 == 1));
    const size_t o = (size_t)k * nr + n;
    pv[k] = psi_on ? Xs[o] : 0.0;
    D2p[k] = psi_on ? d2[o] : 0.0;
    Tv[k] = ts_on ? Xs[N + o] : 0.0;
    Sv[k] = ts_on ? Xs[2 * N + o] : 0.0;
  }
  const double Ra = a.Ra[b], Ras = a.Ra_s[b], ir2 = a.ir2s[n], rsq = a.rsq[n];
  const double gd = a.dt * a.Pr * a.gr[n], dd = a.dt * a.dT0[n];
  __syncthreads();
  parity_suffix<double>(pv, Sc, M);
  next_kernel_may_start();
  double* R = a.rhs + (size_t)b * a.rhs_stride;
  for (int k = tid; k < M; k += bd) {
    const double k1 = fx_int(k + 1), k2 = fx_int(k + 2);
    const double jt = lin_jt(k, k1, k > 0 ? pv[k - 1] : 0.0, (k + 1 < M) ? Sc[k + 1] : 0.0);
    const double om = lin_a2(D2p[k], k1, k2, ir2, pv[k], (k + 2 < M) ? Sc[k + 2] : 0.0);
    const size_t o = (size_t)k * nr + n;
    R[o] = k < M - 1 ? lin_psi_rhs(om, k1, gd, Ra, Ras, Tv[k + 1], Sv[k + 1]) : om;
    R[N + o] = lin_ts_rhs(rsq, Tv[k], dd, jt);
    R[2 * N + o] = lin_ts_rhs(rsq, Sv[k], dd, jt);
  }
}

// The same right-hand sides in FP32, for Jacobian products inside GMRES solves whose tolerance is far
// above FP32 rounding: X from its FP32 copy, D2s and Dr Q in FP32, the nonlinear-term outputs rounded once,
// written to rhs32.  FP64 arithmetic (and FP64<->FP32 conversion) runs on the GPU's narrow FP64 pipe; here
// only the conversions of the nonlinear-term outputs and of the per-CTA scalars remain on it.  (Staging the
// psi and Q rows in shared memory was measured slower: the 66 KB per CTA cut the resident CTAs that hide
// the latency of these row reads.)
__global__ void __launch_bounds__(kFxThreads) k_rhs32(RhsArgs a) {
  after_previous_kernel();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float scal[8];
  const int M = a.M, nr = a.nr;
  const int n = blockIdx.x, b = blockIdx.y;
  if (a.active && !a.active[b]) return;
  const int tid = threadIdx.x, bd = blockDim.x;
  float* sm = reinterpret_cast<float*>(smem_raw);
  float* pv = sm;
  float* Sc = pv + M;
  float* D2p = Sc + M;
  float* DrQ = D2p + M;
  float* Tv = DrQ + M;
  float* Sv = Tv + M;
  float* opr = Sv + M;                      // Dr row n, D2s row n
  for (int m = tid; m < nr; m += bd) {
    opr[m] = a.Dr32[n * nr + m];
    opr[nr + m] = a.D2s32[n * nr + m];
  }
  if (tid == 0) {
    scal[0] = (float)a.dt;
    scal[1] = (float)(a.dt * a.Pr);
    scal[2] = (float)a.Ra[b];
    scal[3] = (float)a.Ra_s[b];
    scal[4] = (float)a.ir2s[n];
    scal[5] = (float)a.rsq[n];
    scal[6] = (float)a.dT0[n];
    scal[7] = (float)a.gr[n];
  }
  const int N = M * nr;
  const float* Xs = a.X32 + (size_t)b * a.x32_stride;
  const double* O4 = a.linear ? nullptr : a.out4 + (size_t)b * a.out_stride;
  __syncthreads();                          // opr / scal are visible
  for (int k = tid; k < M; k += bd) {
    const bool psi_on = !(a.sym && (k % 2 == 0));
    const bool ts_on = !(a.sym && (k % 2 == 1));
    const float* ps = Xs + (size_t)k * nr;
    float d2 = 0.0f, pn = 0.0f, q = 0.0f;
    if (psi_on) {
      for (int m = 0; m < nr; ++m) d2 = fmaf(opr[nr + m], ps[m], d2);
      pn = ps[n];
    }
    if (O4) {
      const float* qs = a.q32 + (size_t)b * M * nr + (size_t)k * nr;
      for (int m = 0; m < nr; ++m) q = fmaf(opr[m], qs[m], q);
    }
    pv[k] = pn;
    D2p[k] = d2;
    DrQ[k] = q;
    Tv[k] = ts_on ? Xs[N + (size_t)k * nr + n] : 0.0f;
    Sv[k] = ts_on ? Xs[2 * N + (size_t)k * nr + n] : 0.0f;
  }
  __syncthreads();
  parity_suffix<float>(pv, Sc, M);
  __syncthreads();
  const float dt = scal[0], dtPr = scal[1], Ra = scal[2], Ras = scal[3];
  const float ir2 = scal[4], rsq = scal[5], dT0 = scal[6], gr = scal[7];
  float* R = a.rhs32 + (size_t)b * a.rhs_stride;
  for (int k = tid; k < M; k += bd) {
    // k as a float without an int->float conversion: the bits of 2^23 + k, minus 2^23 (exact for k < 2^23)
    const float k1 = (__int_as_float(0x4B000000 | k) - 8388608.0f) + 1.0f;
    const float s1 = (k + 1 < M) ? Sc[k + 1] : 0.0f;
    const float JP = (k == 0) ? s1 : k1 * pv[k - 1] + 2.0f * s1;                                // J_theta_RT
    const float s2 = (k + 2 < M) ? Sc[k + 2] : 0.0f;
    const float Om = D2p[k] - k1 * ir2 * ((k1 + 1.0f) * pv[k] + 2.0f * s2);                    // A2_SINE
    const float grv = (k < M - 1) ? (-k1 * gr) * (Ra * Tv[k + 1] - Ras * Sv[k + 1]) : 0.0f;
    float nxp = 0.0f, nxt = 0.0f, nxs = 0.0f;
    const size_t o = (size_t)k * nr + n;
    if (O4) {
      nxp = -dt * (DrQ[k] - (float)O4[N + o]);
      nxt = -dt * (float)O4[2 * N + o];
      nxs = -dt * (float)O4[3 * N + o];
    }
    const float psiT0 = dT0 * JP;                                                            // DT0_theta
    R[o] = nxp + (Om + dtPr * grv);
    R[N + o] = nxt + (rsq * Tv[k] - dt * psiT0);
    R[2 * N + o] = nxs + (rsq * Sv[k] - dt * psiT0);
  }
}

// ---- standalone theta recurrences (J_theta_RT, A2_SINE_R2, A2_SINE, DT0_theta) ------------------
struct ThetaArgs {
  int op, M, nr, sym;
  const double* D2;
  const double* ir;
  const double* dT0;
  const double* g;
  double* f;
};

__global__ void __launch_bounds__(kFxThreads) k_theta_op(ThetaArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, nr = a.nr;
  const int n = blockIdx.x, b = blockIdx.y;
  const int tid = threadIdx.x, bd = blockDim.x;
  double* sm = reinterpret_cast<double*>(smem_raw);
  double* pv = sm;
  double* Sc = pv + M;
  double* D2p = Sc + M;
  double* opr = D2p + M;
  const bool a2 = (a.op == 1 || a.op == 2);
  if (a2)
    for (int m = tid; m < nr; m += bd) opr[m] = a.D2[n * nr + m];
  __syncthreads();
  const double* g = a.g + (size_t)b * M * nr;
  for (int k = tid; k < M; k += bd) {
    const bool on = !(a.sym && (k % 2 == 0));
    double d2 = 0, pn = 0;
    if (on) {
      const double* ps = g + (size_t)k * nr;
      if (a2)
        for (int m = 0; m < nr; ++m) d2 = fma(opr[m], ps[m], d2);
      pn = ps[n];
    }
    pv[k] = pn;
    D2p[k] = d2;
  }
  __syncthreads();
  parity_suffix<double>(pv, Sc, M);
  __syncthreads();
  double* f = a.f + (size_t)b * M * nr;
  for (int k = tid; k < M; k += bd) {
    const double s1 = (k + 1 < M) ? Sc[k + 1] : 0.0;
    const double s2 = (k + 2 < M) ? Sc[k + 2] : 0.0;
    double v;
    if (a2) {
      v = D2p[k] - (double)(k + 1) * (a.ir[n] * ((k + 2.0) * pv[k] + 2.0 * s2));
      if (a.sym && (k % 2 == 0)) v = 0.0;
    } else {
      const double jp = (k == 0) ? 1.0 * s1 : (k + 1.0) * pv[k - 1] + 2.0 * s1;
      v = (a.op == 3) ? a.dT0[n] * jp : jp;
      if (a.sym && (k % 2 == 1)) v = 0.0;
    }
    f[(size_t)k * nr + n] = v;
  }
}

// ---- standalone batched transforms (Transforms.py) -------------------------------------------
struct TrArgs {
  int kind, rows, n_in, n_out, L;
  StageArgs st;
  const int4* w;
  const int4* e;
  const double* in;
  double* out;
};

constexpr int kTrPairs = 2;

__global__ void __launch_bounds__(kFxThreads) k_transform(TrArgs a) {
  using C = longlong2;
  using Tr = RowTr<double>;
  constexpr int kRows = 2 * kTrPairs;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = a.L;
  C* RA = reinterpret_cast<C*>(smem_raw);
  C* RB = RA + kTrPairs * L;
  int4* Wt = reinterpret_cast<int4*>(RB + kTrPairs * L);
  int4* Et = Wt + L;
  double* scl = reinterpret_cast<double*>(Et + L);   // the rows' exponents
  void* red = scl + 8;                               // 4*32 reduction words of 8 bytes
  const int tid = threadIdx.x, bd = blockDim.x;
#pragma unroll 1
  for (int i = tid; i < L; i += bd) {
    Wt[i] = a.w[i];
    Et[i] = a.e[i];
  }
  const int r0 = blockIdx.x * kRows;
  const bool inverse = (a.kind == SDD_IDCT || a.kind == SDD_IDST);
  const bool sine = (a.kind == SDD_IDST || a.kind == SDD_DST);
  const int n_in = a.n_in, n_out = a.n_out;
  // the rows as they enter the transforms (DCT3: x_k, a sine row by its mirrored wavenumbers; DCT2: f_i with
  // the alternating sign of a sine row), in RB, free until the FFT
  double* XV = reinterpret_cast<double*>(RB);
#pragma unroll 1
  for (int t = 0; t < kRows; ++t) {
    const int r = r0 + t;
    const double* src = a.in + (size_t)r * n_in;
#pragma unroll 1
    for (int k = tid; k < L; k += bd) {
      double v = 0.0;
      if (r < a.rows) {
        if (!inverse) v = neg_if(src[k], sine && (k & 1));
        else if (!sine) v = (k < n_in) ? src[k] : 0.0;
        else if (k == 0) v = (L < n_in) ? 0.5 * src[L] : 0.0;
        else v = (L - k <= n_in - 1) ? src[L - k] : 0.0;
      }
      XV[t * L + k] = v;
    }
  }
  rows_to_fixed(XV, L, kRows, red, reinterpret_cast<int*>(scl));
  if (inverse) {
#pragma unroll 1
    for (int idx = tid; idx < kTrPairs * L; idx += bd) {
      const int p = idx / L;
      RA[idx] = Tr::pack(XV, L, 2 * p, true, idx - p * L, Et, scl);
    }
    __syncthreads();
    C* res = fft_rows<double, false>(RA, RB, kTrPairs, a.st, Wt);
#pragma unroll 1
    for (int idx = tid; idx < kRows * L; idx += bd) {
      const int t = idx / L;
      const int i = idx - t * L;
      const int r = r0 + t;
      if (r >= a.rows) continue;
      const int src = (i & 1) ? (L - 1 - (i >> 1)) : (i >> 1);
      const double val = Tr::out(res[(t >> 1) * L + src], t & 1, t & ~1, kRows, scl);
      a.out[(size_t)r * n_out + i] = neg_if(val, sine && (i & 1));
    }
  } else {
#pragma unroll 1
    for (int idx = tid; idx < kTrPairs * L; idx += bd) {
      const int p = idx / L;
      RA[idx] = Tr::load(XV, L, 2 * p, makhoul_src(idx - p * L, L), scl);
    }
    __syncthreads();
    C* Z = fft_rows<double, false>(RA, RB, kTrPairs, a.st, Wt);
#pragma unroll 1
    for (int idx = tid; idx < kTrPairs * n_out; idx += bd) {
      const int p = idx / n_out;
      const int s = idx - p * n_out;
      const int r = r0 + 2 * p;
      double ya = 0.0, yb = 0.0;
      if (!(sine && s == 0)) {
        const int k = sine ? L - s : s;
        Tr::unpack(Z + p * L, L, k, 2 * p, kRows, Et, scl, (!sine && k == 0) ? 1.0 / L : 2.0 / L, ya, yb);
      }
      if (r < a.rows) a.out[(size_t)r * n_out + s] = ya;
      if (r + 1 < a.rows) a.out[(size_t)(r + 1) * n_out + s] = yb;
    }
  }
}

// ---- F in state layout from the four spectral outputs (NLIN_FX/NLIN_DFX drop-ins) --------------
struct FinishArgs {
  int M, nr;
  const double* Dr;
  const double* out4;
  size_t out_stride;
  double* F;
  size_t f_stride;
};

__global__ void __launch_bounds__(kFxThreads) k_fx_finish(FinishArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* opr = reinterpret_cast<double*>(smem_raw);
  const int M = a.M, nr = a.nr, n = blockIdx.x, b = blockIdx.y;
  for (int m = threadIdx.x; m < nr; m += blockDim.x) opr[m] = a.Dr[n * nr + m];
  __syncthreads();
  const int N = M * nr;
  const double* O4 = a.out4 + (size_t)b * a.out_stride;
  double* F = a.F + (size_t)b * a.f_stride;
  for (int k = threadIdx.x; k < M; k += blockDim.x) {
    const double* qs = O4 + (size_t)k * nr;
    double q = 0;
    for (int m = 0; m < nr; ++m) q = fma(opr[m], qs[m], q);
    const size_t o = (size_t)k * nr + n;
    F[o] = q - O4[N + o];
    F[N + o] = O4[2 * N + o];
    F[2 * N + o] = O4[3 * N + o];
  }
}

static int fx_sm_count() {
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  return sms;
}

// ---- launchers ---------------------------------------------------------------------------------
// The tensor-core contractions of a mixed launch (a.deriv_t): every state row of the batch at once.
static cudaError_t launch_tc_for(const FxArgs& a, int batch, cudaStream_t s) {
  TcArgs t;
  t.M = a.M; t.nr = a.nr; t.sym = a.sym; t.KP = a.tcKP; t.NP = a.tcNP;
  t.rows = batch * 3 * a.M;
  t.X32 = a.X32; t.x32_stride = a.x32_stride;
  t.X = a.X; t.x_stride = a.x_stride;
  t.active = a.active;
  t.B = a.tcB;
  t.out = reinterpret_cast<float*>(a.deriv);
  t.out_stride = a.deriv_stride;
  t.err = a.tc_err;
  return launch_deriv_tc(t, s);
}

// The most dynamic shared memory a k_fx_rows launch of precision prec can take: the opt-in limit less the
// kernel's static shared memory (the parity scans' chunk totals), over its three modes.
size_t fx_rows_max_dynamic_smem(int prec) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  size_t stat = 0;
  auto take = [&](const void* f) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, f) == cudaSuccess) stat = fa.sharedSizeBytes > stat ? fa.sharedSizeBytes : stat;
    else cudaGetLastError();
  };
  if (prec == SDD_PREC_MIXED) {
    take(reinterpret_cast<const void*>(k_fx_rows<float, 0>));
    take(reinterpret_cast<const void*>(k_fx_rows<float, 1>));
    take(reinterpret_cast<const void*>(k_fx_rows<float, 2>));
  } else {
    take(reinterpret_cast<const void*>(k_fx_rows<double, 0>));
    take(reinterpret_cast<const void*>(k_fx_rows<double, 1>));
    take(reinterpret_cast<const void*>(k_fx_rows<double, 2>));
  }
  return (size_t)optin > stat ? (size_t)optin - stat : 0;
}

// k_fx_deriv where it has something to do: FP64 contractions, FP32 ones of the split path that are not on the
// tensor cores, the fused right-hand side's D2 psi, a pending correction.  Modes per CTA: with nr > 32 (one CTA an
// SM: 130 KB of operators) as many as make one wave, up to 8 (540 x 65: 37 us with 4, 64 us with 1); otherwise two
// (a pending correction takes two at once), and more as the batch grows, the operators loaded once for them.
template <typename T>
static cudaError_t launch_deriv(const FxArgs& a, int batch, bool split, cudaStream_t s) {
  const bool f32 = sizeof(T) == 4 && split && !a.deriv_t;
  if (sizeof(T) == 4 && !f32 && !a.fuse_rhs && !a.fix.on) return cudaSuccess;
  using Deriv = void (*)(FxArgs, T*, size_t, int, int);
  static const Deriv derivs[6] = {k_fx_deriv<T, 8>,  k_fx_deriv<T, 16>, k_fx_deriv<T, 24>,
                                  k_fx_deriv<T, 32>, k_fx_deriv<T, 48>, k_fx_deriv<T, 64>};
  static unsigned long long done[6] = {};
  const int ldi = a.nr <= 32 ? (a.nr - 1) / 8 : (a.nr <= 48 ? 4 : 5);   // fx_ld(nr)
  cudaError_t e;
  if ((e = ensure_smem_attr(derivs[ldi], &done[ldi])) != cudaSuccess) return e;
  const bool d2s = a.fuse_rhs != 0;
  int km = 2;
  if (a.nr > 32)
    km = min(8, max(1, (int)(((long)a.M * batch + fx_sm_count() - 1) / fx_sm_count())));
  else if (!a.fix.on)
    while (km < 16 && (long)a.M * batch >= 8l * km * fx_sm_count()) km *= 2;
  e = launch_kernel(derivs[ldi], dim3((a.M + km - 1) / km, batch), dim3(32 * deriv_warps(fx_ld(a.nr))),
                    fx_deriv_smem_bytes<T>(a.nr, d2s, a.fix.on != 0, km, f32), s, a, reinterpret_cast<T*>(a.deriv),
                    a.deriv_stride, km, f32 ? 1 : 0);
  ktimer_mark(SDD_K_FX_DERIV, s);
  return e;
}

// Threads of a k_fx_rows CTA.  A row's transforms leave most of an SM's issue slots empty behind their barriers, so
// several small CTAs serve it better than a large one: the SM's threads (512 at the FP64 kernel's 128 registers,
// 1024 FP32) are shared among the CTAs that shared memory lets in and the launch has.  us, 512 threads against the
// rule: FP64 64 shells of 256 x 30 (2 CTAs of 256) 321 / 248, 16 of 128 x 28 (3 of 160) 54 / 35, 32 of 64 x 20 (4 of 128) 63 /
// 26; FP32 64 shells of 256 x 30 (4 of 256) 107 / 82; 540 x 65 FP64 (one CTA fits) 113 with 512, 132 with 256.
template <typename T>
static int fx_row_threads(size_t smem, long ctas) {
  static const int sm_smem = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    return n;
  }();
  const long fit = (long)(sm_smem / (smem + 1024 + 512));   // (a CTA's reserved and static shared memory)
  const long want = (ctas + fx_sm_count() - 1) / fx_sm_count();
  const int n = (int)std::max(1l, std::min({fit, want, 8l}));
  const int total = sizeof(T) == 8 ? 512 : 1024;
  return std::max(128, std::min(kFxRowThreads, total / n / 32 * 32));
}

template <typename T, int MODE>
static cudaError_t launch_fx_t(const FxArgs& a, int batch, cudaStream_t s) {
  const size_t smem = fx_smem_bytes(a.M, a.P, sizeof(T) == 4 ? SDD_PREC_MIXED : SDD_PREC_FP64);
  static unsigned long long done = 0;
  cudaError_t e = ensure_smem_attr(k_fx_rows<T, MODE>, &done);
  if (e != cudaSuccess) return e;
  if (a.deriv && (e = launch_deriv<T>(a, batch, false, s)) != cudaSuccess) return e;
  if (sizeof(T) == 4 && a.deriv_t && (e = launch_tc_for(a, batch, s)) != cudaSuccess) return e;
  e = launch_kernel(k_fx_rows<T, MODE>, dim3(a.nr, batch), dim3(fx_row_threads<T>(smem, (long)a.nr * batch)), smem, s, a);
  ktimer_mark(SDD_K_FX_ROWS, s);
  return e;
}

// Threads of the split kernels' CTAs.  While every CTA has an SM of its own, what counts is the latency of the loops over
// the row's P elements: as many threads as give each loop its fewest rounds (P = 384: one of 384 instead of two of 256;
// us a step, 256 threads / this rule: 256 x 30 41.5 / 40.2, its residual 46.2 / 43.6, 540 x 65 138.5 / 136.8); with
// more CTAs than SMs, 256, of which two share an SM.
static int fx_split_threads(int P, long ctas) {
  if (ctas > fx_sm_count()) return kFxSplitThreads;
  const int passes = (P + kFxRowThreads - 1) / kFxRowThreads;
  return std::max(128, ((P + passes - 1) / passes + 31) / 32 * 32);
}

template <typename T, int MODE>
static cudaError_t launch_fx_split_t(const FxArgs& a, int batch, cudaStream_t s) {
  const int prec = sizeof(T) == 4 ? SDD_PREC_MIXED : SDD_PREC_FP64;
  // grid rows go to the caller's cache when one is given (modes 0 and 2), else to the scratch
  T* grid = reinterpret_cast<T*>((MODE != 1 && a.base) ? a.base : a.grid);
  const size_t gs = (MODE != 1 && a.base) ? a.base_stride : a.grid_stride;
  cudaError_t e;
  if ((e = launch_deriv<T>(a, batch, true, s)) != cudaSuccess) return e;
  // (the tensor cores' contractions follow on the corrected state)
  if (sizeof(T) == 4 && a.deriv_t && (e = launch_tc_for(a, batch, s)) != cudaSuccess) return e;
  {
    static unsigned long long done = 0;
    if ((e = ensure_smem_attr(k_fx_grid<T>, &done)) != cudaSuccess) return e;
    e = launch_kernel(k_fx_grid<T>, dim3(a.nr, 5, batch), dim3(fx_split_threads(a.P, 5L * a.nr * batch)),
                      fx_grid_smem_bytes(a.M, a.P, prec), s, a, grid, gs);
    ktimer_mark(SDD_K_FX_GRID, s);
    if (e != cudaSuccess || MODE == 2) return e;
  }
  constexpr int PM = MODE == 1 ? 1 : 0;
  static unsigned long long done = 0;
  if ((e = ensure_smem_attr(k_fx_prod<T, PM>, &done)) != cudaSuccess) return e;
  e = launch_kernel(k_fx_prod<T, PM>, dim3(a.nr, 2, batch), dim3(fx_split_threads(a.P, 2L * a.nr * batch)),
                    fx_prod_smem_bytes(a.P, prec), s, a, (const T*)grid, gs);
  ktimer_mark(SDD_K_FX_PROD, s);
  return e;
}

// The split path is taken when forced (split = 2) or, automatically, while the fused kernel would leave
// most SMs idle (nr * batch CTAs below half the SMs); it needs a grid scratch (or none: mode 2 and
// cached mode 0 write the cache).  A batch that shares the GPU with other launches (the captured
// multi-group graphs) is better served by the fused kernel; its autotuner sets the choice per plan.
bool fx_split_rule(int split, int nr, int batch) {
  if (split == 1) return false;
  return split == 2 || 2 * nr * batch <= fx_sm_count();
}

bool fx_uses_split(const FxArgs& a, int batch, int mode) {
  const bool has_grid = (mode != 1 && a.base) || a.grid;
  if (!has_grid || !a.deriv) return false;
  return fx_split_rule(a.split, a.nr, batch);
}

cudaError_t launch_fx(const FxArgs& a_in, int batch, int mode, int prec, cudaStream_t s) {
  FxArgs a = a_in;
  // mixed plans with tensor-core tables: the radial contractions go to k_deriv_tc (needs the deriv scratch)
  a.deriv_t = (prec == SDD_PREC_MIXED && a.tcB && a.deriv) ? 1 : 0;
  if (fx_uses_split(a, batch, mode)) {
    if (prec == SDD_PREC_MIXED) {
      if (mode == 0) return launch_fx_split_t<float, 0>(a, batch, s);
      if (mode == 1) return launch_fx_split_t<float, 1>(a, batch, s);
      return launch_fx_split_t<float, 2>(a, batch, s);
    }
    if (mode == 0) return launch_fx_split_t<double, 0>(a, batch, s);
    if (mode == 1) return launch_fx_split_t<double, 1>(a, batch, s);
    return launch_fx_split_t<double, 2>(a, batch, s);
  }
  if (prec == SDD_PREC_MIXED) {
    if (mode == 0) return launch_fx_t<float, 0>(a, batch, s);
    if (mode == 1) return launch_fx_t<float, 1>(a, batch, s);
    return launch_fx_t<float, 2>(a, batch, s);
  }
  if (mode == 0) return launch_fx_t<double, 0>(a, batch, s);
  if (mode == 1) return launch_fx_t<double, 1>(a, batch, s);
  return launch_fx_t<double, 2>(a, batch, s);
}

cudaError_t launch_rhs(const RhsArgs& a, int batch, cudaStream_t s) {
  if (a.rhs32) {   // needs X32, D2s32, Dr32 and (with a nonlinear term) q32
    if (!a.X32 || !a.D2s32 || !a.Dr32 || (!a.linear && !a.q32)) return cudaErrorInvalidValue;
    const size_t smem32 = (6 * (size_t)a.M + 2 * (size_t)a.nr) * sizeof(float);
    static unsigned long long done32 = 0;
    cudaError_t e = ensure_smem_attr(k_rhs32, &done32);
    if (e != cudaSuccess) return e;
    const cudaError_t er = launch_kernel(k_rhs32, dim3(a.nr, batch), dim3(kFxThreads), smem32, s, a);
    ktimer_mark(SDD_K_RHS, s);
    if (er != cudaSuccess) return er;
    return cudaGetLastError();
  }
  const size_t smem = (7 * (size_t)a.M + 3 + 2 * (size_t)a.nr) * sizeof(double);
  static unsigned long long done = 0;
  cudaError_t e = ensure_smem_attr(k_rhs, &done);
  if (e != cudaSuccess) return e;
  const cudaError_t er = launch_kernel(k_rhs, dim3(a.nr, batch), dim3(kFxThreads), smem, s, a);
  ktimer_mark(SDD_K_RHS, s);
  if (er != cudaSuccess) return er;
  return cudaGetLastError();
}

cudaError_t launch_rhs_lin(const RhsArgs& a, const double* d2psi, size_t d2_stride, int batch, cudaStream_t s) {
  const cudaError_t e = launch_kernel(k_rhs_lin, dim3(a.nr, batch), dim3(kFxThreads), 5 * (size_t)a.M * sizeof(double), s,
                                      a, d2psi, d2_stride);
  ktimer_mark(SDD_K_RHS, s);
  return e;
}

cudaError_t launch_theta_op(int op, int M, int nr, int sym, const double* D2, const double* ir,
                            const double* dT0, const double* g, double* f, int batch, cudaStream_t s) {
  ThetaArgs a{op, M, nr, sym, D2, ir, dT0, g, f};
  const size_t smem = (3 * (size_t)M + (size_t)nr) * sizeof(double);
  static unsigned long long done = 0;
  cudaError_t e = ensure_smem_attr(k_theta_op, &done);
  if (e != cudaSuccess) return e;
  k_theta_op<<<dim3(nr, batch), kFxThreads, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_fx_finish(int M, int nr, const double* Dr, const double* out4, size_t out_stride,
                             double* F, size_t f_stride, int batch, cudaStream_t s) {
  FinishArgs a{M, nr, Dr, out4, out_stride, F, f_stride};
  k_fx_finish<<<dim3(nr, batch), kFxThreads, nr * sizeof(double), s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_transform(int kind, int rows, int n_in, int n_out, const FftPlan* fp,
                             const double* in, double* out, cudaStream_t s) {
  TrArgs a;
  a.kind = kind;
  a.rows = rows;
  a.n_in = n_in;
  a.n_out = n_out;
  a.L = fp->L;
  a.st = stage_args(fp);
  a.w = fp->wfx;
  a.e = fp->efx;
  a.in = in;
  a.out = out;
  const size_t smem = (2 * kTrPairs + 2) * (size_t)fp->L * sizeof(longlong2) + (4 * 32 + 8) * 8;
  static unsigned long long done = 0;
  cudaError_t e = ensure_smem_attr(k_transform, &done);
  if (e != cudaSuccess) return e;
  const int grid = (rows + 2 * kTrPairs - 1) / (2 * kTrPairs);
  k_transform<<<grid, kFxThreads, smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace sdd
