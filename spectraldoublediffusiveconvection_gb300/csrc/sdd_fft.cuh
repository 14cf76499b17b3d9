// Shared-memory FFT building blocks for the theta transforms.
//
// The reference's transforms (Transforms.py:73-129) are scipy DCT-II/III and DST-II/III on the
// midpoint grid theta_i = pi(2i+1)/(2P).  Here every one of them is reduced to
//   DCT3:  f_i = sum_{k<P} x_k cos(k theta_i)            (inverse direction)
//   DCT2:  y_k = sum_{i<P} f_i cos(k theta_i)            (forward direction)
// and both are evaluated for two real rows at once with one complex FFT of length P (Makhoul's
// even/odd reordering; the pair rides in the real and imaginary parts):
//   DCT3: W_k = V_A(k) + i V_B(k),  V(k) = 0.5 e^{i pi k/2P} (x_k - i x_{P-k}) (k>=1), V(0) = x_0,
//         v = IDFT(W) (unnormalised),  f_{2n} = v_n,  f_{2n+1} = v_{P-1-n}  (A = Re, B = Im)
//   DCT2: z_n = f_A[src(n)] + i f_B[src(n)],  Z = DFT(z),
//         y_A[k] = c (Z_k + Z_{-k})_re/2 + s (Z_k - Z_{-k})_im/2,
//         y_B[k] = c (Z_k + Z_{-k})_im/2 - s (Z_k - Z_{-k})_re/2,   (c, s) = (cos, sin)(pi k/2P).
// The DCT twiddle table holds 0.5 (cos, sin)(pi k/2P), the factor 1/2 of both formulas folded in.
// Sine transforms use sin(w theta_i) = (-1)^i cos((P-w) theta_i).
// The complex FFT is a Stockham autosort FFT (natural order in and out) with radix-2/3/4/5/7 passes,
// ping-ponging between two shared-memory buffers; twiddles come from a table exp(-2 pi i k/L) built on
// the host.
//
// FP32 transforms run in FP32.  FP64 transforms run in 64-bit fixed point on the integer pipe (sdd_fixed.cuh): each row
// scaled by a power of two above its 1-norm, which bounds every value inside its transform; a complex product is 12 wide
// multiply-adds, a radix-4 butterfly with its twiddles 36, of 4.5 to 5 cycles each.
// N_r=30, N_theta=256, FP64 / fixed point: grid kernel 18.9 / 14.6 us, product kernel 14.4 / 10.2 us, row kernel of 64
// shells 712 / 492 us.
#pragma once
#include <cuda_runtime.h>
#include "sdd_fixed.cuh"
#include "sdd_internal.cuh"

namespace sdd {

// Element and twiddle types of a transform of T data: FP32 complex, or 64-bit fixed point with twiddles in
// two 32-bit digits per component.
template <typename T> struct Cplx;
template <> struct Cplx<double> { using type = longlong2; using tw = int4; };
template <> struct Cplx<float> { using type = float2; using tw = float2; };

template <typename C> __device__ __forceinline__ C cmk(decltype(C::x) a, decltype(C::x) b) {
  C r; r.x = a; r.y = b; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return cmk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return cmk<C>(a.x - b.x, a.y - b.y); }
// Every multiply-add is an explicit fma (the translation units that include this file are compiled
// without automatic contraction), so the rounding of a transform does not depend on the kernel it is
// inlined into.
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return cmk<float2>(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
}
// a times the twiddle (inverse direction: its conjugate)
template <bool INV> __device__ __forceinline__ float2 ctw(float2 a, float2 w) {
  return cmul(a, cmk<float2>(w.x, INV ? -w.y : w.y));
}
template <bool INV> __device__ __forceinline__ longlong2 ctw(longlong2 a, int4 w) { return fx_cmul<INV>(a, w); }
// multiply by -i (forward) or +i (inverse)
template <typename C, bool INV> __device__ __forceinline__ C cmul_mi(C a) {
  return INV ? cmk<C>(-a.y, a.x) : cmk<C>(a.y, -a.x);
}

// In-register radix-R DFT of v[0..R-1] (R a compile-time constant); w is the length-L twiddle table.
template <typename T, bool INV, int R>
__device__ __forceinline__ void butterfly(typename Cplx<T>::type (&v)[R], const typename Cplx<T>::tw* w, int L) {
  using C = typename Cplx<T>::type;
  if constexpr (R == 2) {
    C a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    C t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    C t2 = cadd(v[1], v[3]), t3 = cmul_mi<C, INV>(csub(v[1], v[3]));
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3);
    v[3] = csub(t1, t3);
  } else if constexpr (sizeof(T) == 8) {
    // odd radix in fixed point: with a_r = v_r + v_{R-r}, d_r = v_r - v_{R-r},
    //   out_q, out_{R-q} = (v_0 + sum_r cos(2 pi q r / R) a_r)  -+ i sum_r sin(2 pi q r / R) d_r   (forward)
    constexpr int H = (R - 1) / 2;
    const int step = L / R;
    C a[H], d[H], o[R];
    o[0] = v[0];
#pragma unroll
    for (int r = 0; r < H; ++r) {
      a[r] = cadd(v[r + 1], v[R - 1 - r]);
      d[r] = csub(v[r + 1], v[R - 1 - r]);
      o[0] = cadd(o[0], a[r]);
    }
#pragma unroll
    for (int q = 1; q <= H; ++q) {
      C A = v[0], B = cmk<C>(0, 0);
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        const int4 t = w[((q * r) % R) * step];        // (cos, -sin) in digits
        A = cadd(A, cmk<C>(fx_rmul(a[r - 1].x, t.x, t.y), fx_rmul(a[r - 1].y, t.x, t.y)));
        B = cadd(B, cmk<C>(fx_rmul(d[r - 1].x, t.z, t.w), fx_rmul(d[r - 1].y, t.z, t.w)));
      }
      // forward: i B with B = -sum sin d;  inverse: its negative
      const C iB = INV ? cmk<C>(B.y, -B.x) : cmk<C>(-B.y, B.x);
      o[q] = cadd(A, iB);
      o[R - q] = csub(A, iB);
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = o[q];
  } else if constexpr (R == 3) {
    const T h = (T)0.86602540378443864676;  // sqrt(3)/2
    C s = cadd(v[1], v[2]);
    C d = csub(v[1], v[2]);
    C t = cmk<C>(fma((T)-0.5, s.x, v[0].x), fma((T)-0.5, s.y, v[0].y));
    C u = cmul_mi<C, INV>(d);  // -i d forward
    v[0] = cadd(v[0], s);
    v[1] = cmk<C>(fma(h, u.x, t.x), fma(h, u.y, t.y));
    v[2] = cmk<C>(fma(-h, u.x, t.x), fma(-h, u.y, t.y));
  } else {  // small prime radix (5, 7): direct DFT with roots of unity from the table
    C o[R];
    const int step = L / R;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      C acc = v[0];
#pragma unroll
      for (int r = 1; r < R; ++r) acc = cadd(acc, ctw<INV>(v[r], w[((q * r) % R) * step]));
      o[q] = acc;
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = o[q];
  }
}

// One Stockham pass of radix R over nf FFTs of length L stored back to back (stride L); fnb, fns divide by
// nb = L / R and by Ns, tws = L / (Ns R) (precomputed per stage).
template <typename T, bool INV, int R>
__device__ __forceinline__ void fft_pass_r(const typename Cplx<T>::type* __restrict__ in,
                                           typename Cplx<T>::type* __restrict__ out, int L, int nf, int Ns,
                                           const typename Cplx<T>::tw* w, FastDiv fnb, FastDiv fns, int tws) {
  using C = typename Cplx<T>::type;
  const int nb = L / R;
  const int total = nf * nb;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int f = (int)fast_div((unsigned)t, fnb);
    const int j = t - f * nb;
    const C* src = in + f * L;
    C* dst = out + f * L;
    const int jq = (int)fast_div((unsigned)j, fns);
    const int k = j - jq * Ns;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[j + r * nb];
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = ctw<INV>(v[r], w[k * r * tws]);
    }
    butterfly<T, INV, R>(v, w, L);
    const int idxD = jq * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[idxD + r * Ns] = v[r];
  }
}

// The same pass in fixed point, out of line: the buffers and the table by their byte offsets in the block's
// dynamic shared memory (a generic pointer would cost the shared-memory loads).  Kept small: the row kernel
// once had 200 KB of inlined and unrolled code, and its warps waited for instructions more than for anything
// else.
template <int R>
static __device__ __noinline__ void fft_pass_fx(int in, int out, int w, int L, int nf, int Ns, FastDiv fnb, FastDiv fns,
                                                int tws) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const longlong2* I = reinterpret_cast<const longlong2*>(smem_raw + in);
  longlong2* O = reinterpret_cast<longlong2*>(smem_raw + out);
  const int4* W = reinterpret_cast<const int4*>(smem_raw + w);
  const int nb = L / R;
  const int total = nf * nb;
#pragma unroll 1
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int f = (int)fast_div((unsigned)t, fnb);
    const int j = t - f * nb;
    const int jq = (int)fast_div((unsigned)j, fns);
    const int k = j - jq * Ns;
    longlong2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = I[f * L + j + r * nb];
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = fx_cmul<false>(v[r], W[k * r * tws]);
    }
    butterfly<double, false, R>(v, W, L);
    const int d = f * L + jq * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) O[d + r * Ns] = v[r];
  }
}

template <typename T, bool INV, bool OUTLINE>
__device__ __forceinline__ void fft_pass(typename Cplx<T>::type* in, typename Cplx<T>::type* out, int L, int nf, int R,
                                         int Ns, const typename Cplx<T>::tw* w, FastDiv fnb, FastDiv fns, int tws) {
  if constexpr (sizeof(T) == 8 && OUTLINE) {
    static_assert(!INV, "FP64 inverse transforms are forward ones of swapped pairs (dct3_pack_fx)");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto off = [&](const void* p) { return (int)(reinterpret_cast<const unsigned char*>(p) - smem_raw); };
    const int i = off(in), o = off(out), wo = off(w);
    switch (R) {
      case 4: fft_pass_fx<4>(i, o, wo, L, nf, Ns, fnb, fns, tws); break;
      case 2: fft_pass_fx<2>(i, o, wo, L, nf, Ns, fnb, fns, tws); break;
      case 3: fft_pass_fx<3>(i, o, wo, L, nf, Ns, fnb, fns, tws); break;
      case 5: fft_pass_fx<5>(i, o, wo, L, nf, Ns, fnb, fns, tws); break;
      default: fft_pass_fx<7>(i, o, wo, L, nf, Ns, fnb, fns, tws); break;
    }
  } else {
    switch (R) {
      case 4: fft_pass_r<T, INV, 4>(in, out, L, nf, Ns, w, fnb, fns, tws); break;
      case 2: fft_pass_r<T, INV, 2>(in, out, L, nf, Ns, w, fnb, fns, tws); break;
      case 3: fft_pass_r<T, INV, 3>(in, out, L, nf, Ns, w, fnb, fns, tws); break;
      case 5: fft_pass_r<T, INV, 5>(in, out, L, nf, Ns, w, fnb, fns, tws); break;
      default: fft_pass_r<T, INV, 7>(in, out, L, nf, Ns, w, fnb, fns, tws); break;
    }
  }
}

// Full FFT of nf rows in buffer a (b is scratch of the same size).  Returns the buffer holding the
// result.  OUTLINE: FP64 passes out of line, for kernels with many rows per CTA and more than one transform; the
// split path's one-transform kernels inline them (10.2 against 12.2 us for the product kernel).  Must be called by all threads of the block; ends with a __syncthreads().
template <typename T, bool INV, bool OUTLINE = true>
__device__ typename Cplx<T>::type* fft_rows(typename Cplx<T>::type* a, typename Cplx<T>::type* b, int nf,
                                            const StageArgs& st, const typename Cplx<T>::tw* w) {
  using C = typename Cplx<T>::type;
  C* in = a;
  C* out = b;
  int Ns = 1;
#pragma unroll 1
  for (int s = 0; s < st.nst; ++s) {
    const int R = st.rad[s];
    fft_pass<T, INV, OUTLINE>(in, out, st.L, nf, R, Ns, w, st.nb[s], st.ns[s], st.tws[s]);
    __syncthreads();
    Ns *= R;
    C* tmp = in; in = out; out = tmp;
  }
  return in;
}

// DCT3 packing in fixed point (rows A, B of a pair at k and P - k): V_A(k) + i V_B(k) with
// V(k) = e_k (x_k - i x_{P-k}), that is e_k ((x_A,k + x_B,P-k) - i (x_A,P-k - x_B,k)).
__device__ __forceinline__ longlong2 dct3_pack_fx(int4 e, i64 xa, i64 xar, i64 xb, i64 xbr) {
  longlong2 z;
  z.x = xa + xbr;
  z.y = xb - xar;
  z = fx_cmul<false>(z, e);
  return make_longlong2(z.y, z.x);                     // swapped: the inverse transform is a forward one
}
// y_A, y_B of a DCT2 pair in fixed point from Z_k, Z_{-k} and e_k = 0.5 (cos, sin)(pi k/2P).
__device__ __forceinline__ void dct2_unpack_fx(longlong2 Zk, longlong2 Zm, int4 e, i64& ya, i64& yb) {
  const i64 u = Zk.x + Zm.x, v = Zk.y - Zm.y, s = Zk.y + Zm.y, t = Zm.x - Zk.x;
  const int u0 = fx_lo(u), u1 = fx_hi(u), v0 = fx_lo(v), v1 = fx_hi(v);
  const int s0 = fx_lo(s), s1 = fx_hi(s), t0 = fx_lo(t), t1 = fx_hi(t);
  const i64 R = 1ll << 29;
  const i64 a2 = fx_mad(u1, e.x, (i64)v1 * e.z);
  const i64 a1 = fx_mad(u1, e.y, fx_mad(u0, e.x, fx_mad(v1, e.w, fx_mad(v0, e.z, R))));
  const i64 b2 = fx_mad(s1, e.x, (i64)t1 * e.z);
  const i64 b1 = fx_mad(s1, e.y, fx_mad(s0, e.x, fx_mad(t1, e.w, fx_mad(t0, e.z, R))));
  ya = (a2 << 2) + (a1 >> 30);
  yb = (b2 << 2) + (b1 >> 30);
}

// Makhoul source index of reordered slot n (forward direction): v_n = f_{src(n)}.
__device__ __forceinline__ int makhoul_src(int n, int P) {
  return (n < (P + 1) / 2) ? 2 * n : 2 * (P - 1 - n) + 1;
}

}  // namespace sdd
