// Device Krylov kernels for the matrix-free Newton-GMRES of Main.py:523-536 (the reference calls
// scipy.sparse.linalg.lgmres on a LinearOperator wrapping PDFX).  Here: restarted GMRES(m) with
// classical Gram-Schmidt, the pass repeated for a column only where the first one cancelled w below
// kReorthEta of its norm, FP64 throughout, one Krylov space per shell of a batch.
//
// Reductions are deterministic: every dot product is a fixed-order two-level sum (per-CTA partials over
// fixed element chunks, then a fixed-order sum of the partials), so a shell's result does not depend
// on the other shells in the batch.
//
// Vector layout: V[i][b][ld]: Krylov vector i of shell b has n used doubles at stride ld (n = 3*N_fm*nr
// for Newton, n+1 with the continuation parameter appended for the bordered arclength system).
//
// FP32 basis (the VT = float instances): the Krylov vectors are stored rounded to FP32 and the
// Gram-Schmidt products run in FP32 arithmetic (per-thread FP32 partial sums over a few elements, the
// cross-thread sums in FP64); w, the norms, the Hessenberg matrix and the rotations stay FP64.  For inner
// solves whose tolerance (relative 1e-4 in Newton) is far above FP32 rounding: the outer residual is FP64,
// so the converged state is unchanged in accuracy.  The FP64 products are bound by the FP64 multiply-add
// rate (one per element of V), the FP32 ones by the bytes of V, half as many.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "sdd_fixed.cuh"
#include "sdd_internal.cuh"
#include "sdd_krylov.cuh"
#include "sdd_rowops.cuh"

namespace sdd {

constexpr int kDotThreads = 256;

// part[(b*(nv) + i)*nchunk + c] = sum over chunk c of V_i[b] . w[b],  i < nv.
// The chunk of w sits in registers (kDotPer elements per thread); the vectors go kDotVecs at a time, so
// each thread has kDotVecs * kDotPer independent loads in flight and a block reduction serves kDotVecs
// dot products (the products are FP64-throughput bound on this GPU, about 5 TB/s of V).  Each partial is
// a fixed-order sum: per thread over its elements in index order, then the warp's transposed shuffle
// tree (warp_sum4), then the warps in order.
constexpr int kDotPer = kDotChunk / kDotThreads;
constexpr int kSubPer = kSubChunk / kDotThreads;
static_assert(kSubChunk % kDotThreads == 0, "update chunk must be a multiple of the block");
constexpr int kDotVecs = 4;
static_assert(kDotChunk % kDotThreads == 0, "dot chunk must be a multiple of the block");

// warp_sum4 in FP32 (the FP32 basis's projections: conversions and FP64 additions hold the FP64 pipe, the
// FP32 ones do not); the same lane pattern.
__device__ __forceinline__ float warp_sum4f(const float (&sv)[4], int lane) {
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
  float k0 = h16 ? sv[2] : sv[0], k1 = h16 ? sv[3] : sv[1];
  const float s0 = h16 ? sv[0] : sv[2], s1 = h16 ? sv[1] : sv[3];
  k0 += __shfl_xor_sync(0xffffffffu, s0, 16);
  k1 += __shfl_xor_sync(0xffffffffu, s1, 16);
  float k = h8 ? k1 : k0;
  const float t = h8 ? k0 : k1;
  k += __shfl_xor_sync(0xffffffffu, t, 8);
  k += __shfl_xor_sync(0xffffffffu, k, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 1);
  return k;
}

// The last CTA of a shell to finish (ticket[b], one counter per shell, zero between launches) sums the
// shell's partials in chunk order and writes h: the reduction of k_dot_reduce, without its launch.
__device__ __forceinline__ bool last_chunk_of_shell(int* ticket, int b, int nblocks) {
  __shared__ int s_last;
  __syncthreads();                                   // this CTA's partials are written
  if (threadIdx.x == 0) {
    __threadfence();
    const int last = atomicAdd(ticket + b, 1) == nblocks - 1;
    if (last) {
      __threadfence();
      ticket[b] = 0;                                 // ready for the next launch
    }
    s_last = last;
  }
  __syncthreads();
  return s_last != 0;
}

__device__ __forceinline__ void reduce_partials(const double* part, int b, int nv, int nchunk, double* h, int ldh,
                                                int accumulate) {
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    double t = 0.0;
    const volatile double* p = part + ((size_t)b * nv + i) * nchunk;
    for (int c = 0; c < nchunk; ++c) t += p[c];
    if (accumulate) h[(size_t)b * ldh + i] += t;
    else h[(size_t)b * ldh + i] = t;
  }
}

// blockIdx.z selects the vectors [z vpb, (z+1) vpb) of the CTA (vpb a multiple of kDotVecs): small batches
// spread the vectors over more CTAs; every partial is summed the same way whatever the split.
template <typename VT>
__global__ void __launch_bounds__(kDotThreads) k_dot_partials(const VT* __restrict__ V, size_t vstride_i,
                                                             const double* __restrict__ w, int n, int ld, int nv,
                                                             int chunk, double* part,
                                                             const int* __restrict__ active, int* ticket,
                                                             double* h, int ldh, int accumulate, int vpb) {
  __shared__ double red[kDotVecs][kDotThreads / 32];
  const int c = blockIdx.x, b = blockIdx.y, nchunk = gridDim.x;
  const int ib = blockIdx.z * vpb, ie = min(nv, ib + vpb);
  if (active && !active[b]) {                         // skipped shell: zero partials (its results are unused)
    for (int i = ib + threadIdx.x; i < ie; i += blockDim.x) part[((size_t)b * nv + i) * nchunk + c] = 0.0;
  } else {
    const int e0 = c * chunk;
    const double* wb = w + (size_t)b * ld;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    VT wr[kDotPer];
#pragma unroll
    for (int k = 0; k < kDotPer; ++k) {
      const int e = e0 + threadIdx.x + k * kDotThreads;
      wr[k] = e < n ? (VT)wb[e] : (VT)0;
    }
    for (int i0 = ib; i0 < ie; i0 += kDotVecs) {
      VT sp[kDotVecs];
#pragma unroll
      for (int u = 0; u < kDotVecs; ++u) {
        sp[u] = (VT)0;
        if (i0 + u < ie) {
          const VT* vb = V + (size_t)(i0 + u) * vstride_i + (size_t)b * ld;
          VT x[kDotPer];                               // (all loads in flight before the first multiply-add)
#pragma unroll
          for (int k = 0; k < kDotPer; ++k) {
            const int e = e0 + threadIdx.x + k * kDotThreads;
            x[k] = e < n ? vb[e] : (VT)0;
          }
#pragma unroll
          for (int k = 0; k < kDotPer; ++k)
            if (e0 + k * kDotThreads + (int)threadIdx.x < n) sp[u] = fma(x[k], wr[k], sp[u]);
        }
      }
      static_assert(kDotVecs == 4, "warp_sum4 reduces four vectors");
      double ws;
      if constexpr (sizeof(VT) == 4) {
        ws = (double)warp_sum4f(sp, lane);             // the warp's 256 products in FP32, then FP64
      } else {
        ws = warp_sum4(sp, lane);
      }
      if ((lane & 7) == 0) red[lane >> 3][warp] = ws;
      __syncthreads();
      if (threadIdx.x < kDotVecs && i0 + threadIdx.x < ie) {
        double t = 0.0;
        for (int q = 0; q < kDotThreads / 32; ++q) t += red[threadIdx.x][q];
        part[((size_t)b * nv + i0 + threadIdx.x) * nchunk + c] = t;
      }
      __syncthreads();
    }
  }
  if (ticket && last_chunk_of_shell(ticket, b, nchunk * gridDim.z))
    reduce_partials(part, b, nv, nchunk, h, ldh, accumulate);
}

// w[b] -= sum_{i<nv} V_i[b] coef[b*ldc + i] for the shells with sub_mask[b] (per element, the products summed
// in index order), then nrm2[b] = |w[b]|^2 for the shells with norm_mask[b] (0 for the others): per thread over its elements
// in index order, the warp tree of k_dot_partials, the warps in order, the chunks of kSubChunk elements in
// order.  The chunks are a quarter of the dot products' (the update's dependent multiply-adds over the
// basis dominate, so one shell's update spreads over four times the CTAs).  With reo != nullptr the shell's
// last CTA also sets the second-pass flag of column j: active and |w'|^2 < eta^2 (|w'|^2 + |h|^2), where
// |w|^2 = |w'|^2 + |h|^2 for an orthonormal basis.
template <typename VT>
__global__ void __launch_bounds__(kDotThreads) k_sub_norm(const VT* __restrict__ V, size_t vstride_i, double* w,
                                                         const double* __restrict__ coef, int ldc, int n, int ld,
                                                         int nv, const int* __restrict__ sub_mask,
                                                         const int* __restrict__ norm_mask, double* part,
                                                         int* ticket, double* nrm2, GmresState gs, int j,
                                                         double eta2, int set_reo) {
  __shared__ double red[kDotVecs][kDotThreads / 32];
  __shared__ VT cs[kMaxRestart + 1];                   // the coefficients in the basis's precision
  const int c = blockIdx.x, b = blockIdx.y, nchunk = gridDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e0 = c * kSubChunk;
  double* wb = w + (size_t)b * ld;
  const bool sub = !sub_mask || sub_mask[b];
  const bool nrm = !norm_mask || norm_mask[b];
  const double* cb = coef + (size_t)b * ldc;
  for (int i = threadIdx.x; i < nv && i <= kMaxRestart; i += blockDim.x) cs[i] = (VT)cb[i];
  __syncthreads();
  double sv[kDotVecs] = {0.0, 0.0, 0.0, 0.0};
  // per element the products summed in index order; the thread's elements side by side, so that their
  // loads of one basis vector are in flight together
  VT t[kSubPer];
#pragma unroll
  for (int k = 0; k < kSubPer; ++k) t[k] = (VT)0;
  if (sub) {
    const VT* vb = V + (size_t)b * ld + e0 + threadIdx.x;
    const int kmax = min(kSubPer, max(0, (n - e0 - (int)threadIdx.x + kDotThreads - 1) / kDotThreads));
    if (kmax == kSubPer) {
#pragma unroll 4
      for (int i = 0; i < nv; ++i) {
#pragma unroll
        for (int k = 0; k < kSubPer; ++k) t[k] += vb[(size_t)i * vstride_i + k * kDotThreads] * cs[i];
      }
    } else {
      for (int i = 0; i < nv; ++i)
        for (int k = 0; k < kmax; ++k) t[k] += vb[(size_t)i * vstride_i + k * kDotThreads] * cs[i];
    }
  }
#pragma unroll
  for (int k = 0; k < kSubPer; ++k) {
    const int e = e0 + threadIdx.x + k * kDotThreads;
    if (e < n) {
      double x = wb[e];
      if (sub) {
        x -= (double)t[k];
        wb[e] = x;
      }
      if (nrm) sv[0] = fma(x, x, sv[0]);
    }
  }
  const double ws = warp_sum4(sv, lane);
  if ((lane & 7) == 0) red[lane >> 3][warp] = ws;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int q = 0; q < kDotThreads / 32; ++q) t += red[0][q];
    part[(size_t)b * nchunk + c] = nrm ? t : 0.0;
  }
  if (last_chunk_of_shell(ticket, b, nchunk) && threadIdx.x == 0) {
    double t = 0.0;
    const volatile double* p = part + (size_t)b * nchunk;
    for (int q = 0; q < nchunk; ++q) t += p[q];
    nrm2[b] = t;
    if (set_reo) {
      int r = 0;
      if (gs.active[b]) {
        const double* hc = gs.hcol + (size_t)b * (gs.m + 1);
        double h2 = 0.0;
        for (int i = 0; i <= j; ++i) h2 = fma(hc[i], hc[i], h2);
        r = t < eta2 * (t + h2) ? 1 : 0;
      }
      gs.reo[b] = r;
    }
  }
}

// h[b*ldh + i] (+)= sum_c part[(b*nv+i)*nchunk + c]
__global__ void k_dot_reduce(const double* __restrict__ part, int nv, int nchunk, double* __restrict__ h,
                             int ldh, int accumulate) {
  const int b = blockIdx.x;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    double t = 0.0;
    const double* p = part + ((size_t)b * nv + i) * nchunk;
    for (int c = 0; c < nchunk; ++c) t += p[c];
    if (accumulate) h[(size_t)b * ldh + i] += t;
    else h[(size_t)b * ldh + i] = t;
  }
}

// x[b] += sum_{i<k_b} V_i[b] * y[b*ldy + i]  (the sum in the basis's precision)
template <typename VT>
__global__ void k_add_combination(const VT* __restrict__ V, size_t vstride_i, double* __restrict__ x,
                                  const double* __restrict__ y, int ldy, const int* __restrict__ kb, int n,
                                  int ld) {
  __shared__ VT ys[kMaxRestart];
  const int b = blockIdx.y;
  const int k = min(kb[b], kMaxRestart);
  const double* yb = y + (size_t)b * ldy;
  for (int i = threadIdx.x; i < k; i += blockDim.x) ys[i] = (VT)yb[i];
  __syncthreads();
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    VT s = (VT)0;
    for (int i = 0; i < k; ++i) s += V[(size_t)i * vstride_i + (size_t)b * ld + e] * ys[i];
    x[(size_t)b * ld + e] += (double)s;
  }
}

// out[b] = a[b] * scale[b]  (scale may be per shell); out32 / out2 (nullable): FP32 and FP64 copies
__global__ void k_scale(const double* __restrict__ a, const double* __restrict__ scale, double* __restrict__ out,
                        int n, int ld, float* __restrict__ out32, double* __restrict__ out2) {
  const int b = blockIdx.y;
  const double s = scale[b];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const double v = a[(size_t)b * ld + e] * s;
    out[(size_t)b * ld + e] = v;
    if (out32) out32[(size_t)b * ld + e] = (float)v;
    if (out2) out2[(size_t)b * ld + e] = v;
  }
}

// FP32 basis: out[b] = fl32(a[b] * scale[b]); out32 (nullable) the same FP32 values, out2 (nullable) them
// in FP64 (the vector the next product reads is exactly the stored basis vector)
__global__ void k_scale_to32(const double* __restrict__ a, const double* __restrict__ scale, float* __restrict__ out,
                             int n, int ld, float* __restrict__ out32, double* __restrict__ out2) {
  const int b = blockIdx.y;
  const double s = scale[b];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const float v = (float)(a[(size_t)b * ld + e] * s);
    out[(size_t)b * ld + e] = v;
    if (out32) out32[(size_t)b * ld + e] = v;
    if (out2) out2[(size_t)b * ld + e] = (double)v;
  }
}

// out[e] = (double)in[e]
__global__ void k_widen(const float* __restrict__ in, double* __restrict__ out, size_t n) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    out[e] = (double)in[e];
}

// out = a - b
__global__ void k_sub(const double* __restrict__ a, const double* __restrict__ bb, double* __restrict__ out,
                      size_t n) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
    out[e] = a[e] - bb[e];
}

// X[b] (stride ldx) -= dx[b] (stride ld) where mask[b] != 0
__global__ void k_masked_sub(double* __restrict__ X, const double* __restrict__ dx, const int* __restrict__ mask,
                             int n, int ldx, int ld) {
  const int b = blockIdx.y;
  if (!mask[b]) return;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    X[(size_t)b * ldx + e] -= dx[(size_t)b * ld + e];
}

// Start of a GMRES cycle.  nrm2[b] = ||r_b||^2.  Sets beta, g = [beta,0..], inv = 1/beta, and the
// per-shell activity flag (active while the shell is being solved and beta is above its target).
__global__ void k_cycle_start(GmresState s, const double* __restrict__ nrm2, int B) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const double beta = sqrt(nrm2[b]);
  s.beta[b] = beta;
  double* g = s.g + (size_t)b * (s.m + 1);
  for (int i = 0; i <= s.m; ++i) g[i] = 0.0;
  g[0] = beta;
  const int act = s.solve[b] && beta > s.target[b] && beta > 0.0;
  s.active[b] = act;
  s.kb[b] = 0;
  s.inv[b] = (act && beta > 0.0) ? 1.0 / beta : 0.0;
  s.resid[b] = beta;
}

// One warp: column col[0 .. j] through the previous rotations (csv, snv) into out[0 .. j - 1]; returns the entry a of
// row j that the new rotation takes.  a_{i+1} = -sn_i a_i + cs_i col_{i+1} is a linear recurrence, scanned 32 rows at
// a time (each step of a serial chain would hold the SM sub-partition for four FP64 instructions of 64 cycles).
__device__ __forceinline__ double rotate_rows(const double* col, const double* csv, const double* snv, int j, int lane,
                                              double* out) {
  double a0 = col[0];
  for (int i0 = 0; i0 < j; i0 += 32) {
    const int i = i0 + lane;
    const bool ok = i < j;
    const double c = ok ? csv[i] : 0.0, s = ok ? snv[i] : 0.0, x = ok ? col[i + 1] : 0.0;
    double mul = ok ? -s : 1.0, add = c * x;           // rows past j: the identity
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double m1 = __shfl_up_sync(0xffffffffu, mul, o), q1 = __shfl_up_sync(0xffffffffu, add, o);
      if (lane >= o) {
        add = fma(mul, q1, add);
        mul *= m1;
      }
    }
    const double an = fma(mul, a0, add);               // a_{i+1}
    double ai = __shfl_up_sync(0xffffffffu, an, 1);
    if (lane == 0) ai = a0;
    if (ok) out[i] = fma(c, ai, s * x);
    a0 = __shfl_sync(0xffffffffu, an, 31);
  }
  return a0;
}

// One warp: the new rotation of column j from a and |w|^2, and whether the shell goes on.  The square roots and
// the divisions run in lanes side by side.
struct ArnoldiColumn {
  double cj, sj, r, gj, res, inv;
  int act;
};
__device__ __forceinline__ ArnoldiColumn new_rotation(double a, double nrm2, double gj, double beta, double target, int j,
                                                      int m, int lane) {
  ArnoldiColumn o;
  const double r2 = fma(a, a, nrm2);
  double root = sqrt(lane == 0 ? nrm2 : r2);
  if (!(r2 > 1e-280 && r2 < 1e290) && lane != 0) root = hypot(a, sqrt(nrm2));   // (a a out of range, or zero)
  const double hnext = __shfl_sync(0xffffffffu, root, 0);
  o.r = __shfl_sync(0xffffffffu, root, 1);
  const double q = (lane == 0 ? a : (lane == 1 ? hnext : 1.0)) / (lane < 2 ? o.r : hnext);
  o.cj = __shfl_sync(0xffffffffu, q, 0);
  o.sj = __shfl_sync(0xffffffffu, q, 1);
  o.inv = __shfl_sync(0xffffffffu, q, 2);
  if (!(o.r > 0.0)) {
    o.cj = 1.0;
    o.sj = 0.0;
  }
  o.gj = gj;
  o.res = fabs(-o.sj * gj);
  const bool breakdown = !(hnext > 1e-300 * beta);
  o.act = !(o.res <= target || breakdown || j + 1 == m);
  if (!o.act || !(hnext > 0.0)) o.inv = 0.0;
  return o;
}
__device__ __forceinline__ void store_column(const GmresState& s, int b, int j, const ArnoldiColumn& o) {
  const int m = s.m;
  double* H = s.H + (size_t)b * (m + 1) * m;
  double* g = s.g + (size_t)b * (m + 1);
  s.cs[(size_t)b * m + j] = o.cj;
  s.sn[(size_t)b * m + j] = o.sj;
  H[j * m + j] = o.r;
  H[(j + 1) * m + j] = 0.0;
  g[j + 1] = -o.sj * o.gj;
  g[j] = o.cj * o.gj;
  s.resid[b] = o.res;
  s.kb[b] = j + 1;
  s.active[b] = o.act;
  s.inv[b] = o.inv;
}

// After Gram-Schmidt for column j: hcol + h2 [b][0..j] hold the projections, nrm2[b] = ||w||^2.  Stores the
// column in H, applies the previous Givens rotations, makes the new one, updates g and the residual estimate.
__global__ void __launch_bounds__(32) k_arnoldi_finish(GmresState s, const double* __restrict__ nrm2, int j,
                                                        int B) {
  // one warp per shell: the column (hcol + h2) and the previous rotations in shared memory
  __shared__ double col[kMaxRestart + 1], csv[kMaxRestart], snv[kMaxRestart], out[kMaxRestart];
  const int b = blockIdx.x, lane = threadIdx.x;
  if (b >= B) return;
  const int m = s.m;
  const double* hc = s.hcol + (size_t)b * (m + 1);
  const double* hd = s.h2 + (size_t)b * (m + 1);
  if (!s.active[b]) {
    if (lane == 0) s.inv[b] = 0.0;
    return;
  }
  for (int i = lane; i <= j; i += 32) col[i] = hc[i] + hd[i];
  for (int i = lane; i < j; i += 32) {
    csv[i] = s.cs[(size_t)b * m + i];
    snv[i] = s.sn[(size_t)b * m + i];
  }
  const double gj = s.g[(size_t)b * (m + 1) + j], beta = s.beta[b], target = s.target[b];
  __syncwarp();
  const double a = rotate_rows(col, csv, snv, j, lane, out);
  const ArnoldiColumn o = new_rotation(a, nrm2[b], gj, beta, target, j, m, lane);
  if (lane == 0) store_column(s, b, j, o);
  __syncwarp();
  double* H = s.H + (size_t)b * (m + 1) * m;           // H[row*m + col]
  for (int i = lane; i < j; i += 32) H[i * m + j] = out[i];
}

template <typename E>
__device__ __forceinline__ void cp_async_one(E* smem, const E* gmem) {
  static_assert(sizeof(E) == 4 || sizeof(E) == 8, "element size");
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (sizeof(E) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem));
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem));
}

// Everything of column j after the product in one launch, for short vectors: w = A V_j is orthogonalised against
// V_0 .. V_j (the second pass where the first cancelled w below eta of its norm), the column of H rotated,
// V_{j+1} = w / |w| written (out; out2 and out32: its FP64 and FP32 copies).  A cluster of kOrthCtas CTAs per shell,
// each with a slice of w in shared memory; the partial projections and norms meet in distributed shared memory,
// every CTA sums them in rank order, so that all of a cluster hold the same column and the same 1 / |w|.
// As separate launches (two passes of two, the rotations, the scaling) each step pays a launch, a global reduction
// and a ticket.  This kernel is bound by about 14 dependent FP64 sums and five cluster barriers (11 us), then by its
// multiply-adds, which run on kOrthCtas SMs a shell only: longer vectors keep the launches.  us a column with its
// product, launches / one launch: FP64, n = 3648 104 / 67, 7488 114 / 83, 11808 120 / 109, 15744 128 / 132; FP32 basis,
// 8 shells, n = 4416 113 / 80, 15744 182 / 180.
// The rule goes by the vector's length alone, so that a shell's solve has the same bits alone and in any batch (the two
// forms sum in different orders).  Large batches pay for that: a cluster takes 16 SMs, nine run at a time.  Launches /
// one launch, 64 shells: FP64 n = 336 128 / 103, 3648 241 / 252, 6624 378 / 409, 11808 697 / 768; FP32 basis 336 110 / 112,
// 3648 155 / 164, 8832 268 / 277, 15744 507 / 598.  With 12 shells or fewer one launch is the faster one at every length
// it takes (the closest: FP64 n = 11808, 12 shells, 218 / 209).
// Projections: a warp takes four vectors and (few vectors) a quarter or a half of the slice; FP64 sums, or with an
// FP32 basis FP32 sums of at most 256 products, as in k_dot_partials.
// STAGE: the slice's part of V_0 .. V_j waits in shared memory (both passes read it twice), where it fits.
template <typename VT, bool STAGE>
__global__ void __launch_bounds__(kDotThreads + 32) k_orth(const VT* __restrict__ V, size_t vstride_i, const double* w, int n,
                                                     int ld, int j, GmresState s, double eta2, VT* out, float* out32,
                                                     double* out2, int* flags) {
  extern __shared__ __align__(16) unsigned char orth_smem[];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double sw[kOrthSlice];
  __shared__ double ps[4][kMaxRestart], pd[2][kMaxRestart], pn[2];
  __shared__ double hcol[kMaxRestart], hrot[kMaxRestart], h[kMaxRestart], csv[kMaxRestart], snv[kMaxRestart];
  __shared__ VT hv[kMaxRestart];
  __shared__ double red[kDotThreads / 32], s_nrm, s_h2, s_inv, s_a;
  const int rank = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nv = j + 1, m = s.m;
  const int ne = (n + kOrthCtas * 32 - 1) / (kOrthCtas * 32) * 32;   // the slice, at most kOrthSlice
  const int e0 = rank * ne, cnt = max(0, min(ne, n - e0));
  const double* wb = w + (size_t)b * ld + e0;
  const VT* Vg = V + (size_t)b * ld + e0;
  VT* Vs = reinterpret_cast<VT*>(orth_smem);           // [vector][ne]
  const VT* Vb = STAGE ? Vs : Vg;
  const size_t vstr = STAGE ? (size_t)ne : vstride_i;
  const size_t ob = (size_t)b * ld + e0;
  const int act = s.active[b];                         // (in flight with the copies below)
  if (STAGE) {
    for (int i = warp; i < nv; i += kDotThreads / 32 + 1)
      for (int e = lane; e < cnt; e += 32) cp_async_one(Vs + (size_t)i * ne + e, Vg + (size_t)i * vstride_i + e);
    cp_async_commit();
  }
  if (!act) {                                          // (the whole cluster) a shell that has stopped
    cp_async_wait<0>();
    if (rank == 0 && tid == 0) {
      s.inv[b] = 0.0;
      if (flags) flags[b] = 0;
    }
    if (out)
      for (int e = tid; e < cnt; e += blockDim.x) {
        const double v = wb[e] * 0.0;
        out[ob + e] = (VT)v;
        if (out32) out32[ob + e] = (float)v;
        if (out2) out2[ob + e] = (double)(VT)v;
      }
    return;
  }
  const bool rot = warp == kDotThreads / 32;           // the last warp only rotates the column
  for (int e = tid; e < ne; e += blockDim.x) sw[e] = e < cnt ? wb[e] : 0.0;
  if (tid < j) {                                       // (j < kMaxRestart threads)
    csv[tid] = s.cs[(size_t)b * m + tid];
    snv[tid] = s.sn[(size_t)b * m + tid];
  }
  const double gj = s.g[(size_t)b * (m + 1) + j], beta = s.beta[b], target = s.target[b];
  const int ng = (nv + 3) / 4, nseg = ng == 1 ? 4 : (ng == 2 ? 2 : 1);
  const int seg = (ne / nseg + 31) / 32 * 32;          // elements of a segment, whole warps of them
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (STAGE && pass == 0) cp_async_wait<0>();
    __syncthreads();                                   // sw, the slice of V
    for (int t = rot ? ng * nseg : warp; t < ng * nseg; t += kDotThreads / 32) {
      const int i0 = t / nseg * 4, q = t % nseg, a0 = q * seg, a1 = min(cnt, a0 + seg);
      double sum = 0.0;
      VT sp[4] = {(VT)0, (VT)0, (VT)0, (VT)0};
      const VT* vb = Vb + (size_t)i0 * vstr + lane;
      const int nu = min(4, nv - i0);
      for (int c0 = a0; c0 < a1; c0 += 256) {
        const int c1 = min(a1, c0 + 256);
#pragma unroll 4
        for (int c = c0; c < c1; c += 32) {
          const bool in = c + lane < c1;
          const VT x = in ? (VT)sw[c + lane] : (VT)0;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (u < nu) sp[u] = fma(in ? vb[(size_t)u * vstr + c] : (VT)0, x, sp[u]);
        }
        if constexpr (sizeof(VT) == 4) {
          sum += (double)warp_sum4f(sp, lane);
#pragma unroll
          for (int u = 0; u < 4; ++u) sp[u] = (VT)0;
        }
      }
      if constexpr (sizeof(VT) == 8) sum = warp_sum4(sp, lane);
      if ((lane & 7) == 0) ps[q][i0 + (lane >> 3)] = sum;
    }
    __syncthreads();
    if (tid < nv) {
      double t = ps[0][tid];
      for (int q = 1; q < nseg; ++q) t += ps[q][tid];
      pd[pass][tid] = t;
    }
    cluster.sync();
    if (tid < 4 * kMaxRestart) {                       // h_i over the ranks, four of them a thread
      const int i = tid >> 2, q = tid & 3;
      double t = 0.0;
      if (i < nv) {
        double v[kOrthCtas / 4];
#pragma unroll
        for (int r = 0; r < kOrthCtas / 4; ++r) v[r] = *cluster.map_shared_rank(&pd[pass][i], q * (kOrthCtas / 4) + r);
        t = v[0];
#pragma unroll
        for (int r = 1; r < kOrthCtas / 4; ++r) t += v[r];
      }
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      if (q == 0 && i < nv) {
        h[i] = t;
        hv[i] = (VT)t;
        hcol[i] = pass ? hcol[i] + t : t;
      }
    }
    __syncthreads();
    if (rot) {                                         // beside the update: the rotations so far, and |h|^2
      const double a = rotate_rows(hcol, csv, snv, j, lane, hrot);
      double t = lane < nv ? h[lane] * h[lane] : 0.0;
      for (int i = lane + 32; i < nv; i += 32) t = fma(h[i], h[i], t);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) {
        s_a = a;
        if (pass == 0) s_h2 = t;
      }
    }
    double nn = 0.0;
    for (int e = rot ? cnt : tid; e < cnt; e += kDotThreads) {
      VT t = (VT)0;
      const VT* vb = Vb + e;
#pragma unroll 8
      for (int i = 0; i < nv; ++i) t += vb[(size_t)i * vstr] * hv[i];
      const double x = sw[e] - (double)t;
      sw[e] = x;
      nn = fma(x, x, nn);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
    if (lane == 0 && !rot) red[warp] = nn;
    __syncthreads();
    if (warp == 0) {
      double t = lane < kDotThreads / 32 ? red[lane] : 0.0;
#pragma unroll
      for (int o = kDotThreads / 64; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) pn[pass] = t;
    }
    cluster.sync();
    if (warp == 0) {
      double t = lane < kOrthCtas ? *cluster.map_shared_rank(&pn[pass], lane) : 0.0;
#pragma unroll
      for (int o = kOrthCtas / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) s_nrm = t;
    }
    __syncthreads();
    const double t = s_nrm;
    if (pass == 0 && !(t < eta2 * (t + s_h2))) break;  // (the same numbers in every CTA of the cluster)
  }
  ArnoldiColumn col;
  if (warp == 0) {
    col = new_rotation(s_a, s_nrm, gj, beta, target, j, m, lane);
    if (lane == 0) s_inv = col.inv;
  }
  cluster.sync();                                      // all have read the shell's state; remote reads are done
  if (rank == 0) {
    if (tid == 0) {
      store_column(s, b, j, col);
      if (flags) flags[b] = col.act;
    }
    double* H = s.H + (size_t)b * (m + 1) * m;
    for (int i = tid; i < j; i += blockDim.x) H[i * m + j] = hrot[i];
  }
  if (out) {
    const double inv = s_inv;
    for (int e = tid; e < cnt; e += blockDim.x) {
      const double v = sw[e] * inv;
      out[ob + e] = (VT)v;
      if (out32) out32[ob + e] = (float)v;
      if (out2) out2[ob + e] = (double)(VT)v;
    }
  }
}

// Back substitution R y = g over the first kb[b] columns, one warp per shell: R in shared memory, lane l the rows l
// and l + 32; y_i = t_i / R_ii goes to all lanes, which take its column off their rows (one thread for a whole
// shell: 37 us at 50 columns, now about 20; the rows' divisions are 10 of them, which reciprocals formed ahead would save
// at the price of one more rounding an entry).
__global__ void __launch_bounds__(32) k_solve_y(GmresState s) {
  extern __shared__ __align__(16) double R[];
  const int b = blockIdx.x, lane = threadIdx.x;
  const int m = s.m, k = s.kb[b];
  const double* H = s.H + (size_t)b * (m + 1) * m;
  const double* g = s.g + (size_t)b * (m + 1);
  double* y = s.y + (size_t)b * m;
#pragma unroll 8
  for (int q = lane; q < k * m; q += 32) R[q] = H[q];
  __syncwarp();
  double t[2], d[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = lane + 32 * u;
    t[u] = r < k ? g[r] : 0.0;
    d[u] = r < k ? R[r * m + r] : 0.0;
  }
  for (int i = k - 1; i >= 0; --i) {
    const int u = i >> 5;
    const double di = u ? d[1] : d[0];
    const double yi = __shfl_sync(0xffffffffu, di != 0.0 ? (u ? t[1] : t[0]) / di : 0.0, i & 31);
    if (lane == 0) y[i] = yi;
#pragma unroll
    for (int v = 0; v < 2; ++v)
      if (lane + 32 * v < i) t[v] -= R[(lane + 32 * v) * m + i] * yi;
  }
}

// ---- pseudo-arclength continuation helpers (Main.py:829-837, 910-917) ------------------------------
// g[b][k][n] = dtPr * (-(k+1)) gr[n] T[b][k+1][n] for k < M-1, 0 for k = M-1: the psi right-hand side of
// PDFmu (kGR_RT applied to T, Matrix_Operators.py:97-128); symmetric plans drop the odd T slots.
__global__ void k_grk_T(const double* __restrict__ X, int ldx, double* __restrict__ g, int M, int nr,
                        const double* __restrict__ gr, double dtPr, int sym) {
  const int b = blockIdx.y;
  const int N = M * nr;
  const double* T = X + (size_t)b * ldx + N;
  double* gb = g + (size_t)b * 3 * N;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 3 * N; e += gridDim.x * blockDim.x) {
    double v = 0.0;
    if (e < N) {
      const int k = e / nr, n = e - k * nr;
      if (k < M - 1 && !(sym && ((k + 1) & 1))) v = dtPr * ((-(double)(k + 1) * gr[n]) * T[(size_t)(k + 1) * nr + n]);
    }
    gb[e] = v;
  }
}

// out[b][0..N) += v[b][n] * Jmu[b][0..N)  (psi block; Jmu stride ldj);  out[b][n] = delta*dot[b] + (1-delta)*mudot[b]*v[b][n]
__global__ void k_border(const double* __restrict__ v, double* __restrict__ out, int n, int ld,
                         const double* __restrict__ Jmu, int ldj, int Npsi, const double* __restrict__ dot,
                         const double* __restrict__ mudot, double delta) {
  const int b = blockIdx.y;
  const double vl = v[(size_t)b * ld + n];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < Npsi; e += gridDim.x * blockDim.x)
    out[(size_t)b * ld + e] += vl * Jmu[(size_t)b * ldj + e];
  if (blockIdx.x == 0 && threadIdx.x == 0) out[(size_t)b * ld + n] = delta * dot[b] + (1.0 - delta) * mudot[b] * vl;
}

// dst[b][e] (stride ldd) = a * src[b][e] (stride lds), e < n; optionally dst[b][n] = last[b]
__global__ void k_copy_scaled(const double* __restrict__ src, int lds, double* __restrict__ dst, int ldd, int n,
                              double a, const double* __restrict__ last) {
  const int b = blockIdx.y;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    dst[(size_t)b * ldd + e] = a * src[(size_t)b * lds + e];
  if (last && blockIdx.x == 0 && threadIdx.x == 0) dst[(size_t)b * ldd + n] = last[b];
}

// y[b] (stride ldy) = x0[b] (stride ldx0) + c[b] * d[b] (stride ldd), e < n
__global__ void k_axpy_shell(const double* __restrict__ x0, int ldx0, const double* __restrict__ d, int ldd,
                             const double* __restrict__ c, double* __restrict__ y, int ldy, int n) {
  const int b = blockIdx.y;
  const double cb = c[b];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    y[(size_t)b * ldy + e] = x0[(size_t)b * ldx0 + e] + cb * d[(size_t)b * ldd + e];
}

// ---- host wrappers ------------------------------------------------------------------------------
static int grid_x(int n) {
  int g = (n + 255) / 256;
  return g < 1 ? 1 : (g > 1024 ? 1024 : g);
}

static int sm_count_dev() {
  static int n = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 1;
  }();
  return n;
}

template <typename VT>
static cudaError_t krylov_dots_t(const VT* V, size_t vstride_i, const double* w, int n, int ld, int nv, int B,
                                 double* part, double* h, int ldh, int accumulate, cudaStream_t st, const int* active,
                                 int* ticket) {
  const int nchunk = (n + kDotChunk - 1) / kDotChunk;
  // with the one-launch reduction, spread the vectors over CTAs until the launch has ~2 CTAs per SM
  int nvg = 1;
  if (ticket) {
    const int want = (2 * sm_count_dev() + B * nchunk - 1) / (B * nchunk);
    nvg = std::max(1, std::min((nv + kDotVecs - 1) / kDotVecs, want));
  }
  int vpb = (nv + nvg - 1) / nvg;
  vpb = (vpb + kDotVecs - 1) / kDotVecs * kDotVecs;
  nvg = (nv + vpb - 1) / vpb;
  k_dot_partials<VT><<<dim3(nchunk, B, nvg), kDotThreads, 0, st>>>(V, vstride_i, w, n, ld, nv, kDotChunk, part,
                                                                   active, ticket, h, ldh, accumulate, vpb);
  if (!ticket) k_dot_reduce<<<B, 64, 0, st>>>(part, nv, nchunk, h, ldh, accumulate);
  return cudaGetLastError();
}
cudaError_t krylov_dots(const double* V, size_t vstride_i, const double* w, int n, int ld, int nv, int B,
                        double* part, double* h, int ldh, int accumulate, cudaStream_t st, const int* active,
                        int* ticket) {
  return krylov_dots_t(V, vstride_i, w, n, ld, nv, B, part, h, ldh, accumulate, st, active, ticket);
}
cudaError_t krylov_dots(const float* V, size_t vstride_i, const double* w, int n, int ld, int nv, int B,
                        double* part, double* h, int ldh, int accumulate, cudaStream_t st, const int* active,
                        int* ticket) {
  return krylov_dots_t(V, vstride_i, w, n, ld, nv, B, part, h, ldh, accumulate, st, active, ticket);
}

template <typename VT>
static cudaError_t krylov_sub_norm_t(const VT* V, size_t vstride_i, double* w, const double* coef, int ldc, int n,
                                     int ld, int nv, int B, const int* sub_mask, const int* norm_mask, double* part,
                                     int* ticket, double* nrm2, const GmresState* reo_of, int j, double eta,
                                     cudaStream_t st) {
  if (!ticket || nv > kMaxRestart + 1) return cudaErrorInvalidValue;
  const int nchunk = (n + kSubChunk - 1) / kSubChunk;
  GmresState gs{};
  if (reo_of) gs = *reo_of;
  k_sub_norm<VT><<<dim3(nchunk, B), kDotThreads, 0, st>>>(V, vstride_i, w, coef, ldc, n, ld, nv, sub_mask, norm_mask,
                                                          part, ticket, nrm2, gs, j, eta * eta, reo_of ? 1 : 0);
  return cudaGetLastError();
}
cudaError_t krylov_sub_norm(const double* V, size_t vstride_i, double* w, const double* coef, int ldc, int n, int ld,
                            int nv, int B, const int* sub_mask, const int* norm_mask, double* part, int* ticket,
                            double* nrm2, const GmresState* reo_of, int j, double eta, cudaStream_t st) {
  return krylov_sub_norm_t(V, vstride_i, w, coef, ldc, n, ld, nv, B, sub_mask, norm_mask, part, ticket, nrm2, reo_of,
                           j, eta, st);
}
cudaError_t krylov_sub_norm(const float* V, size_t vstride_i, double* w, const double* coef, int ldc, int n, int ld,
                            int nv, int B, const int* sub_mask, const int* norm_mask, double* part, int* ticket,
                            double* nrm2, const GmresState* reo_of, int j, double eta, cudaStream_t st) {
  return krylov_sub_norm_t(V, vstride_i, w, coef, ldc, n, ld, nv, B, sub_mask, norm_mask, part, ticket, nrm2, reo_of,
                           j, eta, st);
}

cudaError_t krylov_add_combination(const double* V, size_t vstride_i, double* x, const double* y, int ldy,
                                   const int* kb, int n, int ld, int B, cudaStream_t st) {
  k_add_combination<double><<<dim3(grid_x(n), B), 256, 0, st>>>(V, vstride_i, x, y, ldy, kb, n, ld);
  return cudaGetLastError();
}
cudaError_t krylov_add_combination(const float* V, size_t vstride_i, double* x, const double* y, int ldy,
                                   const int* kb, int n, int ld, int B, cudaStream_t st) {
  k_add_combination<float><<<dim3(grid_x(n), B), 256, 0, st>>>(V, vstride_i, x, y, ldy, kb, n, ld);
  return cudaGetLastError();
}

cudaError_t krylov_scale(const double* a, const double* scale, double* out, int n, int ld, int B, cudaStream_t st,
                         float* out32, double* out2) {
  k_scale<<<dim3(grid_x(n), B), 256, 0, st>>>(a, scale, out, n, ld, out32, out2);
  return cudaGetLastError();
}
cudaError_t krylov_scale(const double* a, const double* scale, float* out, int n, int ld, int B, cudaStream_t st,
                         float* out32, double* out2) {
  k_scale_to32<<<dim3(grid_x(n), B), 256, 0, st>>>(a, scale, out, n, ld, out32, out2);
  return cudaGetLastError();
}

cudaError_t krylov_widen(const float* in, double* out, size_t n, cudaStream_t st) {
  k_widen<<<grid_x((int)(n > (1u << 30) ? (1u << 30) : n)), 256, 0, st>>>(in, out, n);
  return cudaGetLastError();
}

cudaError_t krylov_sub(const double* a, const double* b, double* out, size_t n, cudaStream_t st) {
  k_sub<<<grid_x((int)(n > (1u << 30) ? (1u << 30) : n)), 256, 0, st>>>(a, b, out, n);
  return cudaGetLastError();
}

cudaError_t krylov_masked_sub(double* X, const double* dx, const int* mask, int n, int ldx, int ld, int B,
                              cudaStream_t st) {
  k_masked_sub<<<dim3(grid_x(n), B), 256, 0, st>>>(X, dx, mask, n, ldx, ld);
  return cudaGetLastError();
}

cudaError_t krylov_cycle_start(const GmresState& s, const double* nrm2, int B, cudaStream_t st) {
  k_cycle_start<<<(B + 63) / 64, 64, 0, st>>>(s, nrm2, B);
  return cudaGetLastError();
}

cudaError_t krylov_arnoldi_finish(const GmresState& s, const double* nrm2, int j, int B, cudaStream_t st) {
  if (s.m > kMaxRestart || j >= s.m) return cudaErrorInvalidValue;
  k_arnoldi_finish<<<B, 32, 0, st>>>(s, nrm2, j, B);
  return cudaGetLastError();
}

constexpr int kOrthStage = 160 * 1024;                 // bytes of V's slice in shared memory at most

static cudaLaunchConfig_t orth_config(int B, size_t smem, cudaLaunchAttribute* at, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kOrthCtas, B);
  cfg.blockDim = dim3(kDotThreads + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = kOrthCtas;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}
// Clusters of 16 CTAs are above the portable 8: whether this device takes them (asked once).
template <typename VT, bool STAGE>
static bool orth_fits() {
  cudaLaunchAttribute at = {};
  const size_t smem = STAGE ? kOrthStage : 0;
  const cudaLaunchConfig_t cfg = orth_config(1, smem, &at, nullptr);
  const auto k = k_orth<VT, STAGE>;
  int n = 0;
  const bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess &&
                  cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n > 0;
  if (!ok) cudaGetLastError();
  return ok;
}
bool krylov_orth_takes(int n, bool basis32) {
  if (n > (basis32 ? kOrthMax : kOrthMax / 4 * 3)) return false;
  static std::atomic<int> state[64][2];                // per device and basis: 0 not asked, 1 yes, 2 no
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  std::atomic<int>& q = state[dev & 63][basis32];
  if (q.load() == 0)
    q.store((basis32 ? orth_fits<float, false>() && orth_fits<float, true>()
                     : orth_fits<double, false>() && orth_fits<double, true>()) ? 1 : 2);
  return q.load() == 1;
}

template <typename VT>
static cudaError_t krylov_orth_t(const VT* V, size_t vstride_i, const double* w, int n, int ld, int j, int B,
                                 const GmresState& s, double eta, VT* out, float* out32, double* out2, int* flags,
                                 cudaStream_t st) {
  if (n > kOrthMax || s.m > kMaxRestart || j >= s.m) return cudaErrorInvalidValue;
  const int ne = (n + kOrthCtas * 32 - 1) / (kOrthCtas * 32) * 32;
  const size_t slice = (size_t)(j + 1) * ne * sizeof(VT);
  const bool stage = slice <= kOrthStage;
  cudaLaunchAttribute at = {};
  const cudaLaunchConfig_t cfg = orth_config(B, stage ? slice : 0, &at, st);
  return cudaLaunchKernelEx(&cfg, stage ? k_orth<VT, true> : k_orth<VT, false>, V, vstride_i, w, n, ld, j, s, eta * eta,
                            out, out32, out2, flags);
}
cudaError_t krylov_orth(const double* V, size_t vstride_i, const double* w, int n, int ld, int j, int B,
                        const GmresState& s, double eta, double* out, float* out32, double* out2, int* flags,
                        cudaStream_t st) {
  return krylov_orth_t(V, vstride_i, w, n, ld, j, B, s, eta, out, out32, out2, flags, st);
}
cudaError_t krylov_orth(const float* V, size_t vstride_i, const double* w, int n, int ld, int j, int B,
                        const GmresState& s, double eta, float* out, float* out32, double* out2, int* flags,
                        cudaStream_t st) {
  return krylov_orth_t(V, vstride_i, w, n, ld, j, B, s, eta, out, out32, out2, flags, st);
}

cudaError_t contin_grk_T(const double* X, int ldx, double* g, int M, int nr, const double* gr, double dtPr, int sym,
                         int B, cudaStream_t st) {
  k_grk_T<<<dim3(grid_x(3 * M * nr), B), 256, 0, st>>>(X, ldx, g, M, nr, gr, dtPr, sym);
  return cudaGetLastError();
}

cudaError_t contin_border(const double* v, double* out, int n, int ld, const double* Jmu, int ldj, int Npsi,
                          const double* dot, const double* mudot, double delta, int B, cudaStream_t st) {
  k_border<<<dim3(grid_x(Npsi), B), 256, 0, st>>>(v, out, n, ld, Jmu, ldj, Npsi, dot, mudot, delta);
  return cudaGetLastError();
}

cudaError_t krylov_copy_scaled(const double* src, int lds, double* dst, int ldd, int n, double a, const double* last,
                               int B, cudaStream_t st) {
  k_copy_scaled<<<dim3(grid_x(n), B), 256, 0, st>>>(src, lds, dst, ldd, n, a, last);
  return cudaGetLastError();
}

cudaError_t krylov_axpy_shell(const double* x0, int ldx0, const double* d, int ldd, const double* c, double* y,
                              int ldy, int n, int B, cudaStream_t st) {
  k_axpy_shell<<<dim3(grid_x(n), B), 256, 0, st>>>(x0, ldx0, d, ldd, c, y, ldy, n);
  return cudaGetLastError();
}

cudaError_t krylov_solve_y(const GmresState& s, int B, cudaStream_t st) {
  if (s.m > kMaxRestart) return cudaErrorInvalidValue;
  k_solve_y<<<B, 32, (size_t)s.m * s.m * sizeof(double), st>>>(s);   // (at most 32 KB)
  return cudaGetLastError();
}

}  // namespace sdd
