// Per-step diagnostics of _Time_Step (Main.py:285-296): the 2-norm of the state, the volume-averaged
// kinetic energy (Kinetic_Energy, Main.py:71-134) and the Nusselt numbers of T and S (Nusselt,
// Main.py:41-68), on the device.
//
// Kinetic energy.  With JPSI = J_theta_RT(psi) (Matrix_Operators.py:437), the reference forms for every
// interior radius r_n the cosine row JPSI_k(r_n)/r_n and the sine row (Dr psi_k)(r_n) (shifted to the
// sinusoid convention), transforms both to the 3 N_fm midpoint grid (IDCT / IDST with n = 3 N_fm) and
// integrates |.|^2 by the trapezoidal rule over r (x = R interior) and then over theta with sin(theta).
// Both rules are weighted sums, so KE = (1/2V) sum_n wr_n sum_i wt_i sin(theta_i) (J^2 + D^2)(r_n, theta_i):
// a CTA computes the inner sum of one radius (the two transforms ride in one complex FFT of length 3 N_fm, in
// fixed point like the other FP64 transforms) and the last one of a shell the outer sums.
//
// Nusselt.  Nu - 1 at r = R[0] is (R[0]^2/A_T) sum_{k even} (D TT_k)[0]/(1 - k^2), TT_k the zero-padded
// radial profile of mode k: a fixed weighted sum of the even-mode coefficients (weights from the plan).
#include <cuda_runtime.h>

#include "sdd_fft.cuh"
#include "sdd_rowops.cuh"
#include "sdd_internal.cuh"

namespace sdd {

size_t diag_rows_smem_bytes(int M, int L) {
  return (4 * (size_t)L * 2 + 5 * (size_t)M + 8) * sizeof(double) + 4 * 32 * 8;
}

// One CTA per (interior radius n, shell): the inner kinetic-energy sum of its radius, and a slice of the sums over the
// state (|X|^2, Nu_T, Nu_S); the shell's last CTA adds the partial sums in order.  (As a kernel of one CTA a shell
// the outer sums took longer than the rows: 12.0 + 17.5 us at 90 x 23, now 15 us, most of it the latency of the
// transform's passes and of a few dozen dependent FP64 operations.)
// Two CTAs an SM (128 registers): of the 196 that the widest pass takes unbounded one CTA fits, and batches, whose small
// CTAs wait at their barriers, took longer than with FP64 transforms.  us a call, FP64 / 196 / 128 registers: 12 x 65, 64
// shells 152 / 234 / 129, 24 x 34 78 / 118 / 65, 64 x 20 56 / 72 / 42, one shell 21 / 12 / 11; 90 x 23 29 / 13.3 / 13.0.
__global__ void __launch_bounds__(256, 2) k_diag(DiagArgs a) {
  using C = longlong2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int M = a.M, nr = a.nr, L = a.L;
  const int n = blockIdx.x, b = blockIdx.y;
  const int tid = threadIdx.x, bd = blockDim.x;
  C* RA = reinterpret_cast<C*>(smem_raw);
  C* RB = RA + L;
  int4* Wt = reinterpret_cast<int4*>(RB + L);
  int4* Et = Wt + L;
  double* pv = reinterpret_cast<double*>(Et + L);
  double* Sc = pv + M;
  double* dp = Sc + M;
  double* Ar = dp + M;        // cosine row: J_theta_RT(psi)_k(r_n) / r_n
  double* Br = Ar + M;        // sine row: (Dr psi)_{k-1}(r_n), [0] = 0
  double* scl = Br + M;       // the two rows' exponents
  unsigned* red = reinterpret_cast<unsigned*>(scl + 8);
#pragma unroll 1
  for (int i = tid; i < L; i += bd) {
    cp_async16(Wt + i, a.w + i);
    cp_async16(Et + i, a.e + i);
  }
  cp_async_commit();
  after_previous_kernel();                             // (the tables are the plan's)
  const double* ps = a.X + (size_t)b * a.x_stride;
#pragma unroll 1
  for (int k = tid; k < M; k += bd) pv[k] = (a.sym && (k % 2 == 0)) ? 0.0 : ps[(size_t)k * nr + n];
  // the slice of the state's sums: 3 M elements, (M + 1) / 2 Nusselt weights
  double v[4] = {0.0, 0.0, 0.0, 0.0};                  // |X|^2, KE, NuT, NuS
  {
    const size_t N = (size_t)M * nr;
    const double* xs = ps + (size_t)n * 3 * M;
#pragma unroll 4
    for (int q = tid; q < 3 * M; q += bd) v[0] = fma(xs[q], xs[q], v[0]);
    const int ne = (M + 1) / 2;
    for (int q = tid; q < ne; q += bd) {
      const int e = n * ne + q, kk = e / nr, m = e - kk * nr;
      const size_t o = (size_t)(2 * kk) * nr + m;
      const double w = a.nuw[e];
      v[2] = fma(w, ps[N + o], v[2]);
      v[3] = fma(w, ps[2 * N + o], v[3]);
    }
  }
  const double* drn = a.Dr + (size_t)n * nr;
  const int half = (nr + 1) / 2;
#pragma unroll 1
  for (int i = tid; i < (2 * M + 31) / 32 * 32; i += bd) {   // two lanes a mode (whole warps)
    const int k = min(i >> 1, M - 1), m0 = (i & 1) * half, m1 = min(nr, m0 + half);
    const double* pk = ps + (size_t)k * nr;
    double acc = 0.0;
#pragma unroll 8
    for (int m = m0; m < m1; ++m) acc = fma(__ldg(drn + m), pk[m], acc);
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    if (i < 2 * M && (i & 1) == 0) dp[k] = acc;
  }
  __syncthreads();
  parity_suffix<double>(pv, Sc, M);   // as J_theta_RT
  __syncthreads();
  const double irn = a.ir[n], wrn = a.wr[n];
#pragma unroll 1
  for (int k = tid; k < M; k += bd) {
    const double s1 = (k + 1 < M) ? Sc[k + 1] : 0.0;
    double jp = (k == 0) ? 1.0 * s1 : (k + 1.0) * pv[k - 1] + 2.0 * s1;
    if (a.sym && (k % 2 == 1)) jp = 0.0;
    Ar[k] = irn * jp;
    Br[k] = k >= 1 ? dp[k - 1] : 0.0;
  }
  cp_async_wait<0>();                                  // the twiddles
  __syncthreads();
  // DCT3 inputs with n_in = M on length L (see k_transform): cosine x_k = A_k; sine x_k = B_{L-k}
  double* XV = reinterpret_cast<double*>(RB);
#pragma unroll 1
  for (int k = tid; k < L; k += bd) {
    const double xa = (k < M) ? Ar[k] : 0.0;
    const double xb = (L - k <= M - 1 && k > 0) ? Br[L - k] : 0.0;
    XV[k] = xa;
    XV[L + k] = xb;
  }
  int* E = reinterpret_cast<int*>(scl);
  rows_to_fixed(XV, L, 2, red, E);
  const i64* XA = reinterpret_cast<const i64*>(XV);
  const i64* XB = XA + L;
#pragma unroll 1
  for (int k = tid; k < L; k += bd)
    RA[k] = k == 0 ? make_longlong2(XB[0], XA[0]) : dct3_pack_fx(Et[k], XA[k], XA[L - k], XB[k], XB[L - k]);
  __syncthreads();
  C* res = fft_rows<double, false>(RA, RB, 1, a.st, Wt);
  next_kernel_may_start();
  const bool bad = E[0] == kFxBad || E[1] == kFxBad;
  double ke = 0.0;
#pragma unroll 2
  for (int i = tid; i < L; i += bd) {
    const int src = (i & 1) ? (L - 1 - (i >> 1)) : (i >> 1);
    const C c = res[src];
    const double ja = bad ? fx_nan() : fx2d(c.y, 60 - E[0]), db = fx2d(c.x, 60 - E[1]);   // (db's sign drops out)
    ke = fma(a.tw[i], fma(ja, ja, db * db), ke);
  }
  v[1] = wrn * ke;
  const int lane = tid & 31, warp = tid >> 5;
  const double t4 = warp_sum4(v, lane);
  double* rd = reinterpret_cast<double*>(red);
  __syncthreads();                      // (the exponents are read before the sums reuse the reduction words)
  if ((lane & 7) == 0) rd[(lane >> 3) * 8 + warp] = t4;
  __syncthreads();
  __shared__ int s_last;
  if (warp == 0) {                      // lane 8 q + w: warp w's sum of value q
    double t = rd[lane];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((lane & 7) == 0) a.part[((size_t)b * nr + n) * 4 + (lane >> 3)] = t;
    __threadfence();
    __syncwarp();
    if (lane == 0) {
      int* cnt = a.ticket + (size_t)b * 6 + 5;
      const int last = atomicAdd(cnt, 1) == nr - 1;
      if (last) *cnt = 0;               // ready for the next launch
      s_last = last;
    }
  }
  __syncthreads();
  if (!s_last || warp >= 4) return;
  __threadfence();
  // warp q adds value q over the radii
  const double* p = a.part + (size_t)b * nr * 4 + warp;
  double t = lane < nr ? __ldcg(p + 4 * lane) : 0.0;
  if (lane + 32 < nr) t += __ldcg(p + 4 * (lane + 32));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) a.out[(size_t)b * 4 + warp] = warp == 0 ? sqrt(t) : (warp == 1 ? a.ke_scale * t : t);
}

cudaError_t launch_diag(const DiagArgs& a, int batch, cudaStream_t s) {
  static unsigned long long done = 0;
  const cudaError_t e = ensure_smem_attr(k_diag, &done);
  if (e != cudaSuccess) return e;
  return launch_kernel(k_diag, dim3(a.nr, batch), dim3(256), diag_rows_smem_bytes(a.M, a.L), s, a);
}

}  // namespace sdd
