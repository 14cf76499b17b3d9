// Internal declarations shared by the CUDA translation units of libsdd_gb300.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>

#include "../../include/sdd_gb300.h"
#include "sdd_fixed.cuh"

namespace sdd {

constexpr int kMaxStages = 16;   // FFT stages (radices) per length
constexpr int kMaxRadix = 7;     // largest radix handled by the butterflies (2,3,4,5,7)
constexpr int kMaxNr = 64;       // interior radial points supported by the chain kernel
constexpr int kMaxM = 1024;      // theta modes supported
constexpr int kFxThreads = 256;  // threads of the rhs / theta / transform row kernels
constexpr int kFxRowThreads = 512;  // threads of the nonlinear-term row kernel

void set_cuda_error(cudaError_t e);

// Kernel launch through cudaLaunchKernelEx with the launch error returned, as a programmatic dependent of the kernel
// before it in the stream: it is launched once every CTA of that kernel has ended or called next_kernel_may_start().
// EVERY kernel launched this way calls after_previous_kernel(), which waits for the completion (and the writes) of all
// kernels before it, ahead of anything it reads that a kernel writes and of every write to global memory.  Before it
// stand only loads of the plan's tables (operators, twiddles, blocks, chain scalars: written and synchronised when the
// plan or its chunk tables are made).  The kernel is resident while the one before it still writes, so only those tables
// go through __ldg: a read-only load promises that its data do not change during the whole kernel, and the compiler may
// move it across the wait.  Everything that a kernel writes (states, derivatives, right-hand sides, products) is read by
// plain loads after the wait.  Dependents hide most of a launch's latency: single steps of 64 x 20 47.5 -> 31
// us, 256 x 30 62.8 -> 46.5, 64 shells 618 -> 606; inside the captured step graphs 44.6 -> 43.4.
// next_kernel_may_start() stands where a kernel's last phase begins: the next kernel's CTAs come up and load their
// tables beside it (us a step: 256 x 30 43.5 -> 41.5, 540 x 65 146 -> 139, 3 shells of 128 x 28 mixed 44.4 -> 41.7, 90 x
// 23 with diagnostics 50 -> 45; the tables ahead of the wait alone 42.9, 145, 44.3, 50).  Before the transforms
// instead of after them it is slower (42.1, 140, 42.8), at a kernel's start far slower (256 x 30 50, 64 shells 606 ->
// 667): the CTAs that wait then take the room where the next kernel's others would spread over the SMs.
#ifdef __CUDACC__
__device__ __forceinline__ void after_previous_kernel() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_kernel_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                 Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Per-kernel timing for sdd_step_kernel_profile: while a KernelTimer is installed on the calling thread,
// every launcher records an event after each launch, tagged with the kernel's id (SDD_K_* in the public
// header).  Off (one thread-local load per launch) otherwise, and always off during graph capture.
struct KernelTimer {
  static constexpr int kMax = 64;
  cudaEvent_t ev[kMax];
  int id[kMax];
  int n;
};
extern thread_local KernelTimer* g_ktimer;
inline void ktimer_mark(int id, cudaStream_t s) {
  KernelTimer* t = g_ktimer;
  if (t && t->n < KernelTimer::kMax && cudaEventRecord(t->ev[t->n], s) == cudaSuccess) t->id[t->n++] = id;
}

// Raises a kernel's dynamic shared-memory limit to the device's opt-in maximum once per device, so
// launches do not pay a cudaFuncSetAttribute call each.  max_carveout: also prefer the largest
// shared-memory share of the L1/shared storage, for kernels whose many CTAs must be resident at once.
template <typename F>
inline cudaError_t ensure_smem_attr(F* fn, unsigned long long* done_mask, bool max_carveout = false) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (__atomic_load_n(done_mask, __ATOMIC_ACQUIRE) & bit) return cudaSuccess;
  int optin = 0;
  e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(fn));
  if (e != cudaSuccess) return e;
  // the dynamic limit may not exceed the opt-in maximum less the kernel's static shared memory
  e = cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           optin - (int)fa.sharedSizeBytes);
  if (e == cudaSuccess && max_carveout)
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) __atomic_fetch_or(done_mask, bit, __ATOMIC_ACQ_REL);
  return e;
}

// Twiddle tables and radix plan of one complex FFT length L (used for DCT-II/III of length L).
struct FftPlan {
  int L = 0;
  int nst = 0;
  int rad[kMaxStages] = {0};
  int4* wfx = nullptr;      // exp(-2 pi i k / L), k < L, in 32-bit digits (re hi, lo, im hi, lo) of 2^62
  int4* efx = nullptr;      // 0.5 exp(+i pi k / (2L)), k < L, the same
  float2* w32 = nullptr;
  float2* e32 = nullptr;
};

// Returns a cached device FFT plan for length L (nullptr if L has a prime factor > kMaxRadix).
const FftPlan* get_fft_plan(int L);

// Kernel argument blocks -----------------------------------------------------------------------

// Division of n < 2^31 by an invariant d >= 1 with one multiply-high and a shift (Granlund and Montgomery,
// "Division by invariant integers using multiplication", 1994): with l = ceil(log2 d) and p = 31 + l,
// m = ceil(2^p / d) < 2^32 and floor(n / d) = floor(n m / 2^p), because m d - 2^p < d <= 2^l and
// n < 2^31 keep the error below one.  m = 0 encodes d = 1.
struct FastDiv {
  unsigned m;
  int s;                     // p - 32
};
inline FastDiv make_fastdiv(unsigned d) {
  if (d <= 1) return FastDiv{0u, 0};
  int l = 0;
  while ((1ull << l) < d) ++l;
  const int p = 31 + l;
  return FastDiv{(unsigned)(((1ull << p) + d - 1) / d), p - 32};
}
__device__ __forceinline__ unsigned fast_div(unsigned n, FastDiv f) { return f.m ? (__umulhi(n, f.m) >> f.s) : n; }

struct StageArgs {           // radices passed by value, with each stage's divisors precomputed
  int L, nst;
  int rad[kMaxStages];
  int tws[kMaxStages];       // twiddle stride L / (Ns R) of the stage
  FastDiv nb[kMaxStages];    // division by L / R (butterflies per transform)
  FastDiv ns[kMaxStages];    // division by Ns (product of the earlier radices)
};

inline StageArgs stage_args(const FftPlan* fp) {
  StageArgs st{};
  st.L = fp->L;
  st.nst = fp->nst;
  int Ns = 1;
  for (int i = 0; i < kMaxStages; ++i) {
    st.rad[i] = fp->rad[i];
    if (i < fp->nst) {
      const int R = fp->rad[i];
      st.tws[i] = fp->L / (Ns * R);
      st.nb[i] = make_fastdiv((unsigned)(fp->L / R));
      st.ns[i] = make_fastdiv((unsigned)Ns);
      Ns *= R;
    }
  }
  return st;
}

struct FxOps {               // FP64 or FP32 copies of the operators the nonlinear term needs
  const void* Dr;            // nr*nr
  const void* D2r2;          // nr*nr
  const void* ir4r2;         // nr
  const i64* fxDr;           // Dr as a two-digit block, D^2/r^2 and A2_SINE's D2 as three-digit blocks
  const int* wx[2];          // (sdd_fixed.cuh)
  const void* w;             // FFT twiddles (P): FP32 complex, or fixed-point digits (FP64)
  const void* e;             // DCT twiddles (P), the same
};

struct RhsArgs {
  int M, nr, sym, linear;
  double dt, Pr;
  const double* Dr;          // nr*nr
  const double* D2s;         // nr*nr (A2_SINE)
  const double* ir2s, *rsq, *dT0, *gr;
  const double* X;           // state (or perturbation) the linear terms act on
  size_t x_stride;
  const double* out4;        // FX spectral outputs (ignored when linear)
  size_t out_stride;
  const double* Ra, *Ra_s;   // per shell
  double* rhs;               // [shell][3][M][nr]
  size_t rhs_stride;
  // mixed plans: Q (out4's first block) also in FP32, [shell][M][nr]; then Dr Q is an FP32 contraction
  // (part of the FP32 nonlinear term) with Dr32, converted to FP64 once
  const float* q32;
  const float* Dr32;
  const int* active;         // nullable: per-shell flags; kernels skip shells whose flag is 0
  // FP32 right-hand sides (Jacobian products of Newton solves whose GMRES tolerance is far above FP32
  // rounding): k_rhs32 reads the FP32 copy X32 of X and writes rhs32 [shell][3][M][nr] instead of rhs
  const float* X32;
  size_t x32_stride;         // floats between shells in X32
  float* rhs32;
  const float* D2s32;        // nr*nr (A2_SINE) in FP32
  // Crank-Nicolson / Adams-Bashforth 2 (cnab2 != 0; the plan's operators are those of dt/2, dt above is
  // the full step): rhs = 2 lin + dt (3/2 E - 1/2 E_prev) with E the explicit terms per unit time
  // (psi: -(Dr Q - R) + Pr gr_k(Ra T - Ra_s S); T/S: -N - psi_T0), lin = A2_SINE(psi), r^2 T, r^2 S.
  // hist [shell][3][M][nr] (stride rhs_stride) holds E_prev on entry when hist_valid (else the explicit
  // part is Euler, dt E) and E of this step on exit.
  int cnab2;
  int hist_valid;
  double* hist;
};

// A chunk correction of the state left pending by the previous time step (layouts 3 / 11, sdd_step): the split
// nonlinear term's k_fx_deriv applies X[jj] += G_jj s_c(jj) to its mode before using it, with the
// arithmetic of k_mode_mv (the same bits), and writes the corrected rows back (and their FP32
// copy).  The previous step's chunk end states and carry products are still in dbuf / pbuf: this step's
// chains overwrite them only after the nonlinear term.
struct FixArgs {
  int on;
  int kc, nch, np, ldd, ldl;
  const i64* GA4, *GT, *GS;
  const double* dbuf, *pbuf;
  size_t d_stride, p_stride;
  double* X;                 // the state being corrected in place (the nonlinear term's input)
  float* X32;                // nullable: its FP32 copy
};

struct FxArgs {
  int M, nr, P, sym;
  StageArgs st;
  FxOps ops;
  const double* X;           // state whose nonlinear term (FX) or perturbation (DFX) is formed
  size_t x_stride;           // doubles between shells in X
  const float* X32;          // nullable: X rounded to FP32, read by the FP32 kernels instead of converting X
  size_t x32_stride;         // floats between shells in X32
  float* q32;                // nullable (FP32 kernels): Q also written in FP32, [shell][M][nr]
  const int* active;         // nullable: per-shell flags; kernels skip shells whose flag is 0 (their
                             // outputs are left as they were: Krylov solves mask those shells out)
  void* base;                // base-state grid cache [shell][nr][9][P] (T precision), nullable
  size_t base_stride;        // elements between shells in base
  double* out4;              // [shell][4][M][nr] : Qhat, Rhat, NJ_T hat, NJ_S hat
  size_t out_stride;         // doubles between shells in out4
  size_t fx_stride;
  void* grid;                // nullable: grid-field scratch [shell][nr][9][P] (T precision) of the split path
  size_t grid_stride;        // elements between shells in grid
  int split;                 // 0 auto, 1 fused row kernel, 2 split (needs grid or a cache)
  void* deriv;               // split path: radial derivatives [shell][5][M][nr] (T): Dr psi, D2r2 psi, Dr T, Dr S
                             // (and, with fuse_rhs, D2s psi in FP64 as the fifth block)
  size_t deriv_stride;       // elements between shells in deriv
  // fuse_rhs: the right-hand sides' linear parts (the terms of Main.py:262-280 that do not involve the nonlinear term)
  // are written into rl.rhs, by k_fx_grid (split path) or k_rhs_lin; the chains' h kernel adds the nonlinear
  // parts from out4.  rl carries the operators, parameters and the rhs buffer; deriv's fifth block the FP64
  // D2 psi that they need.
  int fuse_rhs;
  RhsArgs rl;
  FixArgs fix;               // split path: a pending correction of X (see FixArgs)
  // mixed plans: the FP32 radial contractions on the tensor cores (k_deriv_tc, 3xTF32).  tcB: the plan's
  // split operator tiles (nullable: CUDA-core FP32 contractions); tcKP / tcNP: nr rounded up to 8.  When
  // they are used, deriv's four FP32 blocks hold the transposed layout [op][n][k] (deriv_t, set by
  // launch_fx) and the row kernels read them instead of contracting.
  const float* tcB;
  int tcKP, tcNP;
  int* tc_err;               // nullable: set by a tensor-core kernel whose wait timed out
  int deriv_t;
};

// k_deriv_tc: the four radial contractions of Derivatives for every state row of a batch, 3xTF32 on the
// tensor cores, into out[shell][op][n][k] (op 0 Dr psi, 1 (D^2/r^2) psi, 2 Dr T, 3 Dr S; FP32).
struct TcArgs {
  int M, nr, sym, KP, NP;
  int rows;                  // batch * 3 * M state rows
  const float* X32;          // the state in FP32 (nullable: X is converted)
  size_t x32_stride;
  const double* X;
  size_t x_stride;
  const int* active;         // nullable: per-shell flags; rows of shells whose flag is 0 are skipped
  const float* B;            // [hi | lo] operator tiles (build_tc_operator), 16-byte aligned
  float* out;
  size_t out_stride;         // floats between shells in out
  int* err;                  // nullable: set to 1 when a wait for the tensor cores timed out
};



// Tables of one chunking of the chains (see k_chain_fx): chunk length kc, nch chunks per chain, the
// corrections G_jj of every mode and the carried-state maps, either per chunk (Phi_c, the sequential
// carry of layout 2) or as the products P_{j,i} = Phi_{j-1} ... Phi_{i+1}, i <= j - 2 (np per chain,
// row j after row j-1; the parallel carry of layout 3).
struct ChunkSet {
  int kc, nch, np;
  const i64* GA4, *GT, *GS;           // G_jj: [M][2] blocks (psi: f_e, bf_e half), [M] blocks (T, S)
  const i64* PhiA4, *PhiT, *PhiS;     // Phi_c: [2 parity][nch] x 4 blocks (row half, operand half) or 1
  const i64* PA4, *PT, *PS;           // P_{j,i}: [2 parity][np] x 4 blocks or 1
};

struct ChainArgs {
  int M, nr, ldl, sym;
  int field0;                // first field handled (blockIdx.x/2 + field0)
  int layout;                // the requested layout (0 automatic; resolve_chain_layout)
  int type0, fmask;          // set by launch_chain: first chain type (0 psi, 1 T and S), fields to solve
  size_t field_off;          // doubles between field blocks (N_fm*nr, or 0 when g/f point at one block)
  const double* g;           // rhs [shell][3][M][nr]
  size_t g_stride;
  double* f;                 // solution [shell][3][M][nr]
  size_t f_stride;
  float* f32;                // nullable: the final solution also rounded to FP32 (the next mixed step's X32)
  size_t f32_stride;
  const double* sub;         // nullable: f -= sub (Newton residual), same layout
  size_t sub_stride;
  // fixed-point blocks (sdd_fixed.cuh): Linv of every mode, and the psi step matrices [A_j B_j] as two
  const i64* LinvA4, *LinvT, *LinvS, *ABA4;
  double* h;                 // [shell][3][M][nr] h = Linv g
  size_t h_stride;           // doubles between shells in h
  const double* coefA4;      // [M][4] per jj: (dt bjt, dt bjt bj, bj, bjt), dt = Pr*dt, j = M - jj
  const double* coefT, *coefS;  // [M][4] per jj: (2 dt (j+2), 0.5 if j == 0 else 1, 0, 0), j = M-1-jj
  // fuse_rhs: g is not read; the h kernel forms g from the linear parts in `lin` and the nonlinear-term
  // outputs in out4 (psi: -dt (Dr Q - R) + lin; T, S: -dt N + lin)
  int fuse_rhs;
  const double* lin;         // [shell][3][M][nr] linear parts (k_fx_grid), stride g_stride
  const double* out4;        // [shell][4][M][nr]
  size_t out_stride;
  const int* wxDr;           // Dr as a three-digit block (sdd_fixed.cuh)
  const float* q32, *Dr32;   // mixed plans: Dr Q in FP32 (see RhsArgs)
  int split_fx;              // the nonlinear term runs split over CTAs (one small batch): resolve_chain_layout
  double dt;                 // the step's dt
  // chunked (parallel-in-modes) chains, layout 2: every chain of S = N_fm/2 steps is cut into nch chunks
  // of kc steps.  Chunk c runs from a zero carried state (f_local, end state d_c); the carried states
  // s_c at the chunk starts follow s_{c+1} = Phi_c s_c + d_c; then f += G_jj s_c for the chunk's modes.
  int kc, nch;               // chunk length (steps) and chunks per chain
  int ldd;                   // doubles per (field, parity, chunk) slot of dbuf / cbuf (>= 2 nr, even)
  const i64* GA4, *GT, *GS;           // G_jj: [M][2] blocks (psi: f_e, bf_e half), [M] blocks (T, S)
  const i64* PhiA4, *PhiT, *PhiS;     // Phi_c: [2 parity][nch] x 4 blocks (row half, operand half) or 1
  double* dbuf;              // [shell][3][2][nch][ldd] chunk end states from a zero start
  double* cbuf;              // [shell][3][2][nch][ldd] carried states at the chunk starts (c >= 1)
  size_t d_stride;           // doubles per shell in dbuf / cbuf
  int* counter;              // [shell][6] chunks finished per chain (the last one runs the carry), zeroed
  // layouts 3 / 11 (parallel carry): the chunks only write their end states; k_carry_fx forms
  // part_{j,i} = P_{j,i} d_i for every product in parallel and the corrections sum
  // s_j = d_{j-1} + sum_i part_{j,i} (index order)
  int carry_seq;             // 1: the last-finishing chunk CTA runs the sequential carry (layouts 2 / 10)
  int np;                    // products per chain
  const i64* PA4, *PT, *PS;
  double* pbuf;              // [shell][6][np][ldd] products P_{j,i} d_i
  size_t p_stride;           // doubles per shell in pbuf
  ChunkSet cset[2];          // the chunkings of layouts 2 and 3 (launch_chain copies one into the fields above)
  int defer_fix;             // layouts 3 / 11: leave the correction to the next step's nonlinear term (FixArgs)
  const int* active;         // nullable: per-shell flags; kernels skip shells whose flag is 0
  // nullable: FP32 right-hand sides (k_rhs32, stride g_stride): h = Linv g is then formed in FP32 with the
  // FP32 copies of the Linv blocks (k_mode_mv32) and stored in FP64 for the chains
  const float* g32;
  const float* Linv32A4, *Linv32T, *Linv32S;
};

struct DiagArgs {
  int M, nr, sym, L;         // L = 3 M: the kinetic-energy grid
  StageArgs st;              // FFT of length L
  const int4* w;             // FFT twiddles of length L (fixed-point digits)
  const int4* e;             // DCT twiddles of length L
  const double* Dr;          // nr*nr interior D
  const double* ir;          // nr  1/R interior
  const double* tw;          // L   trapezoid weight * sin(theta_i) on the L-point midpoint grid
  const double* wr;          // nr  trapezoid weights over the interior radii
  const double* nuw;         // ceil(M/2)*nr  Nusselt weights of the even modes
  double ke_scale;           // 1/(2V), V = (2/3)(r_o^3 - r_i^3)
  const double* X;           // states [shell][3][M][nr]
  size_t x_stride;
  double* part;              // [shell][nr][4] partial sums of |X|^2, KE, Nu_T, Nu_S
  int* ticket;               // six counters a shell of which the last one counts its CTAs (zero between launches)
  double* out;               // [shell][4]
};

// launchers (return cudaError_t of the launch)
cudaError_t launch_diag(const DiagArgs& a, int batch, cudaStream_t s);
size_t diag_rows_smem_bytes(int M, int L);
cudaError_t launch_fx(const FxArgs& a, int batch, int mode, int prec, cudaStream_t s);
cudaError_t launch_deriv_tc(const TcArgs& a, cudaStream_t s);
size_t tc_smem_bytes(int KP, int NP);
// [hi | lo] tiles of B = [Dr ; D^2/r^2] (2 NP rows of KP) in the tensor cores' canonical shared-memory
// layout: 2 * 2 NP * KP floats
void build_tc_operator(const double* Dr, const double* D2r2, int nr, int KP, int NP, float* out);
// whether launch_fx takes the split path for these arguments
bool fx_uses_split(const FxArgs& a, int batch, int mode);
// the largest dynamic shared memory a k_fx_rows launch of this precision can take on the current device
size_t fx_rows_max_dynamic_smem(int prec);
// the split-or-fused rule alone (split: 0 automatic, 1 fused, 2 split), for a plan whose scratch is not yet
// reserved
bool fx_split_rule(int split, int nr, int batch);
cudaError_t launch_rhs(const RhsArgs& a, int batch, cudaStream_t s);
// the linear parts alone, with D2 psi formed ([shell][M][nr], stride d2_stride)
cudaError_t launch_rhs_lin(const RhsArgs& a, const double* d2psi, size_t d2_stride, int batch, cudaStream_t s);
cudaError_t launch_chain(const ChainArgs& a, int batch, int nfields, cudaStream_t s);
// the chain layout launch_chain runs for a.layout (0 = automatic) and this launch size
int resolve_chain_layout(const ChainArgs& a, int batch, int nfields);
// fixed-point blocks from FP64 matrices on the device (setup)
cudaError_t launch_to_fixed(const double* src, size_t src_stride, int rs, int cs, int nrows, int r0, int c0, int nr,
                            int ldl, i64* out, size_t out_stride, int nblk, cudaStream_t s);
cudaError_t launch_to_wide(const double* src, int nr, int ld, int* out, cudaStream_t s);
cudaError_t launch_chunk_fix(const ChainArgs& a, int batch, int nfields, cudaStream_t s);
cudaError_t launch_theta_op(int op, int M, int nr, int sym, const double* D2, const double* ir,
                            const double* dT0, const double* g, double* f, int batch,
                            cudaStream_t s);
cudaError_t launch_transform(int kind, int rows, int n_in, int n_out, const FftPlan* fp,
                             const double* in, double* out, cudaStream_t s);
size_t fx_smem_bytes(int M, int P, int prec);

}  // namespace sdd
