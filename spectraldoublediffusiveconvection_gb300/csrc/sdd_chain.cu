// Mode-coupled implicit solves: the back-substitution chains of
//   A4_BSub_TSTEP_V2   (Matrix_Operators.py:1115-1194)  -- psi: (A^2 - dt Pr A^4) psi = g
//   NAB2_BSub_TSTEP_V2 (Matrix_Operators.py:1033-1086)  -- T, S: (r^2 - dt r^2 Lap) f = g
// In the sin/cos basis each operator couples mode j to j+2, j+4, ... so a solve is two sequential
// chains (one per mode parity) of N_fm/2 steps.
//
// Restructured for a short critical path (exact algebra):
//   h_j = Linv_j g_j for every mode first (k_mode_mv, all SMs in parallel, off the chains), then
//   psi:  f_j = h_j + A_j f_e + B_j bf_e,  A_j = Linv_j (dt bjt D2 + diag(alpha_j)),  B_j = Linv_j diag(beta_j),
//         alpha_j = dt bjt bj IR4 - bjt IR2,  beta_j = dt bjt IR4   (b_test of :1155, expanded)
//         f_e += f_j,  bf_e += bj f_j + bjt f_e   (:1153, :1159)
//   T, S: b += 2 dt (j+2) f_{j+2},  f_j = h_j - (j==0 ? 0.5 : 1) Linv_j b   (:1058-1083)
// so each chain step is ONE dependent matvec ([A_j B_j] over 2 nr columns, or Linv_j) plus three
// elementwise updates.
//
// Arithmetic.  An FP64 warp instruction holds its SM sub-partition for 64 cycles on GB300, and a chain is one
// dependent matvec after another, so with FP64 matvecs a chain step cost (columns per lane) x 64 cycles.  Every
// block matvec here runs in 64-bit fixed point (sdd_fixed.cuh): blocks as digits scaled per row by its
// 1-norm, the operand scaled by its largest entry to 61 bits, three IMAD.WIDE (13 to 15 cycles) a column instead
// of 64.  The carried states (f_e, bf_e, b) stay FP64; h, the matvec and its parts are summed in fixed point and
// rounded once.  Error of a matvec against extended precision: 1e-18 to 2e-17 of the result, FP64's 1e-16 to 5e-16
// (row by row: sdd_fixed.cuh).
// An operand with an infinity takes an FP64 path with the same blocks (fx_dot_slow); one with a NaN gives NaN.
//
// k_chain_fx: a CTA holds one parity's chains of psi (two groups of warps: one carries f_e and multiplies by
// A_j, the other bf_e and B_j; the halves meet in shared memory) or of T and S (a group each), one lane per
// row, for one shell or two (which then share the blocks' way through shared memory).  The next blocks stream
// in with cp.async; one barrier a step (nr > 32: two).
// Layouts:
//   whole chains (1, 4 to 9: one kernel, the numbers are kept for callers that select them);
//   chunked (2, 3, 10, 11): the S = N_fm/2 steps of a chain are cut into nch chunks of kc steps that
//     run concurrently, each from a zero carried state.  The chain's carried state s (psi: [f_e; bf_e], 2 nr;
//     T/S: b, nr) enters every later step linearly, so with the plan's precomputed Phi_c (state over a whole
//     chunk) and G_jj (state -> f_jj):
//       2, 10: s_1 = d_0,  s_{c+1} = Phi_c s_c + d_c   (by the chain's last-finishing chunk CTA)
//       3, 11: s_c = d_{c-1} + sum_{i<=c-2} P_{c,i} d_i, P_{c,i} = Phi_{c-1}...Phi_{i+1} precomputed,
//              every product at once (k_carry_fx), the row sums in the corrections
//       f_jj += G_jj s_c(jj)                    (k_mode_mv, all modes in parallel)
//     The critical path drops from S dependent steps to kc + (nch - 2) carried matvecs + one matvec
//     (2, 10), or kc steps + one product + one matvec (3, 11, shorter chunks).
#include <cuda_runtime.h>
#include <algorithm>
#include <type_traits>

#include "sdd_fixed.cuh"
#include "sdd_internal.cuh"

namespace sdd {

// Operand x of one row (ignored where !ok) published as digits for column exponent cx; returns the exponent of
// the warp's rows.
__device__ __forceinline__ int publish(double x, int cx, bool ok, int2* xs) {
  const int em = __reduce_max_sync(0xffffffffu, ok ? fx_key(x, cx) : -0x10000);
  if (ok) *xs = fx_digits(x, cx, em);
  return em;
}

// One block's product with a published operand, row r of the block (LD x LD, in shared memory): the columns
// [32 w, 32 w + 32) of each warp segment w carry their own exponent em[w].  Returns the value v 2^e.
template <int LD, int W>
__device__ __forceinline__ FxVal block_row(const i64* blk, int nr, int r, const int2* xs, const int* em) {
  const int2* A = reinterpret_cast<const int2*>(blk) + r;
  const int ea = fx_row_exp(blk, LD)[r];
  int worst = ea;                                      // kFxBad: a NaN (or such a row), kFxInf: an infinity
#pragma unroll
  for (int w = 0; w < W; ++w) worst = max(worst, em[w]);
  FxVal o;
  if constexpr (W == 1) {
    o.v = fx_dot<LD, LD>(A, xs);
    o.e = ea + em[0] - kFxMvExp;
  } else {
    const i64 v0 = fx_dot<(LD < 32 ? LD : 32), LD>(A, xs), v1 = fx_dot<(LD > 32 ? LD - 32 : 0), LD>(A + 32 * LD, xs + 32);
    const int mx = max(em[0], em[1]);
    o.v = fx_shr(v0, mx - em[0]) + fx_shr(v1, mx - em[1]);
    o.e = ea + mx - kFxMvExp;
  }
  if (worst >= kFxInf) {
    double d = worst == kFxBad ? fx_nan() : 0.0;
#pragma unroll
    for (int w = 0; w < W; ++w)
      if (worst == kFxInf) d += fx_dot_slow(blk, LD, r, xs, 32 * w, min(nr, 32 * (w + 1)), em[w]);
    o.v = __double_as_longlong(d);
    o.e = kFxBad;
  }
  return o;
}

__device__ __forceinline__ void copy_words(i64* dst, const i64* src, int words, int t, int nt) {
  for (int c = t; c < words / 2; c += nt) cp_async16(dst + 2 * c, src + 2 * c);
}
// barrier 1: the compute warps of a k_chain_fx CTA, without its loader
__device__ __forceinline__ void compute_sync(int nt) { asm volatile("bar.sync 1, %0;\n" ::"r"(nt) : "memory"); }

// The chains of psi (type 0) or of T and S (type 1) of one parity and `spc` shells: steps [s0, s1) of the
// S = (M - par + 1)/2 chain steps, all of them or (CHUNK) chunk blockIdx.z of a.kc steps from a zero carried
// state; its end state goes to dbuf (psi: [f_e; bf_e]; T/S: b + k_next f_last, the b the next chunk's first
// step uses).  a.h holds h = Linv g.  W = ceil(nr / 32) warps a group, LD = fx_ld(nr), D ring slots of the two
// groups' blocks, streamed in by one more warp (its copies would be a tenth of the chain warps' instructions).
// Step s: publish the operand (W = 1: inside the warp), the block's product, then (psi) the two groups swap
// their halves through shared memory; the one barrier that orders the swap also frees the slot of step s and
// makes the block of step s + 1 visible.  A step is bound by the latency of that sequence (about a dozen
// conversions, shared-memory round trips and three FP64 operations), not by its 3 LD IMAD.WIDE.
// N_r=30, N_theta=256 (FP64 matvecs before): 16.4 -> 12.3 us for one shell's chunks, 288 -> 125 us (and 41 us of
// h = Linv g, which the FP64 form for batches did without) for 64 shells' whole chains.
template <int LD, bool CHUNK, int D>
__global__ void __launch_bounds__(160) k_chain_fx(ChainArgs a, int spc, int batch) {
  constexpr int W = (LD + 31) / 32;
  constexpr int bw = (int)fx_block_words(LD);
  extern __shared__ __align__(16) i64 csm[];
  __shared__ __align__(16) int2 s_x[2][2][32 * W];     // [shell][group] operand digits
  __shared__ int s_e[2][2][W];                         // their exponents
  __shared__ i64 s_pv[2][2][2][32 * W];                // [step parity][shell][group] halves of a product
  __shared__ int s_pe[2][2][2][32 * W];
  __shared__ int s_last;
  const int type = a.type0 + (blockIdx.x >> 1);
  const int par = blockIdx.x & 1;                      // first jj of the chains
  const int tid = threadIdx.x, lane = tid & 31;
  const int nt = 64 * W * spc;                         // compute threads; the last warp loads
  const bool loader = tid >= nt;
  const int sh = loader ? 0 : tid / (64 * W), g = (tid / (32 * W)) & 1, w = (tid >> 5) % W;
  const int b = blockIdx.y * spc + sh;
  const int M = a.M, nr = a.nr;
  const int field = type == 0 ? 0 : 1 + g;
  const int i = 32 * w + lane;
  const bool ok = i < nr;
  const int ir = ok ? i : nr - 1;
  const int S = (M - par + 1) / 2;
  const int chunk = CHUNK ? (int)blockIdx.z : 0;
  const int s0 = CHUNK ? chunk * a.kc : 0;
  const int s1 = CHUNK ? min(S, s0 + a.kc) : S;
  if (s0 >= S) {
    after_previous_kernel();
    return;
  }
  const int nsteps = s1 - s0;
  const size_t foff = (size_t)field * a.field_off;
  const int bs = b < batch ? b : batch - 1;
  const int chain = type == 0 ? par : (1 + g) * 2 + par;
  const size_t dslot = CHUNK ? (size_t)bs * a.d_stride + (size_t)chain * a.nch * a.ldd : 0;
  double* dout = CHUNK ? a.dbuf + dslot + (size_t)chunk * a.ldd : nullptr;
  const int e = (type == 0 && g == 1 ? nr : 0) + ir;   // this row's element of the carried state
  // the rows of f (f32, sub, h) of step s: row M - 1 - (par + 2 (s0 + s)), 2 nr apart
  const ptrdiff_t row0 = (ptrdiff_t)(M - 1 - (par + 2 * s0)) * nr + ir, drow = -2 * (ptrdiff_t)nr;
  double* f = a.f + (size_t)bs * a.f_stride + foff + row0;
  float* f32 = a.f32 ? a.f32 + (size_t)bs * a.f32_stride + foff + row0 : nullptr;   // final values only (no sub)
  const double* sub = a.sub ? a.sub + (size_t)bs * a.sub_stride + foff + row0 : nullptr;
  const double* h = a.h + (size_t)bs * a.h_stride + foff + row0;

  i64* ring = csm;                                     // D slots of the two groups' blocks
  double2* cf = reinterpret_cast<double2*>(ring + 2 * D * bw);   // [group][nsteps + 1] scalars
  const int jj0 = par + 2 * s0;
  // psi: (bj, bjt);  T/S: (k, -) with b += k f_{j+2} at the step's start
  const bool idle = a.sym && par != (type == 0 ? 0 : 1);   // (symmetric: only the "evens" loops run)
  for (int q = idle ? 2 * (nsteps + 1) : tid; q < 2 * (nsteps + 1); q += blockDim.x) {
    const int gg = q / (nsteps + 1), jj = jj0 + 2 * (q - gg * (nsteps + 1));
    const double* c = type == 0 ? a.coefA4 + 2 : (gg == 0 ? a.coefT : a.coefS);
    cf[q] = jj < M ? make_double2(c[(size_t)jj * 4], c[(size_t)jj * 4 + 1]) : make_double2(0.0, 0.0);
  }

  auto fetch_step = [&](int s) {                       // the blocks of step s (step 0 needs none: zero state)
    if (s < nsteps) {
      const size_t jj = jj0 + 2 * s;
      i64* dst = ring + (s % D) * 2 * bw;
      if (type == 0) {
        copy_words(dst, a.ABA4 + jj * 2 * bw, 2 * bw, lane, 32);
      } else {
        copy_words(dst, a.LinvT + jj * bw, bw, lane, 32);
        copy_words(dst + bw, a.LinvS + jj * bw, bw, lane, 32);
      }
    }
    cp_async_commit();
  };
  if (loader && !idle) {                               // (plan tables, as are the scalars)
#pragma unroll
    for (int s = 1; s <= D; ++s) fetch_step(s);
  }
  after_previous_kernel();
  const bool on = !loader && b < batch && (a.fmask >> field & 1) && !(a.active && !a.active[b]);
  const bool wr = on && ok && (type == 1 || g == 0);   // the lanes that write f

  // symmetric: the other parity's rows stay 0
  if (idle) {
    if (wr)
      for (int s = 0; s < nsteps; ++s) {
        f[s * drow] = 0.0;
        if (f32) f32[s * drow] = 0.0f;
      }
    if (CHUNK && on && ok) dout[e] = 0.0;
    return;
  }

  if (loader) {
    cp_async_wait<D - 1>();
    __syncthreads();
    for (int s = 1; s < nsteps; ++s) {
      cp_async_wait<D - 2>();
      __syncthreads();
      fetch_step(s + D);
    }
    cp_async_wait<0>();
  } else {
    // h and sub of this row, two steps ahead in registers
    double hn0 = on ? h[0] : 0.0, hn1 = on && nsteps > 1 ? h[drow] : 0.0;
    double sn0 = sub && wr ? sub[0] : 0.0, sn1 = sub && wr && nsteps > 1 ? sub[drow] : 0.0;
    __syncthreads();                                   // step 1's blocks and the scalars are visible
    const double2* cg = cf + g * (nsteps + 1);
    int2* xs = s_x[sh][g];
    double fe = 0.0, bfe = 0.0;                        // psi: f_e, bf_e (group 1 only);  T/S: b in fe
    ptrdiff_t o = 0;                                   // s drow
    for (int s = 0; s < nsteps; ++s, o += drow) {
      if (s + 2 >= nsteps) next_kernel_may_start();
      const double hi = hn0, si = sn0;
      hn0 = hn1;
      sn0 = sn1;
      if (s + 2 < nsteps) {
        if (on) hn1 = h[o + 2 * drow];
        if (sub && wr) sn1 = sub[o + 2 * drow];
      }
      double fi = hi;
      double pre = 0.0;
      if (s > 0) {
        const i64* blk = ring + ((s % D) * 2 + g) * bw;
        const int em = publish(type == 0 && g == 1 ? bfe : fe, fx_col_exp(blk, LD)[ir], ok, xs + i);
        int ems[W];
        if (W == 1) {
          __syncwarp();
          ems[0] = em;
        } else {
          if (lane == 0) s_e[sh][g][w] = em;
          compute_sync(nt);
#pragma unroll
          for (int q = 0; q < W; ++q) ems[q] = s_e[sh][g][q];
        }
        if (type == 0 && g == 1) pre = fma(cg[s].y, fe, bfe);   // bf_e + bjt f_e, off the product's path
        FxVal p = block_row<LD, W>(blk, nr, ir, xs, ems);
        const int q = s & 1;
        if (type == 0) {
          s_pv[q][sh][g][i] = p.v;
          s_pe[q][sh][g][i] = p.e;
        }
        __syncthreads();
        if (type == 0) {
          const FxVal t{s_pv[q][sh][1 - g][i], s_pe[q][sh][1 - g][i]};
          fi = g == 0 ? fx_sum<true>(hi, p, t) : fx_sum<true>(hi, t, p);
        } else {
          const bool half = jj0 + 2 * s == M - 1;      // j = 0: 0.5 b
          if (p.e == kFxBad) {
            p.v = __double_as_longlong((half ? -0.5 : -1.0) * __longlong_as_double(p.v));
          } else {
            p.v = -p.v;
            p.e -= half ? 1 : 0;
          }
          fi = fx_sum<true>(hi, p);
        }
      }
      if (type == 0) {
        if (g == 1) bfe = fma(cg[s].x, fi, pre);
        fe += fi;
      } else {
        fe = fma(cg[s + 1].x, fi, fe);                 // the b of the next step (of the next chunk after the last)
      }
      if (wr) {
        f[o] = sub ? fi - si : fi;                     // (sub: the Newton residual)
        if (f32 && chunk == 0) f32[o] = (float)fi;     // later chunks: final after the correction
      }
    }
    if (CHUNK && chunk + 1 < a.nch && on && ok) {      // end state of the chunk from a zero start
      const double v = type == 0 && g == 1 ? bfe : fe;
      dout[e] = v;
      if (a.carry_seq && a.nch == 2) a.cbuf[dslot + a.ldd + e] = v;   // s_1 = d_0 only
    }
  }

  if (CHUNK && a.carry_seq && a.nch > 2) {
    // the last chunk CTA of these chains to finish runs the carried-state recurrence s_1 = d_0,
    // s_{c+1} = Phi_c s_c + d_c (c = 1 .. nch - 2), Phi_c streaming through the ring
    __syncthreads();                                   // this chunk's end states before the ticket
    if (tid == 0) {
      int* cnt = a.counter + (size_t)blockIdx.y * spc * 6 + type * 2 + par;
      __threadfence();
      const int last = atomicAdd(cnt, 1) == a.nch - 1;
      if (last) {
        __threadfence();
        *cnt = 0;                                      // ready for the next launch
      }
      s_last = last;
    }
    __syncthreads();
    if (!s_last) return;
    const int per = type == 0 ? 4 : 2;                 // blocks of one Phi_c (psi: row half x operand half; T, S)
    const int slots = 2 * D / per, last = a.nch - 2;
    const double* d = a.dbuf + dslot;
    double* cb = a.cbuf + dslot;
    auto fetch = [&](int c) {
      if (c <= last) {
        i64* dst = ring + ((c - 1) % slots) * per * bw;
        const size_t m = (size_t)par * a.nch + c;
        if (type == 0) {
          copy_words(dst, a.PhiA4 + m * 4 * bw, 4 * bw, tid, blockDim.x);
        } else {
          copy_words(dst, a.PhiT + m * bw, bw, tid, blockDim.x);
          copy_words(dst + bw, a.PhiS + m * bw, bw, tid, blockDim.x);
        }
      }
      cp_async_commit();
    };
    for (int c = 1; c <= slots; ++c) fetch(c);
    const bool act = on && ok;
    double st = act ? __ldcg(d + e) : 0.0;             // s_1 = d_0
    if (act) cb[a.ldd + e] = st;
    for (int c = 1; c <= last; ++c) {
      if (slots > 1) cp_async_wait<1>();
      else cp_async_wait<0>();
      __syncthreads();                                 // Phi_c landed
      const i64* P = ring + ((c - 1) % slots) * per * bw;
      if (!loader) {
        // (the two row halves of a psi column share their column exponents)
        const int em = publish(st, fx_col_exp(P + g * bw, LD)[ir], act, &s_x[sh][g][i]);
        if (lane == 0) s_e[sh][g][w] = em;
      }
      __syncthreads();                                 // s_c visible
      if (!loader) {
        const double dc = act ? __ldcg(d + (size_t)c * a.ldd + e) : 0.0;
        if (type == 0) {
          const FxVal p0 = block_row<LD, W>(P + (2 * g) * bw, nr, ir, s_x[sh][0], s_e[sh][0]);
          const FxVal p1 = block_row<LD, W>(P + (2 * g + 1) * bw, nr, ir, s_x[sh][1], s_e[sh][1]);
          st = fx_sum<true>(dc, p0, p1);
        } else {
          st = fx_sum<true>(dc, block_row<LD, W>(P + g * bw, nr, ir, s_x[sh][g], s_e[sh][g]));
        }
        if (act) cb[(size_t)(c + 1) * a.ldd + e] = st;
      }
      __syncthreads();                                 // Phi_c and s_c are done with
      fetch(c + slots);
    }
    cp_async_wait<0>();
  }
}

static size_t chain_fx_smem_bytes(int nsteps, int ld, int D) {
  return 2 * D * fx_block_words(ld) * sizeof(i64) + 2 * ((size_t)nsteps + 1) * sizeof(double2);
}

// Parallel carry of the chunked chains (layouts 3 and 11).  One CTA per (psi or T and S, parity; shell; product
// (j, i)), i <= j - 2: part_{j,i} = P_{j,i} d_i, the blocks staged in shared memory by one round of cp.async.
// Four groups of W warps: psi (row half, operand half); T/S (field, half of the columns); the two halves of a
// product meet in shared memory.  The corrections sum each row (carried_state):
//   s_j = d_{j-1} + part_{j,0} + part_{j,1} + ... + part_{j,j-2},
// the exact algebra of s_{c+1} = Phi_c s_c + d_c.
template <int LD>
__global__ void __launch_bounds__(LD > 32 ? 256 : 128) k_carry_fx(ChainArgs a) {
  constexpr int W = (LD + 31) / 32;
  constexpr int bw = (int)fx_block_words(LD);
  extern __shared__ __align__(16) i64 psm[];
  __shared__ __align__(16) int2 s_x[4][W][32 * W];     // each warp's own copy of its operand digits
  __shared__ i64 s_v[4][32 * W];
  __shared__ int s_e[4][32 * W];
  const int type = a.type0 + (blockIdx.x >> 1), par = blockIdx.x & 1;
  const int b = blockIdx.y, pidx = blockIdx.z;
  if (a.sym && par != (type == 0 ? 0 : 1)) {           // inactive chains: their carried states are not read
    after_previous_kernel();
    return;
  }
  int j = 2;
  while (j * (j - 1) / 2 <= pidx) ++j;                 // row j holds products (j-1)(j-2)/2 .. j(j-1)/2 - 1
  const int ii = pidx - (j - 1) * (j - 2) / 2;
  const int nr = a.nr;
  const int tid = threadIdx.x, lane = tid & 31, q = tid / (32 * W), w = (tid >> 5) % W;
  const int i = 32 * w + lane, ir = min(i, nr - 1);
  const size_t m = (size_t)par * a.np + pidx;
  if (type == 0) {
    copy_words(psm, a.PA4 + m * 4 * bw, 4 * bw, tid, blockDim.x);
  } else {
    copy_words(psm, a.PT + m * bw, bw, tid, blockDim.x);
    copy_words(psm + bw, a.PS + m * bw, bw, tid, blockDim.x);
  }
  cp_async_commit();
  after_previous_kernel();                             // (the blocks are the plan's)
  if (a.active && !a.active[b]) {
    cp_async_wait<0>();
    return;
  }
  const int chain = type == 0 ? par : (1 + (q >> 1)) * 2 + par;
  const double* d = a.dbuf + (size_t)b * a.d_stride + ((size_t)chain * a.nch + ii) * a.ldd +
                    (type == 0 ? (q & 1) * nr : 0);
  int2* xs = s_x[q][w];
  double x[W];
#pragma unroll
  for (int p = 0; p < W; ++p) x[p] = 32 * p + lane < nr ? d[32 * p + lane] : 0.0;
  cp_async_wait<0>();
  __syncthreads();
  const i64* blk = psm + (type == 0 ? q : q >> 1) * bw;
  int cx[W];
#pragma unroll
  for (int p = 0; p < W; ++p) cx[p] = 32 * p + lane < nr ? fx_col_exp(blk, LD)[32 * p + lane] : 0;
  next_kernel_may_start();
  const int em = publish_regs<W>(x, cx, nr, lane, xs);
  const int ea = fx_row_exp(blk, LD)[ir];
  // psi: all columns of block (row half, operand half); T/S: half the columns of the field's
  constexpr int H = LD / 2;
  const int c0 = type == 0 ? 0 : (q & 1) * H, c1 = type == 0 || (q & 1) ? LD : H;
  const int2* A = reinterpret_cast<const int2*>(blk) + ir;
  FxVal p;
  p.v = type == 0 ? fx_dot<LD, LD>(A, xs) : fx_dot<H, LD>(A + c0 * LD, xs + c0);
  p.e = ea + em - kFxMvExp;
  if (em >= kFxInf || ea == kFxBad) {
    p.v = __double_as_longlong(em == kFxInf ? fx_dot_slow(blk, LD, ir, xs, c0, min(c1, nr), em) : fx_nan());
    p.e = kFxBad;
  }
  s_v[q][i] = p.v;
  s_e[q][i] = p.e;
  __syncthreads();
  if ((q & 1) == 0 && i < nr) {
    const FxVal t{s_v[q + 1][i], s_e[q + 1][i]};
    const int oc = type == 0 ? par : chain;
    double* y = a.pbuf + (size_t)b * a.p_stride + ((size_t)oc * a.np + pidx) * a.ldd + (type == 0 && q ? nr : 0);
    y[i] = fx_sum<true>(0.0, p, t);
  }
}

// Element e of the carried state s_c (c >= 1) of chain `chain` under layouts 3 / 11: d_{c-1} plus the row's
// products (k_carry_fx), summed in index order.
__device__ __forceinline__ double carried_state(const ChainArgs& a, int b, size_t chain, int c, int e) {
  const double* d = a.dbuf + (size_t)b * a.d_stride + chain * a.nch * a.ldd;
  double v = d[(size_t)(c - 1) * a.ldd + e];
  if (c >= 2) {
    const double* row = a.pbuf + (size_t)b * a.p_stride + (chain * a.np + (size_t)(c - 1) * (c - 2) / 2) * a.ldd;
    const int nt = c - 1;                              // in index order, the terms loaded eight at a time
    for (int u0 = 0; u0 < nt; u0 += 8) {
      double tv[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) tv[k] = (u0 + k < nt) ? row[(size_t)(u0 + k) * a.ldd + e] : 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (u0 + k < nt) v += tv[k];
    }
  }
  return v;
}

// Independent per-mode matvecs, one warp per (field, mode, 32 rows) and up to kMvShells shells, one lane per
// row; the lane's row of the block sits in registers for all shells of the group (the block is read once per
// group, its loads all in flight at once), the next shell's inputs load beside a shell's product (corrections of 8
// shells of 384 x 36: 41 us without, 31 with; h of batches is bound by the integer pipe, 61 us at 64 shells of
// 256 x 30, 21 of it the three-digit Dr Q):
//   FIX = false:  h_jj = Linv_jj g_jj                          (the chains' right-hand sides)
//   FIX = true:   f_jj += G_jj s_c(jj) for the modes of chunks c >= 1   (chunked chains' correction)
constexpr int kMvShells = 4;

// The right-hand side of FIX = false is a.g, or (fuse_rhs) formed here, each operation rounded by itself:
//   psi: (-dt (Dr Q - R)) + lin,  T: (-dt NT) + lin,  S: (-dt NS) + lin,
// Dr Q in fixed point like the other matvecs, or (mixed plans' FP32 nonlinear term) in FP32.
template <bool FIX, int LD>
__global__ void __launch_bounds__(128) k_mode_mv(ChainArgs a, int nfields, int batch, int group) {
  constexpr int NP = (LD + 31) / 32;
  constexpr int bw = (int)fx_block_words(LD);
  extern __shared__ __align__(16) int msm[];           // fused right-hand side: Dr's block, or Dr^T in FP32
  __shared__ int4 s_w[FIX ? 1 : 4][32 * NP];           // Q's digits
  __shared__ __align__(16) int2 s_x[4][32 * NP];
  __shared__ float s_q[4][32 * NP];
  __shared__ double s_dq[FIX || NP == 1 ? 1 : 2][4][32];   // [buffer][warp] Dr Q of the warp's rows
  __shared__ i64 s_pv[FIX ? 4 : 1][kMvShells][32];     // psi's first half of a correction, per shell
  __shared__ int s_pe[FIX ? 4 : 1][kMvShells][32];
  const int M = a.M, nr = a.nr;
  const int wid = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool fuse = !FIX && a.fuse_rhs;
  if (fuse && a.field0 == 0 && blockIdx.x * 4 < M * NP) {   // (a CTA with a psi mode; uniform)
    if (a.q32) {
      float* Dt = reinterpret_cast<float*>(msm);
      for (int e = threadIdx.x; e < nr * nr; e += blockDim.x) {
        const int n = e / nr, c = e - n * nr;
        Dt[c * nr + n] = __ldg(a.Dr32 + e);
      }
    } else {
      for (int e = threadIdx.x; e < (int)wx_block_ints(LD) / 4; e += blockDim.x) cp_async16(msm + 4 * e, a.wxDr + 4 * e);
      cp_async_commit();
    }
  }
  const bool in_range = wid < nfields * M * NP;        // (the last CTA's spare warps: field and mode 0)
  const int fm = in_range ? wid / NP : 0, r = in_range ? (wid - fm * NP) * 32 + lane : lane;
  const int fl = fm / M, jj = fm - fl * M;
  const int field = a.field0 + fl;
  const int row = M - 1 - jj;
  const size_t N = (size_t)M * nr, ro = (size_t)row * nr;
  const size_t foff = (size_t)field * a.field_off + ro;
  const bool a4 = field == 0;
  const int rr = min(r, nr - 1);
  const int par = jj & 1;
  const int c = FIX ? (jj >> 1) / a.kc : 0;
  const bool mine = in_range && !(FIX && (c == 0 || (a.sym && !(a4 ? par == 0 : par == 1))));
  const int nseg = FIX && a4 ? 2 : 1;
  const i64* blk = FIX ? (a4 ? a.GA4 + (size_t)jj * 2 * bw : (field == 1 ? a.GT : a.GS) + (size_t)jj * bw)
                       : (a4 ? a.LinvA4 : (field == 1 ? a.LinvT : a.LinvS)) + (size_t)jj * bw;
  const size_t chain = (size_t)(field * 2 + par);
  const int b0 = blockIdx.y * group, b1 = min(batch, b0 + group);
  int2* xs = s_x[wl];
  FxRow<LD, NP> m;
  if (!FIX || mine) m.load(blk, rr);                   // (the plan's, like Dr's block)
  after_previous_kernel();
  if (fuse && a.field0 == 0 && blockIdx.x * 4 < M * NP) {
    cp_async_wait<0>();
    __syncthreads();
  }
  if (!mine) return;
  for (int sg = 0; sg < nseg; ++sg) {
    const i64* B = blk + (size_t)sg * bw;
    if (FIX && sg > 0) m.load(B, rr);
    // a shell's inputs, loaded one shell ahead of their use
    struct In {
      double x[NP], ln[NP], q[NP];
    };
    auto load = [&](int b) {
      In v;
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const int e = p * 32 + lane;
        v.x[p] = v.ln[p] = v.q[p] = 0.0;
        if (FIX) {
          if (e < nr)
            v.x[p] = a.carry_seq ? a.cbuf[(size_t)b * a.d_stride + (chain * a.nch + c) * a.ldd + sg * nr + e]
                                 : carried_state(a, b, chain, c, sg * nr + e);
        } else if (!fuse) {
          if (e < nr) v.x[p] = a.g[(size_t)b * a.g_stride + foff + e];
        } else if (e < nr) {
          const double* o4 = a.out4 + (size_t)b * a.out_stride + ro;
          v.x[p] = o4[(size_t)(field + 1) * N + e];      // psi: R
          v.ln[p] = a.lin[(size_t)b * a.g_stride + foff + e];
          if (a4) v.q[p] = a.q32 ? (double)a.q32[(size_t)b * N + ro + e] : o4[e];
        }
      }
      if (FIX && sg + 1 == nseg && r < nr) v.ln[0] = a.f[(size_t)b * a.f_stride + foff + r];
      return v;
    };
    In in = load(b0);
    int turn = 0;                                      // s_dq's buffer: alternates over the shells that are not skipped
#pragma unroll 1
    for (int b = b0; b < b1; ++b) {
      const int u = b - b0;
      const In cur = in;
      if (b + 1 < b1) in = load(b + 1);
      else next_kernel_may_start();
      if (a.active && !a.active[b]) continue;
      double x[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) x[p] = cur.x[p];
      if (fuse) {
        if (a4) {
          double dq[NP];
          // (nr > 32: the two warps of a mode form Dr Q's rows of their own and swap them)
          constexpr int P1 = NP == 1 ? 1 : 2;
          const int own = NP == 1 ? 0 : wl & 1;
          const int e = min(own * 32 + lane, nr - 1);
          double d;
          if (a.q32) {
#pragma unroll
            for (int p = 0; p < NP; ++p)
              if (p * 32 + lane < nr) s_q[wl][p * 32 + lane] = (float)cur.q[p];
            __syncwarp();
            const float* Dt = reinterpret_cast<const float*>(msm) + e;
            float acc = 0.0f;
            for (int cc = 0; cc < nr; ++cc) acc = fmaf(Dt[cc * nr], s_q[wl][cc], acc);
            __syncwarp();
            d = (double)acc;
          } else {
            int cx[NP];
#pragma unroll
            for (int p = 0; p < NP; ++p) cx[p] = p * 32 + lane < nr ? msm[3 * LD * LD + LD + p * 32 + lane] : 0;
            const int em = publish_wide<NP>(cur.q, cx, nr, lane, s_w[wl]);
            d = fx_val(wx_dot<LD>(msm, nr, e, s_w[wl], em));
            __syncwarp();                              // the digits are read before the next shell's replace them
          }
          dq[0] = d;
          if constexpr (NP > 1) {
            s_dq[turn][wl][lane] = d;
            asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (wl >> 1)) : "memory");
#pragma unroll
            for (int p = 0; p < P1; ++p) dq[p] = s_dq[turn][(wl & 2) + p][lane];
            turn ^= 1;
          }
#pragma unroll
          for (int p = 0; p < NP; ++p) x[p] = __dsub_rn(dq[p], x[p]);
        }
#pragma unroll
        for (int p = 0; p < NP; ++p)
          if (p * 32 + lane < nr) x[p] = __dadd_rn(__dmul_rn(-a.dt, x[p]), cur.ln[p]);
      }
      const int em = publish_regs<NP>(x, m.cx, nr, lane, xs);
      const FxVal p = m.times(B, nr, rr, xs, em);
      __syncwarp();                                    // the digits are read before the next shell's replace them
      if (FIX) {
        if (sg + 1 < nseg) {
          s_pv[wl][u][lane] = p.v;                     // (read back by the same lane)
          s_pe[wl][u][lane] = p.e;
        } else if (r < nr) {
          double* y = a.f + (size_t)b * a.f_stride + foff + r;
          const double v = nseg == 2 ? fx_sum(cur.ln[0], FxVal{s_pv[wl][u][lane], s_pe[wl][u][lane]}, p)
                                     : fx_sum(cur.ln[0], p);
          *y = v;
          if (a.f32) a.f32[(size_t)b * a.f32_stride + foff + r] = (float)v;
        }
      } else if (r < nr) {
        a.h[(size_t)b * a.h_stride + foff + r] = fx_val(p);
      }
    }
  }
}

// h = Linv g in FP32 from the FP32 right-hand sides (k_rhs32) and the FP32 copies of the Linv blocks: one
// warp per (field, mode) and group of up to kMv32Shells shells, one lane per row.  The lane keeps its row
// of the block in registers for all shells of the group (the block is read once per group, not once per
// shell); each shell's g row is loaded once per lane and broadcast by shuffles.  h is stored in FP64 for
// the chains.  NP: passes of 32 rows (nr <= 32 NP).
constexpr int kMv32Shells = 16;

template <int NP>
__global__ void __launch_bounds__(128) k_mode_mv32(ChainArgs a, int nfields, int batch) {
  after_previous_kernel();
  const int M = a.M, nr = a.nr, ldl = a.ldl;
  const int wid = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (wid >= nfields * M) return;
  const int fl = wid / M, jj = wid - fl * M;
  const int field = a.field0 + fl;
  const size_t foff = (size_t)field * a.field_off + (size_t)(M - 1 - jj) * nr;   // this mode's row
  const float* A = (field == 0 ? a.Linv32A4 : (field == 1 ? a.Linv32T : a.Linv32S)) + (size_t)jj * nr * ldl;
  const int b0 = blockIdx.y * kMv32Shells;
  const int b1 = min(batch, b0 + kMv32Shells);
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int r = p * 32 + lane;
    const bool rok = r < nr;
    float Ar[32 * NP];
#pragma unroll
    for (int c = 0; c < 32 * NP; ++c) Ar[c] = (rok && c < nr) ? __ldg(A + (size_t)c * ldl + r) : 0.0f;
    for (int b = b0; b < b1; ++b) {
      if (a.active && !a.active[b]) continue;
      const float* x = a.g32 + (size_t)b * a.g_stride + foff;
      float xv[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) xv[q] = (q * 32 + lane < nr) ? x[q * 32 + lane] : 0.0f;
      float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
      for (int c = 0; c < 32 * NP; c += 4) {
        s0 = fmaf(Ar[c], __shfl_sync(0xffffffffu, xv[c / 32], c % 32), s0);
        s1 = fmaf(Ar[c + 1], __shfl_sync(0xffffffffu, xv[(c + 1) / 32], (c + 1) % 32), s1);
        s2 = fmaf(Ar[c + 2], __shfl_sync(0xffffffffu, xv[(c + 2) / 32], (c + 2) % 32), s2);
        s3 = fmaf(Ar[c + 3], __shfl_sync(0xffffffffu, xv[(c + 3) / 32], (c + 3) % 32), s3);
      }
      if (rok) a.h[(size_t)b * a.h_stride + foff + r] = (double)((s0 + s1) + (s2 + s3));
    }
  }
}

// f(std::integral_constant<int, LD>) for the padded block size of a plan (fx_ld)
template <typename F>
static cudaError_t with_ld(int ld, F&& f) {
  switch (ld) {
    case 8: return f(std::integral_constant<int, 8>{});
    case 16: return f(std::integral_constant<int, 16>{});
    case 24: return f(std::integral_constant<int, 24>{});
    case 32: return f(std::integral_constant<int, 32>{});
    case 48: return f(std::integral_constant<int, 48>{});
    case 64: return f(std::integral_constant<int, 64>{});
    default: return cudaErrorInvalidValue;
  }
}

static int sm_count() {
  static const int sms = [] {  // thread-safe one-time initialisation (host threads may launch concurrently)
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  return sms;
}


// h = Linv g (FIX = false) or the chunk corrections.  A warp takes more shells as soon as the launch would
// still give every SM 32 warps: the block is then read once for all of them (bits do not depend on it).
template <bool FIX>
static cudaError_t launch_mode_mv(const ChainArgs& a, int batch, int nfields, cudaStream_t s) {
  if (!FIX && a.g32) {   // FP32 right-hand sides: the FP32 matvecs, whatever the chain layout
    if (!a.Linv32A4 || !a.Linv32T || !a.Linv32S || a.fuse_rhs) return cudaErrorInvalidValue;
    const dim3 grid((nfields * a.M + 3) / 4, (batch + kMv32Shells - 1) / kMv32Shells);
    const cudaError_t e = a.nr <= 32 ? launch_kernel(k_mode_mv32<1>, grid, dim3(128), 0, s, a, nfields, batch)
                                     : launch_kernel(k_mode_mv32<2>, grid, dim3(128), 0, s, a, nfields, batch);
    ktimer_mark(SDD_K_MODE_H, s);
    return e;
  }
  const int np = a.nr <= 32 ? 1 : 2;
  const long warps = (long)nfields * a.M * np;
  int group = 1;
  while (group < kMvShells && warps * batch / (2 * group) >= 32l * sm_count()) group *= 2;
  const dim3 grid((unsigned)((warps + 3) / 4), (batch + group - 1) / group);
  const size_t smem = FIX || !a.fuse_rhs || a.field0 != 0 ? 0
                      : a.q32                            ? (size_t)a.nr * a.nr * sizeof(float)
                                                         : wx_block_ints(a.ldl) * sizeof(int);
  const cudaError_t e = with_ld(a.ldl, [&](auto ld) {
    constexpr int LD = decltype(ld)::value;
    static unsigned long long done = 0;
    const cudaError_t er = smem > 40 * 1024 ? ensure_smem_attr(k_mode_mv<FIX, LD>, &done) : cudaSuccess;
    if (er != cudaSuccess) return er;
    return launch_kernel(k_mode_mv<FIX, LD>, grid, dim3(128), smem, s, a, nfields, batch, group);
  });
  ktimer_mark(FIX ? SDD_K_MODE_FIX : SDD_K_MODE_H, s);
  return e;
}

// The chains themselves: whole (nch = 1 CTA per pair of chains) or chunked.  Two shells share a CTA (and the
// blocks' way through shared memory) once a CTA per shell would give every SM more than one.  Blocks of 48 rows: a ring of
// four slots while every CTA has an SM of its own, of two slots beyond, of which three CTAs share an SM and hide each
// other's waits (a ring of four takes 150 KB; FP64 chains before ran two an SM).  us a linear step, four / two slots (and
// FP64 chains): 24 x 34, 64 shells 62 / 51 (58), 128 shells 114 / 91 (96); 96 x 36, 128 shells 339 / 266 (305), 8 shells
// in chunks (160 CTAs) 58 / 55; one CTA an SM: 24 x 34, 32 shells 34 / 37, 192 x 36, 4 shells in chunks 59 / 67.
template <int LD, bool CHUNK, int D>
static cudaError_t launch_chains_ring(const ChainArgs& a, int batch, int ntypes, int nch, int nsteps, int spc,
                                      cudaStream_t s) {
  constexpr int W = (LD + 31) / 32;
  static unsigned long long done = 0;
  const cudaError_t e = ensure_smem_attr(k_chain_fx<LD, CHUNK, D>, &done);
  if (e != cudaSuccess) return e;
  return launch_kernel(k_chain_fx<LD, CHUNK, D>, dim3(2 * ntypes, (batch + spc - 1) / spc, nch), dim3(64 * W * spc + 32),
                       chain_fx_smem_bytes(nsteps, LD, D), s, a, spc, batch);
}
template <bool CHUNK>
static cudaError_t launch_chains(const ChainArgs& a, int batch, int ntypes, int nch, int nsteps, cudaStream_t s) {
  const bool many = 2l * ntypes * batch * nch > sm_count();
  const cudaError_t e = with_ld(a.ldl, [&](auto ld) {
    constexpr int LD = decltype(ld)::value;
    if constexpr (LD == 48) {
      if (many) return launch_chains_ring<LD, CHUNK, 2>(a, batch, ntypes, nch, nsteps, 1, s);
    }
    return launch_chains_ring<LD, CHUNK, (LD > 48 ? 3 : 4)>(a, batch, ntypes, nch, nsteps, LD <= 32 && many ? 2 : 1, s);
  });
  ktimer_mark(SDD_K_CHAIN, s);
  return e;
}

static cudaError_t launch_chunked(const ChainArgs& a, int batch, int nfields, int ntypes, cudaStream_t s) {
  cudaError_t e;
  if ((e = launch_chains<true>(a, batch, ntypes, a.nch, a.kc, s)) != cudaSuccess) return e;
  if (a.nch < 2) return cudaSuccess;
  if (!a.carry_seq) {   // layouts 3 / 11: the products in parallel, then the corrections
    if (a.np > 0) {
      e = with_ld(a.ldl, [&](auto ld) {
        constexpr int LD = decltype(ld)::value;
        static unsigned long long done = 0;
        const cudaError_t er = ensure_smem_attr(k_carry_fx<LD>, &done, true);
        if (er != cudaSuccess) return er;
        return launch_kernel(k_carry_fx<LD>, dim3(2 * ntypes, batch, a.np), dim3(LD > 32 ? 256 : 128),
                             4 * fx_block_words(LD) * sizeof(i64), s, a);
      });
      ktimer_mark(SDD_K_CHAIN_CARRY, s);
      if (e != cudaSuccess) return e;
    }
    if (a.defer_fix) return cudaSuccess;   // the next step's nonlinear term applies the correction
  }
  return launch_mode_mv<true>(a, batch, nfields, s);
}

static void use_chunk_set(ChainArgs& a, const ChunkSet& c) {
  a.kc = c.kc; a.nch = c.nch; a.np = c.np;
  a.GA4 = c.GA4; a.GT = c.GT; a.GS = c.GS;
  a.PhiA4 = c.PhiA4; a.PhiT = c.PhiT; a.PhiS = c.PhiS;
  a.PA4 = c.PA4; a.PT = c.PT; a.PS = c.PS;
}

// The layout-3 / 11 correction f += G_jj s_c on its own (a correction left pending by the last step of a
// sequence; a.f is the state, a.f32 its FP32 copy or null).
cudaError_t launch_chunk_fix(const ChainArgs& a_in, int batch, int nfields, cudaStream_t s) {
  ChainArgs a = a_in;
  use_chunk_set(a, a.cset[1]);
  a.carry_seq = 0;
  if (a.nch < 2) return cudaSuccess;
  return launch_mode_mv<true>(a, batch, nfields, s);
}

// The number a layout request resolves to (sdd_plan_chain_choice).  The whole-chain layouts run one kernel
// (k_chain_fx); whether 8 and 9 are reported as such follows the shared memory that three step-matrix rings in one CTA
// would take at this shape, so that callers keep the numbers they have stored.
static size_t layout_bytes(int layout, int M, int nr, int ldl) {
  const size_t blk = (size_t)nr * ldl, ns = 4 * ((size_t)(M + 1) / 2 + 1), v = nr;
  return ((layout == 8 ? 4 : 6) * blk + ns + 4 * v + 2 * (3 * blk + ns + (layout == 8 ? 2 : 4) * v)) * sizeof(double);
}

int resolve_chain_layout(const ChainArgs& a, int batch, int nfields) {
  const int sms = sm_count();
  static const int optin = [] {   // less a margin for the chain kernels' static shared memory (a few words)
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return n - 256;
  }();
  int layout = a.layout;
  const ChunkSet& c2 = a.cset[0];
  const ChunkSet& c3 = a.cset[1];
  // layout 8 needs all three fields of a step with full right-hand sides, and its three rings in one CTA
  if (layout == 8 && (nfields != 3 || a.field0 != 0 || a.split_fx || a.g32 ||
                      layout_bytes(8, a.M, a.nr, a.ldl) > (size_t)optin))
    layout = 6;
  // layout 9 needs all three fields and its three rings in one CTA
  if (layout == 9 && (nfields != 3 || a.field0 != 0 || layout_bytes(9, a.M, a.nr, a.ldl) > (size_t)optin))
    layout = 5;
  // (the numbers 4 to 11 are kept for callers that select or record them: 10 / 11 are the chunks of 2 / 3, reported as
  // 2 / 3 with an FP32 right-hand side)
  if ((layout == 10 || layout == 11) && a.g32) layout -= 8;
  // Chunks shorten the chains' critical path and add a correction matvec per mode (nr > 32: two, or their columns
  // in halves), so what decides is the batch.  Parallel carry while its chunks and products fit the chip (us a
  // step, parallel / sequential carry: 256 x 30, 4 shells 77 / 82, 8: 128 / 123; 64 x 20, 8 shells 44 / 48; 192 x 36,
  // 2 shells 68 / 78, 4: 100 / 90); sequential carry against whole chains: 256 x 30, 8 shells 123 / 206, 32: 343 /
  // 384, 64: 605 / 608; 64 x 20, 32 shells 114 / 119, 64: 195 / 192; 192 x 36, 8 shells 137 / 174, 16: 203 / 206, 32:
  // 361 / 278; 540 x 65, 8 shells 610 / 752, 16: 1072 / 1077.  Short chains gain nothing (16 x 8: 27.0 parallel, 25.9
  // whole; 24 x 20, 24 shells 69 sequential, 67 whole).
  const bool wide = a.nr > 32;
  if (layout == 0 && a.M > 16 && c3.nch > 1 && c3.GA4 && 4 * nfields * batch * c3.nch <= (wide ? 3 : 7) * sms) layout = 3;
  if (layout == 0 && a.M >= 40 && c2.nch > 1 && c2.GA4 && (wide ? 4 : 1) * nfields * batch <= sms) layout = 2;
  // (the same chunks; the number says that the full FP64 right-hand side is there)
  if (a.layout == 0 && (layout == 2 || layout == 3) && !a.split_fx && !a.g32) layout += 8;
  // layouts 6 / 7 need the full right-hand side in FP64: with the fused or the FP32 one, the pre-pass form
  if ((layout == 6 || layout == 7) && (a.split_fx || a.g32)) layout = 5;
  // a launch that fills the SMs (one kernel; the number as in layout_bytes)
  if (layout == 0) {
    if (2 * nfields * batch <= sms) layout = 4;
    else if (a.split_fx || a.g32) layout = 5;
    else if (nfields == 3 && a.field0 == 0 && layout_bytes(8, a.M, a.nr, a.ldl) <= (size_t)optin) layout = 8;
    else layout = 6;
  }
  if (layout == 5 && a.nr > 32) layout = 4;
  return layout;
}


// The chains of fields field0 .. field0 + nfields - 1.  a.g holds the right-hand sides (or they are formed from
// a.lin and a.out4, fuse_rhs); a.h receives h = Linv g, which is what the chains read.
cudaError_t launch_chain(const ChainArgs& a_in, int batch, int nfields, cudaStream_t s) {
  ChainArgs a = a_in;
  const int layout = resolve_chain_layout(a, batch, nfields);
  a.fmask = ((1 << nfields) - 1) << a.field0;
  a.type0 = a.field0 == 0 ? 0 : 1;
  const int ntypes = a.field0 == 0 && nfields == 3 ? 2 : 1;
  cudaError_t e = launch_mode_mv<false>(a, batch, nfields, s);   // h = Linv g
  if (e != cudaSuccess) return e;
  if (layout == 2 || layout == 3 || layout == 10 || layout == 11) {
    const bool seq = layout == 2 || layout == 10;
    const ChunkSet& c = a.cset[seq ? 0 : 1];
    if (!c.GA4 || c.kc < 1 || c.nch < 1) return cudaErrorInvalidValue;
    use_chunk_set(a, c);
    a.carry_seq = seq;
    return launch_chunked(a, batch, nfields, ntypes, s);
  }
  if ((e = launch_chains<false>(a, batch, ntypes, 1, (a.M + 1) / 2, s)) != cudaSuccess) return e;
  return cudaGetLastError();
}

// ---- blocks to fixed point ------------------------------------------------------------------------
// The scales of an nr x nr block at a (element (r, c) at a[r rs + c cs]), padded to ld: cx[c] with |A_rc| < 2^cx down
// the column (over nrows rows from r = -r0 on, which share it), ea[r] with sum_c |A_rc| 2^-cx < 2^ea along the row
// (kFxBad: a row with an infinity or NaN).  A row's sum is of whole numbers, 18 bits of its largest entry, each rounded
// up: so a single entry stays 2^-24 below 2^ea, which the high digits (31 bits and the sign) need.  One thread a column,
// then a row (with FP64 sums and scalings the conversions of a plan of 64 x 20 took 0.35 ms).
// Ends with a barrier.
__device__ __forceinline__ void block_scales(const double* a, int rs, int cs, int nrows, int r0, int nr, int ld, int* cx,
                                             int* ea) {
  for (int c = threadIdx.x; c < ld; c += blockDim.x) {
    unsigned m = 0;
    if (c < nr) {
      const double* col = a + (ptrdiff_t)c * cs - (ptrdiff_t)r0 * rs;
#pragma unroll 8
      for (int r = 0; r < nrows; ++r) {
        const unsigned h = abs_hi(col[(size_t)r * rs]);
        if (h < 0x7ff00000u) m = max(m, h);
      }
    }
    cx[c] = m >> 20 ? (int)(m >> 20) - 1022 : 0;
  }
  __syncthreads();
  for (int r = threadIdx.x; r < ld; r += blockDim.x) {
    const double* row = a + (size_t)r * rs;
    const int n = r < nr ? nr : 0;
    int em = -0x10000, bad = 0;
#pragma unroll 8
    for (int c = 0; c < n; ++c) {
      const unsigned h = abs_hi(row[(size_t)c * cs]);
      bad |= h >= 0x7ff00000u;
      if (h) em = max(em, max((int)(h >> 20), 1) - cx[c]);
    }
    unsigned tot = 0;
#pragma unroll 8
    for (int c = 0; c < n; ++c) {
      const unsigned h = abs_hi(row[(size_t)c * cs]);
      int e1;
      const unsigned m = fx_mant_hi(h, e1);
      if (h) tot += (m >> min(em - (e1 - cx[c]) + 3, 31)) + 1;
    }
    ea[r] = bad ? kFxBad : max(tot ? em - 1040 + (32 - __clz((int)tot)) : -1022, -1022);
  }
  __syncthreads();
}

constexpr int kConvThreads = 256;

// Block m of `out` (stride out_stride words) from rows [r0, r0 + nr) and columns [c0, c0 + nr) of the m-th
// source matrix (element (r, c) at r rs + c cs, stride src_stride, nrows rows: the column exponents are those of whole
// columns, so that the row halves of a column share them).
__global__ void __launch_bounds__(kConvThreads) k_to_fixed(const double* src, size_t src_stride, int rs, int cs, int nrows,
                                                           int r0, int c0, int nr, int ldl, i64* out, size_t out_stride) {
  __shared__ int cx[kMaxNr], ea[kMaxNr];
  const double* a = src + (size_t)blockIdx.x * src_stride + (size_t)r0 * rs + (size_t)c0 * cs;
  i64* o = out + (size_t)blockIdx.x * out_stride;
  block_scales(a, rs, cs, nrows, r0, nr, ldl, cx, ea);
  for (int q = threadIdx.x; q < ldl * ldl; q += blockDim.x) {
    const int c = q / ldl, r = q - c * ldl;
    const bool in = r < nr && c < nr && ea[r] != kFxBad;
    const i64 A = in ? d2fx(a[(size_t)r * rs + (size_t)c * cs], 1084 - kMvA + ea[r] + cx[c]) : 0;
    reinterpret_cast<int2*>(o)[q] = mv_digits(A);
  }
  int* rexp = reinterpret_cast<int*>(o + (size_t)ldl * ldl);
  for (int q = threadIdx.x; q < ldl; q += blockDim.x) {
    rexp[q] = ea[q];
    rexp[ldl + q] = cx[q];
  }
}

// A radial operator (row-major nr x nr on the device) as a three-digit block.
__global__ void __launch_bounds__(kConvThreads) k_to_wide(const double* src, int nr, int ld, int* out) {
  __shared__ int cx[kMaxNr], ea[kMaxNr];
  block_scales(src, nr, 1, nr, 0, nr, ld, cx, ea);
  for (int q = threadIdx.x; q < ld * ld; q += blockDim.x) {
    const int c = q / ld, r = q - c * ld;
    int d2 = 0, d1 = 0, d0 = 0;
    if (r < nr && c < nr && ea[r] != kFxBad) {
      const double x = src[r * nr + c];
      wx_split(x, 1022 + cx[c] + ea[r] - (int)(abs_hi(x) >> 20), d2, d1, d0);
    }
    out[q] = d2;
    out[ld * ld + q] = d1;
    out[2 * ld * ld + q] = d0;
  }
  int* rexp = out + 3 * ld * ld;
  for (int q = threadIdx.x; q < ld; q += blockDim.x) {
    rexp[q] = ea[q];
    rexp[ld + q] = cx[q];
  }
}

cudaError_t launch_to_wide(const double* src, int nr, int ld, int* out, cudaStream_t s) {
  k_to_wide<<<1, kConvThreads, 0, s>>>(src, nr, ld, out);
  return cudaGetLastError();
}

cudaError_t launch_to_fixed(const double* src, size_t src_stride, int rs, int cs, int nrows, int r0, int c0, int nr,
                            int ldl, i64* out, size_t out_stride, int nblk, cudaStream_t s) {
  k_to_fixed<<<nblk, kConvThreads, 0, s>>>(src, src_stride, rs, cs, nrows, r0, c0, nr, ldl, out, out_stride);
  return cudaGetLastError();
}

}  // namespace sdd
