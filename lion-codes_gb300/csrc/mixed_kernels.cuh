// Kernels of the mixed-precision batched complex LUP determinant, shared by
// the complex128 (lup_mixed.cu), coordinate (lup_mixed_lll.cu) and complex64
// (lup_mixed_c64.cu) entry points and by the CF call (cf.cu).
//
// Per matrix (one warp, shared memory), with FP64 used only where accuracy
// needs it and almost all arithmetic on the FP32 and integer pipes, which on
// GB300 run far faster than FP64:
//  1. power-of-two column-then-row equilibration A^ = D_r^-1 A D_c^-1, chosen
//     from the exponent fields (exact; log|det D| is added back in FP64);
//  2. split of every scaled FP64 entry into float hi + lo by integer
//     operations (48 significant bits kept);
//  3. FP32 complex LUP of hi with partial pivoting on |Re|+|Im|; alongside,
//     the residual R = P A^ - L U is accumulated exactly in float-float
//     (Ogita-Rump-Oishi Dot2: TwoProd + TwoSum per real product, the real
//     and imaginary parts as packed FP32 pairs), starting from hi + lo, so R
//     carries FP64-level accuracy although every operation is an FP32 one;
//  4. E = U^-1 L^-1 R by FP32 triangular solves;
//  5. log det(I + E) by an unpivoted FP32 LU that keeps the identity implicit
//     (only the small offsets are stored), log1p/atan2 of each pivot, or, for
//     the register-tiled sizes when ||E|| is small enough that the dropped
//     terms stay below 1e-12 max(1, |log|det||), by tr E - tr(E^2)/2;
//  6. log|det| = log|prod u_jj| (complex float-float product, one FP64 log
//     and atan2 per matrix, deferred and done for 32 matrices at once by the
//     32 lanes) + equilibration + Re log det(I+E); phase likewise.
// A matrix whose ||E||_F exceeds the threshold, or whose FP32 factorisation
// meets a zero or non-finite pivot, is refactorised by the FP64 warp routine
// (reference pivot rule, fused arithmetic) and flagged LUFQHE_ST_FALLBACK.
// The permutation parity reported is that of the pivoting actually used.
//
// Warps take matrices from a work counter rather than a fixed grid stride: a
// matrix refactorised in FP64 costs many times an accepted one, and a fixed
// share of the batch per warp would leave the kernel waiting on the warps
// that drew the most of them. At n = 24 and 32 the refinements and FP64
// refactorisations run after the FP32 pass, in a second kernel on the same
// stream that has the whole GPU: the FP32 pass saves a matrix whose
// correction is within theta but beyond what FP32 solves carry (its L\U and
// Y = L^-1 R) for one refinement step of the back substitution, and appends
// the index of a rejected matrix to the call's pending list; the second
// kernel deals the list's entries out to its warps at a fixed stride for FP64
// while the other warps refine the saved matrices, so the FP64 and FP32 pipes
// work side by side; a third corrects the FP64 factors it listed. For n <= 16, where
// the FP64 refactorisations are cheap and rare enough that a second launch costs
// more than it saves, the FP32 pass refines and refactorises in place, and so does
// the n = 24, 32 variant that reads its batch over the host link
// (lup_mixed_tile_kernel); at 17 <= n <= 31 without a register-tiled rule the
// rejected matrices go to lup_mixed_fallback_kernel, but for small batches of
// n <= 23. The FP32 pass of every n <= 32 is the lane-grid kernel
// (mixed_grid.cuh). The kernels take their matrices from a source: dense matrices in
// the reference layout, or matrices built from coordinates or permutations.
//
// Every call owns its state: the work counter, the pending list (room for the
// whole batch), the saved matrices and the factor list sit in one block from the
// library's stream-ordered pool whose head is zeroed on the call's stream before
// the first kernel. Nothing is shared between calls, so any number of them may be
// in flight on any streams, and a captured call replays on its own memory. A call
// whose batch fits in two strides of its grid needs no counter (warps take
// matrices at a fixed stride) and, without a list, takes no block.

#pragma once

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "bulk_copy.cuh"
#include "lup_fp64_sub.cuh"
#include "mixed_core.cuh"
#include "mixed_grid.cuh"

namespace lufqhe {

extern int g_tile_warps;     // warps per CTA of the tile kernels (option 2)
extern int g_mixed_refine;   // refinement of the back substitution (option 5)
extern float g_mixed_theta;  // ||E||_F threshold (option 1)
unsigned int fp64_share_64k(int n);
size_t mixed_smem_per_warp(int n);

namespace {

using namespace mixed;

// Warps per CTA and CTAs per SM the register-tiled kernels are compiled for:
// the register budget this leaves (65536 / (32 warps blocks)) is what lets the
// SM hold that many warps, whichever of registers or shared memory binds.
// n = 24: 3-warp CTAs, 5 per SM (15 KB of shared memory per warp); n = 32:
// shared memory allows 8 warps whatever the registers.
constexpr int tile_max_warps(int n) { return n == 24 ? 3 : 4; }
constexpr int tile_min_ctas(int n) { return n == 24 ? 5 : 1; }

// Head of a call's state block (zeroed on the call's stream before the first
// kernel). Behind it: the pending list of the FP64 pass (one entry per matrix
// of the batch at most), then the saved matrices of the refinement.
struct CallHead {
  unsigned long long claim;           // FP32 pass: claims after each warp's first matrix
  unsigned long long refine_saved;    // saved matrices (may exceed the capacity)
  unsigned long long refine_claimed;  // claimed by the finish kernel
  unsigned int pend_count;            // entries of the pending list
  unsigned int pad;
  unsigned long long corr_count;      // host-link variant: matrices listed for the correction
};
constexpr size_t kHeadBytes = 256;

// A warp's first matrix is its own index in the grid; later ones come from the
// call's counter (after the grid's warps), or, for a call that needs none (a batch
// within two strides of the grid), at the grid's stride. Small batches, where
// most warps take one matrix, then make no same-address atomics at the start
// (n=8, 4096 matrices: 31.0 -> 28.9 us).
__device__ __forceinline__ long long claim_matrix(CallHead *head, int lane, long long prev) {
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  if (prev < 0) return (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (!head) return prev + warps;
  unsigned long long b = 0;
  if (lane == 0) b = atomicAdd(&head->claim, 1ull);
  return (long long)__shfl_sync(kFull, b, 0) + warps;
}

// List entries: the matrix index, with this bit set for the FP64 route (status
// flag LUFQHE_ST_FP64) rather than a rejection (LUFQHE_ST_FALLBACK).
constexpr unsigned int kPendRouted = 0x80000000u;

// Matrices per SM up to which a batch of 17 <= n <= 23 refactorises in place: one
// launch and no state block (64 Gaussian matrices of n = 20: 39.0 us with a second
// kernel, 35.5 in place; 500 LLL 147, 136; 1000 LLL 160, 150). Beyond that the
// rejected matrices of an SM wait for one another (2280 LLL: 176 listed, 196).
constexpr long long kInplaceMaxPerSm = 8;
// The same of the lane-grid kernels: shared memory holds 16 warps an SM at
// NP = 16 (13.5 KB each), 15 at 24 (14.8 KB) and 8 at 32 (25.7 KB).
constexpr int grid_warps(int np) { return np == 24 ? 3 : 4; }
// (n = 32 itself is compiled for 3 CTAs although 2 fit: with 168 registers instead
// of 255 the compiler moves less code ahead of its use, 412 us instead of 557
// for 8192 LLL matrices; the padded sizes gain from the 255.)
constexpr int grid_min_ctas(int np, int nc) { return np == 24 ? 5 : np == 32 ? (nc ? 3 : 2) : 4; }
// Warps of the FP64 pass's CTA (one CTA per SM).
constexpr int kFallbackMaxWarps = 20;
// Warps of a CTA of the correction pass after the finish kernel.
constexpr int kFacCorrectWarps = 4;

// Hand matrix b to the FP64 pass (the list has room for every matrix).
__device__ __forceinline__ void defer_fp64(CallHead *head, unsigned int *pend, long long b,
                                           int lane, bool routed) {
  if (lane == 0) {
    const unsigned int pos = atomicAdd(&head->pend_count, 1u);
    pend[pos] = (unsigned int)b | (routed ? kPendRouted : 0u);
  }
}

// Matrices the FP32 pass leaves for a refinement of the back substitution
// (TILE_REFINE): per matrix a header and the warp's L\U and Y = L^-1 R as they
// lie in shared memory (row stride N + 1), in the call's state block (counted
// by the head's refine_saved / refine_claimed).
struct RefineHead {
  long long b;
  int exp_sum, par, prod_e, pad;
  float xh, xl, yh, yl;
};
template <int N>
constexpr size_t refine_entry_bytes() {
  return (sizeof(RefineHead) + 2 * (size_t)N * (N + 1) * sizeof(float2) + 15) & ~(size_t)15;
}
// Share of a batch the refinement buffer has room for (the rest go straight
// to the FP64 pass): on lowest-Landau-level n = 24 matrices about 9% qualify.
constexpr double kRefineShare = 0.25;

// The host-link variant refactorises rejected matrices in place (it waits on
// the link and has compute to spare) but hands their extended-precision
// correction, whose latency would hold the warp off the link for the length
// of several factorisations, to a pass of its own (the factor list with the
// matrix from the warp's device copy, FacList); the device path's finish
// kernel lists its factorisations the same way, without the copy. Share of a
// batch the list has room for (beyond it the warp corrects in place):
constexpr double kCorrShare = 0.25;
// Sources whose matrices the correction pass reads from a copy in the list:
// all but a dense device batch (rows built from coordinates would be built
// again entry by entry for the residual).
template <class Src>
constexpr int fac_copies() {
  return std::is_same<Src, DenseSource>::value ? 0 : 1;
}

// Save a TILE_REFINE matrix (F at row stride ldf); false (warp-uniform) if the
// buffer is full.
template <int N>
__device__ __noinline__ bool save_refine(CallHead *head, unsigned char *buf, long long cap, long long b,
                            const float2 *F, int ldf, const float2 *Rm, const CFF &prod,
                            int exp_sum, int par, int lane) {
  constexpr int NL = N * (N + 1);
  unsigned long long k = 0;
  if (lane == 0) k = atomicAdd(&head->refine_saved, 1ull);
  k = __shfl_sync(kFull, k, 0);
  if (k >= (unsigned long long)cap) return false;
  unsigned char *e = buf + k * refine_entry_bytes<N>();
  float2 *dF = reinterpret_cast<float2 *>(e + sizeof(RefineHead));
  float2 *dY = dF + NL;
  for (int q = lane; q < NL; q += 32) {
    dF[q] = F[q + q / (N + 1) * (ldf - (N + 1))];
    dY[q] = Rm[q];
  }
  if (lane == 0) {
    RefineHead h;
    h.b = b;
    h.exp_sum = exp_sum;
    h.par = par;
    h.prod_e = prod.e;
    h.pad = 0;
    h.xh = prod.xh;
    h.xl = prod.xl;
    h.yh = prod.yh;
    h.yl = prod.yl;
    *reinterpret_cast<RefineHead *>(e) = h;
  }
  return true;
}

// The FP32 pass above n = 32, where the precision policy takes it (a share below 1
// under LUFQHE_OPT_FP64_SHARE): a warp per matrix in shared memory, the rejected
// matrices to the call's pending list.
template <class Src>
__global__ void __launch_bounds__(kMaxWarpsMixed * 32)
    lup_mixed_kernel(Src src, int n, long long batch,
                     float theta2, unsigned int share64k, CallHead *head, unsigned int *pend,
                     double *__restrict__ logabs, double *__restrict__ phase,
                     int8_t *__restrict__ parity, int32_t *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int lds = n + 1;
  const size_t nl = (size_t)n * lds;
  MixedSmem S;
  unsigned char *base = smem_raw;
  S.SC = reinterpret_cast<float4 *>(base) + warp * nl;
  base += warps * nl * sizeof(float4);
  S.Af = reinterpret_cast<float2 *>(base) + warp * nl;
  base += warps * nl * sizeof(float2);
  S.hold = reinterpret_cast<double *>(base) + warp * 2 * n;
  base += warps * 2 * (size_t)n * sizeof(double);
  S.er = reinterpret_cast<int *>(base) + warp * 2 * n;
  S.ec = S.er + n;
  const CorrScratch cs{S.Af, S.er, S.hold};

  DeferredOut out;
  for (long long b = claim_matrix(head, lane, -1); b < batch; b = claim_matrix(head, lane, b)) {
    __syncwarp();
    double2 *M = reinterpret_cast<double2 *>(S.SC);
    if (share64k && route_fp64_entry(src.first(b, n), share64k)) {
      fallback_fp64_src(src, b, n, M, lds, S.hold, lane, b, logabs, phase, parity, status,
                        LUFQHE_ST_FP64, &cs);
      continue;
    }
    if (src.load(b, n, M, lds, lane)) {
      emit_nonfinite(lane, b, logabs, phase, parity, status);
      continue;
    }
    CFF prod;
    int exp_sum, par;
    float2 corr;
    if (mixed_factor(S, n, lane, theta2, prod, exp_sum, corr, par))
      out.push(lane, b, prod, exp_sum, corr, par, logabs, phase, parity, status);
    else
      defer_fp64(head, pend, b, lane, false);
  }
  out.flush(lane, logabs, phase, parity, status);
}


// The FP32 pass of the lane-grid path: each warp takes Grid::G consecutive
// matrices at a time. NC = n for the register-tiled sizes, 0 for the generic
// rule. FORM says where the matrices go that it does not accept:
//  GRID_DEFER: to the call's pending list, and (n = 24, 32) those to refine to the
//    saved matrices;
//  GRID_INPLACE: refined or refactorised in FP64 right away, one at a time by the
//    whole warp;
//  .._ROUTED: so too, and the matrices that the policy routes to FP64 (share64k) to
//    the pending list, or, in place where a warp takes one matrix at a time, to FP64
//    right away. Forms of their own, so that a call without a routed share runs
//    none of that code (with one code for both: 65536 LLL x n=16 669 us against 648,
//    8192 LLL x n=27 750 against 704). GRID_DEFER keeps grid_unit's own look at the
//    share, which never finds one there: without it the compiler's schedule of the
//    padded n = 25..31 is 4% slower (8192 Gaussian x n=27 430 us against 416).
enum GridForm { GRID_INPLACE, GRID_INPLACE_ROUTED, GRID_DEFER, GRID_DEFER_ROUTED };
constexpr bool grid_defers(int form) { return form == GRID_DEFER || form == GRID_DEFER_ROUTED; }
constexpr bool grid_routes(int form) {
  return form == GRID_INPLACE_ROUTED || form == GRID_DEFER_ROUTED;
}
template <int NP, int LPM, int NC, int FORM, class Src>
__global__ void __launch_bounds__(grid_warps(NP) * 32, grid_min_ctas(NP, NC))
    lup_mixed_grid_kernel(Src src, int n_rt, long long batch, float theta2,
                          unsigned int share64k, CallHead *claims, CallHead *head,
                          unsigned int *pend, int refine, unsigned char *saved, long long saved_cap,
                          int bulk, double *__restrict__ logabs, double *__restrict__ phase,
                          int8_t *__restrict__ parity, int32_t *__restrict__ status) {
  using Gd = Grid<NP, LPM>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr bool DEFER = grid_defers(FORM);
  constexpr bool BULK = std::is_same<Src, DenseSource>::value;
  const int n = NC ? NC : n_rt;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char *base = smem_raw + (size_t)warp * Gd::kWarpBytes;
  float4 *HLw = reinterpret_cast<float4 *>(base);
  float2 *Fw = reinterpret_cast<float2 *>(HLw + Gd::G * Gd::kHL);
  int *Iw = reinterpret_cast<int *>(Fw + Gd::G * Gd::kF);
  double2 *M = reinterpret_cast<double2 *>(HLw);
  __shared__ __align__(8) uint64_t bars[grid_warps(NP)];
  WarpBulk wb;
  if constexpr (BULK)
    if (bulk) wb.init(&bars[warp], lane);

  DeferredOut out;
  const long long units = (batch + Gd::G - 1) / Gd::G;
  long long u = claim_matrix(claims, lane, -1);
  long long nu = u < units ? claim_matrix(claims, lane, u) : units;
  for (; u < units; u = nu, nu = u < units ? claim_matrix(claims, lane, u) : units) {
    const long long b0 = u * Gd::G;
    const int cnt = (int)min((long long)Gd::G, batch - b0);
    // a unit of routed matrices alone is not staged
    if (grid_routes(FORM) && share64k) {
      const int grp = lane / Gd::LPM;
      if (__all_sync(kFull, grp >= cnt || route_fp64_entry(src.first(b0 + grp, n), share64k))) {
        if constexpr (DEFER || Gd::G > 1)
          for (int q = 0; q < cnt; ++q) defer_fp64(head, pend, b0 + q, lane, true);
        else
          grid_refactor<NP>(src, b0, n, HLw, Fw, Iw, lane, b0, logabs, phase, parity, status,
                            LUFQHE_ST_FP64);
        continue;
      }
    }
    __syncwarp();
    bool staged = false;
    if constexpr (BULK) {
      if (bulk && !wb.broken) {
        if (nu < units && lane == 0) {
          const int ncnt = (int)min((long long)Gd::G, batch - nu * Gd::G);
          prefetch_rows_l2(src.A + (size_t)(nu * Gd::G) * n * src.lda, ncnt * n, n, src.lda);
        }
        if (!wb.load_rows(src.A + (size_t)b0 * n * src.lda, cnt * n, n, src.lda, M, Gd::LDH, NP,
                          lane)) {
          for (int q = 0; q < cnt; ++q)
            emit_wait_timeout(lane, b0 + q, logabs, phase, parity, status);
          continue;
        }
        staged = true;
      }
    }
    if (!staged) load_rows(src, b0, cnt * n, n, M, Gd::LDH, NP, lane);
    __syncwarp();
    // DEFER: a matrix within theta but above the FP32 solves' cap gets its back
    // substitution refined by the next pass, if the buffer has room; the others
    // are listed for FP64
    grid_unit<NP, LPM, NC, !DEFER, false>(
        src, b0, b0, cnt, n, HLw, Fw, Iw, lane, theta2,
        FORM == GRID_INPLACE || (!DEFER && Gd::G == 1) ? 0u : share64k, refine != 0,
        [](int q) { return q; },
        [&](long long b, bool routed, bool can_refine, const CFF &prod, int exp_sum, int par) {
          if constexpr (NC != 0)
            if (can_refine && saved &&
                save_refine<NC>(head, saved, saved_cap, b, Fw, Gd::LDF,
                                reinterpret_cast<const float2 *>(HLw), prod, exp_sum, par, lane))
              return;
          defer_fp64(head, pend, b, lane, routed);
        },
        out, logabs, phase, parity, status);
  }
  out.flush(lane, logabs, phase, parity, status);
}


// n = 24 and 32, a batch in mapped host memory: the FP32 path with everything
// else in place (the kernel waits on the link and has compute to spare), except
// the corrections of its FP64 refactorisations, which are listed for a pass of
// their own.
template <int N>
__global__ void __launch_bounds__(tile_max_warps(N) * 32, tile_min_ctas(N))
    lup_mixed_tile_kernel(DenseSource src, long long batch, float theta2, unsigned int share64k,
                          CallHead *head, double2 *spill, int refine, unsigned char *corr_list,
                          long long corr_cap, double *__restrict__ logabs,
                          double *__restrict__ phase, int8_t *__restrict__ parity,
                          int32_t *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LDS = N + 1;
  constexpr size_t NL = (size_t)N * LDS;
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  unsigned char *base = smem_raw;
  float4 *HL = reinterpret_cast<float4 *>(base) + warp * NL;
  base += warps * NL * sizeof(float4);
  float2 *F = reinterpret_cast<float2 *>(base) + warp * NL;
  base += warps * NL * sizeof(float2);
  double *hold = reinterpret_cast<double *>(base) + warp * 2 * N;
  base += warps * 2 * (size_t)N * sizeof(double);
  int *er = reinterpret_cast<int *>(base) + warp * 2 * N;
  int *ec = er + N;
  const CorrScratch cs{F, er, hold};
  // this warp's copy of its current matrix in global memory (a few KB per warp,
  // so the copies stay in L2); an FP64 refactorisation reloads it from there
  // instead of reading the matrix over the host link again
  double2 *own = spill + ((size_t)blockIdx.x * warps + warp) * N * N;

  DeferredOut out;
  long long b = claim_matrix(head, lane, -1);
  long long nb = b < batch ? claim_matrix(head, lane, b) : batch;
  for (; b < batch; b = nb, nb = b < batch ? claim_matrix(head, lane, b) : batch) {
    __syncwarp();
    double2 *M = reinterpret_cast<double2 *>(HL);
    if (share64k && route_fp64_entry(src.first(b, N), share64k)) {
      fallback_fp64_src(src, b, N, M, LDS, hold, lane, b, logabs, phase, parity, status,
                        LUFQHE_ST_FP64, &cs);
      continue;
    }
    if (src.load(b, N, M, LDS, lane)) {
      emit_nonfinite(lane, b, logabs, phase, parity, status);
      continue;
    }
    {
      BlockWalk w(lane, N);
      for (int e = lane; e < N * N; e += 32) {
        own[e] = M[w.i * LDS + w.k];
        w.next(N);
      }
    }
    CFF prod;
    int exp_sum, par;
    float2 corr;
    const int code =
        mixed_factor_tile_ex<N, true>(HL, F, er, ec, lane, theta2, prod, exp_sum, corr, par);
    if (code == TILE_ACCEPT ||
        (code == TILE_REFINE && refine &&
         mixed_refine_tile<N>(F, reinterpret_cast<float2 *>(HL),
                              reinterpret_cast<float2 *>(HL) + N * (N + 1),
                              reinterpret_cast<float2 *>(er), lane, theta2,
                              tile_la_est(prod, exp_sum), corr))) {
      out.push(lane, b, prod, exp_sum, corr, par, logabs, phase, parity, status);
    } else {
      // the factors (and the warp's copy of the matrix) are listed for the
      // correction pass, so that no warp stops reading the link for one
      const FacList fl{&head->corr_count, corr_list, corr_cap, 1};
      fallback_fp64_src<DenseSource, true>(DenseSource{own, N}, 0, N, M, LDS, hold, lane, b,
                                           logabs, phase, parity, status, LUFQHE_ST_FALLBACK,
                                           &cs, &fl);
    }
  }
  out.flush(lane, logabs, phase, parity, status);
}

// The passes after the FP32 pass, as one kernel in the tile path's
// shared-memory layout (n = 24, 32): the FP64 refactorisations of the matrices
// the FP32 pass rejected, dealt out at a fixed stride over the grid's warps
// first, while the warps without one refine the saved matrices (claimed one at
// a time; a refinement that fails is refactorised in FP64 on the spot). The
// FP64 pipe and the FP32 pipes then work side by side instead of one pass
// after the other.
template <int N, class Src>
__global__ void __launch_bounds__(tile_max_warps(N) * 32, tile_min_ctas(N))
    lup_mixed_finish_kernel(Src src, CallHead *head, const unsigned int *pend,
                            const unsigned char *refine, long long refine_cap, float theta2,
                            unsigned char *fac, long long fac_cap,
                            double *__restrict__ logabs, double *__restrict__ phase,
                            int8_t *__restrict__ parity, int32_t *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LDS = N + 1;
  constexpr size_t NL = (size_t)N * LDS;
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  unsigned char *base = smem_raw;
  float4 *HL = reinterpret_cast<float4 *>(base) + warp * NL;
  double2 *M = reinterpret_cast<double2 *>(HL);
  float2 *Rm = reinterpret_cast<float2 *>(HL);
  base += warps * NL * sizeof(float4);
  float2 *F = reinterpret_cast<float2 *>(base) + warp * NL;
  base += warps * NL * sizeof(float2);
  double *hold = reinterpret_cast<double *>(base) + warp * 2 * N;
  base += warps * 2 * (size_t)N * sizeof(double);
  float2 *diag = reinterpret_cast<float2 *>(reinterpret_cast<int *>(base) + warp * 2 * N);
  const CorrScratch cs{F, reinterpret_cast<int *>(diag), hold};
  // the corrections of the FP64 factorisations go to lup_mixed_fac_correct_kernel
  const FacList fl{&head->corr_count, fac, fac_cap, fac_copies<Src>()};
  // 1. the FP32 pass's rejections, dealt out
  const unsigned long long listed = head->pend_count;
  const unsigned long long stride = (unsigned long long)warps * gridDim.x;
  for (unsigned long long j = (unsigned long long)warp * gridDim.x + blockIdx.x; j < listed;
       j += stride) {
    const unsigned int e = pend[j];
    const long long b = e & ~kPendRouted;
    fallback_fp64_src(src, b, N, M, LDS, hold, lane, b, logabs, phase, parity, status,
                      (e & kPendRouted) ? LUFQHE_ST_FP64 : LUFQHE_ST_FALLBACK, &cs, &fl);
  }
  // 2. the saved matrices, claimed; a failed refinement is refactorised here
  DeferredOut out;
  if (refine) {
    unsigned long long *claimed = const_cast<unsigned long long *>(&head->refine_claimed);
    const unsigned long long saved = min(head->refine_saved, (unsigned long long)refine_cap);
    for (;;) {
      unsigned long long k = saved;
      if (lane == 0 && *(volatile unsigned long long *)claimed < saved)
        k = atomicAdd(claimed, 1ull);
      k = __shfl_sync(kFull, k, 0);
      if (k >= saved) break;
      const unsigned char *e = refine + k * refine_entry_bytes<N>();
      const RefineHead h = *reinterpret_cast<const RefineHead *>(e);
      const float2 *sF = reinterpret_cast<const float2 *>(e + sizeof(RefineHead));
      const float2 *sY = sF + NL;
      __syncwarp();
      for (int q = lane; q < (int)NL; q += 32) {
        F[q] = __ldcg(sF + q);
        Rm[q] = __ldcg(sY + q);
      }
      __syncwarp();
      const CFF prod = {h.xh, h.xl, h.yh, h.yl, h.prod_e};
      float2 corr;
      if (mixed_refine_tile<N>(F, Rm, Rm + NL, diag, lane, theta2, tile_la_est(prod, h.exp_sum),
                               corr))
        out.push(lane, h.b, prod, h.exp_sum, corr, h.par, logabs, phase, parity, status);
      else
        fallback_fp64_src(src, h.b, N, M, LDS, hold, lane, h.b, logabs, phase, parity, status,
                          LUFQHE_ST_FALLBACK, &cs, &fl);
    }
  }
  out.flush(lane, logabs, phase, parity, status);
}

// The corrections of the finish kernel's FP64 factorisations (n = 24, 32):
// entry j of the list by CTA j % grid with all its warps (the inlined
// fp64_correct_group, whose result is fp64_correct_warp's bit for bit), on the
// listed L\U and pivot order and the source's matrix. One warp per matrix,
// the factorisation (~92 us on a sub-partition's shared FP64 pipe) and then
// the correction (120-177 us) on the same warp had been the finish kernel's
// critical path.
// COPY: the entries carry the matrix (the host-link variant's list), which is
// the source of the residual instead of src.
// Compiled for 8 CTAs per SM (32768 LLL x n=24, us: 114 without a bound, 107.5
// for 8, 111 for 9; n = 32 the same, whose shared memory allows 8).
template <int N, class Src, bool COPY = false>
__global__ void __launch_bounds__(kFacCorrectWarps * 32, 8)
    lup_mixed_fac_correct_kernel(Src src, const CallHead *head, const unsigned char *fac,
                                 long long fac_cap, double *__restrict__ logabs,
                                 double *__restrict__ phase, int8_t *__restrict__ parity,
                                 int32_t *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long red[3 * kFacCorrectWarps];
  constexpr int LDS = N + 1;
  const int tid = threadIdx.x, nthr = blockDim.x;
  double2 *M = reinterpret_cast<double2 *>(smem_raw);
  double *hold = reinterpret_cast<double *>(M + (size_t)N * LDS);
  float2 *F = reinterpret_cast<float2 *>(hold + 2 * N);
  int *ints = reinterpret_cast<int *>(F + (size_t)N * LDS);
  const CorrScratch cs{F, ints, hold};
  const unsigned long long listed = min(head->corr_count, (unsigned long long)fac_cap);
  for (unsigned long long j = blockIdx.x; j < listed; j += gridDim.x) {
    const unsigned char *e = fac + j * fac_entry_bytes(N, COPY);
    const FacHead h = *reinterpret_cast<const FacHead *>(e);
    const int *pe = reinterpret_cast<const int *>(e + sizeof(FacHead));
    const double2 *fe = reinterpret_cast<const double2 *>(e + fac_factors_offset(N));
    __syncthreads();  // the previous entry's correction is done with the scratch
    for (int i = tid; i < N; i += nthr) ints[i] = __ldcg(pe + i);
    for (int q = tid; q < N * N; q += nthr) M[(q / N) * LDS + q % N] = __ldcg(fe + q);
    __syncthreads();
    double2 c;
    if constexpr (COPY)
      c = fp64_correct_group(DenseSource{reinterpret_cast<const double2 *>(e + fac_copy_offset(N)),
                                         N},
                             0, N, M, LDS, cs, tid, nthr, CtaBarrier(),
                             reinterpret_cast<float *>(red));
    else
      c = fp64_correct_group(src, h.b, N, M, LDS, cs, tid, nthr, CtaBarrier(),
                             reinterpret_cast<float *>(red));
    if (tid == 0) {
      logabs[h.b] = h.la + c.x;
      if (phase) phase[h.b] = h.ph + c.y;
      if (parity) parity[h.b] = (int8_t)h.par;
      if (status) status[h.b] = h.flag;
    }
  }
}

// The FP64 pass of the sizes without a register-tiled kernel (17 <= n <= 31, and
// above 32): one CTA per SM; its warps refactorise the pending list's matrices
// (reference pivot rule, fused arithmetic, status flag LUFQHE_ST_FALLBACK, or
// LUFQHE_ST_FP64 for the routed share). Every factorisation of one n costs the
// same, so the entries are dealt out at a fixed stride: entry j goes to warp
// j / G of CTA j % G (G CTAs), so the first G entries land on warp 0 of every
// SM, the next G on warp 1 (the next SM sub-partition), and no sub-partition's
// FP64 pipe holds more than ceil(count / (4 G)) of them when the list is
// short. (First-come claims piled up to five matrices on some sub-partitions
// while others idled.)
template <class Src>
__global__ void __launch_bounds__(kFallbackMaxWarps * 32)
    lup_mixed_fallback_kernel(Src src, int n, const CallHead *head, const unsigned int *pend,
                              double *__restrict__ logabs, double *__restrict__ phase,
                              int8_t *__restrict__ parity, int32_t *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int lds = n + 1;
  double2 *M = reinterpret_cast<double2 *>(smem_raw) + (size_t)warp * n * lds;
  double *hold_all = reinterpret_cast<double *>(reinterpret_cast<double2 *>(smem_raw) +
                                                (size_t)warps * n * lds);
  double *hold = hold_all + warp * 2 * n;
  // n <= kCorrectMaxN: the correction's scratch after the row scales
  // (fallback_smem_per_warp)
  float2 *F_all = reinterpret_cast<float2 *>(hold_all + (size_t)warps * 2 * n);
  const CorrScratch cs{F_all + (size_t)warp * n * lds,
                       reinterpret_cast<int *>(F_all + (size_t)warps * n * lds) + warp * 2 * n,
                       hold};
  const unsigned long long listed = head->pend_count;
  const unsigned long long stride = (unsigned long long)warps * gridDim.x;
  for (unsigned long long j = (unsigned long long)warp * gridDim.x + blockIdx.x; j < listed;
       j += stride) {
    const unsigned int e = pend[j];
    const long long b = e & ~kPendRouted;
    fallback_fp64_src(src, b, n, M, lds, hold, lane, b, logabs, phase, parity, status,
                      (e & kPendRouted) ? LUFQHE_ST_FP64 : LUFQHE_ST_FALLBACK,
                      n <= kCorrectMaxN ? &cs : nullptr);
  }
}

// The FP64 pass of the routed share at n <= 16 (LUFQHE_OPT_FP64_SHARE): the
// listed matrices several per warp, as the plain kernels take them (lup_fp64_warp's
// bits). In the FP32 pass, a warp per matrix between its units, they cost twice as
// much and held up the other half of a unit (65536 x n=16, a quarter routed, us:
// Gaussian 985 in place, 785 listed; n=8 361 and 196).
template <int LPM, class Src>
__global__ void __launch_bounds__(128)
    lup_mixed_routed_kernel(Src src, int n, const CallHead *head, const unsigned int *pend,
                            double *__restrict__ logabs, double *__restrict__ phase,
                            int8_t *__restrict__ parity, int32_t *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int G = 32 / LPM;
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane / LPM, sub = lane % LPM, lds = n | 1;
  const unsigned gmask = ((1u << LPM) - 1u) << (grp * LPM);
  double2 *Mw = reinterpret_cast<double2 *>(smem_raw) + (size_t)warp * G * n * lds;
  double2 *M = Mw + (size_t)grp * n * lds;
  double *hold = reinterpret_cast<double *>(reinterpret_cast<double2 *>(smem_raw) +
                                            (size_t)warps * G * n * lds) +
                 (size_t)(warp * G + grp) * 2 * n;
  const long long listed = head->pend_count;
  const long long stride = (long long)gridDim.x * warps * G;
  for (long long j0 = ((long long)blockIdx.x * warps + warp) * G; j0 < listed; j0 += stride) {
    const int cnt = (int)min((long long)G, listed - j0);
    const bool valid = grp < cnt;
    const unsigned int b = valid ? pend[j0 + grp] & ~kPendRouted : 0u;
    __syncwarp();
    for (int q = 0; q < cnt; ++q)
      load_rows(src, __shfl_sync(kFull, b, q * LPM), n, n, Mw + (size_t)q * n * lds, lds, n, lane);
    __syncwarp();
    int par = 0;
    const int st = lup_fp64_sub<ARITH_FUSED, LPM>(M, lds, hold, n, sub, gmask, valid, &par);
    double la, ph;
    logdet_from_diag_sub<LPM>(M, lds, n, sub, valid && st == 0, par, &la, &ph);
    if (!valid || sub != 0) continue;
    if (st != 0) {
      la = st == LUFQHE_ST_SINGULAR ? -INFINITY : NAN;
      ph = st == LUFQHE_ST_SINGULAR ? 0.0 : NAN;
      if (st != LUFQHE_ST_SINGULAR) par = 0;
    }
    logabs[b] = la;
    if (phase) phase[b] = ph;
    if (parity) parity[b] = (int8_t)par;
    if (status) status[b] = st == LUFQHE_ST_NONFINITE ? st : st | LUFQHE_ST_FP64;
  }
}

// the bulk-copy staging for complex128 matrices in device memory only
inline int bulk_for(const DenseSource &s) { return g_bulk_loads && is_device_memory(s.A); }
template <class S>
inline int bulk_for(const S &) {
  return 0;
}

// A call's state block: the head, the pending list (pend_cap entries), the
// saved matrices of the refinement (refine_bytes) and the host-link copies
// (spill_bytes), each 256-byte aligned; the head is zeroed on `stream`.
struct CallState {
  unsigned char *block = nullptr;
  CallHead *head = nullptr;
  unsigned int *pend = nullptr;
  unsigned char *refine = nullptr;
  double2 *spill = nullptr;
  unsigned char *corr = nullptr;

  int acquire(size_t pend_cap, size_t refine_bytes, size_t spill_bytes, cudaStream_t stream,
              size_t corr_bytes = 0) {
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t pend_bytes = up(pend_cap * sizeof(unsigned int));
    const size_t total =
        kHeadBytes + pend_bytes + up(refine_bytes) + up(spill_bytes) + up(corr_bytes);
    int rc = lib_malloc_async((void **)&block, total, stream);
    if (rc) return rc;
    head = reinterpret_cast<CallHead *>(block);
    unsigned char *p = block + kHeadBytes;
    pend = pend_cap ? reinterpret_cast<unsigned int *>(p) : nullptr;
    p += pend_bytes;
    refine = refine_bytes ? p : nullptr;
    p += up(refine_bytes);
    spill = spill_bytes ? reinterpret_cast<double2 *>(p) : nullptr;
    p += up(spill_bytes);
    corr = corr_bytes ? p : nullptr;
    return check_cuda(cudaMemsetAsync(block, 0, kHeadBytes, stream), "memset(call state)");
  }
  int release(cudaStream_t stream, int rc) {
    if (!block) return rc;
    const int r2 = lib_free_async(block, stream);
    block = nullptr;
    return rc ? rc : r2;
  }
};

// Whether warps must claim matrices from a counter: a batch beyond two strides
// of the grid. (The calls at n = 24 and 32, which take a state block anyway, and
// those above 32 claim from the block's zeroed counter regardless.)
inline bool needs_counter(long long batch, long long grid_warps) {
  return batch > 2 * grid_warps;
}

// Shared memory of one warp of the FP64 pass: the matrix and its row scales;
// for n <= kCorrectMaxN also the correction's float2 matrix and 2n ints.
inline size_t fallback_smem_per_warp(int n) {
  size_t b = (size_t)n * (n + 1) * sizeof(double2) + 2 * (size_t)n * sizeof(double);
  if (n <= kCorrectMaxN) b += (size_t)n * (n + 1) * sizeof(float2) + 2 * (size_t)n * sizeof(int);
  return b;
}

// Shared-memory limit, and the grid of `warps`-warp CTAs over `units` units.
template <class K>
int grid_geometry(K kern, int warps, size_t smem, long long units, int *grid) {
  int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem),
                      "cudaFuncSetAttribute(mixed)");
  if (rc) return rc;
  int per_sm = 0;
  rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, smem),
                  "occupancy(mixed)");
  if (rc) return rc;
  const long long want = (units + warps - 1) / warps;
  const long long cap = (long long)device_sm_count() * std::max(1, per_sm);
  *grid = (int)std::min(want, cap);
  return LUFQHE_SUCCESS;
}

template <class Src>
int launch_fallback(Src src, int n, const CallHead *head, const unsigned int *pend,
                    long long batch, double *logabs, double *phase, int8_t *parity,
                    int32_t *status, cudaStream_t stream) {
  const size_t per_warp = fallback_smem_per_warp(n);
  int warps = (int)(device_smem_optin() / per_warp);
  if (warps > kFallbackMaxWarps) warps = kFallbackMaxWarps;
  if (warps < 1) warps = 1;
  const size_t smem = per_warp * warps;
  auto kern = lup_mixed_fallback_kernel<Src>;
  int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem),
                      "cudaFuncSetAttribute(mixed fallback)");
  if (rc) return rc;
  int per_sm = 0;
  rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, smem),
                  "occupancy(mixed fallback)");
  if (rc) return rc;
  if (per_sm < 1) {
    set_error("mixed fallback: n=%d does not fit on an SM", n);
    return LUFQHE_ERR_UNSUPPORTED_N;
  }
  // one CTA per SM (the list's length is known only on the device)
  long long want = (batch + warps - 1) / warps;
  long long cap = (long long)device_sm_count();
  int grid = (int)(want < cap ? want : cap);
  KernelTimer timer("lup_mixed_fallback_kernel", n, stream);
  kern<<<grid, warps * 32, smem, stream>>>(src, n, head, pend, logabs, phase, parity, status);
  timer.stop();
  return check_cuda(cudaGetLastError(), "lup_mixed_fallback_kernel launch");
}

template <int LPM, class Src>
int launch_routed(Src src, int n, const CallHead *head, const unsigned int *pend, long long batch,
                  double *logabs, double *phase, int8_t *parity, int32_t *status,
                  cudaStream_t stream) {
  auto kern = lup_mixed_routed_kernel<LPM, Src>;
  const int warps = sub_warps(n, LPM);
  const size_t smem = sub_smem(n, LPM);
  int grid = 0;
  const int rc = grid_geometry(kern, warps, smem, (batch + 32 / LPM - 1) / (32 / LPM), &grid);
  if (rc) return rc;
  KernelTimer timer("lup_mixed_routed_kernel", n, stream);
  kern<<<grid, warps * 32, smem, stream>>>(src, n, head, pend, logabs, phase, parity, status);
  timer.stop();
  return check_cuda(cudaGetLastError(), "lup_mixed_routed_kernel launch");
}

// The correction pass over a factor list of capacity cap (its length is
// known only on the device): as many CTAs as fit, at most one per entry.
template <int N, class Src, bool COPY>
int launch_fac_correct(Src src, const CallHead *head, const unsigned char *list, long long cap,
                       double *logabs, double *phase, int8_t *parity, int32_t *status,
                       cudaStream_t stream) {
  auto k = lup_mixed_fac_correct_kernel<N, Src, COPY>;
  const size_t smem = fallback_smem_per_warp(N);
  int rc = check_cuda(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem),
                      "cudaFuncSetAttribute(mixed fac correct)");
  int per_sm = 0;
  if (!rc)
    rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k,
                                                                  kFacCorrectWarps * 32, smem),
                    "occupancy(mixed fac correct)");
  if (rc) return rc;
  const long long fit = (long long)device_sm_count() * std::max(1, per_sm);
  const int grid = (int)std::min<long long>(cap, fit);
  KernelTimer timer(COPY ? "lup_mixed_fac_correct_kernel_hostlink" : "lup_mixed_fac_correct_kernel",
                    N, stream);
  k<<<grid, kFacCorrectWarps * 32, smem, stream>>>(src, head, list, cap, logabs, phase, parity,
                                                   status);
  timer.stop();
  return check_cuda(cudaGetLastError(), "lup_mixed_fac_correct_kernel launch");
}

// Warps per CTA of a register-tiled size's kernel that takes up to `most` (option 2).
inline int tuned_warps(int most) {
  return g_tile_warps > 0 && g_tile_warps < most ? g_tile_warps : most;
}
// The same of the in-place and finish kernels, in the tile layout.
template <int N>
int tile_warps() {
  return std::min((int)(device_smem_optin() / tile_smem_per_warp<N>()),
                  tuned_warps(tile_max_warps(N)));
}
// Room for `share` of a batch.
inline long long share_cap(double share, long long batch) {
  return std::min(batch, std::max<long long>(256, (long long)(share * (double)batch)));
}

// n = 24 and 32, a batch read over the host link: one kernel, then the
// corrections of its FP64 refactorisations.
template <int N>
int launch_mixed_hostlink(DenseSource src, long long batch, float theta2, double *logabs,
                          double *phase, int8_t *parity, int32_t *status, cudaStream_t stream) {
  auto kern = lup_mixed_tile_kernel<N>;
  const int warps = tile_warps<N>();
  const size_t smem = tile_smem_per_warp<N>() * warps;
  int grid = 0;
  int rc = grid_geometry(kern, warps, smem, batch, &grid);
  if (rc) return rc;
  const long long corr_cap = share_cap(kCorrShare, batch);
  CallState cs;
  rc = cs.acquire(0, 0, (size_t)grid * warps * N * N * sizeof(double2), stream,
                  (size_t)corr_cap * (size_t)fac_entry_bytes(N, true));
  if (rc) return cs.release(stream, rc);
  {
    KernelTimer timer("lup_mixed_tile_kernel_hostlink", N, stream);
    kern<<<grid, warps * 32, smem, stream>>>(src, batch, theta2, fp64_share_64k(N), cs.head,
                                             cs.spill, g_mixed_refine, cs.corr, corr_cap, logabs,
                                             phase, parity, status);
    timer.stop();
  }
  rc = check_cuda(cudaGetLastError(), "lup_mixed_tile_kernel launch");
  if (!rc)
    rc = launch_fac_correct<N, DenseSource, true>(src, cs.head, cs.corr, corr_cap, logabs, phase,
                                                  parity, status, stream);
  return cs.release(stream, rc);
}

// n = 24 and 32: the FP32 pass on the lane grid; the refinements and the FP64
// refactorisations it leaves, side by side in one kernel; the corrections of
// those refactorisations, each by a whole CTA.
template <int N, class Src>
int launch_mixed_tile(Src src, long long batch, float theta2, double *logabs, double *phase,
                      int8_t *parity, int32_t *status, cudaStream_t stream) {
  using Gd = Grid<N, 32>;
  auto kern = fp64_share_64k(N) ? lup_mixed_grid_kernel<N, 32, N, GRID_DEFER_ROUTED, Src>
                                : lup_mixed_grid_kernel<N, 32, N, GRID_DEFER, Src>;
  auto fk = lup_mixed_finish_kernel<N, Src>;
  const int gwarps = tuned_warps(grid_warps(N));
  const size_t gsmem = Gd::kWarpBytes * gwarps;
  const int fwarps = tile_warps<N>();
  const size_t fsmem = tile_smem_per_warp<N>() * fwarps;
  int grid = 0, fgrid = 0;
  int rc = grid_geometry(kern, gwarps, gsmem, batch, &grid);
  if (!rc) rc = grid_geometry(fk, fwarps, fsmem, batch, &fgrid);
  if (rc) return rc;
  const long long refine_cap = g_mixed_refine ? share_cap(kRefineShare, batch) : 0;
  // the list of FP64 factors (an overflow is corrected in the finish kernel)
  const long long fac_cap = share_cap(kCorrShare, batch);
  CallState cs;
  rc = cs.acquire((size_t)batch, (size_t)refine_cap * refine_entry_bytes<N>(), 0, stream,
                  (size_t)fac_cap * (size_t)fac_entry_bytes(N, fac_copies<Src>()));
  if (rc) return cs.release(stream, rc);
  {
    KernelTimer timer("lup_mixed_tile_kernel", N, stream);
    kern<<<grid, gwarps * 32, gsmem, stream>>>(src, N, batch, theta2, fp64_share_64k(N), cs.head,
                                               cs.head, cs.pend, g_mixed_refine, cs.refine,
                                               refine_cap, bulk_for(src), logabs, phase, parity,
                                               status);
    timer.stop();
  }
  rc = check_cuda(cudaGetLastError(), "lup_mixed_grid_kernel launch");
  if (!rc) {
    KernelTimer timer("lup_mixed_finish_kernel", N, stream);
    fk<<<fgrid, fwarps * 32, fsmem, stream>>>(src, cs.head, cs.pend, cs.refine, refine_cap, theta2,
                                              cs.corr, fac_cap, logabs, phase, parity, status);
    timer.stop();
    rc = check_cuda(cudaGetLastError(), "lup_mixed_finish_kernel launch");
  }
  if (!rc)
    rc = launch_fac_correct<N, Src, fac_copies<Src>() != 0>(src, cs.head, cs.corr, fac_cap, logabs,
                                                            phase, parity, status, stream);
  return cs.release(stream, rc);
}

template <int NP, int LPM, int NC, int FORM, class Src>
int launch_mixed_grid(Src src, int n, long long batch, float theta2, double *logabs,
                      double *phase, int8_t *parity, int32_t *status, cudaStream_t stream) {
  using Gd = Grid<NP, LPM>;
  auto kern = lup_mixed_grid_kernel<NP, LPM, NC, FORM, Src>;
  const int warps = NC ? tuned_warps(grid_warps(NP)) : grid_warps(NP);
  const size_t smem = Gd::kWarpBytes * warps;
  const long long units = (batch + Gd::G - 1) / Gd::G;
  int grid = 0;
  int rc = grid_geometry(kern, warps, smem, units, &grid);
  if (rc) return rc;
  // several matrices per warp: a routed share is listed
  constexpr bool list = grid_defers(FORM) || (grid_routes(FORM) && Gd::G > 1);
  // (a list alone does not make the warps claim: within two strides the first
  // ones to claim sat together on few SMs, 3000 x n=17 87 us by stride, 119 claimed)
  const bool counter = needs_counter(units, (long long)grid * warps);
  CallState cs;
  if (list || counter) {
    rc = cs.acquire(list ? (size_t)batch : 0, 0, 0, stream);
    if (rc) return cs.release(stream, rc);
  }
  {
    // (recorded under the names of the two rules)
    KernelTimer timer(NC ? "lup_mixed_tile_kernel" : "lup_mixed_kernel", n, stream);
    kern<<<grid, warps * 32, smem, stream>>>(src, n, batch, theta2, fp64_share_64k(n),
                                             counter ? cs.head : nullptr, cs.head, cs.pend,
                                             g_mixed_refine, nullptr, 0, bulk_for(src), logabs,
                                             phase, parity, status);
    timer.stop();
  }
  rc = check_cuda(cudaGetLastError(), "lup_mixed_grid_kernel launch");
  if constexpr (grid_defers(FORM)) {
    if (!rc)
      rc = launch_fallback(src, n, cs.head, cs.pend, batch, logabs, phase, parity, status, stream);
  } else if constexpr (list) {
    if (!rc)
      rc = launch_routed<Gd::LPM / 2>(src, n, cs.head, cs.pend, batch, logabs, phase, parity,
                                      status, stream);
  }
  return cs.release(stream, rc);
}

// n <= 16: several matrices per warp, except in a batch of at most one matrix
// per SM sub-partition, where a warp each has the least latency (64 LLL matrices
// of n = 16: 23.2 us a call with two per warp, 18.7 us with one). With a routed
// share a warp each up to two of the grid's strides, where the call then needs no
// list (a tenth / half routed, us, a warp each | listed: 4096 x n=8 46/58 | 55/55,
// n=16 83/113 | 111/111; listed 16384 x n=16 186/298, where the routed matrices
// between the FP32 ones of a warp took 243/413).
template <int NP, int NC, class Src>
int launch_mixed_small(Src src, int n, long long batch, float theta2, double *logabs,
                       double *phase, int8_t *parity, int32_t *status, cudaStream_t stream) {
  constexpr int LPM = SmallGrid<NP>::LPM;
  constexpr int NP1 = NP == 12 ? 16 : NP;  // whole 8-column slots
  if (fp64_share_64k(n) != 0) {
    if (batch <= 32ll * device_sm_count())
      return launch_mixed_grid<NP1, 32, NC, GRID_INPLACE_ROUTED>(src, n, batch, theta2, logabs,
                                                                 phase, parity, status, stream);
    return launch_mixed_grid<NP, LPM, NC, GRID_INPLACE_ROUTED>(src, n, batch, theta2, logabs,
                                                               phase, parity, status, stream);
  }
  if (batch <= 4ll * device_sm_count())
    return launch_mixed_grid<NP1, 32, NC, GRID_INPLACE>(src, n, batch, theta2, logabs, phase,
                                                        parity, status, stream);
  return launch_mixed_grid<NP, LPM, NC, GRID_INPLACE>(src, n, batch, theta2, logabs, phase,
                                                      parity, status, stream);
}

// 17 <= n <= 31 without a register-tiled rule, padded to NP; the smaller of them in
// place in small batches.
template <int NP, class Src>
int launch_mixed_padded(Src src, int n, long long batch, float theta2, double *logabs,
                        double *phase, int8_t *parity, int32_t *status, cudaStream_t stream) {
  if constexpr (NP == 24)
    if (batch <= kInplaceMaxPerSm * device_sm_count())
      return launch_mixed_grid<NP, 32, 0, GRID_INPLACE_ROUTED>(src, n, batch, theta2, logabs, phase,
                                                               parity, status, stream);
  if (fp64_share_64k(n))
    return launch_mixed_grid<NP, 32, 0, GRID_DEFER_ROUTED>(src, n, batch, theta2, logabs, phase,
                                                           parity, status, stream);
  return launch_mixed_grid<NP, 32, 0, GRID_DEFER>(src, n, batch, theta2, logabs, phase, parity,
                                                  status, stream);
}

// Sources whose matrices are always of odd order (CF matrices, n = 2Q + 3)
// never reach the register-tiled kernels, which exist for even n only.
template <class S, class = void>
struct has_even_n : std::true_type {};
template <class S>
struct has_even_n<S, std::void_t<decltype(S::kOddN)>> : std::false_type {};

// plain_fp64: the plain fused kernel on the same source (the all-FP64 route)
template <class Src, class PlainFn>
int launch_mixed_src(Src src, int n, long long batch, double *logabs, double *phase,
                     int8_t *parity, int32_t *status, cudaStream_t stream, PlainFn plain_fp64,
                     bool inplace = false) {
  if (batch == 0) return LUFQHE_SUCCESS;
  // every matrix on the FP64 route: the plain fused kernel, whose shared
  // memory layout holds more warps per SM than the mixed kernels'
  if (fp64_share_64k(n) >= 65536u)
    return plain_fp64();
  const float th2 = g_mixed_theta * g_mixed_theta;
  if constexpr (has_even_n<Src>::value) {
    switch (n) {
      case 6: return launch_mixed_small<8, 6>(src, n, batch, th2, logabs, phase, parity, status, stream);
      case 8: return launch_mixed_small<8, 8>(src, n, batch, th2, logabs, phase, parity, status, stream);
      case 12: return launch_mixed_small<12, 12>(src, n, batch, th2, logabs, phase, parity, status, stream);
      case 16: return launch_mixed_small<16, 16>(src, n, batch, th2, logabs, phase, parity, status, stream);
      case 24:
        if constexpr (std::is_same<Src, DenseSource>::value)
          if (inplace) return launch_mixed_hostlink<24>(src, batch, th2, logabs, phase, parity, status, stream);
        return launch_mixed_tile<24>(src, batch, th2, logabs, phase, parity, status, stream);
      case 32:
        if constexpr (std::is_same<Src, DenseSource>::value)
          if (inplace) return launch_mixed_hostlink<32>(src, batch, th2, logabs, phase, parity, status, stream);
        return launch_mixed_tile<32>(src, batch, th2, logabs, phase, parity, status, stream);
      default: break;
    }
  }
  // other sizes on the lane grid of the next size up
  if (n <= kSmallMaxN) {
    switch (small_np(n)) {
      case 8: return launch_mixed_small<8, 0>(src, n, batch, th2, logabs, phase, parity, status, stream);
      case 12: return launch_mixed_small<12, 0>(src, n, batch, th2, logabs, phase, parity, status, stream);
      default: return launch_mixed_small<16, 0>(src, n, batch, th2, logabs, phase, parity, status, stream);
    }
  }
  if (n <= 24) return launch_mixed_padded<24>(src, n, batch, th2, logabs, phase, parity, status, stream);
  if (n <= 32) return launch_mixed_padded<32>(src, n, batch, th2, logabs, phase, parity, status, stream);
  const size_t per_warp = mixed_smem_per_warp(n);
  const size_t optin = device_smem_optin();
  int warps = (int)(optin / per_warp);
  if (warps > 4) warps = 4;
  if (warps < 1) {
    set_error("n=%d needs %zu bytes of shared memory per matrix; the device offers %zu", n,
              per_warp, optin);
    return LUFQHE_ERR_UNSUPPORTED_N;
  }
  const size_t smem = per_warp * warps;
  auto kern = lup_mixed_kernel<Src>;
  int rc = check_cuda(cudaFuncSetAttribute(kern,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                      "cudaFuncSetAttribute(mixed)");
  if (rc) return rc;
  int per_sm = 0;
  rc = check_cuda(
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, smem),
      "occupancy(mixed)");
  if (rc) return rc;
  if (per_sm < 1) per_sm = 1;
  long long want = (batch + warps - 1) / warps;
  long long cap = (long long)device_sm_count() * per_sm;
  int grid = (int)(want < cap ? want : cap);
  const float theta2 = g_mixed_theta * g_mixed_theta;
  CallState cs;
  rc = cs.acquire((size_t)batch, 0, 0, stream);
  if (rc) return cs.release(stream, rc);
  {
    KernelTimer timer("lup_mixed_kernel", n, stream);
    kern<<<grid, warps * 32, smem, stream>>>(src, n, batch, theta2, fp64_share_64k(n),
                                             cs.head, cs.pend, logabs, phase, parity, status);
    timer.stop();
  }
  rc = check_cuda(cudaGetLastError(), "lup_mixed_kernel launch");
  if (!rc)
    rc = launch_fallback(src, n, cs.head, cs.pend, batch, logabs, phase, parity, status, stream);
  return cs.release(stream, rc);
}

}  // namespace

}  // namespace lufqhe
