// Plain FP64 batched complex LUP determinant.
//
// A warp factorises 1 to 8 matrices at a time (n <= 32, by size and batch; a
// CTA takes one above), looping over the batch with a grid stride. The matrices
// sit in shared memory (odd row stride, so a column read by a group of lanes
// hits different banks); the right-looking update of each (n-1-j)^2 trailing
// block is spread over the matrix's lanes. The factorisation itself (pivot
// rule, arithmetic) lives in lup_fp64.cuh and lup_fp64_sub.cuh.
// The determinant is returned in log-polar form: the reference multiplies the
// diagonal directly (LU-fqhe/src/LUCoreCPU.cu:256-265), which overflows for
// lowest-Landau-level matrices.

#include <cmath>

#include <type_traits>

#include "bulk_copy.cuh"
#include "cf_source.cuh"
#include "fp64_correct.cuh"
#include "lup_fp64.cuh"
#include "lup_fp64_sub.cuh"

namespace lufqhe {

namespace {

constexpr int kMaxWarpsPlain = 8;

// The mixed mode's FP64 route for 17 <= n <= 32, where the policy sends a whole
// batch there: one warp per matrix, whose log-determinant gets the
// extended-precision correction (fp64_correct_warp; its scratch follows the row
// scales in shared memory).
template <class Src>
__global__ void __launch_bounds__(kMaxWarpsPlain * 32)
    lup_plain_correct_kernel(Src src, int n, long long batch, double *__restrict__ logabs,
                             double *__restrict__ phase, int8_t *__restrict__ parity,
                             int32_t *__restrict__ status, int status_or, int bulk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int lds = n + 1;
  double2 *M = reinterpret_cast<double2 *>(smem_raw) + (size_t)warp * n * lds;
  double *hold_all = reinterpret_cast<double *>(reinterpret_cast<double2 *>(smem_raw) +
                                                (size_t)warps * n * lds);
  double *hold = hold_all + warp * 2 * n;
  float2 *F_all = reinterpret_cast<float2 *>(hold_all + (size_t)warps * 2 * n);
  const CorrScratch cs{F_all + (size_t)warp * n * lds,
                       reinterpret_cast<int *>(F_all + (size_t)warps * n * lds) + warp * 2 * n,
                       hold};
  const int nn = n * n;

  // complex128 device batches: each matrix staged by bulk copies (bulk != 0),
  // the next one prefetched into L2 meanwhile
  constexpr bool BULK = std::is_same<Src, DenseSource>::value;
  __shared__ __align__(8) uint64_t bars[kMaxWarpsPlain];
  WarpBulk wb;
  if constexpr (BULK)
    if (bulk) wb.init(&bars[warp], lane);
  const long long stride = (long long)gridDim.x * warps;
  for (long long b = (long long)blockIdx.x * warps + warp; b < batch; b += stride) {
    __syncwarp();
    int par = 0;
    int st = -1;
    if constexpr (BULK) {
      if (bulk && !wb.broken) {
        if (b + stride < batch && lane == 0)
          prefetch_matrix_l2(src.A + (size_t)(b + stride) * n * src.lda, n, src.lda);
        if (wb.load(src.A + (size_t)b * n * src.lda, n, src.lda, M, lds, lane)) {
          bool bad = false;
          BlockWalk w(lane, n);
          for (int e = lane; e < nn; e += 32) {
            bad |= !finite_c(M[w.i * lds + w.k]);
            w.next(n);
          }
          st = __any_sync(kFull, bad) ? LUFQHE_ST_NONFINITE : 0;
        } else {
          st = LUFQHE_ST_WAIT_TIMEOUT;
        }
      }
    }
    if (st < 0) st = src.load(b, n, M, lds, lane) ? LUFQHE_ST_NONFINITE : 0;
    if (!st) st = lup_fp64_warp<ARITH_FUSED>(M, lds, hold, n, lane, &par, cs.ints);

    double la, ph;
    if (st == 0) {
      logdet_from_diag(M, lds, n, lane, par, &la, &ph);
      fp64_correct_warp(src, b, n, M, lds, cs, lane, &la, &ph);
    } else if (st == LUFQHE_ST_SINGULAR) {
      la = -INFINITY;
      ph = 0.0;
    } else {
      la = NAN;
      ph = NAN;
      par = 0;
    }

    if (lane == 0) {
      logabs[b] = la;
      if (phase) phase[b] = ph;
      if (parity) parity[b] = (int8_t)par;
      if (status) status[b] = st | status_or;
    }
  }
}

// n <= 32, all but that route: 32 / LPM consecutive matrices per warp at a time
// (lup_fp64_sub). Out: element type of the in-place factors (double2, or float2
// for the reference's complex64 buffers).
template <int ARITH, int LPM, class Src, class Out = double2>
__global__ void __launch_bounds__(kMaxWarpsPlain * 32)
    lup_plain_sub_kernel(Src src, Out *__restrict__ Aout, int n, int lda, long long batch,
                         double *__restrict__ logabs, double *__restrict__ phase,
                         int8_t *__restrict__ parity, int32_t *__restrict__ status,
                         int status_or, int bulk) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int G = 32 / LPM;
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane / LPM, sub = lane % LPM;
  const unsigned gmask = LPM == 32 ? kFull : ((1u << (LPM & 31)) - 1u) << (grp * LPM);
  const int lds = n | 1;  // odd: a column read hits distinct banks
  double2 *Mw = reinterpret_cast<double2 *>(smem_raw) + (size_t)warp * G * n * lds;
  double2 *M = Mw + (size_t)grp * n * lds;
  double *hold = reinterpret_cast<double *>(reinterpret_cast<double2 *>(smem_raw) +
                                            (size_t)warps * G * n * lds) +
                 (size_t)(warp * G + grp) * 2 * n;
  constexpr bool BULK = std::is_same<Src, DenseSource>::value;
  __shared__ __align__(8) uint64_t bars[kMaxWarpsPlain];
  WarpBulk wb;
  if constexpr (BULK)
    if (bulk) wb.init(&bars[warp], lane);
  const long long stride = (long long)gridDim.x * warps * G;
  for (long long b0 = ((long long)blockIdx.x * warps + warp) * G; b0 < batch; b0 += stride) {
    const int cnt = (int)min((long long)G, batch - b0);
    const bool valid = grp < cnt;
    __syncwarp();
    int st = 0, par = 0;
    bool staged = false;
    if constexpr (BULK) {
      if (bulk && !wb.broken) {
        if (b0 + stride < batch && lane == 0)
          prefetch_rows_l2(src.A + (size_t)(b0 + stride) * n * src.lda,
                           (int)min((long long)G, batch - b0 - stride) * n, n, src.lda);
        if (!wb.load_rows(src.A + (size_t)b0 * n * src.lda, cnt * n, n, src.lda, Mw, lds, n,
                          lane))
          st = LUFQHE_ST_WAIT_TIMEOUT;
        staged = true;
      }
    }
    if (!staged) load_rows(src, b0, cnt * n, n, Mw, lds, n, lane);
    __syncwarp();
    if (st == 0) st = lup_fp64_sub<ARITH, LPM>(M, lds, hold, n, sub, gmask, valid, &par);
    double la, ph;
    logdet_from_diag_sub<LPM>(M, lds, n, sub, valid && st == 0, par, &la, &ph);
    if (st == LUFQHE_ST_SINGULAR) {
      la = -INFINITY;
      ph = 0.0;
    } else if (st != 0) {
      la = NAN;
      ph = NAN;
      par = 0;
    }
    if (!valid) continue;
    const long long b = b0 + grp;
    if (Aout && (st == 0 || st == LUFQHE_ST_SINGULAR)) {
      Out *dst = Aout + (size_t)b * n * lda;
      StrideWalk w(sub, LPM, n);
      for (int e = sub; e < n * n; e += LPM) {
        store_entry(dst + (size_t)w.i * lda + w.k, M[w.i * lds + w.k]);
        w.next(n);
      }
    }
    if (sub == 0) {
      logabs[b] = la;
      if (phase) phase[b] = ph;
      if (parity) parity[b] = (int8_t)par;
      if (status) status[b] = st | status_or;
    }
  }
}

// Writes exp(logabs + i*phase) into element (0,0); with pair_product the even
// matrix of each pair gets the product of the pair's determinants
// (LU-fqhe/src/LUCoreGPU.cu:403-435).
template <class T>
__global__ void write_det_kernel(T *A, int n, int lda, long long batch,
                                 const double *logabs, const double *phase,
                                 const int32_t *status, int pair_product) {
  long long b = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  double la = logabs[b], ph = phase[b];
  if (pair_product && (b % 2 == 0) && b + 1 < batch) {
    la += logabs[b + 1];
    ph += phase[b + 1];
  }
  double2 v;
  if (la != la || ph != ph) {
    v = make_double2(NAN, NAN);
  } else {
    double m = exp(la);
    double s, c;
    sincos(ph, &s, &c);
    v = make_double2(m * c, m * s);
  }
  store_entry(A + (size_t)b * n * lda, v);
}

}  // namespace

// n > 32: one matrix per CTA of group_warps(n) warps (lup_fp64_group). With one
// warp per matrix an SM holds only the 3-4 matrices its shared memory fits
// (n=64: 66 KB each), too few warps to cover the FP64 pipe's latency.
constexpr int kGroupMaxWarps = 6, kGroupMinCtas = 6;
constexpr int kGroupMinN = kFp64GroupMinN;
// 4 warps up to n = 48, 6 above, where an SM holds 3 or 4 matrices only (2048
// LLL x n=64, us with 4 / 5 / 6 / 8 warps, when the multipliers of a column were
// unrolled: fused 1745 / 1620 / 1621 / 1615, now 1588 with 6; reference arithmetic
// 3592 / 3395 / 3354 / 3410; 4096 x n=48 fused 1424 / 1425 / 1431 / 1471, now 1376
// with 4). Compiled for 56 registers, 9 CTAs of 4 warps (with 60, 2000 x n=36 in
// reference arithmetic took 768 us instead of 716).
constexpr int kWarpMaxN = 40;
constexpr int group_warps(int n) { return n > 48 ? kGroupMaxWarps : kFp64GroupWarps; }

// CORRECT: the mixed mode's FP64 route, whose log-determinants get the
// extended-precision correction (fp64_correct_group; its scratch follows the
// row scales in shared memory).
template <int ARITH, class Src, class Out = double2, bool CORRECT = false>
__global__ void __launch_bounds__(kGroupMaxWarps * 32, kGroupMinCtas)
    lup_plain_group_kernel(Src src, Out *__restrict__ Aout, int n, int lda, long long batch,
                           double *__restrict__ logabs, double *__restrict__ phase,
                           int8_t *__restrict__ parity, int32_t *__restrict__ status,
                           int status_or) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long red[3 * kGroupMaxWarps];
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int lds = n + 1;
  double2 *M = reinterpret_cast<double2 *>(smem_raw);
  double *hold = reinterpret_cast<double *>(M + (size_t)n * lds);
  CorrScratch cs{};
  if constexpr (CORRECT) {
    float2 *F = reinterpret_cast<float2 *>(hold + 2 * n);
    cs = CorrScratch{F, reinterpret_cast<int *>(F + (size_t)n * lds), hold};
  }
  for (long long b = blockIdx.x; b < batch; b += gridDim.x) {
    __syncthreads();
    int par = 0;
    int st = src.load_group(b, n, M, lds, tid, nthr) ? LUFQHE_ST_NONFINITE : 0;
    if (!st)
      st = lup_fp64_group<ARITH>(M, lds, hold, n, tid, nthr, red, &par, CtaBarrier(),
                                 CORRECT ? cs.ints : nullptr);
    __syncthreads();
    if (Aout && (st == 0 || st == LUFQHE_ST_SINGULAR)) {
      Out *dst = Aout + (size_t)b * n * lda;
      StrideWalk w(tid, nthr, n);
      for (int e = tid; e < n * n; e += nthr) {
        store_entry(dst + (size_t)w.i * lda + w.k, M[w.i * lds + w.k]);
        w.next(n);
      }
    }
    double la = 0.0, ph = 0.0;
    if (tid < 32) {
      // warp 0, with the warp routine's own summation order
      if (st == 0) {
        logdet_from_diag(M, lds, n, tid, par, &la, &ph);
      } else if (st == LUFQHE_ST_SINGULAR) {
        la = -INFINITY;
        ph = 0.0;
      } else {
        la = NAN;
        ph = NAN;
        par = 0;
      }
    }
    if constexpr (CORRECT) {
      if (st == 0) {
        __syncthreads();  // the diagonal is read before the correction overwrites M
        const double2 c = fp64_correct_group(src, b, n, M, lds, cs, tid, nthr, CtaBarrier(),
                                             reinterpret_cast<float *>(red));
        la += c.x;
        ph += c.y;
      }
    }
    if (tid == 0) {
      logabs[b] = la;
      if (phase) phase[b] = ph;
      if (parity) parity[b] = (int8_t)par;
      if (status) status[b] = st | status_or;
    }
  }
}

// the bulk-copy staging for complex128 matrices in device memory only
inline int bulk_for(const DenseSource &s) { return g_bulk_loads && is_device_memory(s.A); }
template <class S>
inline int bulk_for(const S &) {
  return 0;
}

size_t plain_smem_per_warp(int n) {
  return (size_t)n * (n + 1) * sizeof(double2) + 2 * (size_t)n * sizeof(double);
}

template <int LPM, class Src, class Out>
int launch_plain_sub(Src src, Out *Aout, int n, int lda, long long batch, int arith,
                     double *logabs, double *phase, int8_t *parity, int32_t *status,
                     cudaStream_t stream, int status_or) {
  constexpr int G = 32 / LPM;
  const int warps = sub_warps(n, LPM);
  const size_t smem = sub_smem(n, LPM);
  auto kern = arith == ARITH_REF ? lup_plain_sub_kernel<ARITH_REF, LPM, Src, Out>
                                 : lup_plain_sub_kernel<ARITH_FUSED, LPM, Src, Out>;
  int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem),
                      "cudaFuncSetAttribute(plain sub)");
  if (rc) return rc;
  int per_sm = 0;
  rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, smem),
                  "occupancy(plain sub)");
  if (rc) return rc;
  const long long want = (batch + warps * G - 1) / (warps * G);
  const long long cap = (long long)device_sm_count() * (per_sm < 1 ? 1 : per_sm);
  const int grid = (int)(want < cap ? want : cap);
  KernelTimer timer(arith == ARITH_REF ? "lup_plain_kernel_ref" : "lup_plain_kernel", n, stream);
  kern<<<grid, warps * 32, smem, stream>>>(src, Aout, n, lda, batch, logabs, phase, parity, status,
                                           status_or, bulk_for(src));
  timer.stop();
  return check_cuda(cudaGetLastError(), "lup_plain_sub_kernel launch");
}

template <class Src, class Out = double2>
int launch_plain_src(Src src, Out *Aout, int n, int lda, long long batch, int arith,
                     double *logabs, double *phase, int8_t *parity, int32_t *status,
                     cudaStream_t stream, int status_or) {
  if (batch == 0) return LUFQHE_SUCCESS;
  // the mixed mode's FP64 route (status_or set, no factors written back)
  const bool correct = status_or != 0 && arith == ARITH_FUSED && Aout == nullptr &&
                       n >= kCorrectMinN && n <= kCorrectMaxN;
  const size_t corr_smem = (size_t)n * (n + 1) * sizeof(float2) + 2 * (size_t)n * sizeof(int);
  // fused, n <= kWarpMaxN: a warp per matrix, without barriers, where the batch
  // fills its rounds. A part-filled round costs a whole one; groups cost 2% more per
  // matrix and a tenth of a round for their tail (us, warps | groups: x n=33 1700
  // 230 | 246, 3500 454 | 462, 8192 (4.5 of 5 rounds) 1055 | 1050; x n=36 4500 (3.7
  // of 4) 749 | 726; x n=40 3500 (2.9 of 3) 725 | 741, 8192 (6.7 of 7) 1679 | 1654).
  // Reference arithmetic gains nothing (4096 x n=40 2219 | 2211).
  bool warp_each = false;
  if (n >= kGroupMinN && n <= kWarpMaxN && !correct && arith == ARITH_FUSED) {
    const long long round = 4ll * (long long)((device_smem_optin() + 1024) /
                                              (sub_smem(n, 32) + 1024)) * device_sm_count();
    const long long rounds = (batch + round - 1) / round;
    warp_each = 102 * batch + 10 * round >= 100 * rounds * round;
  }
  if (n >= kGroupMinN && !warp_each) {
    const int threads = group_warps(n) * 32;
    const size_t smem = (size_t)n * (n + 1) * sizeof(double2) + 2 * (size_t)n * sizeof(double) +
                        (correct ? corr_smem : 0);
    auto kern = correct              ? lup_plain_group_kernel<ARITH_FUSED, Src, Out, true>
                : arith == ARITH_REF ? lup_plain_group_kernel<ARITH_REF, Src, Out>
                                     : lup_plain_group_kernel<ARITH_FUSED, Src, Out>;
    int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem),
                        "cudaFuncSetAttribute(plain group)");
    if (rc) return rc;
    int per_sm = 0;
    rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem),
                    "occupancy(plain group)");
    if (rc) return rc;
    if (per_sm < 1) {
      set_error("n=%d needs %zu bytes of shared memory per matrix", n, smem);
      return LUFQHE_ERR_UNSUPPORTED_N;
    }
    const long long cap = (long long)device_sm_count() * per_sm;
    const int grid = (int)(batch < cap ? batch : cap);
    KernelTimer timer(arith == ARITH_REF ? "lup_plain_group_kernel_ref" : "lup_plain_group_kernel",
                      n, stream);
    kern<<<grid, threads, smem, stream>>>(src, Aout, n, lda, batch, logabs, phase, parity,
                                                   status, status_or);
    timer.stop();
    return check_cuda(cudaGetLastError(), "lup_plain_group_kernel launch");
  }
  if (!correct) {
    switch (sub_lanes(n, batch, arith, device_sm_count(), device_smem_optin() + 1024)) {
      case 4:
        return launch_plain_sub<4>(src, Aout, n, lda, batch, arith, logabs, phase, parity, status,
                                   stream, status_or);
      case 8:
        return launch_plain_sub<8>(src, Aout, n, lda, batch, arith, logabs, phase, parity, status,
                                   stream, status_or);
      case 16:
        return launch_plain_sub<16>(src, Aout, n, lda, batch, arith, logabs, phase, parity,
                                    status, stream, status_or);
      default:
        return launch_plain_sub<32>(src, Aout, n, lda, batch, arith, logabs, phase, parity,
                                    status, stream, status_or);
    }
  }
  const size_t per_warp = plain_smem_per_warp(n) + (correct ? corr_smem : 0);
  const size_t optin = device_smem_optin();
  int warps = (int)(optin / per_warp);
  if (warps > 4) warps = 4;
  if (warps < 1) {
    set_error("n=%d needs %zu bytes of shared memory per matrix; the device offers %zu", n,
              per_warp, optin);
    return LUFQHE_ERR_UNSUPPORTED_N;
  }
  const size_t smem = per_warp * warps;
  auto kern = lup_plain_correct_kernel<Src>;
  int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)smem),
                      "cudaFuncSetAttribute(plain)");
  if (rc) return rc;
  int per_sm = 0;
  rc = check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, smem),
                  "occupancy(plain)");
  if (rc) return rc;
  if (per_sm < 1) per_sm = 1;
  long long want = (batch + warps - 1) / warps;
  long long cap = (long long)device_sm_count() * per_sm;
  int grid = (int)(want < cap ? want : cap);
  KernelTimer timer("lup_plain_kernel", n, stream);
  kern<<<grid, warps * 32, smem, stream>>>(src, n, batch, logabs, phase, parity, status, status_or,
                                           bulk_for(src));
  timer.stop();
  return check_cuda(cudaGetLastError(), "lup_plain_correct_kernel launch");
}

int launch_plain(const double2 *A, double2 *Aout, int n, int lda, long long batch, int arith,
                 double *logabs, double *phase, int8_t *parity, int32_t *status,
                 cudaStream_t stream, int status_or) {
  return launch_plain_src(DenseSource{A, lda}, Aout, n, lda, batch, arith, logabs, phase, parity,
                          status, stream, status_or);
}

int launch_plain32(const float2 *A, float2 *Aout, int n, int lda, long long batch, int arith,
                   double *logabs, double *phase, int8_t *parity, int32_t *status,
                   cudaStream_t stream, int status_or) {
  return launch_plain_src(Dense32Source{A, lda}, Aout, n, lda, batch, arith, logabs, phase,
                          parity, status, stream, status_or);
}

int launch_plain_lll(const double2 *Z, int n, long long batch, int arith, double *logabs,
                     double *phase, int8_t *parity, int32_t *status, cudaStream_t stream,
                     int status_or) {
  return launch_plain_src(LllSource{Z}, static_cast<double2 *>(nullptr), n, n, batch, arith,
                          logabs, phase, parity, status, stream, status_or);
}

int launch_plain_cf(const CfSource &src, int n, long long batch, int arith, double *logabs,
                    double *phase, int8_t *parity, int32_t *status, cudaStream_t stream,
                    int status_or) {
  return launch_plain_src(src, static_cast<double2 *>(nullptr), n, n, batch, arith, logabs, phase,
                          parity, status, stream, status_or);
}

template <class T>
int launch_write_det_t(T *A, int n, int lda, long long batch, const double *logabs,
                       const double *phase, const int32_t *status, int pair_product,
                       cudaStream_t stream) {
  if (batch == 0) return LUFQHE_SUCCESS;
  int threads = 256;
  long long blocks = (batch + threads - 1) / threads;
  write_det_kernel<T><<<(unsigned)blocks, threads, 0, stream>>>(A, n, lda, batch, logabs, phase,
                                                                status, pair_product);
  return check_cuda(cudaGetLastError(), "write_det_kernel launch");
}

int launch_write_det(double2 *A, int n, int lda, long long batch, const double *logabs,
                     const double *phase, const int32_t *status, int pair_product,
                     cudaStream_t stream) {
  return launch_write_det_t(A, n, lda, batch, logabs, phase, status, pair_product, stream);
}

int launch_write_det32(float2 *A, int n, int lda, long long batch, const double *logabs,
                       const double *phase, const int32_t *status, int pair_product,
                       cudaStream_t stream) {
  return launch_write_det_t(A, n, lda, batch, logabs, phase, status, pair_product, stream);
}

}  // namespace lufqhe
