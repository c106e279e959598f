// The FP64 factorisation of lup_fp64.cuh with 32 / LPM matrices per warp, LPM
// lanes each, for n <= 2 LPM.
//
// FP64 instructions are the scarce resource on GB300: one costs its pipe the
// same with one lane active as with 32. With a warp per matrix, the trailing
// updates of n = 16 are 384 of the 1023 FP64 instructions a matrix took; the
// rest (pivot keys, the pivot's reciprocal, multipliers, the logs) ran on a few
// lanes, or on all lanes for one value. Here one instruction does those for 2,
// 4 or 8 matrices, and the trailing blocks fill their lanes better. Every
// matrix sees the operations of lup_fp64_warp in the same order, so factors,
// pivots, parity and results are the same bits. The whole GPU, us, one matrix a
// warp -> now: 131072 x n=8 3295 -> 836 (reference arithmetic), 2005 -> 489
// (fused); 65536 x n=16 4010 -> 2171, 2109 -> 1066; 32768 x n=24 4225 -> 3470,
// 2071 -> 1682. The FP64 pipe stays the bound: it is over 80% busy.
#pragma once

#include "lup_fp64.cuh"

namespace lufqhe {

// Lane `sub` of a group of LPM lanes (gmask in the warp), on its group's matrix
// M (row stride lds) with 2n doubles of scratch at hold. Also checks that the
// entries are finite. Group-uniform result: 0, LUFQHE_ST_NONFINITE,
// LUFQHE_ST_SCALE_TINY or LUFQHE_ST_SINGULAR (M as it was when the zero pivot
// was met). All lanes of the warp call it together; a group past the end of the
// batch passes valid = false and touches nothing.
template <int ARITH, int LPM>
__device__ int lup_fp64_sub(double2 *M, int lds, double *hold, int n, int sub, unsigned gmask,
                            bool valid, int *parity) {
  constexpr int R = 2;  // rows per lane (n <= 32 has one with 32 lanes)
  double *rhold = hold + n;
  int par = 0, st = 0;
  {
    bool bad = false, tiny = false;
    const long long tiny_bits = __double_as_longlong(1e-24);
    if (valid)
      for (int i = sub; i < n; i += LPM) {
        long long big = 0;
        for (int k = 0; k < n; ++k) {
          const double2 v = M[i * lds + k];
          bad |= !finite_c(v);
          big = max(big, abs_bits(v.x));
        }
        const double h = __longlong_as_double(big);
        hold[i] = h;
        rhold[i] = __drcp_rn(h);
        tiny |= big < tiny_bits;
      }
    if (__ballot_sync(kFull, tiny) & gmask) st = LUFQHE_ST_SCALE_TINY;
    if (__ballot_sync(kFull, bad) & gmask) st = LUFQHE_ST_NONFINITE;
    __syncwarp();
  }
  bool live = valid && st == 0;
  // argmax over the group of (key, row), ties to the larger row
  auto argmax = [](long long &bk, int &bi) {
#pragma unroll
    for (int off = LPM / 2; off; off >>= 1) {
      const long long ok = __shfl_xor_sync(kFull, bk, off);
      const int oi = __shfl_xor_sync(kFull, bi, off);
      if (ok > bk || (ok == bk && oi > bi)) {
        bk = ok;
        bi = oi;
      }
    }
  };
  const long long inf_bits = 0x7ff0000000000000ll;
  const long long safe_lo = 0x0170000000000000ll;  // 2^-1000
  const long long safe_hi = 0x7e70000000000000ll;  // 2^+1000
  for (int j = 0; j < n; ++j) {
    // screened search (see lup_fp64_warp); a NaN quotient is never chosen
    long long key[R], bk = -1;
    int bi = j;
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const int i = j + sub + LPM * q;
      key[q] = -3;
      if (j + LPM * q >= n) continue;  // no row of this slot
      if (live && i < n) {
        const long long a =
            __double_as_longlong(__dmul_rn(fabs(M[i * lds + j].x), rhold[i]));
        key[q] = (a & 0x7fffffffffffffffll) > inf_bits ? -2 : a;
        if (key[q] >= bk) {
          bk = key[q];
          bi = i;
        }
      }
    }
    argmax(bk, bi);
    int near = 0;
#pragma unroll
    for (int q = 0; q < R; ++q)
      near += __popc(__ballot_sync(kFull, key[q] > -3 && key[q] >= bk - 16) & gmask);
    const bool exact = live && (near != 1 || bk < safe_lo || bk > safe_hi);
    if (__any_sync(kFull, exact)) {
      long long ek = -1;
      int ei = j;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const int i = j + sub + LPM * q;
        if (exact && i < n) {
          const double d = __ddiv_rn(fabs(M[i * lds + j].x), hold[i]);
          const long long k = (d == d) ? __double_as_longlong(d) : -2ll;
          if (k >= ek) {
            ek = k;
            ei = i;
          }
        }
      }
      argmax(ek, ei);
      if (exact) bi = ei;
    }
    if (live && bi != j) {
      const int p = bi;
      for (int k = sub; k < n; k += LPM) {
        const double2 t = M[p * lds + k];
        M[p * lds + k] = M[j * lds + k];
        M[j * lds + k] = t;
      }
      if (sub == 0) {
        hold[p] = hold[j];
        rhold[p] = rhold[j];
      }
      par ^= 1;
    }
    __syncwarp();
    const double2 piv = M[j * lds + j];
    if (live && is_zero_c(piv)) {
      st = LUFQHE_ST_SINGULAR;
      live = false;
    }
    if (j == n - 1) break;
    if (ARITH == ARITH_REF) {
      const double den = pivot_den<ARITH_REF>(piv);
      const double y = __drcp_rn(den);
      const long long db = abs_bits(den);
      const bool den_safe = db >= 0x03f0000000000000ll && db <= 0x7bf0000000000000ll;  // [2^-960, 2^960]
      if (live)
        for (int i = j + 1 + sub; i < n; i += LPM) {
          const double2 a = M[i * lds + j];
          const double nx = __dadd_rn(__dmul_rn(a.x, piv.x), __dmul_rn(a.y, piv.y));
          const double ny = __dsub_rn(__dmul_rn(a.y, piv.x), __dmul_rn(a.x, piv.y));
          M[i * lds + j] = make_double2(div_rn_markstein(nx, den, y, den_safe),
                                        div_rn_markstein(ny, den, y, den_safe));
        }
    } else {
      const double d = pivot_den<ARITH>(piv);
      if (live)
        for (int i = j + 1 + sub; i < n; i += LPM)
          M[i * lds + j] = cdiv_pivot<ARITH>(M[i * lds + j], piv, d);
    }
    __syncwarp();
    // trailing update on the m x m block, two entries at a time so that one's
    // loads overlap the other's arithmetic; lanes without an entry read T[-1], a
    // multiplier, which nobody writes
    const int m = n - 1 - j, mm = m * m;
    double2 *T = M + (j + 1) * lds + j + 1;
    const double2 *L = M + (j + 1) * lds + j, *U = M + j * lds + j + 1;
    StrideWalk w(sub, LPM, m);
    for (int e0 = 0; e0 < mm; e0 += 2 * LPM) {
      const int e = e0 + sub;
      const int i0 = w.i, k0 = w.k;
      w.next(m);
      const int i1 = w.i, k1 = w.k;
      w.next(m);
      const bool on0 = live && e < mm, on1 = live && e + LPM < mm;
      if (e0 + LPM < mm) {  // uniform: no FP64 work for a second half that is empty
        const int f0 = on0 ? i0 * lds + k0 : -1, f1 = on1 ? i1 * lds + k1 : -1;
        const double2 s0 = T[f0], l0 = L[on0 ? i0 * lds : 0], u0 = U[on0 ? k0 : 0];
        const double2 s1 = T[f1], l1 = L[on1 ? i1 * lds : 0], u1 = U[on1 ? k1 : 0];
        const double2 r0 = cmsub<ARITH>(s0, l0, u0), r1 = cmsub<ARITH>(s1, l1, u1);
        if (on0) T[f0] = r0;
        if (on1) T[f1] = r1;
      } else if (on0) {
        T[i0 * lds + k0] = cmsub<ARITH>(T[i0 * lds + k0], L[i0 * lds], U[k0]);
      }
    }
    __syncwarp();
  }
  *parity = par;
  return st;
}

// log|det| and phase from the diagonal of each group's factored M, summed in
// the order of logdet_from_diag (entry j on lane j of a warp).
template <int LPM>
__device__ __forceinline__ void logdet_from_diag_sub(const double2 *M, int lds, int n, int sub,
                                                     bool live, int par, double *la_out,
                                                     double *ph_out) {
  double la[2] = {0.0, 0.0}, ph[2] = {0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int j = sub + LPM * q;
    if (live && j < n) {
      double lg, ar;
      log_arg_c(M[j * lds + j], lg, ar);
      la[q] += lg;
      ph[q] += ar;
    }
  }
  double a = la[0] + la[1], p = ph[0] + ph[1];
#pragma unroll
  for (int off = LPM / 2; off; off >>= 1) {
    a += __shfl_xor_sync(kFull, a, off);
    p += __shfl_xor_sync(kFull, p, off);
  }
  if (par) p += kPi;
  *la_out = a;
  *ph_out = wrap_phase(p);
}

// FP64 instructions of one warp pass over 32 / lpm matrices: trailing updates,
// multipliers, the pivot's reciprocal and keys, then the logs.
inline long long sub_pass_cost(int n, int lpm, int arith) {
  const bool ref = arith == ARITH_REF;
  auto passes = [lpm](long long items) { return (items + lpm - 1) / lpm; };
  long long c = 120 * passes(n);
  for (int m = n - 1; m > 0; --m)
    c += passes(m + 1) + 13 + passes(m) * (ref ? 18 : 6) + passes((long long)m * m) * (ref ? 8 : 4);
  return c;
}

// Warps per CTA: small CTAs where a warp's matrices are large, so that an SM
// fills up.
inline int sub_warps(int n, int lpm) { return n > 16 && lpm < 32 ? 2 : 4; }

// Shared memory of a CTA: its matrices and 2n doubles each.
inline size_t sub_smem(int n, int lpm) {
  return (size_t)sub_warps(n, lpm) * (32 / lpm) *
         ((size_t)n * (n | 1) * sizeof(double2) + 2 * (size_t)n * sizeof(double));
}

// Lanes per matrix for a batch: the least time, where a round of W warps on an
// SM takes c max(100, 17 W) cycles, c the FP64 instructions of a warp's pass. A
// warp alone takes about 100 cycles per FP64 instruction (its dependent
// chains), an SM's FP64 pipe 16 to 17 (both within 10% over n = 8..32 and every
// width), and shared memory bounds the warps of a round. A large batch then
// takes the fewest lanes, two rows each; one that would leave SMs short of
// warps that way takes more (n = 16, reference arithmetic, us with 8 / 16 / 32
// lanes: 256 matrices 101 / 66 / 52, 1000 101 / 66 / 79, 4000 169 / 196 / 260).
inline int sub_lanes(int n, long long batch, int arith, int sms, size_t smem_per_sm) {
  int best = 32;
  double best_cost = 0.0;
  for (int lpm = 32; lpm >= 4 && 2 * lpm >= n; lpm /= 2) {
    const int warps = sub_warps(n, lpm);
    const long long fit = (long long)(smem_per_sm / (sub_smem(n, lpm) + 1024));
    const long long ctas_sm = fit < 1 ? 1 : fit > 64 / warps ? 64 / warps : fit;
    const long long per_cta = (long long)warps * (32 / lpm);
    const long long ctas = (batch + per_cta - 1) / per_cta;
    const long long full = (ctas - 1) / (ctas_sm * sms);  // rounds before the last
    const long long last = (ctas - full * ctas_sm * sms + sms - 1) / sms;
    auto round = [&](long long c) { return 17.0 * c * warps > 100.0 ? 17.0 * c * warps : 100.0; };
    const double cost =
        (double)sub_pass_cost(n, lpm, arith) * ((double)full * round(ctas_sm) + round(last));
    if (lpm == 32 || cost < best_cost) {
      best = lpm;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace lufqhe
