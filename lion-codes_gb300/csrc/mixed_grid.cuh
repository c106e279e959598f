// The mixed method's FP32 path for n <= 32, several small matrices per warp.
//
// The steps and every rounded operation are those of mixed_core.cuh (the
// register-tiled path there, and for other sizes the generic one), so an accepted
// matrix has the same bits; only the generic rule's ||E||_F is summed in another
// order (that of a 4 x 8 lane grid), so a matrix within rounding of the acceptance
// bound may be accepted here and refactorised there, or the reverse. What differs
// is where the work sits:
//  * A matrix has GR x GC lanes: 8 for n <= 8, 16 for n <= 16, 32 above, so a
//    warp factorises 4, 2 or 1 matrices in lockstep. At n = 8 the serial parts
//    of a factorisation (pivot searches, reciprocals, reductions, the log
//    bookkeeping) outweigh the arithmetic, and one instruction now serves four
//    matrices of them.
//  * LUP: lane = row, the row in registers, pivoting by position numbers
//    instead of row exchanges. A step is one key maximum, one shared-memory
//    write of the finished row by its lane (to its final position, so F ends up
//    as the pivoted L\U), a broadcast read of its U part and FMAs in registers;
//    the shared-memory form read and wrote every trailing entry and exchanged
//    two rows of F and of the hi/lo copy per step.
//  * Residual, solves, log det(I + E): lane (r, c) of the grid owns entries
//    (GR a + r, GC b + c). R goes from the float-float accumulators straight
//    into the solves' registers. The t loop of the residual is cut into blocks
//    of 2, 4 or 8 steps whose slots are known at compile time, so that only the
//    diagonal blocks carry masks.
//  * Sums over a matrix (||E||_F, tr E, tr E^2) are taken in the order of a
//    4 x 8 lane grid whatever the grid is, so the choice of grid changes no bit.
// Bound by instruction issue and fetch (62% issue, FMA pipe 48% at n = 16; the
// code a warp runs through once per matrix, 4000 instructions, does not fit the
// instruction cache). Measured against the one-matrix-per-warp kernels, Gaussian
// matrices, us: 131072 x n=8 397 -> 179, 65536 x n=12 427 -> 241, 65536 x n=16
// 618 -> 430; generic rule: 131072 x n=4 524 -> 198, 131072 x n=11 1546 -> 552,
// 20011 LLL x n=19 845 -> 624 (with its FP64 pass).
#pragma once

#include "mixed_core.cuh"

namespace lufqhe {
namespace mixed {
namespace {

template <int NP, int LPM_>
struct Grid {
  static constexpr int LPM = LPM_;     // lanes per matrix: 8, 16 or 32
  static constexpr int G = 32 / LPM;   // matrices per warp
  static constexpr int GR = LPM == 8 ? 2 : 4;
  static constexpr int GC = LPM / GR;
  static constexpr int SA = (NP + GR - 1) / GR, SB = (NP + GC - 1) / GC;
  static constexpr int LDH = NP + 1;  // row stride of the double2 matrix and its hi/lo copy
  static constexpr int LDF = NP + 2;  // row stride of F: 16-byte rows for paired accesses
  // shared memory of one matrix: hi/lo copy, F, 2 NP ints. Where several
  // matrices share a warp, F has 64 bytes more, so that the same row of two of
  // them starts in different banks (n = 8: 184 -> 180 us for 131072)
  static constexpr size_t kHL = (size_t)NP * LDH;
  static constexpr size_t kF = (size_t)NP * LDF + (G > 1 ? 8 : 0);
  static constexpr size_t kWarpBytes =
      G * (kHL * sizeof(float4) + kF * sizeof(float2) + 2 * NP * sizeof(int));
};

// The grid of a size n <= 16: padded to NP = 8, 12 or 16, whichever path takes
// it. The kernels dispatch by small_np and reserve small_warp_bytes; both follow
// from here.
constexpr int kSmallMaxN = 16;
__host__ __device__ constexpr int small_np(int n) { return n <= 8 ? 8 : n <= 12 ? 12 : 16; }
template <int NP>
using SmallGrid = Grid<NP, NP == 8 ? 8 : 16>;
// Shared memory of a warp on size n's grid, and of one that takes every size up
// to nm.
__host__ __device__ constexpr size_t small_layout_bytes(int n) {
  return small_np(n) == 8    ? SmallGrid<8>::kWarpBytes
         : small_np(n) == 12 ? SmallGrid<12>::kWarpBytes
                             : SmallGrid<16>::kWarpBytes;
}
__host__ __device__ constexpr size_t small_warp_bytes(int nm) {
  size_t most = 0;
  for (int n = 1; n <= nm; ++n)
    if (small_layout_bytes(n) > most) most = small_layout_bytes(n);
  return most;
}
// Every size fits its grid, and the reservation covers it for every nm >= n.
constexpr bool small_layouts_covered() {
  for (int nm = 1; nm <= kSmallMaxN; ++nm)
    for (int n = 1; n <= nm; ++n)
      if (small_np(n) < n || small_warp_bytes(nm) < small_layout_bytes(n)) return false;
  return true;
}
static_assert(small_layouts_covered(), "a warp's shared memory must hold every size it takes");

// This lane's place in its matrix's grid.
template <int NP, int LPM>
struct GridLane {
  int lane, sub, gb, r, c;
  unsigned gmask;
  __device__ __forceinline__ explicit GridLane(int l) {
    using Gd = Grid<NP, LPM>;
    lane = l;
    sub = l % Gd::LPM;
    gb = l - sub;
    r = sub / Gd::GC;
    c = sub % Gd::GC;
    gmask = Gd::LPM == 32 ? kFull : ((1u << (Gd::LPM & 31)) - 1u) << gb;
  }
  __device__ __forceinline__ int at(int rr, int cc) const { return gb + rr * Grid<NP, LPM>::GC + cc; }
};

template <int LPM>
__device__ __forceinline__ unsigned group_max(unsigned v) {
  if constexpr (LPM == 32) {
    return __reduce_max_sync(kFull, v);
  } else {
#pragma unroll
    for (int off = LPM / 2; off; off >>= 1) v = max(v, __shfl_xor_sync(kFull, v, off));
    return v;
  }
}
template <int LPM>
__device__ __forceinline__ int group_add(int v) {
  if constexpr (LPM == 32) {
    return __reduce_add_sync(kFull, v);
  } else {
#pragma unroll
    for (int off = LPM / 2; off; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
    return v;
  }
}

// split_scaled without branches: hi and lo of x 2^-s, |x| 2^-s < 2, from the
// exponent words. adj is ((s + 1023 - 127) << 20); the subtraction wraps, and
// the true biased exponent lies in [-1918, 127]. lo is the low 29 mantissa
// bits as top 16 + low 13, each exact in float, added with truncation (so 24
// significant bits are kept, as split_scaled keeps them), times a power of two.
__device__ __forceinline__ void split_words(double x, int adj, float &hi, float &lo) {
  const unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const int he = (int)(h & 0x7ff00000u);
  const int ef = (int)((unsigned)he - (unsigned)adj);
  const unsigned mant = __funnelshift_l(l, h, 3) & 0x7fffffu;
  const unsigned mag = (he != 0 && ef > 0) ? (((unsigned)ef << 3) | mant) : 0u;
  const unsigned sign = h & 0x80000000u;
  hi = __uint_as_float(mag | sign);
  const float top = __uint_as_float(((l >> 6) & 0x7fff80u) | 0x3f800000u);   // 1 + top 2^-16
  const float low = __uint_as_float(((l << 10) & 0x7ffc00u) | 0x37800000u);  // 2^-16 + low 2^-29
  const float r = __fadd_rz(__fadd_rn(top, -1.0f - 1.52587890625e-05f), low);
  const int se = max((int)(mag & 0x7f800000u) - (23 << 23), 0);
  float v;
  asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(v) : "f"(r), "f"(__uint_as_float((unsigned)se | sign)));
  lo = v;
}

// Sums of one matrix in the order of a 4 x 8 lane grid: `p[q][w]` is the chain
// of the virtual lane row/column class this lane holds (row class a % NR, column
// class b % NCH). xor 16, 8, 4, 2, 1 of the virtual lane become in-lane adds
// where both partners sit in this lane.
template <int LPM>
struct Chains {
  static constexpr int GR = LPM == 8 ? 2 : 4, GC = LPM / GR;
  static constexpr int NR = 4 / GR, NCH = 8 / GC;
};
template <int LPM>
__device__ __forceinline__ float chain_sum(
    const float (&p)[Chains<LPM>::NR][Chains<LPM>::NCH]) {
  constexpr int GC = Chains<LPM>::GC;
  constexpr int NR = Chains<LPM>::NR, NCH = Chains<LPM>::NCH;
  float s[NCH];
#pragma unroll
  for (int w = 0; w < NCH; ++w) {
    // virtual row bit 1, then bit 0
    float v;
    if constexpr (NR == 2) {
      v = p[0][w] + p[1][w];
    } else {
      v = p[0][w];
      v += __shfl_xor_sync(kFull, v, 2 * GC);
    }
    v += __shfl_xor_sync(kFull, v, GC);
    s[w] = v;
  }
  float t;
  if constexpr (NCH == 2) {
    t = s[0] + s[1];
  } else {
    t = s[0];
    t += __shfl_xor_sync(kFull, t, 4);
  }
  t += __shfl_xor_sync(kFull, t, 2);
  t += __shfl_xor_sync(kFull, t, 1);
  return t;
}

// One LUP step t (compile-time) for every matrix of the warp. x: the lane's
// row; pos: its position in the pivoted order. NC = 0: the generic rule (the
// largest |Re| + |Im|, ties to the smaller position; correctly rounded
// reciprocal); else the register-tiled rule (values within 2^-18 tie). Returns
// false (single-matrix warps only) on a zero or non-finite pivot.
template <int NP, int LPM, int NC, int T>
__device__ __forceinline__ bool lup_step(float2 (&x)[NP], float2 *F, int n,
                                         const GridLane<NP, LPM> &g, int &pos, int &par, bool &fail) {
  using Gd = Grid<NP, LPM>;
  constexpr bool GEN = NC == 0;
  const bool cand = pos >= T && g.sub < n;
  const unsigned mb = __float_as_uint(fabsf(x[T].x) + fabsf(x[T].y));
  float best;
  int bi;
  if constexpr (GEN) {
    const unsigned top = group_max<LPM>(cand ? mb : 0u);
    best = __uint_as_float(top);
    bi = 31 - (int)group_max<LPM>((cand && mb == top) ? 31u - (unsigned)pos : 0u);
  } else {
    const unsigned key = group_max<LPM>(cand ? ((mb & ~31u) | (31u - (unsigned)pos)) : 0u);
    best = __uint_as_float(key & ~31u);
    bi = 31 - (int)(key & 31u);
  }
  if (!(best > 0.0f) || !(best < INFINITY)) {
    if constexpr (Gd::G == 1) return false;
    fail = true;
  }
  if (cand && pos == bi) {
    float4 *row = reinterpret_cast<float4 *>(F + T * Gd::LDF);
#pragma unroll
    for (int k = 0; k < NP; k += 2) row[k / 2] = make_float4(x[k].x, x[k].y, x[k + 1].x, x[k + 1].y);
    pos = T;
  } else if (pos == T) {
    pos = bi;
  }
  par ^= bi != T ? 1 : 0;
  __syncwarp();
  if constexpr (T + 1 < NP) {
    const float2 ut = F[T * Gd::LDF + T];
    const float2 rp = GEN ? crcpf(ut) : crcpf_approx(ut);
    const bool below = pos > T && g.sub < n;
    const float2 l = cmulf(x[T], rp);
    const float2 lz = below ? l : make_float2(0.f, 0.f);
    if (below) x[T] = l;
    const float4 *row = reinterpret_cast<const float4 *>(F + T * Gd::LDF);
#pragma unroll
    for (int k = (T + 1) & ~1; k < NP; k += 2) {
      const float4 u = row[k / 2];
      if (k > T) x[k] = cfms(x[k], lz, make_float2(u.x, u.y));
      x[k + 1] = cfms(x[k + 1], lz, make_float2(u.z, u.w));
    }
  }
  return true;
}
template <int NP, int LPM, int NC, int T>
__device__ __forceinline__ bool lup_steps(float2 (&x)[NP], float2 *F, int n,
                                          const GridLane<NP, LPM> &g, int &pos, int &par, bool &fail) {
  if constexpr (T < (NC ? NC : NP)) {
    if (NC == 0 && T >= n) return true;
    if (!lup_step<NP, LPM, NC, T>(x, F, n, g, pos, par, fail)) return false;
    return lup_steps<NP, LPM, NC, T + 1>(x, F, n, g, pos, par, fail);
  } else {
    return true;
  }
}

// The LUP in shared memory on the 4 x 8 lane grid (one matrix per warp), rows
// of F exchanged, rowat[i] the original row at position i.
template <int NP, int NC>
__device__ __forceinline__ bool lup_shared(float2 *F, int *rowat, int n, int lane, int &par) {
  using Gd = Grid<NP, 32>;
  constexpr int LDF = Gd::LDF, SA = Gd::SA, SB = Gd::SB;
  constexpr bool GEN = NC == 0;
  const int tr = lane >> 3, tc = lane & 7;
  const float2 zero = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    const bool cand = lane >= t && lane < n;
    unsigned mb = 0u;
    float2 v = zero;
    if (cand) {
      v = F[lane * LDF + t];
      mb = __float_as_uint(fabsf(v.x) + fabsf(v.y));
    }
    float best;
    int bi;
    if constexpr (GEN) {
      const unsigned top = __reduce_max_sync(kFull, mb);
      best = __uint_as_float(top);
      bi = 31 - (int)__reduce_max_sync(kFull, (cand && mb == top) ? 31u - (unsigned)lane : 0u);
    } else {
      const unsigned key = __reduce_max_sync(kFull, cand ? ((mb & ~31u) | (31u - (unsigned)lane)) : 0u);
      best = __uint_as_float(key & ~31u);
      bi = 31 - (int)(key & 31u);
    }
    if (!(best > 0.0f) || !(best < INFINITY)) return false;  // zero/NaN/Inf pivot
    // the pivot to all lanes, the multipliers by the lanes' (exchanged) rows
    const float2 ut = shfl2(v, bi), vt = shfl2(v, t);
    if (bi != t) {
      if (lane < n && lane != t) {
        const float2 a = F[bi * LDF + lane];
        F[bi * LDF + lane] = F[t * LDF + lane];
        F[t * LDF + lane] = a;
      }
      if (lane == t) {
        F[t * LDF + t] = ut;
        const int a = rowat[bi];
        rowat[bi] = rowat[t];
        rowat[t] = a;
      }
      if (lane == bi) v = vt;
      par ^= 1;
    }
    const float2 rp = GEN ? crcpf(ut) : crcpf_approx(ut);
    if (lane > t && lane < n) F[lane * LDF + t] = cmulf(v, rp);
    __syncwarp();
    float2 lv[SA], uv[SB];
#pragma unroll
    for (int a = 0; a < SA; ++a) {
      const int i = 4 * a + tr;
      lv[a] = (i > t && i < n) ? F[i * LDF + t] : zero;
    }
#pragma unroll
    for (int b = 0; b < SB; ++b) {
      const int k = 8 * b + tc;
      uv[b] = (k > t && k < n) ? F[t * LDF + k] : zero;
    }
#pragma unroll
    for (int a = 0; a < SA; ++a) {
      if (4 * a + 3 <= t) continue;
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        if (8 * b + 7 <= t) continue;
        const int i = 4 * a + tr, k = 8 * b + tc;
        F[i * LDF + k] = cfms(F[i * LDF + k], lv[a], uv[b]);
      }
    }
    __syncwarp();
  }
  return true;
}

// Residual steps of block TBLK (t in [TB TBLK, TB TBLK + TB), t < n): slots
// whose rows or columns all lie before the block have nothing left to add.
template <int NP, int LPM, int TB, int TBLK>
__device__ __forceinline__ void residual_block(float4 (&acc)[Grid<NP, LPM>::SA][Grid<NP, LPM>::SB],
                                               const float2 *F, int n, const GridLane<NP, LPM> &g) {
  using Gd = Grid<NP, LPM>;
  constexpr int T0 = TBLK * TB;
  if constexpr (T0 < NP) {
    if (T0 >= n) return;
#pragma unroll 1
    for (int t = T0; t < min(T0 + TB, n); ++t) {
      float2 Uv[Gd::SB];
#pragma unroll
      for (int b = 0; b < Gd::SB; ++b) {
        if (Gd::GC * b + Gd::GC <= T0) continue;
        const int k = Gd::GC * b + g.c;
        Uv[b] = F[t * Gd::LDF + k];
        if (Gd::GC * b < T0 + TB && k < t) Uv[b] = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int a = 0; a < Gd::SA; ++a) {
        if (Gd::GR * a + Gd::GR <= T0) continue;
        const int i = Gd::GR * a + g.r;
        float2 l = F[i * Gd::LDF + t];
        if (Gd::GR * a < T0 + TB) {
          if (i < t) l = make_float2(0.f, 0.f);
          if (i == t) l = make_float2(1.f, 0.f);
        }
#pragma unroll
        for (int b = 0; b < Gd::SB; ++b) {
          if (Gd::GC * b + Gd::GC <= T0) continue;
          dot2_csub(acc[a][b], l, Uv[b]);
        }
      }
    }
    residual_block<NP, LPM, TB, TBLK + 1>(acc, F, n, g);
  }
}

// The FP32 path of one matrix per lane group. In: the FP64 matrix in HL (as
// double2, row stride LDH). HL, F, ints: this lane's matrix (Grid::kHL float4,
// Grid::kF float2, 2 NP ints); n the order, NC = n for the register-tiled
// rule or 0 for the generic one. The outcome is uniform over the group:
//  TILE_ACCEPT: prod, exp_sum, corr, par hold the determinant;
//  TILE_REFINE (NC != 0): ||E||_F within theta but above the FP32 solves' cap;
//    F holds L\U in pivoted order and HL's float2 view (row stride n + 1)
//    Y = L^-1 R;
//  TILE_REJECT, TILE_NONFINITE: for the FP64 route, or not finite.
// Lanes of a group past the batch's end run on whatever the group holds; every
// address depends on n and the lane only, or on positions below 32.
template <int NP, int LPM, int NC>
__device__ __forceinline__ int grid_factor(float4 *HL, float2 *F, int *ints, const int n_rt,
                                           int lane, float theta2, CFF &prod, int &exp_sum,
                                           float2 &corr, int &par) {
  using Gd = Grid<NP, LPM>;
  constexpr int GR = Gd::GR, GC = Gd::GC, SA = Gd::SA, SB = Gd::SB;
  constexpr int LDH = Gd::LDH, LDF = Gd::LDF;
  constexpr bool GEN = NC == 0;
  // n = 17..24: the LUP in shared memory and wider residual blocks, whose code
  // is half the size (32768 LLL x n=24, FP32 pass, us: 921 in registers, 825 in
  // shared memory, 767 with blocks of 8; Gaussian 680, 697, 670). n = 32 is
  // faster in registers (8192 LLL 412 against 492 to 547), the padded sizes
  // above 24 in registers with blocks of 8.
  constexpr bool kShared = NP == 24;
  constexpr int kTB = NP == 24 || (NP == 32 && GEN) ? 8 : Gd::GR;
  const int n = GEN ? n_rt : NC;
  const GridLane<NP, LPM> g(lane);
  const int sub = g.sub, r = g.r, c = g.c;
  const float2 zero = make_float2(0.f, 0.f);
  const double2 *A = reinterpret_cast<const double2 *>(HL);
  int *ecs = ints, *ers = ints + NP;

  // 1. exponents, columns first, as the exponent fields' places in the words
  int esum = 0;
  unsigned cm = 0u;
  if (sub < n) {
#pragma unroll 4
    for (int i = 0; i < n; ++i) {
      const uint4 w = *reinterpret_cast<const uint4 *>(A + i * LDH + sub);
      cm = max(cm, max(w.y & 0x7fffffffu, w.w & 0x7fffffffu));
    }
    const int ec = cm < 0x00100000u ? 0 : (int)(cm >> 20) - 1023;
    ecs[sub] = (ec + 1023) << 20;
    esum = ec;
  }
  const bool nonfinite = (__ballot_sync(kFull, cm >= 0x7ff00000u) & g.gmask) != 0u;
  if (Gd::G == 1 && nonfinite) return TILE_NONFINITE;
  __syncwarp();
  if (sub < n) {
    int m = (int)0x80000000;
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
      const uint4 w = *reinterpret_cast<const uint4 *>(A + sub * LDH + k);
      const unsigned raw = max(w.y & 0x7fffffffu, w.w & 0x7fffffffu);
      const int v = (int)raw - ecs[k];
      if (raw >= 0x00100000u) m = max(m, v);
    }
    const int er = m == (int)0x80000000 ? 0 : (m >> 20);
    ers[sub] = (int)((unsigned)(er - 127) << 20);
    esum += er;
  }
  exp_sum = group_add<LPM>(esum);
  __syncwarp();
  // 2. split: hi + lo in place of each entry
  {
    int i = sub / n, k = sub - i * n;
    const int di = LPM / n, dk = LPM - di * n;
#pragma unroll 2
    for (int e = sub; e < n * n; e += LPM) {
      const int idx = i * LDH + k;
      const double2 v = A[idx];
      const int adj = (int)((unsigned)ecs[k] + (unsigned)ers[i]);
      float xh, xl, yh, yl;
      split_words(v.x, adj, xh, xl);
      split_words(v.y, adj, yh, yl);
      HL[idx] = make_float4(xh, yh, xl, yl);
      if constexpr (kShared) F[i * LDF + k] = make_float2(xh, yh);
      i += di;
      k += dk;
      if (k >= n) {
        k -= n;
        ++i;
      }
    }
  }
  __syncwarp();

  // 3. FP32 LUP: lane = row
  bool fail = false;
  par = 0;
  if constexpr (kShared) {
    int *rowat = ints;  // (the exponents are done with)
    if (sub < NP) rowat[sub] = sub;
    if constexpr (NC < NP) {
      // padding: rows and columns past n are zero
      for (int e = lane; e < NP * NP; e += 32) {
        const int i = e / NP, k = e - i * NP;
        if (i >= n || k >= n) F[i * LDF + k] = zero;
      }
    }
    __syncwarp();
    if (!lup_shared<NP, NC>(F, rowat, n, lane, par)) return TILE_REJECT;
  } else {
    float2 x[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      x[k] = zero;
      if (sub < n && k < n) {
        const float4 h = HL[sub * LDH + k];
        x[k] = make_float2(h.x, h.y);
      }
    }
    if ((GEN || NC < NP) && sub >= n && sub < NP) {
      // rows of the padding: zero multipliers
      float4 *row = reinterpret_cast<float4 *>(F + sub * LDF);
#pragma unroll
      for (int k = 0; k < NP; k += 2) row[k / 2] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    int pos = sub;
    if (!lup_steps<NP, LPM, NC, 0>(x, F, n, g, pos, par, fail)) return TILE_REJECT;
    __syncwarp();
    // the row at each position (the exponents are done with); a failed group's
    // positions may be incomplete or out of range, so it starts from the identity
    int *rowat = ints;
    if (sub < NP) rowat[sub] = sub;
    __syncwarp();
    if (sub < n && pos < NP) rowat[pos] = sub;
    __syncwarp();
  }

  // 4. residual R = P A^ - L U in float-float
  float2 Y[SA][SB];
  {
    float4 acc[SA][SB];
#pragma unroll
    for (int a = 0; a < SA; ++a) {
      const int i = GR * a + r;
      const bool row_ok = (NP % GR == 0 && !GEN && NC == NP) || i < n;
      const int row = row_ok ? ints[i] : 0;
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int k = GC * b + c;
        acc[a][b] = (row_ok && ((NP % GC == 0 && !GEN && NC == NP) || k < n))
                        ? HL[row * LDH + k]
                        : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    residual_block<NP, LPM, kTB, 0>(acc, F, n, g);
#pragma unroll
    for (int a = 0; a < SA; ++a)
#pragma unroll
      for (int b = 0; b < SB; ++b)
        Y[a][b] = make_float2(__fadd_rn(acc[a][b].x, acc[a][b].z),
                              __fadd_rn(acc[a][b].y, acc[a][b].w));
  }
  __syncwarp();  // HL is free: its float2 view takes Y or E (Rm), then the diagonal scratch
  float2 *Rm = reinterpret_cast<float2 *>(HL);
  const int ldr = n + 1;
  float2 *diag = Rm + n * ldr;

  // 5. Y = L^-1 R (unit lower)
#pragma unroll
  for (int s = 0; s < SA; ++s) {
#pragma unroll 1
    for (int u = 0; u < GR; ++u) {
      const int t = GR * s + u;
      if (t >= n - 1) break;
      float2 yt[SB];
#pragma unroll
      for (int b = 0; b < SB; ++b) yt[b] = shfl2(Y[s][b], g.at(u, c));
      {
        const bool below = r > u && GR * s + r < n;
        const float2 l = below ? F[(GR * s + r) * LDF + t] : zero;
#pragma unroll
        for (int b = 0; b < SB; ++b) {
          const float2 v = cfms(Y[s][b], l, yt[b]);
          Y[s][b] = below ? v : Y[s][b];
        }
      }
#pragma unroll
      for (int a = s + 1; a < SA; ++a) {
        const float2 l = F[(GR * a + r) * LDF + t];
#pragma unroll
        for (int b = 0; b < SB; ++b) Y[a][b] = cfms(Y[a][b], l, yt[b]);
      }
    }
  }
  if constexpr (!GEN) {
#pragma unroll
    for (int a = 0; a < SA; ++a)
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int i = GR * a + r, k = GC * b + c;
        if (i < n && k < n) Rm[i * ldr + k] = Y[a][b];
      }
  }
  // E = U^-1 Y; the reciprocals of the diagonal first, one per lane
  if (sub < n) diag[sub] = crcpf(F[sub * LDF + sub]);
  __syncwarp();
#pragma unroll
  for (int s = SA - 1; s >= 0; --s) {
#pragma unroll 1
    for (int u = GR - 1; u >= 0; --u) {
      const int t = GR * s + u;
      if (t >= n) continue;
      const float2 dinv = diag[t];
      float2 et[SB];
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        et[b] = cmulf(shfl2(Y[s][b], g.at(u, c)), dinv);
        Y[s][b] = r == u ? et[b] : Y[s][b];
      }
      {
        const bool above = r < u;
        const float2 uu = above ? F[(GR * s + r) * LDF + t] : zero;
#pragma unroll
        for (int b = 0; b < SB; ++b) {
          const float2 v = cfms(Y[s][b], uu, et[b]);
          Y[s][b] = above ? v : Y[s][b];
        }
      }
#pragma unroll
      for (int a = 0; a < s; ++a) {
        const float2 uu = F[(GR * a + r) * LDF + t];
#pragma unroll
        for (int b = 0; b < SB; ++b) Y[a][b] = cfms(Y[a][b], uu, et[b]);
      }
    }
  }

  // 6. product of the diagonal of U in float-float (the lanes past the group's
  // hold the identity of a full warp's product)
  {
    CFF acc = {1.0f, 0.0f, 0.0f, 0.0f, 0};
    if (sub < n) {
      const float2 u = F[sub * LDF + sub];
      CFF v = {u.x, 0.0f, u.y, 0.0f, 0};
      ff_renorm(v);
      acc = ff_cmul(acc, v);
    }
#pragma unroll 1
    for (int off = LPM / 2; off; off >>= 1) acc = ff_cmul(acc, shfl_cff(acc, off, true));
    prod = shfl_cff(acc, g.gb, false);
  }
  // acceptance, from the group's first lane's sum
  float f;
  {
    constexpr int NR = Chains<LPM>::NR, NCH = Chains<LPM>::NCH;
    float p[NR][NCH];
#pragma unroll
    for (int q = 0; q < NR; ++q)
#pragma unroll
      for (int w = 0; w < NCH; ++w) p[q][w] = 0.0f;
#pragma unroll
    for (int a = 0; a < SA; ++a)
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        float &s = p[a % NR][b % NCH];
        s = __fmaf_rn(Y[a][b].x, Y[a][b].x, __fmaf_rn(Y[a][b].y, Y[a][b].y, s));
      }
    f = __shfl_sync(kFull, chain_sum<LPM>(p), g.gb);
  }
  const float la_est = tile_la_est(prod, exp_sum);
  const float rel_cap = kCorrRelCap * fmaxf(1.0f, la_est);
  int code = TILE_ACCEPT;
  if (!(f <= rel_cap * rel_cap)) code = GEN ? TILE_REJECT : TILE_REFINE;
  if (!(f <= theta2) || fail) code = TILE_REJECT;
  if (nonfinite) code = TILE_NONFINITE;
  const bool accept = code == TILE_ACCEPT;
  if (!__any_sync(kFull, accept)) return code;

  // 7. log det(I + E): the series where its bound allows (register-tiled
  // rule), else the elimination; each runs if any matrix of the warp needs it
  const float nf = sqrtf(f);
  const bool series = !GEN && nf * f <= 3e-12f * fmaxf(1.0f, la_est - 1.0f) * (1.0f - nf);
  corr = zero;
  if (!GEN && __any_sync(kFull, accept && series)) {
    constexpr int NR = Chains<LPM>::NR, NCH = Chains<LPM>::NCH;
    float trx[NR][NCH], try_[NR][NCH], t2x[NR][NCH], t2y[NR][NCH];
#pragma unroll
    for (int q = 0; q < NR; ++q)
#pragma unroll
      for (int w = 0; w < NCH; ++w) trx[q][w] = try_[q][w] = t2x[q][w] = t2y[q][w] = 0.0f;
    // entry (t, t), t = GR a + r, sits in slot (a, GR a / GC) of the lane with
    // c = (GR a) % GC + r
#pragma unroll
    for (int a = 0; a < SA; ++a) {
      const int b = GR * a / GC;
      if (c == GR * a % GC + r && GR * a + r < n) {
        trx[a % NR][b % NCH] += Y[a][b].x;
        try_[a % NR][b % NCH] += Y[a][b].y;
      }
    }
    // tr(E^2) = sum_ik E_ik E_ki, the transposed entries through shared memory
    // (a matrix left for refinement keeps its Y there)
    __syncwarp();
    if (accept) {
#pragma unroll
      for (int a = 0; a < SA; ++a)
#pragma unroll
        for (int b = 0; b < SB; ++b) {
          const int i = GR * a + r, k = GC * b + c;
          if (i < n && k < n) Rm[i * ldr + k] = Y[a][b];
        }
    }
    __syncwarp();
#pragma unroll
    for (int a = 0; a < SA; ++a)
#pragma unroll
      for (int b = 0; b < SB; ++b) {
        const int i = GR * a + r, k = GC * b + c;
        if (i < n && k < n) {
          const float2 e = cmulf(Y[a][b], Rm[k * ldr + i]);
          t2x[a % NR][b % NCH] += e.x;
          t2y[a % NR][b % NCH] += e.y;
        }
      }
    const float sx = chain_sum<LPM>(trx), sy = chain_sum<LPM>(try_);
    const float qx = chain_sum<LPM>(t2x), qy = chain_sum<LPM>(t2y);
    corr = make_float2(__shfl_sync(kFull, __fmaf_rn(-0.5f, qx, sx), g.gb),
                       __shfl_sync(kFull, __fmaf_rn(-0.5f, qy, sy), g.gb));
  }
  if (__any_sync(kFull, accept && !series)) {
#pragma unroll
    for (int s = 0; s < SA; ++s) {
      const int q = GR * s / GC;  // column slot of t = GR s + u
#pragma unroll 1
      for (int u = 0; u < GR; ++u) {
        const int t = GR * s + u;
        if (t >= n) break;
        const int ct = GR * s % GC + u;  // grid column of t
        const float2 d = shfl2(Y[s][q], g.at(u, ct));
        if (sub == 0) diag[t] = d;
        if (t == n - 1) break;
        const float2 rp = crcpf(make_float2(1.0f + d.x, d.y));
        float2 et[SB];
#pragma unroll
        for (int b = q; b < SB; ++b) et[b] = shfl2(Y[s][b], g.at(u, c));
#pragma unroll
        for (int a = s; a < SA; ++a) {
          const float2 l = cmulf(shfl2(Y[a][q], g.at(r, ct)), rp);
#pragma unroll
          for (int b = q; b < SB; ++b) Y[a][b] = cfms(Y[a][b], l, et[b]);
        }
      }
    }
    __syncwarp();
    float cre = 0.0f, cim = 0.0f;
    if (sub < n) {
      const float2 d = diag[sub];
      cre = __fmaf_rn(0.5f, log1pf(__fmaf_rn(d.x, d.x, __fmaf_rn(d.y, d.y, 2.0f * d.x))), cre);
      cim += atan2f(d.y, 1.0f + d.x);
    }
#pragma unroll
    for (int off = LPM / 2; off; off >>= 1) {
      cre += __shfl_xor_sync(kFull, cre, off);
      cim += __shfl_xor_sync(kFull, cim, off);
    }
    const float2 e = make_float2(__shfl_sync(kFull, cre, g.gb), __shfl_sync(kFull, cim, g.gb));
    if (!series) corr = e;
  }
  return code;
}

// F of one matrix from the grid path's row stride to stride N + 1, in place.
template <int NP, int N>
__device__ __forceinline__ void repack_f(float2 *F, int lane) {
  constexpr int K = (N * N + 31) / 32;
  float2 v[K];
  __syncwarp();
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int e = lane + 32 * q;
    if (e < N * N) v[q] = F[e / N * (NP + 2) + e % N];
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const int e = lane + 32 * q;
    if (e < N * N) F[e / N * (N + 1) + e % N] = v[q];
  }
  __syncwarp();
}

// FP64 refactorisation of matrix sb of src into output ob, in one matrix's area
// of the lane grid, by the whole warp. The row scales lie in the padding after the
// matrix, or, where there is none (n = NP = 8, 12, 16: sizes without a correction),
// over F; the correction of n >= 17 takes F and the ints.
template <int NP, class Src>
__device__ __forceinline__ void grid_refactor(const Src &src, long long sb, int n, float4 *HL,
                                              float2 *F, int *ints, int lane, long long ob,
                                              double *logabs, double *phase, int8_t *parity,
                                              int32_t *status, int flag) {
  double *hold = n < NP ? reinterpret_cast<double *>(HL + (size_t)n * (n + 1))
                        : reinterpret_cast<double *>(F);
  const CorrScratch cs{F, ints, hold};
  fallback_fp64_src(src, sb, n, reinterpret_cast<double2 *>(HL), n + 1, hold, lane, ob, logabs,
                    phase, parity, status, flag, NP > 16 ? &cs : nullptr);
}
// The same out of line, for a kernel with many sizes. (In the batched kernels
// the call cost more than the code it saves: 65536 LLL x n=16 645 -> 677 us.)
template <int NP, class Src>
__device__ __noinline__ void grid_refactor_call(const Src src, long long sb, int n, float4 *HL,
                                                float2 *F, int *ints, int lane, long long ob,
                                                double *logabs, double *phase, int8_t *parity,
                                                int32_t *status, int flag) {
  grid_refactor<NP>(src, sb, n, HL, F, ints, lane, ob, logabs, phase, parity, status, flag);
}

// One unit of a warp: matrices b0 + at(q), q < cnt, of src, staged in areas
// HLw + q kHL, into outputs ob0 + at(q): the FP32 path, then what it does not
// accept: refined or refactorised right here (INPLACE, NP < 32), or handed to
// defer(b, routed, can_refine, prod, exp_sum, par). share64k: the share routed to
// FP64, for units that hold some of it beside others: it goes to defer in any case
// (the kernels ask for units of such matrices alone before they stage them). CALL:
// FP64 out of line.
template <int NP, int LPM, int NC, bool INPLACE, bool CALL, class Src, class At, class Defer>
__device__ __forceinline__ void grid_unit(const Src &src, long long b0, long long ob0, int cnt,
                                          int n, float4 *HLw, float2 *Fw, int *Iw, int lane,
                                          float theta2, unsigned int share64k, bool refine, At at,
                                          Defer defer, DeferredOut &out, double *logabs,
                                          double *phase, int8_t *parity, int32_t *status) {
  using Gd = Grid<NP, LPM>;
  const int grp = lane / LPM;
  CFF prod;
  int exp_sum, par;
  float2 corr;
  int code = grid_factor<NP, LPM, NC>(HLw + grp * Gd::kHL, Fw + grp * Gd::kF, Iw + grp * 2 * NP, n,
                                      lane, theta2, prod, exp_sum, corr, par);
  bool routed = false;
  if (share64k && grp < cnt && code != TILE_NONFINITE) {
    routed = route_fp64_entry(src.first(b0 + grp, n), share64k);
    if (routed) code = TILE_REJECT;
  }
#pragma unroll 1
  for (int q = 0; q < cnt; ++q) {
    const int from = q * LPM;
    int cq = code, eq = exp_sum, rq = par;
    CFF pq = prod;
    float2 kq = corr;
    if constexpr (Gd::G > 1) {
      cq = __shfl_sync(kFull, code, from);
      pq = shfl_cff(prod, from, false);
      eq = __shfl_sync(kFull, exp_sum, from);
      rq = __shfl_sync(kFull, par, from);
      kq = shfl2(corr, from);
    }
    const long long b = b0 + at(q), ob = ob0 + at(q);
    if (cq == TILE_ACCEPT) {
      out.push(lane, ob, pq, eq, kq, rq, logabs, phase, parity, status);
      continue;
    }
    if (cq == TILE_NONFINITE) {
      emit_nonfinite(lane, ob, logabs, phase, parity, status);
      continue;
    }
    const bool rt = Gd::G > 1 ? share64k && __shfl_sync(kFull, (int)routed, from) != 0 : routed;
    if constexpr (!INPLACE) {
      defer(b, rt, cq == TILE_REFINE && refine, pq, eq, rq);
    } else if (rt) {
      defer(b, true, false, pq, eq, rq);
    } else {
      float4 *HLq = HLw + q * Gd::kHL;
      float2 *Fq = Fw + q * Gd::kF;
      int *Iq = Iw + q * 2 * NP;
      if constexpr (NC != 0) {
        if (cq == TILE_REFINE && refine) {
          float2 *Rm = reinterpret_cast<float2 *>(HLq);
          repack_f<NP, NC>(Fq, lane);
          if (mixed_refine_tile<NC>(Fq, Rm, Rm + NC * (NC + 1),
                                    reinterpret_cast<float2 *>(Iq), lane, theta2,
                                    tile_la_est(pq, eq), kq)) {
            out.push(lane, ob, pq, eq, kq, rq, logabs, phase, parity, status);
            continue;
          }
        }
      }
      if constexpr (CALL)
        grid_refactor_call<NP>(src, b, n, HLq, Fq, Iq, lane, ob, logabs, phase, parity, status,
                               LUFQHE_ST_FALLBACK);
      else
        grid_refactor<NP>(src, b, n, HLq, Fq, Iq, lane, ob, logabs, phase, parity, status,
                          LUFQHE_ST_FALLBACK);
    }
  }
}

}  // namespace
}  // namespace mixed
}  // namespace lufqhe
