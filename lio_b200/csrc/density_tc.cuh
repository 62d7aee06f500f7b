// Tensor-core form of the density contraction (included by engine.cu inside its
// anonymous namespace; uses GroupDev and packed_index).
//
// G^a = A^a . D for the basis kinds a = F (LDA) or F, dF/dx, dF/dy, dF/dz (GGA),
// with D the group's dense density, computed with int8 tensor-core products
// (tcgen05 kind::i8, exact int32 accumulation in TMEM) on Ozaki-style slices:
//   A^a_pj = 2^(e_p) * sum_s a_s[p][j] 128^-(s+1),   |a_s| <= 64  (per point p)
//   D_ji   = 2^(f_T) * sum_t d_t[i][j] 128^-(t+1),   |d_t| <= 64  (per 32-function tile T of i)
// and G_pi = 2^(e_p + f_T - 7(S+1)) * sum_l acc_l[p][i] 128^(S-1-l), where the
// level accumulator acc_l holds every slice pair s + t = l (pairs with
// s + t >= S are dropped). With S = 6 the dropped terms are ~2^-42 of
// max_j|A_pj| * max_(j, i in T)|D_ji| per term, far inside the 1e-7 / 1e-6 Ha
// absolute tolerances. One exponent per tile lets the epilogue scale a whole
// row dot once instead of every G_pi.
//
// Slice pairs in few, wide MMAs: the S slices of a 32-function D tile are
// stacked along N ("tall" B operand, row t * 32 + i holds d_t[i]). For A slice s
// one MMA with N = (S - s) * 32 multiplies a_s by d_0 .. d_(S-1-s) (a prefix of
// the tall operand) into TMEM columns starting at level s, so product (s, t)
// lands on level s + t: S MMAs per K step and kind instead of S(S+1)/2 narrow
// ones (an MMA costs about the same for every N up to 64 on this part).
//
// The row-dot epilogue needs F, dF and d2F at (p, i) in FP64. They are not
// streamed from HBM (80 bytes per point and function, three quarters of the
// kernel's traffic before). Each value is P(r) R(r): a Cartesian monomial of the
// point's displacement from the function's atom times the shell's contracted
// radial part, whose sums t, tg, th (the only exponentials) are computed once per
// geometry (k_radial, 24 bytes per point and shell). The epilogue contracts G
// shell by shell in factored form: with S0 = sum_c P_c G_c, S1_a = sum_c
// dP_c/da G_c and S2_ab = sum_c d2P_c/da db G_c over the shell's components,
//   sum_c F_c G_c        = t S0
//   sum_c dF_c/da G_c    = t S1_a + r_a tg2 S0
//   sum_c d2F_c/dadb G_c = t S2_ab + tg2 (r_b S1_a + r_a S1_b + delta_ab S0) + th4 r_a r_b S0
// (tg2 = -2 tg, th4 = 4 th; the closed forms of g2g/cpu/functions.cpp:81-352
// summed over a shell). The shells of an atom share r, so U0 = sum tg2 S0,
// W0 = sum th4 S0 and V_a = sum tg2 S1_a are summed over them first and meet r
// once per atom:
//   grad_a += r_a U0,   d2_ab += r_a (r_b W0 + V_b) + r_b V_a + delta_ab U0.
// For that the device keeps a group's functions atom by atom (group_order). An s
// shell then costs 3 FP64 operations for kind F and 1 for a gradient kind, a p
// shell 12 and 7.
#pragma once
#include <type_traits>

#include "umma.cuh"

constexpr int kSlices = 6;       // Ozaki slices per operand
constexpr int kTcPoints = 128;   // UMMA M: points per tile
constexpr int kTcFuncs = 32;     // functions per density tile (output columns per level)
constexpr int kTcTall = kSlices * kTcFuncs;  // rows of the stacked D operand
constexpr int kTcEpiWarps = 8;   // two per TMEM lane quadrant
constexpr int kTcCpw = kTcFuncs / 2;         // columns per epilogue warp
constexpr int kTcSliceA = 32 * kTcPoints;    // bytes of one A slice per 32-byte K step
constexpr int kTcStepA = kSlices * kTcSliceA;  // one kind's A slices per K step (contiguous)
constexpr int kTcStepD = 32 * kTcTall;         // one spin's stacked D slices per K step (contiguous)
constexpr int kTcChunk = kTcFuncs * kTcPoints;  // doubles of one blocked basis chunk (kind, 32 functions)

// A batch of MMAs is one kind (F, x, y, z) of a (128-point tile, 32-function tile),
// every spin: NS x S x 32 level columns in TMEM, one buffer at two spins, two at one.
// A unit of the epilogue is KP batches: one kind with both spins, or (one spin, GGA)
// the kinds {F, x} then {y, z}, so that a shell's fixed cost is shared by two values
// per column; LDA: {F}.
constexpr int kTcMaxTileShells = 32;  // shells that 32 functions touch, at most
template <bool GGA, int NS>
struct TcCfg {
  static constexpr int KP = (GGA && NS == 1) ? 2 : 1;
  static constexpr int NA = GGA ? 4 : 1;   // kinds of the contraction
  static constexpr int NP = NA / KP;       // units per function tile
  static constexpr int NQ = GGA ? 10 : 1;
  static constexpr int NR = GGA ? 3 : 1;   // radial sums per (shell, point): t (LDA); t, -2 tg, 4 th (GGA)
  static constexpr int kStage = kTcStepA + NS * kTcStepD;  // a K step of one kind: its A slices, every spin's D slices
  static constexpr int kBufs = NS == 2 ? 1 : 2;            // level buffers
  static constexpr uint32_t kLevels = NS * kSlices * kTcFuncs;
  static constexpr uint32_t kCols = kBufs * kLevels;
  // after the level columns, the unit's G in FP64: per function column c the
  // NS x KP values, two 32-bit TMEM columns each (column kCols + c * kGPer + ...)
  static constexpr uint32_t kGPer = 2 * NS * KP;
  static constexpr uint32_t kTmem = 512;
  static_assert(kCols + kTcFuncs * kGPer <= kTmem, "levels and G fit the 512 TMEM columns");
  // epilogue warps, operand producer, MMA issuer
  static constexpr int kWarps = kTcEpiWarps + 2;
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kProd = kTcEpiWarps, kMma = kTcEpiWarps + 1;
  // Dynamic shared memory, all of it filled by the producer's bulk copies: two tile
  // slots (the group's record, the points' x, y, z and exponents) | one or two shell
  // slots (of a 32-function tile: which shells, their records and radial sums
  // [shell][NR][128 points]) | column group 1 -> 0 hand-off | operand ring.
  // Sized by nrf, the most shells that a 32-function tile of the system's groups
  // touches: two shell slots where two stages still fit beside them.
  static constexpr int kTileXyz = 256, kTileExp = kTileXyz + 3 * kTcPoints * 8;
  static constexpr int kTileSlot = kTileExp + NA * kTcPoints * 2;
  static_assert(sizeof(GroupDev) <= kTileXyz, "a group's record fits its slot");
  static constexpr int kShellRec = 128, kShellRad = kShellRec + kTcMaxTileShells * 32;
  static constexpr int kRed = 4 * NS * NQ * 32 * 8;  // per lane quadrant: [spin][value][lane] FP64
  static constexpr int kMaxStages = 4;
  static constexpr int kMaxSmem = 227 * 1024 - 1024;  // less the static part
  struct Layout {
    int shell_slot, nrb, stages;  // bytes of a shell slot, shell slots, operand stages
    __host__ __device__ constexpr int shells() const { return 2 * kTileSlot; }
    __host__ __device__ constexpr int red() const { return shells() + nrb * shell_slot; }
    __host__ __device__ constexpr int ring() const { return red() + kRed; }
    __host__ __device__ constexpr int total() const { return ring() + stages * kStage; }
  };
  static constexpr Layout layout(int nrf) {
    Layout l{kShellRad + nrf * NR * kTcPoints * 8, 2, 0};
    for (;; l.nrb = 1) {
      l.stages = (kMaxSmem - l.ring()) / kStage;
      if (l.stages > kMaxStages) l.stages = kMaxStages;
      if (l.stages >= 2 || l.nrb == 1) return l;
    }
  }
  static_assert((kMaxSmem - 2 * kTileSlot - kShellRad - kTcMaxTileShells * NR * kTcPoints * 8 - kRed) / kStage >= 2,
                "two stages beside one shell slot of any system");
  // The form's limit on a group's functions, in 32s. Nothing here needs it: shared memory no longer
  // grows with a group's functions (the limit is what it held when each had an entry per spin, beside
  // two stages and per-warp radial sums), and int32 levels hold far more (below). It stays as it is
  // known to callers, who are refused (mode 1) or given the FP64 form (mode 3) above it.
  static constexpr int kMaxFuncs = (227 * 1024 - 256 - 2 * (KP * kTcStepA + NS * kTcStepD) - kTcEpiWarps * 16 * NR * 32 * 8) /
                                   (8 * NS) / 32 * 32;
  static_assert((long long)kSlices * 64 * 64 * kMaxFuncs < (1ll << 31), "level accumulators over a group's functions");
};

// where the layouts change over to one shell slot; tests/test_gpu_shell_slots.py runs both sides
static_assert(TcCfg<true, 2>::layout(20).nrb == 2 && TcCfg<true, 2>::layout(21).nrb == 1 &&
                  TcCfg<true, 1>::layout(24).nrb == 2 && TcCfg<true, 1>::layout(25).nrb == 1 &&
                  TcCfg<false, 2>::layout(32).nrb == 2 && TcCfg<false, 1>::layout(32).nrb == 2,
              "the cases of the shell slot test");

// exponent so that |x| * 2^-e <= 1/2 for every |x| <= amax
__device__ __forceinline__ int slice_exponent(double amax) { return amax > 0.0 ? ilogb(amax) + 2 : 0; }

// exact 2^k as a double (k within the normal range), else ldexp
__device__ __forceinline__ double pow2(int k) {
  return (k > -1022 && k < 1024) ? __longlong_as_double((long long)(k + 1023) << 52) : ldexp(1.0, k);
}

// The S = 6 base-128 digits of x (|x| < 1/2), all from one rounding on the
// FP64 adder: t = 2^52 + B + x 2^42 with B = 64 (128^6 - 1) / 127 (even) rounds
// x 2^42 to the nearest integer N, ties to even, and the low mantissa bits of
// t hold M = N + B >= 0. The base-128 digits m_k of M less 64 are balanced
// digits of N (|m_k - 64| <= 64), so
//   x = sum_s (m_(5-s) - 64) 128^-(s+1) + r,  |r| <= 2^-43,
// with two FP64 operations per value instead of three per digit for a
// digit-by-digit extraction. `s42` is 2^42 times the row's power-of-two scale
// (digit_scale). Returns t's two 32-bit halves (M = bits 0..42).
__device__ __forceinline__ void digits_m(double x, double s42, uint32_t& lo, uint32_t& hi) {
  const double t = fma(x, s42, 4505815965769792.0);  // 2^52 + B
  lo = (uint32_t)__double2loint(t);
  hi = (uint32_t)__double2hiint(t);
}
// `s42` for a row with exponent e: 2^(42 - e), or 0 (every digit zero) for a
// row whose values are all below 2^-981, where 2^(42 - e) would leave the
// double range; the dropped values are far below any tolerance
__device__ __forceinline__ double digit_scale(int e) { return e > -980 ? pow2(42 - e) : 0.0; }

// m_(5-s), the field of slice s (0 = most significant), in the low byte; for
// s >= 1 bit 7 of that byte belongs to the next field and is masked by
// pack_digits. t's exponent bits (from bit 20 of hi) never reach a low byte.
__device__ __forceinline__ uint32_t digit_field(uint32_t lo, uint32_t hi, int s) {
  switch (s) {
    case 0: return hi >> 3;                        // bits 35..42 (m_5 <= 128)
    case 1: return __funnelshift_r(lo, hi, 28);    // bits 28..34
    case 2: return lo >> 21;
    case 3: return lo >> 14;
    case 4: return lo >> 7;
    default: return lo;
  }
}
// four fields (low bytes, first point lowest) -> four int8 digits m - 64,
// byte-wise without carries between bytes; slice 0 keeps its bit 7 (m_5 = 128
// gives digit 64)
__device__ __forceinline__ uint32_t pack_digits(uint32_t f0, uint32_t f1, uint32_t f2, uint32_t f3, bool top) {
  const uint32_t w = __byte_perm(__byte_perm(f0, f1, 0x0040), __byte_perm(f2, f3, 0x0040), 0x5410);
  const uint32_t low = (w & 0x7F7F7F7Fu) + 0x40404040u;
  return top ? low ^ ((w ^ 0xC0C0C0C0u) & 0x80808080u) : low ^ 0x80808080u;
}

// ---------------------------------------------------------------- A slices
// Per geometry: one thread per (group, point) and kind; reads the blocked FP64
// basis (NK kinds per block), writes the per-point exponent and the int8
// slices. Layout per 128-point tile T, kind a and 32-function K step kk: the S
// slices one after the other (kTcStepA bytes, one bulk copy), each in the
// K-major interleaved UMMA layout of a 128-row x 32-byte block.
template <int NA>
__global__ void k_slice_basis(const int2* __restrict__ tiles, const GroupDev* __restrict__ groups,
                              const double* __restrict__ bblk, int NK, int8_t* __restrict__ aslices,
                              int16_t* __restrict__ aexp) {
  const int2 t = tiles[blockIdx.x];
  const GroupDev G = groups[t.x];
  const int r = threadIdx.x;
  const int p = t.y * kTcPoints + r;
  const int nks = G.m32 / 32;
  // value (kind a, function j) of this point
  auto val = [&](int a, int j) {
    return bblk[G.bb_off + ((long long)(t.y * G.nftc + (j >> 5)) * NK + a) * kTcChunk + (j & 31) * kTcPoints + r];
  };
  for (int a = 0; a < NA; a++) {
    double amax = 0.0;
    for (int j = 0; j < G.m; j++) amax = fmax(amax, fabs(val(a, j)));
    const int e = slice_exponent(amax);
    const double s42 = digit_scale(e);
    aexp[G.aexp_off + (long long)a * G.ldp + p] = (int16_t)e;
    int8_t* dst = aslices + G.sl_off + (long long)(t.y * NA + a) * nks * kTcStepA;
    // 16 consecutive functions at a time: per slice their 16 digits are one
    // contiguous 16-byte row segment of the K-major block, one store
    for (int j0 = 0; j0 < G.m32; j0 += 16) {
      uint32_t lo[16], hi[16];
#pragma unroll
      for (int k = 0; k < 16; k++) digits_m(j0 + k < G.m ? val(a, j0 + k) : 0.0, s42, lo[k], hi[k]);
      int8_t* blk = dst + (j0 >> 5) * kTcStepA + lio::umma::kmajor_offset(r, j0 & 31, kTcPoints);
#pragma unroll
      for (int s = 0; s < kSlices; s++) {
        uint32_t w[4];
#pragma unroll
        for (int k4 = 0; k4 < 4; k4++)
          w[k4] = pack_digits(digit_field(lo[4 * k4], hi[4 * k4], s), digit_field(lo[4 * k4 + 1], hi[4 * k4 + 1], s),
                              digit_field(lo[4 * k4 + 2], hi[4 * k4 + 2], s),
                              digit_field(lo[4 * k4 + 3], hi[4 * k4 + 3], s), s == 0);
        *reinterpret_cast<uint4*>(blk + s * kTcSliceA) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

// --------------------------------------------------------------- D slices
// Per solve: one CTA per (group, 32-function tile) and spin (blockIdx.y). Lane r
// of every warp is function i = 32 tile + r; the warps share the j's in pieces of
// 8. Gathers column i of the group's density from the packed matrix (off-diagonal
// packed values halved), takes the tile's exponent (one per 32 columns, from the
// largest |D_ji| of the tile, stored for each of its functions) and writes its S
// slices into the stacked operand: per tile and 32-function K step kk a 192-row x
// 32-byte block (kTcStepD bytes, one bulk copy) whose row t * 32 + i holds d_t[i].
// Bound by the latency of the gathers (the matrices sit in L2): 8 of them in
// flight per thread over 8 warps, and each warp's first piece stays in registers
// between the two passes. One warp per tile that walked all j's one load at a time
// took 94 us per spin at 256 atoms, 74 us at 121 atoms (LDA) and 28 us at 27; this
// takes 54 us for both spins, 25 and 15.
constexpr int kSdWarps = 8;
__global__ void __launch_bounds__(32 * kSdWarps)
    k_slice_density(const int2* __restrict__ tiles, const GroupDev* __restrict__ groups,
                    const int* __restrict__ fn_glob, const double* __restrict__ P_a, const double* __restrict__ P_b,
                    int8_t* __restrict__ dsl_a, int16_t* __restrict__ dexp_a, int8_t* __restrict__ dsl_b,
                    int16_t* __restrict__ dexp_b, int8_t* __restrict__ dhalf_a, int8_t* __restrict__ dhalf_b) {
  __shared__ double wmax[kSdWarps];
  const int2 t = tiles[blockIdx.x];
  const GroupDev& G = groups[t.x];
  const int r = threadIdx.x & 31, warp = threadIdx.x >> 5;  // function within the tile
  const int i = t.y * kTcFuncs + r, m = G.m, M = G.pk_M;
  const int* fg = fn_glob + G.fn_off;
  const double* P = (blockIdx.y == 0 ? P_a : P_b) + G.pk_off;
  const int gi = i < m ? fg[i] : 0;
  auto piece = [&](int j0, double (&v)[8]) {  // D_ji of 8 consecutive j
#pragma unroll
    for (int k = 0; k < 8; k++) {
      v[k] = 0.0;
      if (i < m && j0 + k < m) {
        const int gj = fg[j0 + k];
        v[k] = P[packed_index(gi, gj, M)] * (gi != gj ? 0.5 : 1.0);
      }
    }
  };
  double first[8], amax = 0.0;
  piece(8 * warp, first);
#pragma unroll
  for (int k = 0; k < 8; k++) amax = fmax(amax, fabs(first[k]));
  for (int j0 = 8 * (warp + kSdWarps); j0 < m; j0 += 8 * kSdWarps) {
    double v[8];
    piece(j0, v);
#pragma unroll
    for (int k = 0; k < 8; k++) amax = fmax(amax, fabs(v[k]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (r == 0) wmax[warp] = amax;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kSdWarps; w++) amax = fmax(amax, wmax[w]);
  const int e = slice_exponent(amax);
  const double s42 = digit_scale(e);
  if (warp == 0) (blockIdx.y == 0 ? dexp_a : dexp_b)[G.dexp_off + i] = (int16_t)e;
  int8_t* dst = (blockIdx.y == 0 ? dsl_a : dsl_b) + G.ds_off + (long long)t.y * (G.m32 / 32) * kTcStepD;
  int8_t* dhalf = blockIdx.y == 0 ? dhalf_a : dhalf_b;  // null: not wanted (LDA)
  if (dhalf) dhalf += (G.dexp_off / kTcFuncs + t.y) * kTcStepD;
  for (int j0 = 8 * warp; j0 < G.m32; j0 += 8 * kSdWarps) {
    double v[8];
    if (j0 == 8 * warp) {
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = first[k];
    } else {
      piece(j0, v);
    }
    // per slice the 8 digits are half of a 16-byte row segment
    auto write = [&](int8_t* blk, auto scale) {
      uint32_t lo[8], hi[8];
#pragma unroll
      for (int k = 0; k < 8; k++) digits_m(v[k], scale(j0 + k), lo[k], hi[k]);
#pragma unroll
      for (int s = 0; s < kSlices; s++) {
        uint32_t w[2];
#pragma unroll
        for (int k4 = 0; k4 < 2; k4++)
          w[k4] = pack_digits(digit_field(lo[4 * k4], hi[4 * k4], s), digit_field(lo[4 * k4 + 1], hi[4 * k4 + 1], s),
                              digit_field(lo[4 * k4 + 2], hi[4 * k4 + 2], s),
                              digit_field(lo[4 * k4 + 3], hi[4 * k4 + 3], s), s == 0);
        *reinterpret_cast<uint2*>(blk + lio::umma::kmajor_offset(s * kTcFuncs + r, j0 & 31, kTcTall)) =
            make_uint2(w[0], w[1]);
      }
    };
    write(dst + (j0 >> 5) * kTcStepD, [&](int) { return s42; });
    // the tile's diagonal block as the gradient kinds read it: strict triangle j < i as it is, half of
    // the diagonal (32 entries on a grid one bit coarser; a half of every entry would put all 1024 there)
    if (dhalf && (j0 >> 5) == t.y) write(dhalf, [&](int j) { return j < i ? s42 : (j == i ? 0.5 * s42 : 0.0); });
  }
}

// ------------------------------------------------------- the fused kernel
// K (padded functions) up to which two adjacent levels combine exactly in
// int32: |acc_l| <= (l + 1) * 64 * 64 * K, so |128 acc_4 + acc_5| < 2^31 for K < 813
constexpr int kTcNarrowK = 768;

// sum_l acc_l 128^(S-1-l) of column c in FP64: level pairs in int32 (narrow)
// or each level converted (wide), then combined with one rounding, 2^-53 of
// the leading term and far below the dropped slice pairs. A template parameter: a
// test of it at every value cost 6 to 7 % (density stage at 256 atoms open shell 5.88
// against 5.50 ms, 64 atoms 681 against 629 us; force kernel 583 against 531 us).
template <bool NARROW, int W>
__device__ __forceinline__ double level_sum(const int32_t (&lv)[kSlices][W], int c) {
  double v0, v1, v2;
  if constexpr (NARROW) {
    v0 = (double)(lv[0][c] * 128 + lv[1][c]);
    v1 = (double)(lv[2][c] * 128 + lv[3][c]);
    v2 = (double)(lv[4][c] * 128 + lv[5][c]);
  } else {
    v0 = fma((double)lv[0][c], 128.0, (double)lv[1][c]);
    v1 = fma((double)lv[2][c], 128.0, (double)lv[3][c]);
    v2 = fma((double)lv[4][c], 128.0, (double)lv[5][c]);
  }
  return fma(fma(v0, 16384.0, v1), 16384.0, v2);
}

// named barrier over the two epilogue warps of a TMEM lane quadrant; returns the OR of `pred` over them
__device__ __forceinline__ bool pair_sync_or(int quad, bool pred) {
  uint32_t out;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, %2, 64, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(out)
      : "r"((uint32_t)pred), "r"(1 + quad)
      : "memory");
  return out != 0;
}

// ------------------------------------------------------------- radial sums
// Per geometry: one thread per (group, point) of a 128-point tile; for every
// shell (simple function) of the group the contracted radial sums at the point
// (g2g/cpu/functions.cpp:68-79: primitives with a_k r^2 > 70 skipped),
//   t = sum_k c_k e^(-a_k r^2),  tg2 = -2 sum_k a_k c_k e^(..),  th4 = 4 sum_k a_k^2 c_k e^(..)
// (t only for LDA, NR = 1). Layout per group and tile: [shell][NR][128 points],
// so the shells of one function tile are contiguous.
template <int NR>
__global__ void __launch_bounds__(kTcPoints) k_radial(const int2* __restrict__ tiles,
                                                      const GroupDev* __restrict__ groups,
                                                      const double* __restrict__ px, const double* __restrict__ py,
                                                      const double* __restrict__ pz, const int* __restrict__ sf_glob,
                                                      const int* __restrict__ nuc, const int* __restrict__ ncont,
                                                      const double* __restrict__ ca, const double* __restrict__ cc,
                                                      const double* __restrict__ ax, const double* __restrict__ ay,
                                                      const double* __restrict__ az, double* __restrict__ rad) {
  const int2 t = tiles[blockIdx.x];
  const GroupDev G = groups[t.x];
  const int r = threadIdx.x;
  const long long p = G.pt_off + t.y * kTcPoints + r;
  const double x = px[p], y = py[p], z = pz[p];
  double* out = rad + G.rad_off + (long long)t.y * G.nsimple * NR * kTcPoints + r;
  for (int sh = 0; sh < G.nsimple; sh++) {
    const int gf = sf_glob[G.sf_off + sh];
    const int atom = nuc[gf];
    const double dx = x - ax[atom], dy = y - ay[atom], dz = z - az[atom];
    const double dist = dx * dx + dy * dy + dz * dz;
    double tt = 0.0, tg = 0.0, th = 0.0;
    const int nc = ncont[gf];
    for (int k = 0; k < nc; k++) {
      const double a = ca[gf * 13 + k], c = cc[gf * 13 + k];
      const double expo = a * dist;
      if (expo > 70.0) continue;
      const double t0 = exp(-expo) * c;
      tt += t0;
      tg += t0 * a;
      th += t0 * (a * a);
    }
    out[(long long)sh * NR * kTcPoints] = tt;
    if (NR == 3) {
      out[((long long)sh * NR + 1) * kTcPoints] = -2.0 * tg;
      out[((long long)sh * NR + 2) * kTcPoints] = 4.0 * th;
    }
  }
}

// A shell of a group as the density epilogue reads it, one 32-byte record per
// (group, shell), written per geometry: its atom's position, its type (0 s, 1 p,
// 2 d; plus 4 where its atom is not the previous shell's, 8 where its components
// straddle two windows of 16 functions) and the group-local
// column of its first component. One load per shell instead of a chain through the
// shell's function, its atom and the positions.
struct __align__(16) ShellInfo {
  double x, y, z;
  int type, fcol;
};
static_assert(sizeof(ShellInfo) == 32, "one 32-byte record per shell");
constexpr int kShellNewAtom = 4;
constexpr int kShellSplit = 8;

// The FP64 values of NC adjacent columns, SK per column, parked in TMEM from column
// `col` of this warp's columns [0, wlen) on. With CLIP the shell's first column may
// lie before them or its last after them: those belong to another warp or function
// tile and count as 0.
template <int NC, int SK, bool CLIP>
__device__ __forceinline__ void load_g(uint32_t gbase, int col, int wlen, uint32_t (&raw)[NC][2 * SK]) {
#pragma unroll
  for (int c = 0; c < NC; c++) {
    if (!CLIP || (col + c >= 0 && col + c < wlen)) {  // warp-uniform
      const uint32_t a = gbase + (uint32_t)((col + c) * 2 * SK);
      if constexpr (SK == 2)
        lio::umma::tmem_ld4u(a, raw[c][0], raw[c][1], raw[c][2], raw[c][3]);
      else
        lio::umma::tmem_ld2(a, raw[c][0], raw[c][1]);
    } else {
#pragma unroll
      for (int k = 0; k < 2 * SK; k++) raw[c][k] = 0u;  // the bits of +0.0
    }
  }
}

// The current atom's sums of one (spin, kind), and what a shell or an atom adds:
// kind F straight to the point's q = (rho; grad rho; d2rho xx, yy, zz, xy, xz, yz),
// with t, tg2 and th4 carrying the batch's power-of-two scale; a gradient kind a to
// v_b = sum_i F_b G^a (b = x, y, z), scaled and added to q at its end. G^a of a
// gradient kind holds only the part of D before and half of its diagonal, so
// F_a D F_b = v_b of kind a + v_a of kind b (k_density_tc). The factor 2 of every
// derivative term is applied when q is written.
template <bool GGA, int KIND, int NQ>
struct UnitSums {
  double U0, W0, V[3], v[3];
  __device__ static constexpr int d2(int a, int b) {  // q's entry of d2rho/da db
    return (a == b ? 4 + a : 6 + a + b) % NQ;
  }
  __device__ __forceinline__ void start() {
    start_atom();
    v[0] = v[1] = v[2] = 0.0;
  }
  __device__ __forceinline__ void finish(double (&q)[NQ], double scale) {
    if constexpr (GGA && KIND > 0) {
#pragma unroll
      for (int b = 0; b < 3; b++)
        q[d2(KIND - 1, b)] = fma(b == KIND - 1 ? 2.0 * scale : scale, v[b], q[d2(KIND - 1, b)]);
    }
  }
  __device__ __forceinline__ void start_atom() { U0 = W0 = V[0] = V[1] = V[2] = 0.0; }
  // one shell: G of its components, r the displacement, n the d normalisation
  template <int TYPE>
  __device__ __forceinline__ void shell(const double* g, const double (&r)[3], double t, double tg2, double th4,
                                        double n, double (&q)[NQ]) {
    double S0, S1[3], S2[6];
    if constexpr (TYPE == 0) {
      S0 = g[0];
    } else if constexpr (TYPE == 1) {
      S1[0] = g[0];
      S1[1] = g[1];
      S1[2] = g[2];
      S0 = fma(r[0], g[0], fma(r[1], g[1], r[2] * g[2]));
    } else {  // P = n xx, xy, n yy, xz, yz, n zz: homogeneous of degree 2, so 2 S0 = r . S1
      S2[0] = (2.0 * n) * g[0];
      S2[1] = (2.0 * n) * g[2];
      S2[2] = (2.0 * n) * g[5];
      S2[3] = g[1];
      S2[4] = g[3];
      S2[5] = g[4];
      S1[0] = fma(r[0], S2[0], fma(r[1], S2[3], r[2] * S2[4]));
      S1[1] = fma(r[1], S2[1], fma(r[0], S2[3], r[2] * S2[5]));
      S1[2] = fma(r[2], S2[2], fma(r[0], S2[4], r[1] * S2[5]));
      S0 = 0.5 * fma(r[0], S1[0], fma(r[1], S1[1], r[2] * S1[2]));
    }
    if constexpr (!GGA) {
      q[0] = fma(t, S0, q[0]);
    } else if constexpr (KIND == 0) {
      q[0] = fma(t, S0, q[0]);
      U0 = fma(tg2, S0, U0);
      W0 = fma(th4, S0, W0);
      if constexpr (TYPE > 0) {
#pragma unroll
        for (int a = 0; a < 3; a++) {
          q[(1 + a) % NQ] = fma(t, S1[a], q[(1 + a) % NQ]);
          V[a] = fma(tg2, S1[a], V[a]);
        }
      }
      if constexpr (TYPE == 2) {
#pragma unroll
        for (int h = 0; h < 6; h++) q[(4 + h) % NQ] = fma(t, S2[h], q[(4 + h) % NQ]);
      }
    } else {
      U0 = fma(tg2, S0, U0);
      if constexpr (TYPE > 0) {
#pragma unroll
        for (int b = 0; b < 3; b++) v[b] = fma(t, S1[b], v[b]);
      }
    }
  }
  __device__ __forceinline__ void end_atom(const double (&r)[3], double (&q)[NQ]) {
    if constexpr (!GGA) {
    } else if constexpr (KIND == 0) {
      constexpr int ha[6] = {0, 1, 2, 0, 0, 1}, hb[6] = {0, 1, 2, 1, 2, 2};
      double Y[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        q[(1 + a) % NQ] = fma(r[a], U0, q[(1 + a) % NQ]);
        Y[a] = fma(r[a], W0, V[a]);
      }
#pragma unroll
      for (int h = 0; h < 6; h++) {
        double x = fma(r[ha[h]], Y[hb[h]], q[(4 + h) % NQ]);
        if (h < 3) x += U0;
        q[(4 + h) % NQ] = fma(r[hb[h]], V[ha[h]], x);
      }
    } else {
#pragma unroll
      for (int b = 0; b < 3; b++) v[b] = fma(r[b], U0, v[b]);
    }
  }
};

// One shell of this warp's columns: its components' G from TMEM and their sums per
// spin and kind (kinds FIRST and, with KP = 2, FIRST + 1); sc the batches' scales
// (SCALED: kind F's go into its radial sums); whole: all in this warp's columns.
template <int TYPE, int NS, int KP, int NQ, bool SCALED, class U0T, class U1T>
__device__ __forceinline__ void shell_unit(uint32_t gbase, int col, int wlen, bool whole, const double (&r)[3], double t,
                                           double tg2, double th4, double dnorm, const double (&sc)[NS * KP],
                                           U0T (&u0)[NS], U1T (&u1)[NS], double (&q)[NS][NQ]) {
  constexpr int NC = TYPE == 0 ? 1 : (TYPE == 1 ? 3 : 6), SK = NS * KP;
  uint32_t raw[NC][2 * SK];
  if (TYPE == 0 || whole)  // warp-uniform; an s shell is one column
    load_g<NC, SK, false>(gbase, col, wlen, raw);
  else
    load_g<NC, SK, true>(gbase, col, wlen, raw);
  lio::umma::tmem_wait_ld();
#pragma unroll
  for (int sp = 0; sp < NS; sp++)
#pragma unroll
    for (int kp = 0; kp < KP; kp++) {
      const int sk = sp * KP + kp;
      double g[NC];
#pragma unroll
      for (int c = 0; c < NC; c++) g[c] = __hiloint2double((int)raw[c][2 * sk + 1], (int)raw[c][2 * sk]);
      if (kp == 0) {
        const double f = SCALED ? sc[sk] : 1.0;
        u0[sp].template shell<TYPE>(g, r, SCALED ? t * f : t, SCALED ? tg2 * f : tg2, SCALED ? th4 * f : th4, dnorm,
                                    q[sp]);
      } else {
        u1[sp].template shell<TYPE>(g, r, t, tg2, th4, dnorm, q[sp]);
      }
    }
}

// A unit's contraction (first kind FIRST) over the nsl shells of this warp's
// columns: `rec` their records and `rad` their radial sums in shared memory
// ([shell][NR][128 points], rad at this thread's), w0 the window's first column, p the point, spx and sd the
// point's and the density tile's power-of-two scales.
template <bool GGA, int NS, int KP, int NR, int NA, int NQ, int FIRST>
__device__ __forceinline__ void contract_unit(int nsl, const ShellInfo* rec, const double* rad, int w0,
                                              uint32_t gbase, int wlen, const double (&p)[3], double dnorm,
                                              const double (&spx)[NA], const double (&sd)[NS],
                                              double (&q)[NS][NQ]) {
  UnitSums<GGA, FIRST, NQ> u0[NS];
  UnitSums<GGA, (FIRST + 1 < 4 ? FIRST + 1 : 3), NQ> u1[NS];  // KP = 2 only
  double sc[NS * KP];
  double r[3];
#pragma unroll
  for (int sp = 0; sp < NS; sp++) {
    u0[sp].start();
    sc[sp * KP] = spx[FIRST] * sd[sp];
    if (KP == 2) {
      u1[sp].start();
      sc[sp * KP + KP - 1] = spx[(FIRST + 1) % NA] * sd[sp];
    }
  }
  auto displacement = [&](const ShellInfo& a) {
    const double2 xy = *reinterpret_cast<const double2*>(&a.x);
    r[0] = p[0] - xy.x;
    r[1] = p[1] - xy.y;
    r[2] = p[2] - a.z;
  };
  displacement(rec[0]);  // nsl >= 1
#pragma unroll 1
  for (int s = 0; s < nsl; s++) {
    const int2 tc = *reinterpret_cast<const int2*>(&rec[s].type);
    if ((tc.x & kShellNewAtom) && s > 0) {
#pragma unroll
      for (int sp = 0; sp < NS; sp++) {
        u0[sp].end_atom(r, q[sp]);
        u0[sp].start_atom();
        if (KP == 2) {
          u1[sp].end_atom(r, q[sp]);
          u1[sp].start_atom();
        }
      }
      displacement(rec[s]);
    }
    const double t = rad[(s * NR) * kTcPoints];
    const double tg2 = GGA ? rad[(s * NR + 1) * kTcPoints] : 0.0;
    const double th4 = GGA && FIRST == 0 ? rad[(s * NR + 2) * kTcPoints] : 0.0;
    const int type = tc.x & 3, col = tc.y - w0;  // the first component's column of the window (may be < 0)
    if (type == 0)
      shell_unit<0, NS, KP, NQ, FIRST == 0>(gbase, col, wlen, !(tc.x & kShellSplit), r, t, tg2, th4, dnorm, sc, u0, u1, q);
    else if (type == 1)
      shell_unit<1, NS, KP, NQ, FIRST == 0>(gbase, col, wlen, !(tc.x & kShellSplit), r, t, tg2, th4, dnorm, sc, u0, u1, q);
    else
      shell_unit<2, NS, KP, NQ, FIRST == 0>(gbase, col, wlen, !(tc.x & kShellSplit), r, t, tg2, th4, dnorm, sc, u0, u1, q);
  }
#pragma unroll
  for (int sp = 0; sp < NS; sp++) {
    u0[sp].end_atom(r, q[sp]);
    u0[sp].finish(q[sp], sc[sp * KP]);
    if (KP == 2) {
      u1[sp].end_atom(r, q[sp]);
      u1[sp].finish(q[sp], sc[sp * KP + KP - 1]);
    }
  }
}

// CTA = one per SM, persistent over the 128-point tiles (all groups, largest
// function count first, tile w handled by CTA w mod gridDim.x). Warp roles:
//   warps 0..7  epilogue: TMEM lane quadrant warp % 4 (one lane = one point),
//               columns 16 * (warp / 4) .. of the function tile;
//   warp 8      producer of everything the others read: per tile its slot, per
//               32-function tile its shell slot, per K step of a batch one stage with
//               the kind's A slices (kTcStepA) and every spin's stacked D slices
//               (kTcStepD), by bulk copies;
//   warp 9      MMA issuer: per stage NS x S MMAs into the batch's level columns.
// Per unit an epilogue warp reads each batch's levels (tfull), forms G in FP64,
// hands the level columns back (tempty) so that the next batch's MMAs overlap its
// work, parks G in the TMEM columns after the levels and contracts it shell by shell
// (parking lets the loop over shells address the columns at run time without local
// memory). The two warps of a lane quadrant meet at a tile's end. What an epilogue
// warp reads per tile and function tile (but for the density tile's exponents) comes
// from slots filled ahead of it: chains
// of dependent global loads (tile, group, shells, their atoms and radial sums) at
// the start of each took 15 to 28 % of its time (density stage with them 6.87 ms at
// 256 atoms open shell, 776 us at 64 atoms, 362 at 121 atoms LDA; with the slots, and
// one spin's kinds in two level buffers, 5.88 ms, 681 and 286 us). Every wait is bounded; a
// timeout sets `fail`, which the other roles poll, and the kernel drains its copies
// and MMAs before it frees TMEM and reports the error.
// The gradient kinds use that D is symmetric: only T_ab = sum_ij F_a,i D_ij F_b,j is
// needed of them, and with L the strict triangle of D plus half of its diagonal,
// D = L + L^T and T_ab = F_a L F_b + F_b L F_a. So their K steps of function tile ft
// end at ft (the last, the 32 x 32 diagonal block, from a copy that holds L), 0.66 of all
// at 256 atoms, for 9 products with F_x, F_y, F_z instead of 6 (density stage 256
// atoms open shell 5.50 -> 4.93 ms, 64 atoms closed shell 629 -> 595 us).
template <bool GGA, int NS>
__global__ void __launch_bounds__(TcCfg<GGA, NS>::kThreads, 1)
    k_density_tc(const int2* __restrict__ tiles, int ntiles, const GroupDev* __restrict__ groups,
                 const int8_t* __restrict__ aslices, const int16_t* __restrict__ aexp,
                 const int8_t* __restrict__ dsl_a, const int16_t* __restrict__ dexp_a,
                 const int8_t* __restrict__ dsl_b, const int16_t* __restrict__ dexp_b,
                 const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
                 const int4* __restrict__ ft_info, const ShellInfo* __restrict__ sinfo,
                 const double* __restrict__ rad, double dnorm, double* __restrict__ part_a,
                 double* __restrict__ part_b, int* __restrict__ err, const int8_t* __restrict__ dhalf_a,
                 const int8_t* __restrict__ dhalf_b, typename TcCfg<GGA, NS>::Layout lay) {
  using Cfg = TcCfg<GGA, NS>;
  constexpr int KP = Cfg::KP, NP = Cfg::NP, NA = Cfg::NA, NQ = Cfg::NQ, NR = Cfg::NR, CPW = kTcCpw;
  constexpr int NB = Cfg::kBufs;
  extern __shared__ __align__(128) uint8_t tc_smem[];
  __shared__ uint64_t full[Cfg::kMaxStages], empty[Cfg::kMaxStages], tfull[NB], tempty[NB];
  __shared__ uint64_t sfull[2], sempty[2], rfull[2], rempty[2], drain;
  __shared__ uint32_t tmem_base;
  __shared__ int fail, consumed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nst = lay.stages, nrb = lay.nrb;
  if (warp == 0) lio::umma::tmem_alloc(&tmem_base, Cfg::kTmem);
  if (tid == 0) {
    for (int b = 0; b < nst; b++) {
      lio::umma::mbar_init(&full[b], 1);
      lio::umma::mbar_init(&empty[b], 1);
    }
    for (int b = 0; b < NB; b++) {
      lio::umma::mbar_init(&tfull[b], 1);
      lio::umma::mbar_init(&tempty[b], kTcEpiWarps);
    }
    for (int b = 0; b < 2; b++) {
      lio::umma::mbar_init(&sfull[b], 1);
      lio::umma::mbar_init(&sempty[b], kTcEpiWarps);
      lio::umma::mbar_init(&rfull[b], 1);
      lio::umma::mbar_init(&rempty[b], kTcEpiWarps);
    }
    lio::umma::mbar_init(&drain, 1);
    lio::umma::fence_mbar_init();
    fail = 0;
    consumed = 0;
  }
  lio::umma::fence_before_sync();
  __syncthreads();
  lio::umma::fence_after_sync();
  const uint32_t tbase = tmem_base;
  volatile int* vfail = &fail;
  int issued = 0, tcnt = 0, rcnt = 0;  // producer: stages, tile slots and shell slots issued
  uint8_t* ring = tc_smem + lay.ring();
  uint8_t* shells = tc_smem + lay.shells();

  if (warp == Cfg::kProd) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      const uint64_t keep = lio::umma::l2_evict_last(), drop = lio::umma::l2_evict_first();
      int buf = 0, use = 0;  // stage and its use count
      auto wait = [&](uint64_t* bar, int uses) {  // `uses` uses of the slot before this one
        return uses == 0 || (!*vfail && lio::umma::mbar_wait(bar, (uses - 1) & 1));
      };
      int2 tn = tiles[min((int)blockIdx.x, ntiles - 1)];
      for (int w = blockIdx.x; w < ntiles && !*vfail; w += gridDim.x) {
        const int2 t = tn;
        tn = tiles[min(w + (int)gridDim.x, ntiles - 1)];
        const GroupDev& G = groups[t.x];
        const int nks = G.m32 / 32, nft = G.nftc, nsimple = G.nsimple;
        const long long p0 = G.pt_off + t.y * kTcPoints, sf_off = G.sf_off, ds_off = G.ds_off;
        const long long ft0 = G.dexp_off / kTcFuncs;  // the group's first function tile
        const int4* info = ft_info + ft0;
        const double* trad = rad + G.rad_off + (long long)t.y * nsimple * NR * kTcPoints;
        const int8_t* Abase = aslices + G.sl_off + (long long)t.y * NA * nks * kTcStepA;
        {
          const int b = tcnt & 1;
          if (!wait(&sempty[b], tcnt >> 1)) {
            *vfail = 1;
            break;
          }
          uint8_t* slot = tc_smem + b * Cfg::kTileSlot;
          lio::umma::mbar_expect_tx(&sfull[b], (uint32_t)(sizeof(GroupDev) + 3 * kTcPoints * 8 + NA * kTcPoints * 2));
          lio::umma::bulk_copy_g2s(slot, &G, sizeof(GroupDev), &sfull[b]);
          const double* xyz[3] = {px, py, pz};
          for (int d = 0; d < 3; d++)
            lio::umma::bulk_copy_g2s(slot + Cfg::kTileXyz + d * kTcPoints * 8, xyz[d] + p0, kTcPoints * 8, &sfull[b]);
          for (int a = 0; a < NA; a++)
            lio::umma::bulk_copy_g2s(slot + Cfg::kTileExp + a * kTcPoints * 2,
                                     aexp + G.aexp_off + (long long)a * G.ldp + t.y * kTcPoints, kTcPoints * 2,
                                     &sfull[b]);
          tcnt++;
        }
        for (int ft = 0; ft < nft && !*vfail; ft++) {
          const int4 fi = info[ft];  // first shell, shells, ...
          auto shell_slot = [&]() {
            const int b = nrb == 2 ? rcnt & 1 : 0;
            if (!wait(&rempty[b], nrb == 2 ? rcnt >> 1 : rcnt)) return false;
            uint8_t* slot = shells + b * lay.shell_slot;
            lio::umma::mbar_expect_tx(&rfull[b], (uint32_t)(16 + fi.y * (32 + NR * kTcPoints * 8)));
            lio::umma::bulk_copy_g2s(slot, info + ft, 16, &rfull[b]);
            lio::umma::bulk_copy_g2s(slot + Cfg::kShellRec, sinfo + sf_off + fi.x, (uint32_t)(fi.y * 32), &rfull[b]);
            lio::umma::bulk_copy_g2s_hint(slot + Cfg::kShellRad, trad + (long long)fi.x * NR * kTcPoints,
                                          (uint32_t)(fi.y * NR * kTcPoints * 8), &rfull[b], drop);
            rcnt++;
            return true;
          };
          // with one slot its last readers are a function tile behind: the first kind's stages go first
          if (nrb == 2 && !shell_slot()) {
            *vfail = 1;
            break;
          }
          // A is read again by the tile's next function tile; D by every tile of the group
          const uint64_t pa = ft + 1 < nft ? keep : drop;
          for (int a = 0; a < NA && !*vfail; a++) {
            const int nka = a == 0 ? nks : ft + 1;  // K steps of this kind
            for (int kk = 0; kk < nka; kk++) {
              if (!wait(&empty[buf], use)) {
                *vfail = 1;
                break;
              }
              uint8_t* stage = ring + buf * Cfg::kStage;
              lio::umma::mbar_expect_tx(&full[buf], (uint32_t)Cfg::kStage);
              lio::umma::bulk_copy_g2s_hint(stage, Abase + ((long long)a * nks + kk) * kTcStepA, kTcStepA, &full[buf],
                                            pa);
              for (int sp = 0; sp < NS; sp++)
                lio::umma::bulk_copy_g2s_hint(
                    stage + kTcStepA + sp * kTcStepD,
                    a > 0 && kk == ft ? (sp == 0 ? dhalf_a : dhalf_b) + (ft0 + ft) * kTcStepD
                                      : (sp == 0 ? dsl_a : dsl_b) + ds_off + ((long long)ft * nks + kk) * kTcStepD,
                    kTcStepD, &full[buf], keep);
              issued++;
              if (++buf == nst) buf = 0, use++;
            }
            if (a == 0 && nrb == 1 && !*vfail && !shell_slot()) *vfail = 1;
          }
        }
      }
    }
  } else if (warp == Cfg::kMma) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      // descriptors of the first A slice and of the stacked D of stage 0; a stage or an
      // operand further on adds its byte offset / 16 to the start address field (bits
      // 0-13: shared addresses stay below 2^18 bytes)
      const uint32_t smem0 = lio::umma::smem_u32(ring);
      const uint64_t ad0 = lio::umma::smem_desc(smem0, 16u * kTcPoints, 128u);
      // stacked D: K-major, 192 rows (LBO = 16 * 192 bytes between K halves)
      const uint64_t dd0 = lio::umma::smem_desc(smem0 + kTcStepA, 16u * kTcTall, 128u);
      int buf = 0, use = 0, bcnt = 0;  // stage, its use count; batches
      bool stop = false;
      auto shape = [&](int w) {  // K steps and batches of a tile
        const GroupDev& G = groups[tiles[min(w, ntiles - 1)].x];
        return make_int2(G.m32 / 32, G.nftc * NA);
      };
      int2 nx = shape(blockIdx.x);
      for (int w = blockIdx.x; w < ntiles && !stop; w += gridDim.x) {
        const int nks = nx.x, nbat = nx.y;
        nx = shape(w + gridDim.x);  // read ahead of the next tile
        for (int tt = 0; tt < nbat && !stop; tt++, bcnt++) {
          const int b = bcnt % NB, uses = bcnt / NB;
          if (uses > 0) {  // the buffer's last batch has been read
            if (*vfail || !lio::umma::mbar_wait(&tempty[b], (uses - 1) & 1)) {
              stop = true;
              break;
            }
            lio::umma::fence_after_sync();
          }
          const uint32_t tcol = tbase + (uint32_t)b * Cfg::kLevels;
          const int nka = tt % NA == 0 ? nks : tt / NA + 1;  // K steps of this kind
          for (int kk = 0; kk < nka; kk++) {
            if (*vfail || !lio::umma::mbar_wait(&full[buf], use & 1)) {
              stop = true;
              break;
            }
            consumed = use * nst + buf + 1;
            lio::umma::fence_after_sync();
            const uint64_t so = (uint64_t)((buf * Cfg::kStage) >> 4);
#pragma unroll
            for (int sp = 0; sp < NS; sp++)
#pragma unroll
              for (int s = 0; s < kSlices; s++)
                lio::umma::mma_i8(tcol + (uint32_t)((sp * kSlices + s) * kTcFuncs),
                                  ad0 + so + (uint64_t)((s * kTcSliceA) >> 4), dd0 + so + (uint64_t)((sp * kTcStepD) >> 4),
                                  lio::umma::idesc_i8(kTcPoints, (kSlices - s) * kTcFuncs), (kk > 0 || s > 0) ? 1u : 0u);
            lio::umma::commit(&empty[buf]);
            if (kk == nka - 1) lio::umma::commit(&tfull[b]);
            if (++buf == nst) buf = 0, use++;
          }
        }
      }
      if (stop) *vfail = 1;
      // every MMA issued so far has completed once this arrives
      lio::umma::commit(&drain);
      if (!lio::umma::mbar_wait(&drain, 0)) *vfail = 1;
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int quad = warp & 3, colg = warp >> 2;
    const int row = quad * 32 + lane;  // this thread's point of the tile
    const uint32_t lane_base = tbase + ((uint32_t)(quad * 32) << 16);
    const int cb = colg * CPW;  // this warp's first column of a function tile
    const uint32_t gbase = lane_base + Cfg::kCols + (uint32_t)cb * Cfg::kGPer;  // G of this warp's columns
    // column group 1 -> 0 hand-off at the end of a tile, [spin][value][lane]
    double* red = reinterpret_cast<double*>(tc_smem + lay.red()) + quad * NS * NQ * 32 + lane;
    bool lfail = false;
    int bcnt = 0, tile_n = 0, ft_n = 0;  // batches, tiles and function tiles so far
    auto wait = [&](uint64_t* bar, int uses) {
      if (!__all_sync(0xffffffffu, !*vfail && lio::umma::mbar_wait(bar, uses & 1))) {
        lfail = true;
        *vfail = 1;
      }
      return !lfail;
    };
    auto release = [&](uint64_t* bar) {
      __syncwarp();
      if (lane == 0) lio::umma::mbar_arrive(bar);
    };
    int ty_next = tiles[min((int)blockIdx.x, ntiles - 1)].y;
    for (int w = blockIdx.x; w < ntiles; w += gridDim.x, tile_n++) {
      const int p = ty_next * kTcPoints + row;
      ty_next = tiles[min(w + (int)gridDim.x, ntiles - 1)].y;
      const uint8_t* tslot = tc_smem + (tile_n & 1) * Cfg::kTileSlot;
      double spx[NA], pt[3];  // 2^(point exponent - 7(S+1)) per kind; the point
      int m = 0, ldp = 0, nft = 0;
      bool narrow = false;
      long long dexp_off = 0, part_off = 0;
      if (wait(&sfull[tile_n & 1], tile_n >> 1)) {
        const GroupDev& G = *reinterpret_cast<const GroupDev*>(tslot);
        m = G.m;
        ldp = G.ldp;
        nft = G.nftc;
        narrow = G.m32 <= kTcNarrowK;
        dexp_off = G.dexp_off;
        part_off = G.part_off;
        const double* xyz = reinterpret_cast<const double*>(tslot + Cfg::kTileXyz) + row;
#pragma unroll
        for (int d = 0; d < 3; d++) pt[d] = xyz[d * kTcPoints];
        const int16_t* ex = reinterpret_cast<const int16_t*>(tslot + Cfg::kTileExp) + row;
#pragma unroll
        for (int a = 0; a < NA; a++) spx[a] = pow2(ex[a * kTcPoints] - 7 * (kSlices + 1));
        release(&sempty[tile_n & 1]);
      }
      double q[NS][NQ];
#pragma unroll
      for (int sp = 0; sp < NS; sp++)
#pragma unroll
        for (int k = 0; k < NQ; k++) q[sp][k] = 0.0;
      for (int ft = 0; ft < nft && !lfail; ft++, ft_n++) {
        const int i0 = ft * kTcFuncs;
        double sd[NS];  // 2^(density tile's exponent)
        sd[0] = pow2(dexp_a[dexp_off + i0]);
        if (NS == 2) sd[NS - 1] = pow2(dexp_b[dexp_off + i0]);
        const int w0 = i0 + cb, wlen = min(CPW, m - w0);  // this warp's columns [w0, w0 + wlen)
        const int rb = nrb == 2 ? ft_n & 1 : 0;
        const uint8_t* sslot = shells + rb * lay.shell_slot;
        const ShellInfo* rec = reinterpret_cast<const ShellInfo*>(sslot + Cfg::kShellRec);
        const double* wrad = reinterpret_cast<const double*>(sslot + Cfg::kShellRad) + row;
        int nsl = 0;
#pragma unroll 1
        for (int pass = 0; pass < NP && !lfail; pass++) {
          // ---- the unit's accumulators -> G (FP64, without the scales), parked in the TMEM columns after the levels
          double gk[KP == 2 ? CPW : 1];  // KP = 2: the first kind's G until the second's
#pragma unroll
          for (int kp = 0; kp < KP; kp++, bcnt++) {
            const int b = bcnt % NB;
            if (!wait(&tfull[b], bcnt / NB)) break;
            lio::umma::fence_after_sync();
            if (wlen <= 0) {
              release(&tempty[b]);
              continue;
            }
            const uint32_t lbase = lane_base + (uint32_t)b * Cfg::kLevels + (uint32_t)cb;
            auto read_batch = [&](auto nrw) {
#pragma unroll
              for (int c0 = 0; c0 < CPW; c0 += 8) {
                if (c0 >= wlen) continue;  // no function there (warp-uniform)
                double x[8][NS];
#pragma unroll
                for (int sp = 0; sp < NS; sp++) {
                  int32_t lv[kSlices][8];
#pragma unroll
                  for (int l = 0; l < kSlices; l++)
                    lio::umma::tmem_ld8(lbase + (uint32_t)((sp * kSlices + l) * kTcFuncs + c0), lv[l]);
                  lio::umma::tmem_wait_ld();
                  if ((c0 + 8 == CPW || c0 + 8 >= wlen) && sp == NS - 1) {  // the batch's last: its columns back to the MMA issuer
                    lio::umma::fence_before_sync();
                    release(&tempty[b]);
                  }
#pragma unroll
                  for (int c = 0; c < 8; c++) x[c][sp] = level_sum<decltype(nrw)::value>(lv, c);
                }
                if (KP == 2 && kp == 0) {
#pragma unroll
                  for (int c = 0; c < 8; c++) gk[(c0 + c) % (KP == 2 ? CPW : 1)] = x[c][0];
                  continue;
                }
                // 8 columns x NS x KP doubles: 8 * kGPer consecutive 32-bit TMEM columns
#pragma unroll
                for (int part = 0; part < NS * KP; part++) {
                  uint32_t v[16];
#pragma unroll
                  for (int e = 0; e < 8; e++) {
                    const int idx = part * 8 + e, c = idx / (NS * KP), sk = idx % (NS * KP);
                    const double y = KP == 2 ? (sk == 0 ? gk[(c0 + c) % (KP == 2 ? CPW : 1)] : x[c][0]) : x[c][sk % NS];
                    v[2 * e] = (uint32_t)__double2loint(y);
                    v[2 * e + 1] = (uint32_t)__double2hiint(y);
                  }
                  lio::umma::tmem_st16(gbase + (uint32_t)(c0 * Cfg::kGPer + part * 16), v);
                }
              }
            };
            if (narrow)
              read_batch(std::true_type{});
            else
              read_batch(std::false_type{});
          }
          lio::umma::tmem_wait_st();
          if (pass == 0 && !lfail && wait(&rfull[rb], nrb == 2 ? ft_n >> 1 : ft_n)) {
            // this warp's shells of the tile's: first shell, shells, first of column group 1, last of column group 0
            const int4 fi = *reinterpret_cast<const int4*>(sslot);
            const int first = colg == 0 ? 0 : fi.z;
            nsl = wlen <= 0 ? 0 : (colg == 0 ? fi.w + 1 : fi.y - fi.z);
            rec += first;
            wrad += first * NR * kTcPoints;
          }
          if (lfail || wlen <= 0) continue;
          // ---- shell by shell over this warp's columns
          if (pass == 0)
            contract_unit<GGA, NS, KP, NR, NA, NQ, 0>(nsl, rec, wrad, w0, gbase, wlen, pt, dnorm, spx, sd, q);
          else if (pass == 1)
            contract_unit<GGA, NS, KP, NR, NA, NQ, (GGA ? KP : 0)>(nsl, rec, wrad, w0, gbase, wlen, pt, dnorm, spx, sd, q);
          else if (pass == 2)
            contract_unit<GGA, NS, KP, NR, NA, NQ, (GGA && KP == 1 ? 2 : 0)>(nsl, rec, wrad, w0, gbase, wlen, pt, dnorm,
                                                                             spx, sd, q);
          else
            contract_unit<GGA, NS, KP, NR, NA, NQ, (GGA && KP == 1 ? 3 : 0)>(nsl, rec, wrad, w0, gbase, wlen, pt, dnorm,
                                                                             spx, sd, q);
        }
        if (!lfail) release(&rempty[rb]);
      }
      // tile done: column group 1 hands its sums to column group 0, which writes them
      if (colg == 1) {
#pragma unroll
        for (int sp = 0; sp < NS; sp++)
#pragma unroll
          for (int k = 0; k < NQ; k++) red[(sp * NQ + k) * 32] = q[sp][k];
      }
      if (pair_sync_or(quad, lfail || *vfail)) break;
      if (colg == 0) {
#pragma unroll
        for (int sp = 0; sp < NS; sp++) {
          double* dst = (sp == 0 ? part_a : part_b) + part_off + p;
#pragma unroll
          for (int k = 0; k < NQ; k++) {
            const double v = q[sp][k] + red[(sp * NQ + k) * 32];
            dst[(long long)k * ldp] = k == 0 ? v : 2.0 * v;  // the factor 2 of the derivative terms
          }
        }
      }
      pair_sync_or(quad, false);  // the hand-off area is free again
    }
  }
  __syncthreads();  // every role done
  if (warp == Cfg::kProd && lane == 0) {
    // copies issued but never consumed (after a timeout) land before the CTA exits: the
    // stages past the last consumed one, the latest phase of each slot
    for (int k = consumed; k < issued; k++)
      if (!lio::umma::mbar_wait(&full[k % nst], (k / nst) & 1)) break;
    for (int k = max(0, tcnt - 2); k < tcnt; k++)
      if (!lio::umma::mbar_wait(&sfull[k & 1], (k >> 1) & 1)) break;
    for (int k = max(0, rcnt - nrb); k < rcnt; k++)
      if (!lio::umma::mbar_wait(&rfull[nrb == 2 ? k & 1 : 0], (nrb == 2 ? k >> 1 : k) & 1)) break;
  }
  lio::umma::fence_before_sync();
  __syncthreads();
  if (tid == 0 && fail) atomicExch(err, 1);
  if (warp == 0) lio::umma::tmem_dealloc(tbase, Cfg::kTmem);
}
