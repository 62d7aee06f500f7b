// FP64 form of the two contractions (included by engine.cu inside its anonymous
// namespace; uses GroupDev and packed_index), on the FP64 tensor instruction
// mma.sync m8n8k4 (tcgen05 has no FP64 kind): a warp instruction is 256
// multiply-adds for one value of each operand per lane, where the FFMA-style
// tiles of 4 x 4 per thread it replaces read 8 values from shared memory for 16
// and ran at 0.12 to 0.19 of the FP64 rate.
#pragma once

// D (8 x 8) += A (8 x 4) B (4 x 8), FP64. Lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
// 16-byte asynchronous copy into shared memory, zeros when !valid
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(lio::umma::smem_u32(dst)), "l"(src),
               "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---------------------------------------------------------------- density
// CTA = (group, 64 points), 4 warps, looping over the group's 32-function tiles
// and, per tile, over the functions j in steps of 16. G^a = A^a D for the kinds a
// (F; for GGA also dF/dx, dF/dy, dF/dz): with 4 kinds warp a computes its kind's
// 64 x 32 block (64 accumulators per lane), with one kind each warp 16 points.
// The gradient kinds use D symmetric: for second derivatives only
//   T^ab = sum_ij dF_i/da D_ij dF_j/db (symmetric in a, b)
// is needed, and with D split by tiles into strictly lower part, diagonal blocks
// and strictly upper part, T^ab = sum_i (dF_i/da H^b_i + dF_i/db H^a_i) where
// H^a_i = sum over the j of tiles before i's of D_ij dF_j/da + half the diagonal
// block's: K steps up to i's tile only, a quarter of the work at 3 tiles saved.
// 8-function blocks past m and 4-function steps past m are skipped. After a tile
// the blocks go through shared memory so that a thread per (point, half of the
// functions) reads each basis value once, coalesced. One partial per point (the
// tile loop is inside), read by the functional. Bound by latency: 239 registers leave
// two CTAs (8 warps) on an SM, which wait for their operand loads, for the mma before and
// at the two barriers of a step; in the steps past the gradient kinds' last the warp of
// kind F alone has work. The FP64 tensor pipe is busy 28 % of the time (64 atoms closed
// shell, 1.69 ms). 45 atoms closed shell: 1605 us with 4 x 4 values per thread (groups
// padded to 64 x 64 blocks), 750 us with this.
constexpr int kD64Points = 64, kD64Funcs = 32, kD64K = 16, kD64Threads = 128;
static_assert(kFuncBlock == 2 * kD64Points && kPointPad % kFuncBlock == 0, "two CTAs per block of the functional's list");
constexpr int kD64StrideA = kD64Points + 4, kD64StrideB = kD64Funcs + 4;  // doubles; = 4 mod 16: no bank conflicts
template <int NA>
struct D64Cfg {
  static constexpr int kA = NA * kD64K * kD64StrideA, kB = 2 * kD64K * kD64StrideB;  // doubles per stage (B: full, halved)
  static constexpr int kStage = kA + kB;
  static constexpr int kG = NA * kD64Funcs * (kD64Points + 1);  // exchange area, over the stages
  static constexpr size_t kSmem = sizeof(double) * (2 * kStage > kG ? 2 * kStage : kG);
};

template <int NA>
__global__ void __launch_bounds__(kD64Threads) k_density_fp64(const int2* __restrict__ tiles,
                                                              const GroupDev* __restrict__ groups,
                                                              const int* __restrict__ fn_glob,
                                                              const double* __restrict__ basis,
                                                              const double* __restrict__ P,
                                                              double* __restrict__ partial, long long part_base) {
  using Cfg = D64Cfg<NA>;
  constexpr int NQ = NA == 1 ? 1 : kNQ;
  constexpr int MB = NA == 4 ? kD64Points / 8 : kD64Points / 32;  // 8-point blocks of a warp
  extern __shared__ __align__(16) double d64_smem[];
  // two CTAs per (group, 128-point block) of the list, which the functional reads too
  const int2 t = tiles[blockIdx.x >> 1];
  const GroupDev& G = groups[t.x];
  const int m = G.m, ldp = G.ldp, pt0 = (2 * t.y + (blockIdx.x & 1)) * kD64Points;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kind = NA == 4 ? warp : 0, mb0 = NA == 4 ? 0 : warp * MB;
  const long long kstride = (long long)m * ldp;
  const double* bas = basis + G.bas_off + pt0;
  const int* fg = fn_glob + G.fn_off;
  const double* Pg = P + G.pk_off;
  const int pM = G.pk_M;
  // B values of a step: thread (tid % 32 = function i of the tile, tid / 32) gathers 4 j's
  double bv[4];
  int gi = 0, ft0 = 0;
  auto gather = [&](int j0) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int j = j0 + (tid >> 5) + 4 * k;
      bv[k] = 0.0;
      if (j < m && ft0 + lane < m) {
        const int gj = fg[j];
        bv[k] = Pg[packed_index(gi, gj, pM)] * (gi != gj ? 0.5 : 1.0);
      }
    }
  };
  auto store_b = [&](double* st, int j0) {
    const double half = j0 >= ft0 ? 0.5 : 1.0;  // the diagonal block's share for the gradient kinds
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int o = ((tid >> 5) + 4 * k) * kD64StrideB + lane;
      st[Cfg::kA + o] = bv[k];
      if (NA == 4) st[Cfg::kA + kD64K * kD64StrideB + o] = half * bv[k];
    }
  };
  // A rows of a step: NA kinds x 16 functions x 64 points; gradient kinds past `glimit` are not needed
  auto copy_a = [&](double* st, int j0, int glimit) {
    const int kinds = NA == 4 && j0 >= glimit ? 1 : NA;
    for (int c = tid; c < kinds * kD64K * (kD64Points / 2); c += kD64Threads) {
      const int pp = (c & (kD64Points / 2 - 1)) * 2, kk = (c / (kD64Points / 2)) % kD64K, a = c / (kD64K * kD64Points / 2);
      const bool ok = j0 + kk < m;
      cp_async16(st + (a * kD64K + kk) * kD64StrideA + pp, bas + a * kstride + (long long)(ok ? j0 + kk : 0) * ldp + pp,
                 ok);
    }
    cp_async_commit();
  };
  const int p = tid & (kD64Points - 1), half = tid >> 6;  // epilogue: this thread's point and half of the functions
  double q[NQ];
#pragma unroll
  for (int k = 0; k < NQ; k++) q[k] = 0.0;

  for (ft0 = 0; ft0 < m; ft0 += kD64Funcs) {
    gi = ft0 + lane < m ? fg[ft0 + lane] : 0;
    const int nb = (min(kD64Funcs, m - ft0) + 7) / 8;              // 8-function blocks of this tile
    const int nsteps = (m + kD64K - 1) / kD64K, glimit = ft0 + kD64Funcs;  // F: all j; gradient: j < glimit
    double acc[MB][kD64Funcs / 8][2];
#pragma unroll
    for (int a = 0; a < MB; a++)
#pragma unroll
      for (int b = 0; b < kD64Funcs / 8; b++) acc[a][b][0] = acc[a][b][1] = 0.0;
    copy_a(d64_smem, 0, glimit);
    gather(0);
    store_b(d64_smem, 0);
    for (int s = 0; s < nsteps; s++) {
      double* st = d64_smem + (s & 1) * Cfg::kStage;
      double* nx = d64_smem + ((s + 1) & 1) * Cfg::kStage;
      const bool more = s + 1 < nsteps;
      if (more) {
        copy_a(nx, (s + 1) * kD64K, glimit);
        gather((s + 1) * kD64K);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      const int kmax = min(kD64K, m - s * kD64K);
      if (kind == 0 || s * kD64K < glimit) {
        const double* As = st + kind * kD64K * kD64StrideA + (lane & 3) * kD64StrideA + (lane >> 2) + mb0 * 8;
        const double* Bs = st + Cfg::kA + (kind > 0 ? kD64K * kD64StrideB : 0) + (lane & 3) * kD64StrideB + (lane >> 2);
        for (int k = 0; k < kmax; k += 4) {
          double a[MB], b[kD64Funcs / 8];
#pragma unroll
          for (int r = 0; r < MB; r++) a[r] = As[k * kD64StrideA + r * 8];
#pragma unroll
          for (int c = 0; c < kD64Funcs / 8; c++) b[c] = Bs[k * kD64StrideB + c * 8];
#pragma unroll
          for (int c = 0; c < kD64Funcs / 8; c++)
            if (c < nb) {
#pragma unroll
              for (int r = 0; r < MB; r++) mma_f64(acc[r][c], a[r], b[c]);
            }
        }
      }
      if (more) store_b(nx, (s + 1) * kD64K);  // its last readers are past the barrier above
      __syncthreads();
    }
    // blocks to shared memory: [kind][function][point]
    double* Gs = d64_smem;
#pragma unroll
    for (int r = 0; r < MB; r++)
#pragma unroll
      for (int c = 0; c < kD64Funcs / 8; c++)
#pragma unroll
        for (int e = 0; e < 2; e++)
          Gs[(kind * kD64Funcs + c * 8 + 2 * (lane & 3) + e) * (kD64Points + 1) + (mb0 + r) * 8 + (lane >> 2)] =
              acc[r][c][e];
    __syncthreads();
    const int i1 = min(m - ft0, (half + 1) * (kD64Funcs / 2));
#pragma unroll 4
    for (int i = half * (kD64Funcs / 2); i < i1; i++) {
      const double* v = bas + (long long)(ft0 + i) * ldp + p;
      const double* g = Gs + i * (kD64Points + 1) + p;
      const double g0 = g[0];
      q[0] = fma(v[0], g0, q[0]);
      if constexpr (NA == 4) {
        constexpr int kg = kD64Funcs * (kD64Points + 1);
        const double gX = g[kg], gY = g[2 * kg], gZ = g[3 * kg];
        const double dx = v[kstride], dy = v[2 * kstride], dz = v[3 * kstride];
        q[1] = fma(dx, g0, q[1]);
        q[2] = fma(dy, g0, q[2]);
        q[3] = fma(dz, g0, q[3]);
        q[4] = fma(2.0 * dx, gX, fma(v[4 * kstride], g0, q[4]));
        q[5] = fma(2.0 * dy, gY, fma(v[5 * kstride], g0, q[5]));
        q[6] = fma(2.0 * dz, gZ, fma(v[6 * kstride], g0, q[6]));
        q[7] = fma(dx, gY, fma(dy, gX, fma(v[7 * kstride], g0, q[7])));
        q[8] = fma(dx, gZ, fma(dz, gX, fma(v[8 * kstride], g0, q[8])));
        q[9] = fma(dy, gZ, fma(dz, gY, fma(v[9 * kstride], g0, q[9])));
      }
    }
    __syncthreads();  // the exchange area becomes stages again
  }
  // the two halves of the functions
  double* red = d64_smem;
  if (half == 1)
#pragma unroll
    for (int k = 0; k < NQ; k++) red[k * kD64Points + p] = q[k];
  __syncthreads();
  if (half == 0) {
    double* dst = partial + (G.part_off - part_base) + pt0 + p;
#pragma unroll
    for (int k = 0; k < NQ; k++) {
      const double v = q[k] + red[k * kD64Points + p];
      dst[(long long)k * ldp] = k == 0 ? v : 2.0 * v;
    }
  }
}

// ---------------------------------------------------------------- Kohn-Sham
// Work item = (group, 32-function tiles I <= J, chunk of the points), 4 warps:
// K_ij = sum_p F_ip f_p F_jp. Stages of 64 points (the rows of I and J by 16-byte
// asynchronous copies, double buffered); warp w takes points 16 w .. 16 w + 15 of
// each stage for the whole 32 x 32 tile of every spin, so that no warp idles on
// the diagonal tiles, of which only the 8 x 8 blocks on and above the diagonal are
// computed. The warps' tiles are summed in shared memory and added into the packed
// accumulator(s) with FP64 atomics. Splitting a group over its points fills the
// GPU: 220 CTAs, each over all of its group's points, took 1012 us at 45 atoms closed
// shell (80 took 727 us at 14 atoms open shell); items of at most 32 blocks 110 us, with the
// FP64 tensor pipe busy 63 % of the time (64 atoms closed shell, 205 us).
constexpr int kF64MaxBlocks = 32;
constexpr int kF64Tile = 32, kF64Points = 64, kF64Stride = kF64Points + 4, kF64Threads = 128;
template <int NS>
struct F64Cfg {
  static constexpr int kStage = 2 * kF64Tile * kF64Stride + NS * kF64Points;  // doubles
  static constexpr int kRed = 3 * NS * kF64Tile * kF64Tile;
  static constexpr size_t kSmem = sizeof(double) * (2 * kStage > kRed ? 2 * kStage : kRed);
};

template <int NS>
__global__ void __launch_bounds__(kF64Threads) k_fock_fp64(const int4* __restrict__ tiles,
                                                           const GroupDev* __restrict__ groups,
                                                           const int* __restrict__ fn_glob,
                                                           const double* __restrict__ basis,
                                                           const double* __restrict__ fac_a,
                                                           const double* __restrict__ fac_b,
                                                           double* __restrict__ K_a, double* __restrict__ K_b,
                                                           long long pt_base) {
  using Cfg = F64Cfg<NS>;
  constexpr int NB = kF64Tile / 8;
  extern __shared__ __align__(16) double f64_smem[];
  const int4 t = tiles[blockIdx.x];
  const GroupDev& G = groups[t.x];
  const int m = G.m, ldp = G.ldp, i0 = t.y * kF64Tile, j0 = t.z * kF64Tile;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool diag = t.y == t.z;
  const double* F = basis + G.bas_off;
  // the chunk's stages: an even share of the group's 64-point blocks
  const int nblk = ldp / kF64Points;
  const int s0 = (int)((long long)nblk * t.w / G.nch64), s1 = (int)((long long)nblk * (t.w + 1) / G.nch64);
  auto copy = [&](double* st, int s) {
    const int pb = s * kF64Points;
    const int rows = diag ? kF64Tile : 2 * kF64Tile;
    for (int c = tid; c < rows * (kF64Points / 2); c += kF64Threads) {
      const int pp = (c & (kF64Points / 2 - 1)) * 2, r = c / (kF64Points / 2);
      const int i = r < kF64Tile ? i0 + r : j0 + r - kF64Tile;
      cp_async16(st + r * kF64Stride + pp, F + (long long)(i < m ? i : 0) * ldp + pb + pp, i < m);
    }
    if (tid < NS * (kF64Points / 2)) {
      const int pp = (tid & (kF64Points / 2 - 1)) * 2, sp = tid / (kF64Points / 2);
      cp_async16(st + 2 * kF64Tile * kF64Stride + sp * kF64Points + pp,
                 (sp == 0 ? fac_a : fac_b) + (G.pt_off - pt_base) + pb + pp, true);
    }
    cp_async_commit();
  };
  const int nbi = min(NB, (m - i0 + 7) / 8), nbj = min(NB, (m - j0 + 7) / 8);  // 8-function blocks that exist
  double acc[NS][NB][NB][2];
#pragma unroll
  for (int sp = 0; sp < NS; sp++)
#pragma unroll
    for (int a = 0; a < NB; a++)
#pragma unroll
      for (int b = 0; b < NB; b++) acc[sp][a][b][0] = acc[sp][a][b][1] = 0.0;
  copy(f64_smem, s0);
  for (int s = s0; s < s1; s++) {
    double* st = f64_smem + ((s - s0) & 1) * Cfg::kStage;
    if (s + 1 < s1) {
      copy(f64_smem + ((s + 1 - s0) & 1) * Cfg::kStage, s + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const int k0 = warp * 16 + (lane & 3);
    const double* As = st + (lane >> 2) * kF64Stride + k0;
    const double* Bs = As + (diag ? 0 : kF64Tile * kF64Stride);
    const double* fs = st + 2 * kF64Tile * kF64Stride + k0;
#pragma unroll
    for (int k = 0; k < 16; k += 4) {
      double a[NB], b[NB];
#pragma unroll
      for (int r = 0; r < NB; r++) {
        a[r] = As[r * 8 * kF64Stride + k];
        b[r] = Bs[r * 8 * kF64Stride + k];
      }
#pragma unroll
      for (int sp = 0; sp < NS; sp++) {
        const double f = fs[sp * kF64Points + k];
#pragma unroll
        for (int c = 0; c < NB; c++) {
          if (c >= nbj) continue;
          const double bf = b[c] * f;
#pragma unroll
          for (int r = 0; r < NB; r++)
            if (r < nbi && !(diag && r > c)) mma_f64(acc[sp][r][c], a[r], bf);
        }
      }
    }
    __syncthreads();
  }
  // sum the warps' tiles: warps 1-3 through shared memory into warp 0
  if (warp > 0)
#pragma unroll
    for (int sp = 0; sp < NS; sp++)
#pragma unroll
      for (int r = 0; r < NB; r++)
#pragma unroll
        for (int c = 0; c < NB; c++)
#pragma unroll
          for (int e = 0; e < 2; e++)
            f64_smem[((((warp - 1) * NS + sp) * NB + r) * NB + c) * 64 + e * 32 + lane] = acc[sp][r][c][e];
  __syncthreads();
  const int* fg = fn_glob + G.fn_off;
  // warp 0 sums the others' tiles onto its own, in registers, and adds every block
  if (warp == 0)
#pragma unroll
    for (int sp = 0; sp < NS; sp++)
#pragma unroll
      for (int r = 0; r < NB; r++)
#pragma unroll
        for (int c = 0; c < NB; c++) {
          if (r >= nbi || c >= nbj || (diag && r > c)) continue;
#pragma unroll
          for (int e = 0; e < 2; e++) {
            double v = acc[sp][r][c][e];
#pragma unroll
            for (int w = 0; w < 3; w++) v += f64_smem[(((w * NS + sp) * NB + r) * NB + c) * 64 + e * 32 + lane];
            const int i = i0 + r * 8 + (lane >> 2), j = j0 + c * 8 + 2 * (lane & 3) + e;
            if (i < m && j < m && i <= j)
              atomicAdd((sp == 0 ? K_a : K_b) + G.pk_off + packed_index(fg[i], fg[j], G.pk_M), v);
          }
        }
}
