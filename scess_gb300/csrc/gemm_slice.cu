// FP64 GEMM on BF16 slices with tcgen05 (see gemm_slice.h for the splitting).
//
// A persistent CTA per SM walks work units (problem, 128 x bn output tile, K range),
// bn <= 128:
//   warp 0     TMA producer: per 32-wide K block one stage with the 7 slices of
//              128 A rows and bn B rows (64-byte rows, 64B swizzle);
//   warp 1     owns TMEM (two rotating accumulators of bn columns for S_4 .. S_0,
//              one for S_5, one for S_6 + S_7) and issues the MMAs (M = 128, N = bn, K = 16);
//   warps 4-19 four epilogue warpgroups, bn / 4 columns each: add every drained
//              S_d, an exact integer, into one 64-bit integer per output, and turn
//              integer + FP32 tail into FP64 at the end of the unit.
// The wide tile (an MMA of N = 128 takes 64 cycles, one of N = 80 still 52) leaves TMEM
// room for four accumulators only, hence the rotation and five drains per K block, which
// run beside the MMAs.  Both bound it: 68 MMAs take 4350 cycles of a K block's 6050, the
// drains' arithmetic (about four cycles of a scheduler per column, warp and drain) with
// their waits and releases as long.  What got it there, TFLOP/s at 4096^3: with 28 products
// and S_5 + S_6 in one accumulator two epilogue warps a scheduler 38.8, four 41.8 (they hide
// each other's waits); MMAs issued from uniform registers (see elect_one) 51.6; S_5 between
// S_2 and S_1, and accumulators released before their arithmetic, 52.3.  With 34 products
// and S_5 apart 45.0 with the tail in two places among the diagonals, 50.1 in three (56.6 at
// the tensor pipe's measured rate).
// Joint form (tiles of at most 64 columns): TMEM holds an accumulator for every S_d, in two
// sets up to 32 columns, and the five are drained together, with one wait and one release a
// block; three stages where they fit.  313600 x 16 x 140: 315 us -> 150, where the
// packs' bytes read at 4.9 TB/s bound it; 200000 x 16 x 16: 71 -> 43 (both before the
// magnitudes, below).
// A unit of a product that stands alone begins with the product of the magnitudes: seven K blocks
// of that plane fill the places of a stage's seven digit slices, and what is added up in the
// next free accumulator tells which outputs are left to the FP64 units (slice_left).  A warp takes
// its 32 x 32 outputs at once where their least sum reaches their largest threshold.  Cost, with
// the packs' eighth plane: 4096^3 49.9 -> 47.3 TFLOP/s, 8192 x 8192 x 32 293 -> 344 us,
// 313600 x 16 x 140 161 -> 207; FP64 iterations at o = 10, v = 90 6.9 -> 7.4 ms, at o = 16,
// v = 140 38.1 -> 41.1, a residual gradient at o = 8, v = 47 5.28 -> 5.46.
// Every mbarrier wait is bounded (see mbarrier.cuh).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <cstring>
#include <mutex>

#include "dgemm_tile.cuh"
#include "gemm_slice.h"
#include "launch.cuh"
#include "pack_tiles.cuh"
#include "slice_math.cuh"
#include "split_sum.cuh"
#include "tcgen05.cuh"

namespace scess {

namespace {

constexpr int BM = 128, BN = 128, BK = kSliceBK;
constexpr int STAGES = 2, MAX_STAGES = 3;                             // (narrow tiles: three)
constexpr uint32_t A_SLICE = (uint32_t)BM * BK * 2;                  // one slice of 128 rows
constexpr uint32_t STAGE_BYTES = kSlices * (BM + BN) * BK * 2;       // 112 KiB
constexpr int NDIAG = 5;                                             // S_0 .. S_4 are drained
constexpr int NROT = 2, TAIL = NROT, NACC = NROT + 2;                // accumulators: S_5 at TAIL, then S_6 + S_7
constexpr int kS5Before = 3, kS6Before = 2, kS7Before = 0;           // places in S_4 .. S_0
constexpr int EPI = 4;                                               // epilogue warpgroups
constexpr int HC = BN / EPI;                                         // columns of an epilogue thread
constexpr int BN_JOINT = 64, HC_JOINT = 16;                          // the same of the joint form
constexpr int THREADS = 128 * (1 + EPI);
constexpr int kEpiRegs = 104, kCtlRegs = 56, kLaunchRegs = 96;       // 56 + 4 x 104 <= 5 x 96
static_assert(kSlices == NDIAG + 2, "the tail is S_5 .. S_7");
static_assert(kCtlRegs + EPI * kEpiRegs <= (1 + EPI) * kLaunchRegs, "setmaxnreg draws on the launch's registers");
// First column of epilogue group h (0 .. EPI) of a tile of bn columns: a quarter each, in groups of
// eight; and the group of a column.
__host__ __device__ constexpr int group_start(int bn, int h) { return 8 * ((bn / 8 * h + 3) / 4); }
__device__ __forceinline__ int column_group(int bn, int col) {
  int h = 0;
  while (h < EPI - 1 && col >= group_start(bn, h + 1)) h++;
  return h;
}
struct Ctl {  // behind the stages
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], tfull[NACC], tempty[NACC], done;
  uint32_t tmem;
  alignas(16) int64_t colOff[BN];
  alignas(16) int colE[BN];
};
constexpr size_t SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + sizeof(Ctl);

enum : unsigned { ERR_FULL_WAIT = 1, ERR_EMPTY_WAIT = 2, ERR_ACCUM_WAIT = 3 };

struct SegArgs {
  int mapA, mapB;
  int nkb, kpad;
  int64_t rowA0[3], rowAy[3], rowAz[3], rowB0[3], rowBy[3], rowBz[3];
};
struct SliceMaps {
  CUtensorMap m[6];
};
struct SliceArgs {
  int M, N, tiles_m, tiles_n;
  int bn;      // tile width: a multiple of 16, at most 128 (joint form: 64)
  int stages;  // joint form
  int fs;      // fraction bits kept of the tail (see slice_value)
  int ny, nz, ng, nseg;
  int kb_total, kb_per_split, splits;
  SegArgs seg[4];
  int tri[3], gstart[4];
  const int *expA, *expB;
  int64_t expA0[3];
  // est: sum_k |a_k b_k| first, to find the outputs that are left to the FP64 units (see
  // slice_left).  Per tile 16 flags (32 rows x a column group each); where one is set, bit
  // column - group_start of left[tile][column group][row] marks an output.  Split-K: the sums
  // go to est_partial [split][n][m], and the reduction sets the marks.
  int est;
  int rowsA, rowsB;  // of the statistics behind expA, expB (see SlicedPack)
  float sq_unit;
  uint32_t *left;
  uint8_t *flags;
  float *est_partial;
  double *C;
  int64_t baseC, cy[3], cz[3], cg[3];
  const int64_t *rowC[3], *colC[3];
  double alpha, beta;
  int alpha_pow2, alpha_e, alpha_neg;  // alpha = (-1)^neg 2^e: folded into the exponent
  double *partial;                     // split-K partial sums [split][n][m], or null
  int64_t part_stride;
  unsigned *err;
  long long wait_cycles;
  int withhold_first;
};

// T += i 2^(9 (4 - D)) for the drained S_D = i 2^(-9 D) of one K block: |i| is at most
// 2^17, 2^20, 0.75 2^22, 0.63 2^23, 0.88 2^23 for D = 0 .. 4.  S_0 .. S_2 become
// integers by adding 1.5 2^(23 - 9 D), whose bit pattern then holds the integer in its
// low bits (the constants' own patterns are taken off once per unit); S_3 and S_4 are
// converted.
constexpr int kMagic0 = 0x4B400000;                    // 1.5 2^23
constexpr int kMagic1 = kMagic0 - (9 << 23);           // 1.5 2^14
constexpr int kMagic2 = kMagic0 - (18 << 23);          // 1.5 2^5
template <int D>
__device__ __forceinline__ void add_diag(long long &T, uint32_t raw) {
  const float s = __uint_as_float(raw);
  if constexpr (D == 0) {
    const int b = __float_as_int(s + __int_as_float(kMagic0));
    T += (long long)((unsigned long long)(unsigned)(b << 4) << 32);
  } else if constexpr (D == 1) {
    const int b = __float_as_int(s + __int_as_float(kMagic1));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(T) : "r"(b), "n"(1 << 27));
  } else if constexpr (D == 2) {
    const int b = __float_as_int(s + __int_as_float(kMagic2));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(T) : "r"(b), "n"(1 << 18));
  } else {
    const int b = __float2int_rn(s * __int_as_float((127 + 9 * D) << 23));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(T) : "r"(b), "n"(1 << (9 * (4 - D))));
  }
}
// What the magic constants have added to T after n K blocks (modulo 2^64).
__device__ __forceinline__ long long magic_sum(int n) {
  const unsigned long long c = ((unsigned long long)(unsigned)(kMagic0 << 4) << 32) +
                               ((unsigned long long)kMagic1 << 27) + ((unsigned long long)kMagic2 << 18);
  return (long long)(c * (unsigned long long)n);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// The wait takes the loaded registers as operands: no use is scheduled before it.
__device__ __forceinline__ void tmem_wait8(uint32_t *r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
               :
               : "memory");
}

// Which outputs the slices cannot hold as well as FP64 multiply-adds would.  A value is rounded at
// 2^-61 of its row's largest, so that an output's error is, in rms, 2^-61 |row max| |column max|
// (q / 3)^(1/2) with q = sum (a_k / row max)^2 + (b_k / column max)^2 over the k that both
// sides have (and 2^-13 each for the digit products that are dropped); a chain of
// multiply-adds has about 0.4 2^-53 sum_k |a_k b_k|.  So that sum has to reach 1.44 2^-8 q^(1/2)
// of |row max| |column max|; 2^-7 is asked for.  Exact zeros are exact here too.
struct RangeRow {
  float sq, count;  // sum of (value / largest)^2, values that are not zero; negative sq: Inf or NaN
};
__device__ __forceinline__ RangeRow range_row(const int *exps, int rows, int64_t r, float sq_unit) {
  if (r >= rows) return {0.0f, 0.0f};
  return {exps[r] == kRowNonFinite ? -1.0f : (float)exps[rows + r] * sq_unit, (float)exps[2 * (int64_t)rows + r]};
}
__device__ __forceinline__ bool slice_left(float sum, RangeRow a, RangeRow b) {
  if (a.sq < 0.0f || b.sq < 0.0f) return true;
  const float q = fminf(a.sq, b.count) + fminf(b.sq, a.count) + 0x1p-13f * fminf(a.count, b.count);
  return sum != 0.0f && sum * sum < 0x1p-14f * q;
}

// What bounds it: long K, the drains (above); short K, the outputs (about 45 instructions each).
template <bool JOINT>
__global__ void __launch_bounds__(THREADS, 1)
    slice_gemm_kernel(const __grid_constant__ SliceMaps maps, const __grid_constant__ SliceArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Ctl &ctl = *reinterpret_cast<Ctl *>(smem + STAGES * STAGE_BYTES);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int tiles = a.tiles_m * a.tiles_n;
  const int nprob = a.gstart[a.ng];
  const int units = tiles * nprob * a.splits;
  const int bn = a.bn;
  const uint32_t bslice = (uint32_t)bn * BK * 2;
  const uint32_t stage_bytes = JOINT ? kSlices * (A_SLICE + bslice) : STAGE_BYTES;
  const int nst = JOINT ? a.stages : STAGES;
  const int nset = JOINT && 12 * bn <= 512 ? 2 : 1;                    // sets of S_0 .. S_4
  const uint32_t tail_col = (uint32_t)((JOINT ? nset * NDIAG : TAIL) * bn);

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; s++) {
      mbar_init(&ctl.full[s], 1);
      mbar_init(&ctl.empty[s], 1);
    }
    for (int b = 0; b < NACC; b++) {
      mbar_init(&ctl.tfull[b], 1);
      mbar_init(&ctl.tempty[b], 4 * EPI);  // one arrival per epilogue warp
    }
    mbar_init(&ctl.done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&ctl.tmem)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl.tmem;
  chain();

  // unit -> (tile m, tile n, problem y, z, g, K-block range, split)
  auto unit_coords = [&](int u, int &tm, int &tn, int &py, int &pz, int &pg, int &kb0, int &kb1, int &sp) {
    const int tile = u % tiles;
    const int rest = u / tiles;
    const int q = rest % nprob;
    sp = rest / nprob;
    tn = tile % a.tiles_n;
    tm = tile / a.tiles_n;
    pg = 0;
    while (pg + 1 < a.ng && q >= a.gstart[pg + 1]) pg++;
    const int lq = q - a.gstart[pg];
    if (a.tri[pg]) {  // lq = y (y + 1) / 2 + z, z <= y
      int y = (int)((sqrtf(8.0f * (float)lq + 1.0f) - 1.0f) * 0.5f);
      while (y * (y + 1) / 2 > lq) y--;
      while ((y + 1) * (y + 2) / 2 <= lq) y++;
      py = y;
      pz = lq - y * (y + 1) / 2;
    } else {
      py = lq % a.ny;
      pz = lq / a.ny;
    }
    kb0 = sp * a.kb_per_split;
    kb1 = min(a.kb_total, kb0 + a.kb_per_split);
  };
  auto seg_at = [&](int kb, int &s, int &lkb) {
    s = 0;
    lkb = kb;
    while (s < a.nseg - 1 && lkb >= a.seg[s].nkb) {
      lkb -= a.seg[s].nkb;
      s++;
    }
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kCtlRegs));
  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;          // stage and its phase
      int used = 0;             // stages filled at least once
      uint32_t lastph = 0;      // phases of their last fills, a bit each
      bool withhold = a.withhold_first;  // diagnostics: the first stage is taken but never filled
      bool ok = true;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        int tm, tn, py, pz, pg, kb0, kb1, sp;
        unit_coords(u, tm, tn, py, pz, pg, kb0, kb1, sp);
        // magnitudes: the places of the digits' seven slices take seven K blocks
        for (int kb = kb0; a.est && kb < kb1; kb += kSlices) {
          if (s == nst) {
            s = 0;
            ph ^= 1u;
          }
          const SegArgs &S = a.seg[0];
          const int n = min(kSlices, kb1 - kb), x = kSlices * S.kpad + kb * BK;
          if (!mbar_wait(&ctl.empty[s], ph ^ 1u, a.err, ERR_EMPTY_WAIT, a.wait_cycles)) { ok = false; break; }
          if (withhold) {
            withhold = false;
            s++;
            continue;
          }
          uint8_t *st = smem + s * stage_bytes;
          mbar_expect_tx(&ctl.full[s], n * (A_SLICE + bslice));
          for (int p = 0; p < n; p++) {
            tma_load_2d(st + p * A_SLICE, &maps.m[S.mapA], x + p * BK, tm * BM, &ctl.full[s]);
            tma_load_2d(st + kSlices * A_SLICE + p * bslice, &maps.m[S.mapB], x + p * BK, tn * bn, &ctl.full[s]);
          }
          used |= 1 << s;
          lastph = (lastph & ~(1u << s)) | (ph << s);
          s++;
        }
        for (int kb = kb0; kb < kb1 && ok; kb++) {
          if (s == nst) {
            s = 0;
            ph ^= 1u;
          }
          int sg, lkb;
          seg_at(kb, sg, lkb);
          const SegArgs &S = a.seg[sg];
          const int ya = (int)(S.rowA0[pg] + py * S.rowAy[pg] + pz * S.rowAz[pg]) + tm * BM;
          const int yb = (int)(S.rowB0[pg] + py * S.rowBy[pg] + pz * S.rowBz[pg]) + tn * bn;
          if (!mbar_wait(&ctl.empty[s], ph ^ 1u, a.err, ERR_EMPTY_WAIT, a.wait_cycles)) { ok = false; break; }
          if (withhold) {
            withhold = false;
            s++;
            continue;
          }
          uint8_t *st = smem + s * stage_bytes;
          mbar_expect_tx(&ctl.full[s], kSlices * (A_SLICE + bslice));
#pragma unroll
          for (int p = kSlices - 1; p >= 0; p--) {
            tma_load_2d(st + p * A_SLICE, &maps.m[S.mapA], p * S.kpad + lkb * BK, ya, &ctl.full[s]);
            tma_load_2d(st + kSlices * A_SLICE + p * bslice, &maps.m[S.mapB], p * S.kpad + lkb * BK, yb,
                        &ctl.full[s]);
          }
          used |= 1 << s;
          lastph = (lastph & ~(1u << s)) | (ph << s);
          s++;
        }
      }
      for (int q = 0; q < nst; q++)
        if (used >> q & 1) mbar_drain(&ctl.full[q], lastph >> q & 1u);
    }
  } else if (warp == 1) {
    // all lanes, issues by the elected one (see elect_one)
    int s = 0, c = 0, w = 0;  // stage, rotating fills (joint: K blocks) and units so far
    uint32_t ph = 0;          // phase of the stage
    const uint64_t desc = sw_desc<64>(smem_u32(smem));
    const uint32_t hi = (uint32_t)(desc >> 32), lo = (uint32_t)desc;
    const uint32_t bq = bslice >> 4;
    const bool issuer = elect_one();
    auto wait = [&](uint64_t *barrier, uint32_t parity, unsigned code) {
      return __all_sync(0xffffffffu, mbar_wait(barrier, parity, a.err, code, a.wait_cycles)) != 0;
    };
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x, w++) {
      int tm, tn, py, pz, pg, kb0, kb1, sp;
      unit_coords(u, tm, tn, py, pz, pg, kb0, kb1, sp);
      const uint32_t idesc = idesc_f16kind(BM, min(bn, (a.N - tn * bn + 15) & ~15), 1u);  // BF16
      if (a.est) {  // magnitudes into the next accumulator (joint form: the first of a set)
        const int b = JOINT ? (nset == 2 ? c & 1 : 0) : c % NROT;
        const int f = JOINT ? (nset == 2 ? c >> 1 : c) : c / NROT;  // fills of it before
        const uint32_t col = tmem + (uint32_t)(JOINT ? b * NDIAG * bn : b * bn);
        ok = wait(&ctl.tempty[b], ((uint32_t)f & 1u) ^ 1u, ERR_EMPTY_WAIT);
        for (int kb = kb0; kb < kb1 && ok; kb += kSlices, s++) {
          if (s == nst) {
            s = 0;
            ph ^= 1u;
          }
          if (!wait(&ctl.full[s], ph, ERR_FULL_WAIT)) { ok = false; break; }
          tc_fence_after();
          const uint32_t da = lo + (uint32_t)s * (stage_bytes >> 4), db = da + (kSlices * A_SLICE >> 4);
          if (issuer) {
            const int n = min(kSlices, kb1 - kb);
            for (int p = 0; p < n; p++)
#pragma unroll
              for (int k = 0; k < 2; k++)
                mma_f16kind(col, da + p * (A_SLICE >> 4) + 2 * k, db + p * bq + 2 * k, hi, idesc, kb > kb0 || p || k ? 1u : 0u);
            mma_commit(&ctl.empty[s]);
          }
        }
        if (!ok) break;
        if (issuer) mma_commit(&ctl.tfull[b]);
        c++;
      }
      for (int kb = kb0; kb < kb1 && ok; kb++, s++) {
        if (s == nst) {
          s = 0;
          ph ^= 1u;
        }
        if (!wait(&ctl.full[s], ph, ERR_FULL_WAIT)) { ok = false; break; }
        tc_fence_after();
        // slice offsets are added to the stage's descriptors (address field in units of 16 bytes)
        const uint32_t da = lo + (uint32_t)s * (stage_bytes >> 4), db = da + (kSlices * A_SLICE >> 4);
        auto product = [&](uint32_t col, int p, int q, uint32_t acc) {
#pragma unroll
          for (int k = 0; k < 2; k++)
            mma_f16kind(tmem + col, da + p * (A_SLICE >> 4) + 2 * k, db + q * bq + 2 * k, hi, idesc, k ? 1u : acc);
        };
        // S_5 into one accumulator, where it stays exact as long as it is below 2^24 of its
        // units, S_6 and S_7 into another
        auto tail = [&](auto diag, uint32_t acc) {
          constexpr int d = decltype(diag)::value;
#pragma unroll
          for (int p = d < kSlices ? 0 : d - kSlices + 1; p <= d && p < kSlices; p++, acc = 1u)
            product(tail_col + (uint32_t)(d == NDIAG ? 0 : bn), p, d - p, acc);
        };
        const uint32_t cont = kb == kb0 ? 0u : 1u;
        auto tail_free = [&]() {
          if (!wait(&ctl.tempty[TAIL], ((uint32_t)w & 1u) ^ 1u, ERR_EMPTY_WAIT)) return false;
          tc_fence_after();
          return true;
        };
        if constexpr (JOINT) {
          // S_4 .. S_0 into a set of their own, drained together beside the tail
          const int set = nset == 2 ? c & 1 : 0;
          if (!wait(&ctl.tempty[set], (uint32_t)(nset == 2 ? c >> 1 : c) & 1u ^ 1u, ERR_EMPTY_WAIT)) { ok = false; break; }
          tc_fence_after();
          c++;
          if (issuer) {
#pragma unroll
            for (int d = NDIAG - 1; d >= 0; d--)
#pragma unroll
              for (int p = 0; p <= d; p++) product((uint32_t)((set * NDIAG + d) * bn), p, d - p, p ? 1u : 0u);
            mma_commit(&ctl.tfull[set]);
          }
          if (kb == kb0 && !tail_free()) { ok = false; break; }
          if (issuer) {
            tail(std::integral_constant<int, NDIAG>{}, cont);
            tail(std::integral_constant<int, NDIAG + 1>{}, cont);
            tail(std::integral_constant<int, NDIAG + 2>{}, 1u);
            mma_commit(&ctl.empty[s]);
          }
        } else {
          // The longest diagonals first, S_5 .. S_7 between them: a drain is then done when its
          // accumulator comes round.
#pragma unroll
          for (int d = NDIAG - 1; d >= 0; d--) {
            if (d == kS5Before) {
              if (kb == kb0 && !tail_free()) { ok = false; break; }
              if (issuer) tail(std::integral_constant<int, NDIAG>{}, cont);
            }
            if (d == kS6Before && issuer) tail(std::integral_constant<int, NDIAG + 1>{}, cont);
            if (d == kS7Before && issuer) tail(std::integral_constant<int, NDIAG + 2>{}, 1u);
            const int b = c % NROT;
            if (ok && !wait(&ctl.tempty[b], (((uint32_t)(c / NROT)) & 1u) ^ 1u, ERR_EMPTY_WAIT)) ok = false;
            if (!ok) break;
            tc_fence_after();
            if (issuer) {
#pragma unroll
              for (int p = 0; p <= d; p++) product((uint32_t)(b * bn), p, d - p, p ? 1u : 0u);
              mma_commit(&ctl.tfull[b]);
            }
            c++;
          }
          if (!ok) break;
          if (issuer) mma_commit(&ctl.empty[s]);
        }
      }
      if (ok && issuer) mma_commit(&ctl.tfull[TAIL]);
    }
    if (issuer) mma_commit(&ctl.done);
    mbar_drain(&ctl.done, 0);
  }
  } else {  // epilogue warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
    const int q = warp & 3;
    const int row = 32 * q + lane;
    const int h = (warp - 4) >> 2;                  // column group
    const int h0 = group_start(bn, h), hc = group_start(bn, h + 1) - h0;  // its columns
    constexpr int HCT = JOINT ? HC_JOINT : HC;
    const int et = threadIdx.x - 128 - 128 * h;     // 0..127 within the group
    const int bar = 1 + h;
    int c = 0, w = 0;
    bool ok = true;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)h0;
    // (one answer for a warp: what follows a wait is done by all its lanes or by none)
    auto wait = [&](uint64_t *barrier, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(barrier, parity, a.err, ERR_ACCUM_WAIT, a.wait_cycles)) != 0;
    };
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x, w++) {
      int tm, tn, py, pz, pg, kb0, kb1, sp;
      unit_coords(u, tm, tn, py, pz, pg, kb0, kb1, sp);
      const int m = tm * BM + row;
      asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");  // previous unit's column tables read
      if (et < hc) {
        const int nn = tn * bn + h0 + et;
        const int e = nn < a.N ? a.expB[nn] : kRowNonFinite;
        ctl.colE[h0 + et] = e == 0 ? 1023 : e;  // (all zero: any scale)
        ctl.colOff[h0 + et] =
            e == kRowNonFinite ? -1
            : a.partial ? (int64_t)sp * a.part_stride + (int64_t)a.M * nn
                        : a.baseC + py * a.cy[pg] + pz * a.cz[pg] + a.cg[pg] + a.colC[pg][nn];
      }
      const int eA = m < a.M ? a.expA[a.expA0[pg] + m] : kRowNonFinite;
      const int64_t rowOff = m < a.M ? (a.partial ? (int64_t)m : a.rowC[pg][m]) : 0;
      const unsigned errv = *(volatile unsigned *)a.err;
      auto release = [&](int b) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&ctl.tempty[b])) : "memory");
      };
      uint32_t left = 0;  // columns of this row left to the FP64 units
      if (a.est) {
        const int b = JOINT ? (nset == 2 ? c & 1 : 0) : c % NROT;
        const int f = JOINT ? (nset == 2 ? c >> 1 : c) : c / NROT;
        const int n0 = tn * bn + h0, nv = min(hc, a.N - n0);  // columns inside the product
        const RangeRow ra = range_row(a.expA, a.rowsA, m, a.sq_unit);
        const RangeRow rb = range_row(a.expB, lane < nv ? a.rowsB : 0, n0 + lane, a.sq_unit);  // lane's column
        ok = wait(&ctl.tfull[b], (uint32_t)f & 1u);
        if (ok) {
          c++;
          tc_fence_after();
          const uint32_t t0 = tl + (uint32_t)(JOINT ? b * NDIAG * bn : b * bn);
          // all of a warp's outputs at once, by the largest threshold of theirs; else one by one
          const RangeRow most = {__int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(fmaxf(rb.sq, 0.0f)))),
                                 __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(rb.count)))};
          float least = 3.0e38f;
          float *p = a.est_partial + (int64_t)sp * a.part_stride + (int64_t)a.M * n0 + m;
#pragma unroll
          for (int j = 0; j < HCT; j += 8) {
            if (j >= hc) continue;
            uint32_t r[8];
            tmem_ld8(t0 + (uint32_t)j, r);
            tmem_wait8(r);
#pragma unroll
            for (int i = 0; i < 8; i++) {
              if (j + i >= nv) continue;
              if (!a.partial) least = fminf(least, __uint_as_float(r[i]));
              else if (m < a.M) p[(int64_t)a.M * (j + i)] = __uint_as_float(r[i]);
            }
          }
          const bool sure = a.partial || m >= a.M || (rb.sq >= 0.0f && least != 0.0f && !slice_left(least, ra, most));
          if (!__all_sync(0xffffffffu, sure)) {
#pragma unroll 1
            for (int j = 0; j < hc; j += 8) {
              uint32_t r[8];
              tmem_ld8(t0 + (uint32_t)j, r);
              tmem_wait8(r);
#pragma unroll
              for (int i = 0; i < 8; i++) {
                const RangeRow x = {__shfl_sync(0xffffffffu, rb.sq, j + i), __shfl_sync(0xffffffffu, rb.count, j + i)};
                if (j + i < nv && m < a.M && slice_left(__uint_as_float(r[i]), ra, x)) left |= 1u << (j + i);
              }
            }
          }
          release(b);
          const bool any = __any_sync(0xffffffffu, left != 0u);
          // (split-K: cleared here, set by the reduction)
          if (lane == 0 && sp == 0) a.flags[16 * (u % tiles) + 4 * h + q] = any;
          if (any || (a.partial && sp == 0)) a.left[(int64_t)(u % tiles * EPI + h) * BM + row] = left;
        }
      }
      long long T[HCT];
      const long long off = magic_sum(kb1 - kb0);
#pragma unroll
      for (int j = 0; j < HCT; j++) T[j] = -off;
      auto take = [&](auto diag) -> bool {
        constexpr int D = decltype(diag)::value;
        const int b = c % NROT;
        if (!wait(&ctl.tfull[b], (uint32_t)(c / NROT) & 1u)) return false;
        tc_fence_after();
        const uint32_t t0 = tl + (uint32_t)(b * bn);
        // (8 columns a load: the sums take most of the registers)
#pragma unroll
        for (int j = 0; j < HC; j += 8) {
          if (j < hc) {
            uint32_t r[8];
            tmem_ld8(t0 + (uint32_t)j, r);
            tmem_wait8(r);
            if (j + 8 >= hc) release(b);  // (all columns are in registers)
#pragma unroll
            for (int i = 0; i < 8; i++) add_diag<D>(T[j + i], r[i]);
          }
        }
        c++;
        return true;
      };
      for (int kb = kb0; kb < kb1 && ok; kb++) {
        if constexpr (JOINT) {
          const int set = nset == 2 ? c & 1 : 0;
          ok = wait(&ctl.tfull[set], (uint32_t)(nset == 2 ? c >> 1 : c) & 1u);
          if (!ok) break;
          c++;
          tc_fence_after();
          const uint32_t t0 = tl + (uint32_t)(set * NDIAG * bn);
          if (hc == 0) release(set);
#pragma unroll
          for (int j = 0; j < HCT; j += 8) {
            if (j >= hc) continue;
            uint32_t r[NDIAG][8];
#pragma unroll
            for (int d = 0; d < NDIAG; d++) tmem_ld8(t0 + (uint32_t)(d * bn + j), r[d]);
#pragma unroll
            for (int d = 0; d < NDIAG; d++) tmem_wait8(r[d]);
            if (j + 8 >= hc) release(set);  // (all columns are in registers)
#pragma unroll
            for (int i = 0; i < 8; i++) {
              add_diag<0>(T[j + i], r[0][i]);
              add_diag<1>(T[j + i], r[1][i]);
              add_diag<2>(T[j + i], r[2][i]);
              add_diag<3>(T[j + i], r[3][i]);
              add_diag<4>(T[j + i], r[4][i]);
            }
          }
        } else {
          ok = take(std::integral_constant<int, 4>{}) && take(std::integral_constant<int, 3>{}) &&
               take(std::integral_constant<int, 2>{}) && take(std::integral_constant<int, 1>{}) &&
               take(std::integral_constant<int, 0>{});
          if (!ok) break;
        }
      }
      if (ok && !wait(&ctl.tfull[TAIL], (uint32_t)w & 1u)) ok = false;
      // Column tables of this unit written.  The group's four warps leave together or not at all:
      // one that left alone would be missed at the next unit's barrier, which has no bound.
      if (group_any(bar, !ok || errv)) break;
      tc_fence_after();
      const double mul = a.alpha;
      const bool scaled = !a.partial && !a.alpha_pow2;
      const uint32_t flip = (!a.partial && a.alpha_pow2 && a.alpha_neg) ? 0x80000000u : 0u;
      // value = (T 2^-36 + tail) 2^(EA + EB - 12), E = exps - 1022
      const int sc0 = (eA == 0 ? 1023 : eA) - 2 * 1022 - 12 - 36 + ((!a.partial && a.alpha_pow2) ? a.alpha_e : 0);
      const float ftail = __int_as_float((127 + 36 + a.fs) << 23);  // 2^(36 + fs)
      double *base = (a.partial ? a.partial : a.C) + rowOff;
      const int mode = (a.partial || a.beta == 0.0) ? 0 : (a.beta == 1.0 ? 1 : 2);
      // Plain warps (every row and column inside the product, finite and of a scale that
      // keeps results normal) skip the checks of each output: 42 instructions instead of 90.
      auto fits = [](int e) { return e >= 640 && e <= 1400; };
      const bool rok = fits(eA == 0 ? 1023 : eA) && sc0 >= -1500 && sc0 <= -600;
      const bool cok = lane >= hc || (ctl.colOff[h0 + lane] >= 0 && fits(ctl.colE[h0 + lane]));
      const bool plain = __all_sync(0xffffffffu, rok && cok && !left) && !scaled && mode != 2;
      auto finish = [&](auto is_plain) {
        constexpr bool PLAIN = decltype(is_plain)::value;
#pragma unroll
        for (int j = 0; j < HCT; j += 8) {
          if (j >= hc) continue;
          uint32_t r[8], r6[8];
          tmem_ld8(tl + tail_col + (uint32_t)j, r);
          tmem_ld8(tl + tail_col + (uint32_t)(bn + j), r6);
          int e[8];
          long long co[8];
          *reinterpret_cast<int4 *>(e) = *reinterpret_cast<const int4 *>(&ctl.colE[h0 + j]);
          *reinterpret_cast<int4 *>(e + 4) = *reinterpret_cast<const int4 *>(&ctl.colE[h0 + j + 4]);
#pragma unroll
          for (int i = 0; i < 8; i += 2)
            *reinterpret_cast<longlong2 *>(co + i) = *reinterpret_cast<const longlong2 *>(&ctl.colOff[h0 + j + i]);
          tmem_wait8(r);
          tmem_wait8(r6);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int w = rint_i32(__uint_as_float(r[i]) * ftail) + rint_i32(__uint_as_float(r6[i]) * ftail);
            double *p = base + co[i];
            if (PLAIN) {
              const double v = slice_value_plain(T[j + i], w, a.fs, sc0 + e[i], flip);
              if (mode == 0) *p = v;
              else asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
            } else if (co[i] >= 0 && eA != kRowNonFinite && !(left >> (j + i) & 1u)) {
              double v = slice_value(T[j + i], w, a.fs, sc0 + e[i], flip);
              if (scaled) v *= mul;
              if (mode == 0) *p = v;
              else if (mode == 1) asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
              else *p = fma(a.beta, *p, v);
            }
          }
        }
      };
      if (plain) finish(std::true_type{});
      else finish(std::false_type{});
      release(TAIL);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

struct PartialSum {
  double sum = 0.0;
  float est = 0.0f;
  __device__ void operator+=(const PartialSum &o) {
    sum += o.sum;
    est += o.est;
  }
};
// Split-K: C = alpha sum_z partial_z + beta C over the outputs that are not left.
template <int ZG>
__global__ void __launch_bounds__(256) slice_reduce_kernel(const __grid_constant__ SliceArgs a, int splits) {
  chain();
  const int64_t MN = (int64_t)a.M * a.N;
  auto load = [&](int z, int64_t e) { return PartialSum{a.partial[z * MN + e], a.est_partial[z * MN + e]}; };
  split_sum<ZG, PartialSum>(a.M, a.N, splits, load, [&](int64_t m, int64_t n, const PartialSum &x) {
    const double s = x.sum;
    if (slice_left(x.est, range_row(a.expA, a.rowsA, m, a.sq_unit), range_row(a.expB, a.rowsB, n, a.sq_unit))) {
      const int tn = (int)n / a.bn, tile = (int)m / BM * a.tiles_n + tn, row = (int)m % BM, col = (int)n - tn * a.bn;
      const int h = column_group(a.bn, col);
      a.flags[16 * tile + 4 * h + (row >> 5)] = 1;
      atomicOr(&a.left[(int64_t)(tile * EPI + h) * BM + row], 1u << (col - group_start(a.bn, h)));
      return;
    }
    double *p = a.C + a.baseC + a.rowC[0][m] + a.colC[0][n];
    double val = a.alpha * s;
    if (a.beta != 0.0) val += a.beta * *p;
    *p = val;
  });
}

// ---------------------------------------------------------------------------------------------
// Packs.  One CTA per tile of 2048 / KT rows x KT values of k (KT = 64, or 32, 16 for a K
// that short; rows in the order of RowTiles, so that loads coalesce) and range of K
// chunks.  A launch takes up to two operands.  OWN: the CTA covers the whole K, finds
// its rows' exponents in a first walk (kept in registers when K <= KT) and cuts in a
// second one, whose loads hit L2.  PART / FROM_PART: K spread over CTAs, partial
// exponents first, the cut in a second launch.  EXPS: exponents only, folded into
// exps[expIdx[row]] with atomics.  GIVEN: exponents exps[expIdx[row]], K spread over
// CTAs.
// HBM-bound with long rows (8 B read and 16 B written per element, 3.4 TB/s at
// 4096 x 4096, 2.3 before the loads of the next chunk were in flight while one is cut).
enum PackMode { PACK_OWN, PACK_PART, PACK_FROM_PART, PACK_EXPS, PACK_GIVEN };
struct PackOp {
  const double *src;
  const int64_t *row, *k;  // offset tables, or null: r rs and k ks
  int64_t rs, ks;
  int64_t rows, K, Kpad;
  RowTiles rt;
  int mode, unitK, negate, parts;
  uint16_t *dst;
  int *exps, *part;
  int *stats;     // behind exps: sums of squares, counts (see SlicedPack)
  float sq_unit;
  const int64_t *expIdx;
  int64_t blocks;  // rt.count times the K ranges
};
struct PackOps {
  PackOp op[2];
};

__device__ __forceinline__ int tile_col(int k) { return k + (k >> 3); }

template <int KT>
__global__ void __launch_bounds__(256) slice_pack_kernel(const __grid_constant__ PackOps ops) {
  chain();
  const bool second = blockIdx.x >= ops.op[0].blocks;
  const PackOp &op = ops.op[second ? 1 : 0];
  const int64_t blk = second ? blockIdx.x - ops.op[0].blocks : blockIdx.x;
  // doubles with a gap every 8 columns and a pitch of 1 mod 16: free of bank conflicts both ways
  constexpr int ROWS = 2048 / KT, PITCH = KT == 64 ? 81 : KT == 32 ? 49 : 33;
  __shared__ double tile[ROWS][PITCH];
  __shared__ int64_t sr[ROWS], sk[KT], srow[ROWS];
  __shared__ int se[ROWS];
  const int t = threadIdx.x;
  const int mode = op.mode, unitK = op.unitK;
  const int64_t x0 = blk % op.rt.count, c0 = blk / op.rt.count, cs = op.blocks / op.rt.count;
  const int64_t K = op.K;
  const double *__restrict__ src = op.src;
  if (t < ROWS) {
    const int64_t r = op.rt.row(x0 * ROWS + t);
    srow[t] = r;
    sr[t] = r < 0 ? -1 : (op.row ? op.row[r] : r * op.rs);
    int e = 0;
    if (r >= 0 && mode == PACK_GIVEN) e = op.exps[op.expIdx ? op.expIdx[r] : r];
    if (r >= 0 && mode == PACK_FROM_PART) {
      for (int q = 0; q < op.parts; q++) e = max(e, op.part[(int64_t)q * op.rows + r]);
      if (c0 == 0) op.exps[r] = e;
    }
    se[t] = e;
  }
  auto koff = [&](int64_t k) -> int64_t { return k < K ? (op.k ? op.k[k] : k * op.ks) : -1; };
  double x[8];
  auto load = [&]() {
#pragma unroll
    for (int p = 0; p < 8; p++) {
      const int rr = unitK ? t / KT + (256 / KT) * p : t % ROWS, kk = unitK ? t % KT : t / ROWS + (256 / ROWS) * p;
      const int64_t ro = sr[rr], ko = sk[kk];
      x[p] = (ro >= 0 && ko >= 0) ? src[ro + ko] : 0.0;
    }
  };
  const bool find = mode == PACK_OWN || mode == PACK_PART || mode == PACK_EXPS;
  if (find) {
    int mx[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int64_t c = c0; c * KT < K; c += cs) {
      __syncthreads();
      if (t < KT) sk[t] = koff(c * KT + t);
      __syncthreads();
      load();
#pragma unroll
      for (int p = 0; p < 8; p++) {
        const int hi = __double2hiint(x[p]) & 0x7fffffff;
        const int e = (hi >> 20) ? (hi >> 20) : ((hi | __double2loint(x[p])) ? 1 : 0);
        mx[p] = max(mx[p], e);
      }
    }
    if (unitK) {  // KT lanes share a row (two warps with KT = 64)
#pragma unroll
      for (int p = 0; p < 8; p++) {
        int m = mx[p];
#pragma unroll
        for (int off = (KT < 32 ? KT : 32) / 2; off > 0; off >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off));
        if (t % (KT < 32 ? KT : 32) == 0) atomicMax(&se[t / KT + (256 / KT) * p], m);
      }
    } else {
      int m = 0;
#pragma unroll
      for (int p = 0; p < 8; p++) m = max(m, mx[p]);
      atomicMax(&se[t % ROWS], m);
    }
    __syncthreads();
    if (t < ROWS && srow[t] >= 0) {
      if (mode == PACK_EXPS) atomicMax(&op.exps[op.expIdx ? op.expIdx[srow[t]] : srow[t]], se[t]);
      else if (mode == PACK_PART) {
        op.part[c0 * op.rows + srow[t]] = se[t];
        if (c0 == 0) op.stats[srow[t]] = op.stats[op.rows + srow[t]] = 0;  // (added up by the second launch)
      }
      else op.exps[srow[t]] = se[t];
    }
    if (mode != PACK_OWN) return;
  }
  const int64_t Kpad = op.Kpad, nchunk = (Kpad + KT - 1) / KT;
  if (!(find && K <= KT)) {  // (else x holds the chunk already)
    __syncthreads();
    if (t < KT) sk[t] = koff(c0 * KT + t);
    __syncthreads();
    load();
  }
  const int rr = t / (KT / 8), ch = t % (KT / 8);
  int count = 0;
  float sq = 0.0f;
  for (int64_t c = c0; c < nchunk; c += cs) {
    const bool more = c + cs < nchunk;
    const int64_t nk = (t < KT && more) ? koff((c + cs) * KT + t) : -1;
    __syncthreads();  // the previous chunk's tile and offsets are used up
#pragma unroll
    for (int p = 0; p < 8; p++) {
      const int r = unitK ? t / KT + (256 / KT) * p : t % ROWS, kk = unitK ? t % KT : t / ROWS + (256 / ROWS) * p;
      tile[r][tile_col(kk)] = x[p];
    }
    if (t < KT) sk[t] = nk;
    __syncthreads();
    if (more) load();  // in flight while this chunk is cut
    const int64_t k0 = c * KT, r = srow[rr];
    if (r < 0 || k0 + ch * 8 >= Kpad) continue;
    const int e = se[rr];
    uint32_t w[kSlices + 1][4];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const double xv = tile[rr][9 * ch + j];
      int64_t F = e == kRowNonFinite ? 0 : slice_fixed(xv, e);  // (GIVEN: the caller rejects such rows)
      const float fx = (float)(int)(F >> 32);  // 2^28 x / 2^E
      sq = fmaf(fx, fx, sq);
      const uint32_t mag = slice_magnitude(xv, e);
      count += mag != 0u;
      if (j & 1) w[kSlices][j >> 1] |= mag << 16;
      else w[kSlices][j >> 1] = mag;
      if (op.negate) F = -F;
      const int64_t G = F + kDigitBias;
#pragma unroll
      for (int p = 0; p < kSlices; p++) {
        // digit 2^(-9 p) as a float (exact), of which BF16 keeps the upper half (exact)
        float f;
        if (p == 0)
          f = __int_as_float(0x4B400000 + (int)(G >> 54)) - 12582912.0f;
        else
          f = __int_as_float((0x4B000000 - (9 * p << 23)) | ((int)(G >> (9 * (6 - p))) & 511)) -
              __int_as_float((0x4B000000 - (9 * p << 23)) | 256);
        const uint32_t b = __float_as_uint(f) >> 16;
        if (j & 1) w[p][j >> 1] |= b << 16;
        else w[p][j >> 1] = b;
      }
    }
    uint16_t *d = op.dst + r * kPlanes * Kpad + k0 + ch * 8;
#pragma unroll
    for (int p = 0; p < kPlanes; p++)
      *reinterpret_cast<uint4 *>(d + p * Kpad) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
  }
  if (!op.stats) return;
#pragma unroll
  for (int off = KT / 16; off > 0; off >>= 1) {
    count += __shfl_xor_sync(0xffffffffu, count, off);
    sq += __shfl_xor_sync(0xffffffffu, sq, off);
  }
  if (ch == 0 && srow[rr] >= 0) {
    int *u = op.stats + srow[rr], *n = u + op.rows;
    const int squares = (int)ceilf(sq * 0x1p-56f / op.sq_unit);
    if (cs == 1) {
      *u = squares;
      *n = count;
    } else {
      atomicAdd(u, squares);
      atomicAdd(n, count);
    }
  }
}

// Tile width of a K: no wider than needed.
int pack_kt(int64_t K) { return K <= 16 ? 16 : K <= 32 ? 32 : 64; }

void launch_packs(const PackOp *op, int n, cudaStream_t stream) {  // (the operands have one K)
  PackOps p;
  p.op[0] = op[0];
  p.op[1] = op[n - 1];
  const int64_t blocks = op[0].blocks + (n > 1 ? op[1].blocks : 0);
  if (blocks > INT32_MAX) throw Error(SCESS_ERR_INVALID, "slice pack: too large");
  const int kt = pack_kt(op[0].K);
  if (kt == 16) launch(slice_pack_kernel<16>, (unsigned)blocks, 256, 0, stream, p);
  else if (kt == 32) launch(slice_pack_kernel<32>, (unsigned)blocks, 256, 0, stream, p);
  else launch(slice_pack_kernel<64>, (unsigned)blocks, 256, 0, stream, p);
  SCESS_CHECK_LAUNCH();
}

// The outputs that the slice GEMM has left (see SliceArgs::est), on the FP64 units.  Items are the
// 64 x 64 pieces of the GEMM's tiles, dealt out one by one; a thread looks at an item's tile, of
// 16 flags, and the CTA walks those that have any.  ks CTAs share an item's K where there are few,
// and the last one adds their ranges in order.  Returns at once where nothing was left (3 us).
struct LeftArgs {
  const uint32_t *left;
  const uint8_t *flags;
  int bn, pieces, tiles_n, ks;  // pieces of a tile: two by one or two
  int64_t items, kper;          // items: tiles, pieces, ks
  double *partial;              // ks > 1: [tile, piece][ks][64 x 64]
  int *counters;                // of a tile and piece; zero between launches
};
__global__ void __launch_bounds__(256) slice_left_kernel(TableGemm g, LeftArgs a) {
  chain();
  constexpr int T = kDgemmTile;
  constexpr int FEW = 128;  // outputs of a piece that are computed one by one, a warp each
  __shared__ DgemmShared sh;
  __shared__ int todo[256], ntodo, few[FEW], nfew, last;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  for (int64_t i0 = 0; i0 * gridDim.x + blockIdx.x < a.items; i0 += 256) {
    if (t == 0) ntodo = 0;
    __syncthreads();
    const int64_t mine = (i0 + t) * gridDim.x + blockIdx.x;
    if (mine < a.items) {
      const uint4 f = *reinterpret_cast<const uint4 *>(a.flags + 16 * (mine / a.ks / a.pieces));
      if (f.x | f.y | f.z | f.w) todo[atomicAdd(&ntodo, 1)] = t;
    }
    __syncthreads();
    for (int q = 0; q < ntodo; q++) {
      const int64_t item = (i0 + todo[q]) * gridDim.x + blockIdx.x, piece = item / a.ks;
      const int z = (int)(item % a.ks), tile = (int)(piece / a.pieces), sub = (int)(piece % a.pieces);
      const int64_t M0 = (int64_t)(tile / a.tiles_n) * BM, N0 = (int64_t)(tile % a.tiles_n) * a.bn;
      const int64_t m0 = M0 + (sub & 1) * T, n0 = N0 + (sub >> 1) * T;
      // outputs (m0 + tx + 16 i, n0 + ty + 16 j) at bit 4 i + j
      uint32_t b = 0;
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int row = (int)(m0 - M0) + tx + 16 * i, col = (int)(n0 - N0) + ty + 16 * j;
          if (M0 + row >= g.M || N0 + col >= g.N || col >= a.bn) continue;
          const int h = column_group(a.bn, col);
          if (a.flags[16 * tile + 4 * h + (row >> 5)] &&
              (a.left[(int64_t)(tile * EPI + h) * BM + row] >> (col - group_start(a.bn, h)) & 1u))
            b |= 1u << (4 * i + j);
        }
      if (t == 0) nfew = 0;
      if (!__syncthreads_or(b)) continue;
      auto finish = [&](int x, int y, double acc) {
        const int64_t off = g.baseC + g.rowC[m0 + x] + g.colC[n0 + y];
        double val = g.alpha * acc;
        if (g.beta != 0.0) val += g.beta * g.C[off];
        g.C[off] = val;
      };
      double *p = a.partial + piece * a.ks * (T * T);
      auto store = [&](int x, int y, double acc) {
        if (a.ks == 1) finish(x, y, acc);
        else p[z * (T * T) + x + T * y] = acc;
      };
      for (uint32_t r = b; r; r &= r - 1) {
        const int bit = __ffs((int)r) - 1, at = atomicAdd(&nfew, 1);
        if (at < FEW) few[at] = tx + 16 * (bit >> 2) + T * (ty + 16 * (bit & 3));
      }
      __syncthreads();
      const int64_t kb = z * a.kper, ke = min(g.K, kb + a.kper);
      if (nfew <= FEW) {
        for (int f = t >> 5; f < nfew; f += 8) {
          const int x = few[f] % T, y = few[f] / T;
          const double *A = g.A + g.baseA + g.rowA[m0 + x], *B = g.B + g.baseB + g.colB[n0 + y];
          double acc = 0.0;
#pragma unroll 4
          for (int64_t k = kb + (t & 31); k < ke; k += 32) acc = fma(A[g.kA[k]], B[g.kB[k]], acc);
          for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
          if ((t & 31) == 0) store(x, y, acc);
        }
      } else {
        dgemm_tile(sh, g, m0, n0, kb, ke, [&](int64_t m, int64_t n, double acc) {
          const int x = (int)(m - m0), y = (int)(n - n0);
          if (b >> (4 * (x >> 4) + (y >> 4)) & 1u) store(x, y, acc);
        });
      }
      __syncthreads();
      if (a.ks == 1) continue;
      __threadfence();
      __syncthreads();
      if (t == 0) last = atomicAdd(&a.counters[piece], 1) == a.ks - 1;
      __syncthreads();
      if (!last) continue;
      __threadfence();
      if (t == 0) a.counters[piece] = 0;
      for (uint32_t r = b; r; r &= r - 1) {
        const int bit = __ffs((int)r) - 1, x = tx + 16 * (bit >> 2), y = ty + 16 * (bit & 3);
        double s = 0.0;
        for (int w = 0; w < a.ks; w++) s += __ldcg(p + w * (T * T) + x + T * y);
        finish(x, y, s);
      }
    }
    __syncthreads();  // (the list is used up)
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaDriverEntryPointQueryResult q;
    void *p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  if (!fn) throw Error(SCESS_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
  return fn;
}

}  // namespace

// The kernel's setmaxnreg split assumes it is launched with exactly kLaunchRegs registers a
// thread; its shared memory is an attribute of each device's copy of it.
SliceEngine::SliceEngine(Ctx &ctx) : ctx_(ctx) {
  auto fits = [](void (*kernel)(SliceMaps, SliceArgs)) {
    cudaFuncAttributes fa;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES) == cudaSuccess &&
           cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && fa.numRegs == kLaunchRegs;
  };
  kernel_ok_ = fits(slice_gemm_kernel<false>) && fits(slice_gemm_kernel<true>);
  cudaGetLastError();
  err_.alloc(sizeof(unsigned) * 4);
  SCESS_CUDA(cudaMemsetAsync(err_.as<void>(), 0, sizeof(unsigned) * 4, ctx_.stream));
}

namespace {
// Unit of the rows' sums of squares: as fine as 31 bits allow (a CTA's part is rounded up).
float square_unit(int64_t K) {
  int e = -12;
  while (std::ldexp(1.0, 30 + e) < (double)K) e++;
  return std::ldexp(1.0f, e);
}
// The joint form's tiles are at most 64 wide.
bool joint(int bn) { return bn <= BN_JOINT; }
// Cycles an SM spends on one K block of a unit, measured (152 tiles of 128 rows, K = 1024:
// widths 16 .. 128; 4096^3 for the scale).
double block_cycles(int bn) { return joint(bn) ? 3050.0 + 22.0 * bn : 3450.0 + 20.0 * bn; }
}  // namespace

// The narrow tile where it is cheaper.
int SliceEngine::tile_n(int64_t N) {
  auto width = [&](int most, int unit) { return (int)round_up(ceil_div(N, ceil_div(N, most)), unit); };
  const int wide = width(BN, 16), narrow = width(BN_JOINT, 16);
  const double cw = block_cycles(wide) * (double)ceil_div(N, wide), cn = block_cycles(narrow) * (double)ceil_div(N, narrow);
  return cn < cw || joint(wide) ? narrow : wide;
}

namespace {
// Split-K of a product and its estimated time in us.  Rounds of units over the SMs times
// the K blocks of a unit; a unit's epilogue costs about 90 cycles a column, partial sums
// are written and read again at 5 TB/s, their reduction is one more launch (4 us).
// (9870 x 136 x 9870: 156 tiles take two rounds of 309 blocks; 19 splits take 20 of 17.)
// A unit's K is at most what its 64-bit sums hold.
double plan_us(int64_t M, int64_t N, int64_t Kpad, int64_t &splits) {
  const int bn = SliceEngine::tile_n(N);
  const int64_t nkb = ceil_div(Kpad, BK), tiles = ceil_div(M, BM) * ceil_div(N, bn);
  const double blk = block_cycles(bn) / 1900.0, epi = 90.0 * bn / 1900.0;
  const int64_t least = ceil_div(nkb, 512);
  const int64_t most = std::min<int64_t>(nkb / 2, std::max<int64_t>(64, ceil_div(2 * kNumSMs, tiles)));
  double best = 1e300;
  splits = least;
  for (int64_t z = least; z <= std::max(least, most); z++) {
    if (z > least && z * M * N > (int64_t(64) << 20)) break;
    double us = (double)ceil_div(tiles * z, kNumSMs) * ((double)ceil_div(nkb, z) * blk + epi);
    if (z > 1) us += 4.0 + (double)z * M * N * 16.0 / 5.0e6;
    if (us < 0.97 * best) {
      best = us;
      splits = z;
    }
  }
  return best;
}
}  // namespace

double SliceEngine::estimate_us(int64_t M, int64_t N, int64_t K, bool cUnitM, bool cUnitN) {
  int64_t z = 1;
  if (exchanges(M, N, cUnitM, cUnitN)) std::swap(M, N);
  // packs at 2.9 TB/s, 14 us of launches and latencies (6 x 5766 x 1116, either way round: 105
  // us measured, 94 by this; on the FP64 units 94 and 95)
  return 14.0 + (double)(M + N) * (double)K * 24.0 / 2.9e6 + plan_us(M, N, round_up(std::max<int64_t>(K, 1), BK), z);
}

bool SliceEngine::usable(int64_t M, int64_t N, int64_t K) const {
  return kernel_ok_ && M <= INT32_MAX / 2 && N <= INT32_MAX / 2 && K < (int64_t(1) << 26);
}

CUtensorMap SliceEngine::map_of(const SlicedPack &p, int box_rows) {
  CUtensorMap m;
  std::memset(&m, 0, sizeof(m));
  cuuint64_t dims[2] = {(cuuint64_t)(kPlanes * p.Kpad), (cuuint64_t)p.rows};
  cuuint64_t strides[1] = {(cuuint64_t)(kPlanes * p.Kpad * 2)};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.mem.as<void>(), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw Error(SCESS_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return m;
}

void SliceEngine::alloc(SlicedPack &out, int64_t rows, int64_t K) {
  const int64_t Kpad = round_up(std::max<int64_t>(K, 1), BK);
  const size_t bytes = (size_t)rows * kPlanes * Kpad * sizeof(uint16_t), eb = (size_t)rows * 3 * sizeof(int);
  if (out.mem.bytes() < bytes) out.mem.alloc(bytes);
  if (out.exps.bytes() < eb) out.exps.alloc(round_up((int64_t)eb, 4096));
  out.rows = rows;
  out.K = K;
  out.Kpad = Kpad;
}

void SliceEngine::row_exps(const double *src, const int64_t *rowOff, int64_t rows, const int64_t *kOff,
                           int64_t K, bool unitK, int *exps, const int64_t *expIdx) {
  PackOp op = {};
  op.src = src;
  op.row = rowOff;
  op.k = kOff;
  op.rows = rows;
  op.K = K;
  op.rt = RowTiles::make(rows, 1, rows, 2048 / pack_kt(K));
  op.mode = PACK_EXPS;
  op.unitK = unitK ? 1 : 0;
  op.exps = exps;
  op.expIdx = expIdx;
  op.blocks = op.rt.count * std::max<int64_t>(1, std::min(ceil_div(K, 64), ceil_div(8 * kNumSMs, op.rt.count)));
  launch_packs(&op, 1, ctx_.stream);
}

void SliceEngine::pack_with_exps(const double *src, const int64_t *rowOff, int64_t rows, const int64_t *kOff,
                                 int64_t K, bool unitK, const int *exps, const int64_t *expIdx, bool negate,
                                 SlicedPack &out) {
  alloc(out, rows, K);
  TimedScope ts(ctx_.timer, "slice_pack", 0.0, (double)rows * K * 8 + (double)rows * out.Kpad * 16, ctx_.stream);
  PackOp op = {};
  op.src = src;
  op.row = rowOff;
  op.k = kOff;
  op.rows = rows;
  op.K = K;
  op.Kpad = out.Kpad;
  op.rt = RowTiles::make(rows, 1, rows, 2048 / pack_kt(K));
  op.mode = PACK_GIVEN;
  op.unitK = unitK ? 1 : 0;
  op.negate = negate ? 1 : 0;
  op.dst = out.mem.as<uint16_t>();
  op.exps = const_cast<int *>(exps);
  op.expIdx = expIdx;
  op.blocks = op.rt.count * std::max<int64_t>(1, std::min(ceil_div(out.Kpad, 64), ceil_div(16 * kNumSMs, op.rt.count)));
  launch_packs(&op, 1, ctx_.stream);
}

void SliceEngine::pack(const Gather *g, SlicedPack *const *out, int n) {
  PackOp first[2], second[2];
  int ns = 0;
  double bytes = 0.0;
  for (int i = 0; i < n; i++) {
    SlicedPack &o = *out[i];
    alloc(o, g[i].rows, g[i].K);
    PackOp &op = first[i];
    op = PackOp{};
    const bool aff = g[i].rs >= 0 && g[i].ks >= 0;
    op.src = g[i].src;
    op.row = aff ? nullptr : g[i].row;
    op.k = aff ? nullptr : g[i].k;
    op.rs = g[i].rs;
    op.ks = g[i].ks;
    op.rows = g[i].rows;
    op.K = g[i].K;
    op.Kpad = o.Kpad;
    op.rt = RowTiles::make(g[i].rows, g[i].P, g[i].E > 0 ? g[i].E : g[i].rows, 2048 / pack_kt(g[i].K));
    op.unitK = g[i].unitK ? 1 : 0;
    op.dst = o.mem.as<uint16_t>();
    op.exps = o.exps.as<int>();
    op.stats = op.exps + g[i].rows;
    op.sq_unit = square_unit(g[i].K);
    bytes += (double)g[i].rows * g[i].K * 8 + (double)g[i].rows * o.Kpad * 16;
    const int64_t chunks = ceil_div(o.Kpad, 64);
    // one walk per CTA over its rows' whole K while that fills the device or K is
    // short; else the exponents first, then the cut, each spread over K too
    if (op.rt.count >= 2 * kNumSMs || chunks <= 4) {
      op.mode = PACK_OWN;
      op.blocks = op.rt.count;
      continue;
    }
    op.mode = PACK_PART;
    op.parts = (int)std::min<int64_t>({ceil_div(g[i].K, 64), ceil_div(8 * kNumSMs, op.rt.count), 64});
    op.blocks = op.rt.count * op.parts;
    const size_t need = (size_t)op.parts * g[i].rows * sizeof(int);
    if (o.part.bytes() < need) o.part.alloc(round_up((int64_t)need, 4096));
    op.part = o.part.as<int>();
    PackOp &cut = second[ns++];
    cut = op;
    cut.mode = PACK_FROM_PART;
    cut.blocks = op.rt.count * std::min(chunks, ceil_div(16 * kNumSMs, op.rt.count));
  }
  TimedScope ts(ctx_.timer, "slice_pack", 0.0, bytes, ctx_.stream);
  launch_packs(first, n, ctx_.stream);
  if (ns) launch_packs(second, ns, ctx_.stream);
}

void SliceEngine::launch(const SliceProblemSet &ps, int splits, double *partial) {
  if (!kernel_ok_) throw Error(SCESS_ERR_UNSUPPORTED, "slice gemm: kernel unavailable");
  if (ps.M <= 0 || ps.N <= 0 || ps.ny <= 0 || ps.nz <= 0 || ps.ng <= 0) return;
  if (ps.ng > 3 || ps.nseg < 1 || ps.nseg > 4) throw Error(SCESS_ERR_INVALID, "slice gemm: groups or segments");
  SliceArgs a;
  std::memset(&a, 0, sizeof(a));
  a.M = (int)ps.M;
  a.N = (int)ps.N;
  a.tiles_m = (int)ceil_div(ps.M, BM);
  // column tiles of equal width (the B-side maps have boxes of this many rows)
  a.bn = tile_n(ps.N);
  a.stages = std::min<int>(MAX_STAGES, (int)(STAGES * STAGE_BYTES / (kSlices * (A_SLICE + (uint32_t)a.bn * BK * 2))));
  a.tiles_n = (int)ceil_div(ps.N, a.bn);
  a.ny = ps.ny;
  a.nz = ps.nz;
  a.ng = ps.ng;
  a.nseg = ps.nseg;
  for (int s = 0; s < ps.nseg; s++) {
    const SliceSegment &g = ps.seg[s];
    if (g.Kpad % BK != 0 || g.Kpad <= 0 || kPlanes * g.Kpad > INT32_MAX)
      throw Error(SCESS_ERR_INVALID, "slice gemm: segment K");
    for (int q = 0; q < ps.ng; q++) {
      const int64_t maxA = g.rowA0[q] + (int64_t)(ps.ny - 1) * g.rowAy[q] + (int64_t)(ps.nz - 1) * g.rowAz[q] + a.tiles_m * BM;
      const int64_t maxB = g.rowB0[q] + (int64_t)(ps.ny - 1) * g.rowBy[q] + (int64_t)(ps.nz - 1) * g.rowBz[q] + a.tiles_n * a.bn;
      if (maxA > INT32_MAX || maxB > INT32_MAX || g.rowA0[q] < 0 || g.rowB0[q] < 0 || g.rowAy[q] < 0 ||
          g.rowAz[q] < 0 || g.rowBy[q] < 0 || g.rowBz[q] < 0)
        throw Error(SCESS_ERR_INVALID, "slice gemm: row coordinates");
    }
    SegArgs &d = a.seg[s];
    d.mapA = g.mapA;
    d.mapB = g.mapB;
    d.nkb = (int)(g.Kpad / BK);
    d.kpad = (int)g.Kpad;
    for (int q = 0; q < 3; q++) {
      d.rowA0[q] = g.rowA0[q];
      d.rowAy[q] = g.rowAy[q];
      d.rowAz[q] = g.rowAz[q];
      d.rowB0[q] = g.rowB0[q];
      d.rowBy[q] = g.rowBy[q];
      d.rowBz[q] = g.rowBz[q];
    }
    a.kb_total += d.nkb;
  }
  splits = std::max(1, std::min(splits, a.kb_total));
  a.kb_per_split = (int)ceil_div(a.kb_total, splits);
  a.splits = (int)ceil_div(a.kb_total, a.kb_per_split);
  // the 64-bit sum holds 2^12 k 2^36 per output: K <= 2^14 a unit
  // and the tails, together below 2^10 K in units of the integer, in 31 bits
  a.fs = 20;
  for (int64_t k = (int64_t)a.kb_per_split * BK; k > 1; k >>= 1) a.fs--;
  if (a.kb_per_split > 512) throw Error(SCESS_ERR_INVALID, "slice gemm: K of a unit");
  int64_t start = 0;
  for (int g = 0; g < ps.ng; g++) {
    if (ps.tri[g] && ps.ny != ps.nz) throw Error(SCESS_ERR_INVALID, "slice gemm: triangular groups need ny == nz");
    a.tri[g] = ps.tri[g] ? 1 : 0;
    a.gstart[g] = (int)start;
    start += a.tri[g] ? (int64_t)ps.ny * (ps.ny + 1) / 2 : (int64_t)ps.ny * ps.nz;
    a.expA0[g] = ps.expA0[g];
    a.cy[g] = ps.cy[g];
    a.cz[g] = ps.cz[g];
    a.cg[g] = ps.cg[g];
    a.rowC[g] = ps.rowC[g];
    a.colC[g] = ps.colC[g];
  }
  if (start > INT32_MAX) throw Error(SCESS_ERR_INVALID, "slice gemm: too many problems");
  a.gstart[ps.ng] = (int)start;
  a.expA = ps.expA;
  a.expB = ps.expB;
  a.est = ps.est;
  a.sq_unit = ps.sq_unit;
  a.rowsA = (int)ps.M;
  a.rowsB = (int)ps.N;
  a.left = ps.left;
  a.flags = ps.flags;
  a.C = ps.C;
  a.baseC = ps.baseC;
  a.alpha = ps.alpha;
  a.beta = ps.beta;
  int e = 0;
  const double f = std::frexp(ps.alpha, &e);
  a.alpha_pow2 = std::fabs(f) == 0.5 && e > -500 && e < 500;
  a.alpha_e = e - 1;
  a.alpha_neg = f < 0;
  a.partial = a.splits > 1 ? partial : nullptr;
  a.part_stride = ps.M * ps.N;
  a.est_partial = reinterpret_cast<float *>(partial + a.splits * a.part_stride);
  if (a.est && (start > 1 || ps.nseg > 1)) throw Error(SCESS_ERR_INVALID, "slice gemm: estimates of one problem");
  if (a.splits > 1 && (!partial || !a.est || start > 1)) throw Error(SCESS_ERR_INVALID, "slice gemm: split-K");
  a.err = err_.as<unsigned>();
  const WaitDiag diag = ctx_.take_wait_diag();
  a.wait_cycles = diag.wait_cycles;
  a.withhold_first = diag.withhold_first ? 1 : 0;
  SliceMaps maps;
  for (int i = 0; i < 6; i++) maps.m[i] = ps.maps[std::min(i, ps.nmaps - 1)];
  const int64_t units = (int64_t)a.tiles_m * a.tiles_n * start * a.splits;
  if (units > INT32_MAX) throw Error(SCESS_ERR_INVALID, "slice gemm: too many work units");
  launched_ = true;
  scess::launch(joint(a.bn) ? slice_gemm_kernel<true> : slice_gemm_kernel<false>, (unsigned)std::min<int64_t>(units, kNumSMs), THREADS, SMEM_BYTES, ctx_.stream, maps, a);
  SCESS_CHECK_LAUNCH();
  if (a.splits > 1) {
    const bool groups = split_groups(ps.M * ps.N, a.splits);
    const auto reduce = groups ? slice_reduce_kernel<kSplitGroups> : slice_reduce_kernel<1>;
    scess::launch(reduce, split_blocks(ps.M * ps.N, groups), 256, 0, ctx_.stream, a, a.splits);
    SCESS_CHECK_LAUNCH();
  }
}

void SliceEngine::gemm_grouped(const SliceProblemSet &ps, double flops, const char *name) {
  TimedScope ts(ctx_.timer, name, flops, 0.0, ctx_.stream);
  launch(ps, 1, nullptr);
}

void SliceEngine::product(const TableGemm &g, const SlicedPack &A, const SlicedPack &B, const char *name) {
  SliceProblemSet ps;
  ps.M = g.M;
  ps.N = g.N;
  int64_t splits = 1;
  plan_us(ps.M, ps.N, A.Kpad, splits);
  LeftArgs la = {};
  la.bn = tile_n(g.N);
  la.pieces = la.bn > kDgemmTile ? 4 : 2;
  la.tiles_n = (int)ceil_div(g.N, la.bn);
  la.counters = ctx_.counters.as<int>();
  const int64_t tiles = ceil_div(g.M, BM) * la.tiles_n, pieces = tiles * la.pieces;
  static_assert(2 * kNumSMs <= kSmallCounters, "a counter a piece");
  // few pieces: their K over several CTAs (one takes a millisecond per thousand k)
  const int64_t ks = pieces >= 2 * kNumSMs ? 1 : std::min(4 * kNumSMs / pieces, ceil_div(g.K, 64));
  la.kper = ks == 1 ? g.K : round_up(ceil_div(g.K, ks), 16);
  la.ks = (int)ceil_div(g.K, la.kper);
  la.items = pieces * la.ks;
  // (everything is allocated before anything is launched: the caller falls back to the FP64
  // units when it does not fit)
  auto room = [](DevMem &m, size_t bytes) {
    if (m.bytes() < bytes) m.alloc(bytes);
  };
  const size_t mn = (size_t)g.M * g.N, words = (size_t)tiles * EPI * BM;
  room(left_, words * sizeof(uint32_t) + 16 * tiles);
  room(partial_, std::max(splits > 1 ? splits * mn * (sizeof(double) + sizeof(float)) : 0,
                          la.ks > 1 ? (size_t)la.items * kDgemmTile * kDgemmTile * sizeof(double) : 0));
  ps.est = 1;
  ps.sq_unit = square_unit(g.K);
  ps.left = left_.as<uint32_t>();
  ps.flags = reinterpret_cast<uint8_t *>(ps.left + words);
  la.left = ps.left;
  la.flags = ps.flags;
  la.partial = partial_.d();
  TimedScope ts(ctx_.timer, name, 2.0 * g.M * g.N * g.K, 0.0, ctx_.stream);
  ps.maps[0] = map_of(A, BM);
  ps.maps[1] = map_of(B, tile_n(ps.N));
  ps.nmaps = 2;
  ps.seg[0].Kpad = A.Kpad;
  ps.expA = A.e();
  ps.expB = B.e();
  ps.C = g.C;
  ps.baseC = g.baseC;
  ps.rowC[0] = g.rowC;
  ps.colC[0] = g.colC;
  ps.alpha = g.alpha;
  ps.beta = g.beta;
  launch(ps, (int)splits, partial_.d());
  scess::launch(slice_left_kernel, (unsigned)std::min<int64_t>(la.items, 4 * kNumSMs), 256, 0, ctx_.stream, g, la);
  SCESS_CHECK_LAUNCH();
}

void SliceEngine::release_workspaces() {
  tmpA_ = SlicedPack();
  tmpB_ = SlicedPack();
  partial_.release();
  left_.release();
}

void SliceEngine::reclaim() {
  if (busy_) return;
  release_workspaces();
  spare_.clear();
  cache_.clear();
}

namespace {
struct Busy {
  bool &b;
  explicit Busy(bool &x) : b(x) { b = true; }
  ~Busy() { b = false; }
};
// The same product with its sides exchanged: C^T = B^T A^T.
TableGemm exchanged(const TableGemm &g) {
  TableGemm h = g;
  h.A = g.B;
  h.B = g.A;
  h.rowA = g.colB;
  h.kA = g.kB;
  h.colB = g.rowA;
  h.kB = g.kA;
  h.rowC = g.colC;
  h.colC = g.rowC;
  h.baseA = g.baseB;
  h.baseB = g.baseA;
  h.M = g.N;
  h.N = g.M;
  h.aUnitM = g.bUnitN;
  h.bUnitN = g.aUnitM;
  return h;
}
}  // namespace

bool SliceEngine::table_gemm(const TableGemm &g, const char *name) {
  Busy busy(busy_);
  try {
    const Gather ga[2] = {{g.A + g.baseA, g.rowA, g.M, g.kA, g.K, !g.aUnitM},
                          {g.B + g.baseB, g.colB, g.N, g.kB, g.K, !g.bUnitN}};
    SlicedPack *const out[2] = {&tmpA_, &tmpB_};
    pack(ga, out, 2);
    if (exchanges(g.M, g.N, false, false)) product(exchanged(g), tmpB_, tmpA_, name);
    else product(g, tmpA_, tmpB_, name);
  } catch (const Error &e) {
    if (e.code != SCESS_ERR_OOM) throw;
    return false;
  }
  return true;
}

void SliceEngine::clear_cache(const void *owner) {
  for (auto it = cache_.begin(); it != cache_.end();) {
    if (it->first.owner == owner) it = cache_.erase(it);
    else ++it;
  }
  if (owner) return;
  // the end of an API call: what is kept beyond it is bounded here, the rest by the block cache
  spare_.clear();
  if (workspace_bytes() > kKeptBytes) release_workspaces();
}

void SliceEngine::clear_stable() {
  // the packs' memory serves the next residual's (at most kSpare of them)
  for (auto &kv : reuse_)
    if ((int)spare_.size() < kSpare) spare_.push_back(std::move(kv.second));
  reuse_.clear();
  stable_.clear();
}

void SliceEngine::clear_error() {
  launched_ = false;
  cudaMemsetAsync(err_.as<void>(), 0, sizeof(unsigned), ctx_.stream);
}

void SliceEngine::check_error() {
  if (!launched_) return;
  launched_ = false;
  unsigned h = 0;
  SCESS_CUDA(cudaMemcpyAsync(&h, err_.as<void>(), sizeof(unsigned), cudaMemcpyDeviceToHost, ctx_.stream));
  ctx_.sync();
  if (h != 0) {
    SCESS_CUDA(cudaMemsetAsync(err_.as<void>(), 0, sizeof(unsigned), ctx_.stream));
    throw Error(SCESS_ERR_CUDA, "tensor-core pipeline wait expired (code " + std::to_string(h) + ")");
  }
}

bool SliceEngine::contract(const EinsumPlan &pl, double alpha, const double *A, const double *B, double beta,
                           double *C, bool constA, bool constB) {
  Busy busy(busy_);
  const bool swap = exchanges(pl.M, pl.N, pl.cUnitM, pl.cUnitN);
  const Gather gA{A, pl.d_rowA, pl.M, pl.d_kA, pl.K, pl.aUnitK, pl.aRowStride, pl.aKStride, pl.aRowP, pl.aRowE};
  const Gather gB{B, pl.d_colB, pl.N, pl.d_kB, pl.K, pl.bUnitK, pl.bColStride, pl.bKStride, pl.bColP, pl.bColE};
  Gather todo[2];
  SlicedPack *out[2];
  int n = 0;
  // the operand's pack: kept (constant operands, stable tensors) or still to be made
  auto get = [&](const Gather &g, bool isA, bool isConst, SlicedPack &tmp) -> SlicedPack * {
    SlicedPack *p = &tmp;
    if (isConst || stable_.count(g.src)) {
      uint64_t &hs = isA ? pl.hashA : pl.hashB;
      if (!hs) hs = isA ? table_hash(pl.rowA, pl.kA) : table_hash(pl.colB, pl.kB);
      const Key key{g.src, hs, g.rows, g.K, isConst ? owner_ : nullptr};
      auto &kept = isConst ? cache_ : reuse_;
      auto it = kept.find(key);
      if (it != kept.end()) return it->second.get();
      std::unique_ptr<SlicedPack> np;
      if (!isConst && !spare_.empty()) {
        np = std::move(spare_.back());
        spare_.pop_back();
      } else {
        np = std::make_unique<SlicedPack>();
      }
      p = np.get();
      alloc(*p, g.rows, g.K);  // (before it is listed: an allocation may fail)
      kept[key] = std::move(np);
    }
    todo[n] = g;
    out[n++] = p;
    return p;
  };
  TableGemm g;
  g.A = A;
  g.B = B;
  g.C = C;
  g.rowA = pl.d_rowA;
  g.kA = pl.d_kA;
  g.colB = pl.d_colB;
  g.kB = pl.d_kB;
  g.rowC = pl.d_rowC;
  g.colC = pl.d_colC;
  g.M = pl.M;
  g.N = pl.N;
  g.K = pl.K;
  g.alpha = alpha;
  g.beta = beta;
  g.aUnitM = pl.aUnitM;
  g.bUnitN = pl.bUnitN;
  const std::string tname = "slice_gemm[" + pl.spec + "]";
  try {
    const SlicedPack *pa = get(gA, true, constA, tmpA_), *pb = get(gB, false, constB, tmpB_);
    if (n) pack(todo, out, n);
    if (swap) product(exchanged(g), *pb, *pa, tname.c_str());
    else product(g, *pa, *pb, tname.c_str());
  } catch (const std::exception &x) {
    // packs listed above may not have been made
    reuse_.clear();
    spare_.clear();
    cache_.clear();
    const Error *e = dynamic_cast<const Error *>(&x);
    if (!e || e->code != SCESS_ERR_OOM) throw;
    return false;  // no room for the packs: the DFMA kernel needs none
  }
  return true;
}

}  // namespace scess
