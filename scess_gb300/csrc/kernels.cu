// FP64 contraction engine and bandwidth-bound kernels of the closed-shell CC path.
//
// GB300 runs FP64 at a small fraction of its tensor rate, so the FP64 GEMM is
// DFMA-bound at any reasonable tile size: one 64x64 tile per 256-thread CTA with
// 4x4 register blocking, operands gathered through offset tables (the einsum
// permutation is fused into the tile loads), deterministic split-K when the
// output has too few tiles to cover the 152 SMs.
#include "common.cuh"
#include "dgemm_tile.cuh"
#include "kernels.h"
#include "launch.cuh"

namespace scess {

namespace {

constexpr int BM = kDgemmTile, BN = kDgemmTile, BK = kDgemmBK;

__global__ void __launch_bounds__(256) dgemm_table_kernel(TableGemm g, int64_t kChunk,
                                                          double *partial) {
  chain();
  __shared__ DgemmShared sh;
  const int64_t kb = (int64_t)blockIdx.z * kChunk;
  dgemm_tile(sh, g, (int64_t)blockIdx.x * BM, (int64_t)blockIdx.y * BN, kb, min(g.K, kb + kChunk),
             [&](int64_t m, int64_t n, double acc) {
               if (partial) {
                 partial[(int64_t)blockIdx.z * g.M * g.N + m + g.M * n] = acc;
               } else {
                 const int64_t off = g.baseC + g.rowC[m] + g.colC[n];
                 double val = g.alpha * acc;
                 if (g.beta != 0.0) val += g.beta * g.C[off];
                 g.C[off] = val;
               }
             });
}

__global__ void splitk_reduce_kernel(TableGemm g, int splits, const double *partial) {
  chain();
  const int64_t MN = g.M * g.N;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < MN;
       e += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int z = 0; z < splits; z++) s += partial[(int64_t)z * MN + e];
    const int64_t m = e % g.M, n = e / g.M;
    const int64_t off = g.baseC + g.rowC[m] + g.colC[n];
    double val = g.alpha * s;
    if (g.beta != 0.0) val += g.beta * g.C[off];
    g.C[off] = val;
  }
}

int choose_splits(const TableGemm &g) {
  const int64_t tiles = ceil_div(g.M, BM) * ceil_div(g.N, BN);
  const int64_t target = 2 * kNumSMs;
  if (tiles >= target || g.K <= 4 * BK) return 1;
  int64_t s = ceil_div(target, tiles);
  s = std::min<int64_t>(s, ceil_div(g.K, 4 * BK));
  // keep the partial buffer below 64 Mi doubles
  while (s > 1 && s * g.M * g.N > (int64_t(64) << 20)) s--;
  return (int)std::max<int64_t>(s, 1);
}

}  // namespace

namespace {

// Small FP64 contraction: GB300 issues about two FP64 lanes per cycle and SM, so one
// 64 x 64 x 16 step of dgemm_table_kernel takes an SM 18 us.  Small products are
// therefore cut finely over the whole device: up to 64 outputs a CTA (tm x tn, chosen
// for the least padding), K in ranges of at most kSmallKB staged at once (two dependent
// loads, then arithmetic), the four 64-thread groups taking every fourth k.  With
// several K ranges per tile the last CTA of the tile to finish adds the partial sums in
// order (deterministic) and leaves the tile's counter at zero.  90 x 10 x 90:
// 107 -> 4 us; 10 x 10 x 81000: 134 us on the tensor cores' slices (packs included), 47 here.
constexpr int kSmallOut = 64, kSmallKB = 128, kSmallSide = 16;
__global__ void __launch_bounds__(256) dgemm_small_kernel(TableGemm g, int64_t kper, int splits, int tm, int tn,
                                                          double *__restrict__ partial,
                                                          int *__restrict__ counters) {
  chain();
  __shared__ double As[kSmallKB][kSmallSide + 1], Bs[kSmallKB][kSmallSide + 1];
  __shared__ double red[4][kSmallOut];
  __shared__ int last;
  const int t = threadIdx.x, grp = t >> 6, o = t & 63, i = o % tm, j = o / tm;
  const int im = 65536 / tm + 1, in = 65536 / tn + 1;  // (exact for e below 4096)
  // a staged range: K or kSmallKB, rounded up to a power of two
  const int ks = 32 - __clz((int)min((int64_t)kSmallKB, min(kper, g.K)) - 1), km = (1 << ks) - 1;
  const int64_t ntm = (g.M + tm - 1) / tm;
  const int64_t tile = blockIdx.x / splits, z = blockIdx.x % splits;
  const int64_t m0 = (tile % ntm) * tm, n0 = (tile / ntm) * tn;
  const int64_t kb = z * kper, ke = min(g.K, kb + kper);
  const bool out = j < tn && m0 + i < g.M && n0 + j < g.N;
  double acc = 0.0;
  for (int64_t k0 = kb; k0 < ke; k0 += kSmallKB) {
    const int nk = (int)min((int64_t)kSmallKB, ke - k0);
    __syncthreads();  // the previous range is used up
    // element e of a side: along its unit-stride index, else along k
    for (int e0 = t; e0 < max(tm, tn) << ks; e0 += 4 * 256) {
      int64_t ra[4], rb[4];
      double a[4], b[4];
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const int e = e0 + 256 * p;
        const int qm = (e * im) >> 16, qn = (e * in) >> 16;  // e / tm, e / tn
        const int am = g.aUnitM ? e - qm * tm : e >> ks, ak = g.aUnitM ? qm : e & km;
        const int bm = g.bUnitN ? e - qn * tn : e >> ks, bk = g.bUnitN ? qn : e & km;
        ra[p] = (am < tm && m0 + am < g.M && ak < nk) ? g.rowA[m0 + am] + g.kA[k0 + ak] : -1;
        rb[p] = (bm < tn && n0 + bm < g.N && bk < nk) ? g.colB[n0 + bm] + g.kB[k0 + bk] : -1;
      }
#pragma unroll
      for (int p = 0; p < 4; p++) {
        a[p] = ra[p] >= 0 ? g.A[g.baseA + ra[p]] : 0.0;
        b[p] = rb[p] >= 0 ? g.B[g.baseB + rb[p]] : 0.0;
      }
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const int e = e0 + 256 * p;
        const int qm = (e * im) >> 16, qn = (e * in) >> 16;  // e / tm, e / tn
        const int am = g.aUnitM ? e - qm * tm : e >> ks, ak = g.aUnitM ? qm : e & km;
        const int bm = g.bUnitN ? e - qn * tn : e >> ks, bk = g.bUnitN ? qn : e & km;
        if (am < tm && ak < nk) As[ak][am] = a[p];
        if (bm < tn && bk < nk) Bs[bk][bm] = b[p];
      }
    }
    __syncthreads();
    if (out)
      for (int k = grp; k < nk; k += 4) acc = fma(As[k][i], Bs[k][j], acc);
  }
  red[grp][o] = acc;
  __syncthreads();
  double s = 0.0;
  if (t < kSmallOut) s = (red[0][t] + red[1][t]) + (red[2][t] + red[3][t]);
  if (splits > 1) {
    double *p = partial + tile * splits * kSmallOut;
    if (t < kSmallOut) p[z * kSmallOut + t] = s;
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(&counters[tile], 1) == splits - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    double v = 0.0;
    for (int q = grp; q < splits; q += 4) v += __ldcg(p + q * kSmallOut + o);
    red[grp][o] = v;
    __syncthreads();
    if (t < kSmallOut) s = (red[0][t] + red[1][t]) + (red[2][t] + red[3][t]);
    if (t == 0) counters[tile] = 0;
  }
  if (t < kSmallOut && out) {
    const int64_t off = g.baseC + g.rowC[m0 + i] + g.colC[n0 + j];
    double val = g.alpha * s;
    if (g.beta != 0.0) val += g.beta * g.C[off];
    g.C[off] = val;
  }
}

struct SmallShape {
  int tm = 8, tn = 8, splits = 1;
  int64_t tiles = 0, kper = 0;
};
SmallShape small_shape(const TableGemm &g) {
  SmallShape s;
  // the tile with the fewest padded outputs (whole warps of 32), then the fewest tiles
  int64_t best = INT64_MAX;
  for (int tm = 4; tm <= kSmallSide; tm++) {
    const int tn = std::min(kSmallOut / tm, kSmallSide);
    const int64_t tiles = ceil_div(g.M, tm) * ceil_div(g.N, tn);
    const int64_t cost = tiles * round_up(tm * tn, 32) * 1024 + std::min<int64_t>(tiles, 1023);
    if (cost < best) {
      best = cost;
      s.tm = tm;
      s.tn = tn;
      s.tiles = tiles;
    }
  }
  // about two CTAs an SM, at least 16 k each; a range beyond 128 k is walked in steps
  const int64_t want = s.tiles >= 2 * kNumSMs ? 1 : ceil_div(2 * kNumSMs, s.tiles);
  const int64_t n = std::max<int64_t>(1, std::min(want, ceil_div(g.K, 16)));
  s.kper = round_up(ceil_div(g.K, n), 4);
  s.splits = (int)ceil_div(g.K, s.kper);
  return s;
}

// One row of a matrix-vector product per warp, or, with few rows, per CTA (its
// eight warps then share the K range): four independent partial sums a lane, so
// that four loads are in flight, added in a fixed order.
template <bool CTA>
__global__ void __launch_bounds__(256) dgemv_table_kernel(TableGemm g) {
  chain();
  __shared__ double red[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t step = CTA ? 256 : 32, k0 = CTA ? threadIdx.x : lane;
  const int64_t m1 = CTA ? gridDim.x : ((int64_t)gridDim.x * blockDim.x) >> 5;
  const double *__restrict__ B = g.B + g.baseB + g.colB[0];
  for (int64_t m = CTA ? blockIdx.x : ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; m < g.M; m += m1) {
    const double *__restrict__ A = g.A + g.baseA + g.rowA[m];
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int64_t k = k0;
    for (; k + 3 * step < g.K; k += 4 * step) {
      const int64_t ka0 = g.kA[k], ka1 = g.kA[k + step], ka2 = g.kA[k + 2 * step], ka3 = g.kA[k + 3 * step];
      const int64_t kb0 = g.kB[k], kb1 = g.kB[k + step], kb2 = g.kB[k + 2 * step], kb3 = g.kB[k + 3 * step];
      const double a0 = A[ka0], a1 = A[ka1], a2 = A[ka2], a3 = A[ka3];
      const double b0 = B[kb0], b1 = B[kb1], b2 = B[kb2], b3 = B[kb3];
      s0 = fma(a0, b0, s0);
      s1 = fma(a1, b1, s1);
      s2 = fma(a2, b2, s2);
      s3 = fma(a3, b3, s3);
    }
    for (; k < g.K; k += step) s0 = fma(A[g.kA[k]], B[g.kB[k]], s0);
    double s = (s0 + s1) + (s2 + s3);
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (CTA) {
      __syncthreads();
      if (lane == 0) red[w] = s;
      __syncthreads();
      if (threadIdx.x == 0)
        s = ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
    }
    if (CTA ? threadIdx.x == 0 : lane == 0) {
      const int64_t off = g.baseC + g.rowC[m] + g.colC[0];
      double val = g.alpha * s;
      if (g.beta != 0.0) val += g.beta * g.C[off];
      g.C[off] = val;
    }
  }
}
}  // namespace

double dgemm_small_us(const TableGemm &g) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return 1e30;
  const SmallShape s = small_shape(g);
  if ((double)s.tiles * s.splits > 2.0e9) return 1e30;
  // Measured: 6 us, and the larger of padded multiply-adds at two lanes a cycle and SM
  // (80 % reached) and 88 ns for a thousand outputs (staging, tables, C).
  const double fma = 1.25 * (double)s.tiles * (double)round_up(s.tm * s.tn, 32) * (double)g.K / (2.0 * kNumSMs * 1900.0);
  return 6.0 + std::hypot(fma, 8.8e-5 * (double)g.M * (double)g.N);
}

int64_t dgemm_small_workspace(const TableGemm &g) {
  const SmallShape s = small_shape(g);
  return s.splits > 1 ? s.tiles * s.splits * kSmallOut : 0;
}

void dgemm_small(const TableGemm &g, double *workspace, int *counters, cudaStream_t stream) {
  const SmallShape s = small_shape(g);
  launch(dgemm_small_kernel, (unsigned)(s.tiles * s.splits), 256, 0, stream, g, s.kper, s.splits, s.tm, s.tn,
         workspace, counters);
  SCESS_CHECK_LAUNCH();
}

namespace {
// Tables of a skinny contraction seen from its small side (Sm, s indices) and
// its long side (Lg, l indices); C(m, n) at C[cS[m] + cL[n]].
struct SkinnyArgs {
  const double *Sm, *Lg;
  double *C;
  const int64_t *sR, *sK, *lR, *lK, *cS, *cL;
  int s, sp, K;        // sp: s rounded up to 4
  int chunk, nchunks;  // small indices of a warp's item (a multiple of 32, or all)
  int64_t l;
  double alpha;
  double beta;
};

template <typename T>
__device__ __forceinline__ void skinny_out(double *p, T v, double beta) {
  if (beta == 1.0) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"((double)v) : "memory");
  } else if (beta == 0.0) {
    *p = (double)v;
  } else {
    *p = fma(beta, *p, (double)v);
  }
}

// Persistent: each block stages the small operand once ([k][m], T = FP32 of the mixed form
// or FP64) and its warps walk items of 32 long indices, one per lane, and a chunk of the
// small ones, with the lane's K long values in registers; every shared load of four
// small-side values (16-byte broadcasts) feeds four multiply-adds.  Neighbouring items go
// to different SMs: with few of them (9000 x 10 x 90: 282 tiles of 32) eight to a block would
// leave most SMs idle.  FP64 is bound by its units: 10 x 81000 x 10 takes 42 us
// (dgemm_small 130; sliced 29 and 27 for the packs).
template <typename T, bool STAGE>
__global__ void __launch_bounds__(256) skinny_kernel(SkinnyArgs a) {
  chain();
  extern __shared__ __align__(16) unsigned char sk_raw[];
  T *sS = reinterpret_cast<T *>(sk_raw);                             // [K][sp]
  int64_t *cSs = reinterpret_cast<int64_t *>(sS + a.K * a.sp);       // [s]
  int64_t *lKs = cSs + a.sp;                                         // [K]
  T *stage = reinterpret_cast<T *>(lKs + kSkinnyMaxK);               // [8][32][33] (STAGE)
  for (int e = threadIdx.x; e < a.K * a.sp; e += blockDim.x) {
    const int m = e % a.sp, k = e / a.sp;
    sS[e] = m < a.s ? (T)a.Sm[a.sR[m] + a.sK[k]] : T(0);
  }
  for (int m = threadIdx.x; m < a.s; m += blockDim.x) cSs[m] = a.cS[m];
  for (int k = threadIdx.x; k < a.K; k += blockDim.x) lKs[k] = a.lK[k];
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const T alpha = (T)a.alpha;
  const int64_t items = (a.l + 31) / 32 * a.nchunks;
  for (int64_t it = (int64_t)w * gridDim.x + blockIdx.x; it < items; it += (int64_t)gridDim.x * 8) {
    const int64_t t = it / a.nchunks;
    const int ms = (int)(it - t * a.nchunks) * a.chunk, me = min(a.s, ms + a.chunk);
    const int64_t n = t * 32 + lane;
    const bool ok = n < a.l;
    const int64_t lr = ok ? a.lR[n] : 0, cl = ok ? a.cL[n] : 0;
    T lv[kSkinnyMaxK];
#pragma unroll
    for (int k = 0; k < kSkinnyMaxK; k++) lv[k] = (ok && k < a.K) ? (T)a.Lg[lr + lKs[k]] : T(0);
    // four results C(m .. m + 3, n)
    auto quad = [&](int m, T *c) {
      c[0] = c[1] = c[2] = c[3] = T(0);
#pragma unroll
      for (int k = 0; k < kSkinnyMaxK; k++) {
        if (k < a.K) {
          alignas(16) T q[4];
          const T *src = sS + k * a.sp + m;
          if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4 *>(q) = *reinterpret_cast<const float4 *>(src);
          } else {
            *reinterpret_cast<double2 *>(q) = *reinterpret_cast<const double2 *>(src);
            *reinterpret_cast<double2 *>(q + 2) = *reinterpret_cast<const double2 *>(src + 2);
          }
#pragma unroll
          for (int x = 0; x < 4; x++) c[x] = fma(q[x], lv[k], c[x]);
        }
      }
    };
    if (!STAGE) {
      for (int m = ms; m < me; m += 4) {
        T c[4];
        quad(m, c);
        if (!ok) continue;
#pragma unroll
        for (int x = 0; x < 4; x++)
          if (m + x < a.s) skinny_out(a.C + cSs[m + x] + cl, alpha * c[x], a.beta);
      }
    } else {
      T *st = stage + w * 32 * 33;
      for (int m0 = ms; m0 < me; m0 += 32) {
        // this lane's 32 results C(m0 .. m0 + 31, n) into its row of the stage
#pragma unroll 1
        for (int j = 0; j < 32 && m0 + j < a.sp; j += 4) {
          T c[4];
          quad(m0 + j, c);
#pragma unroll
          for (int x = 0; x < 4; x++) st[lane * 33 + j + x] = alpha * c[x];
        }
        __syncwarp();
        // lanes along the small side: column n' of the tile, rows m0 + lane
        const int m = m0 + lane;
        for (int j = 0; j < 32; j++) {
          const int64_t clj = __shfl_sync(0xffffffffu, cl, j);
          if (t * 32 + j < a.l && m < a.s) skinny_out(a.C + cSs[m] + clj, st[j * 33 + lane], a.beta);
        }
        __syncwarp();
      }
    }
  }
}

// Small indices of an item: with few tiles of 32 long ones, chunks of 32 apart.
int64_t skinny_chunk(int64_t s, int64_t l) {
  const int64_t sp = round_up(s, 4);
  return ceil_div(l, 32) >= 16 * kNumSMs ? sp : std::min<int64_t>(32, sp);
}

template <typename T>
void skinny_launch(SkinnyArgs a, bool stage, cudaStream_t stream) {
  const int64_t tiles = ceil_div(a.l, 32);
  a.chunk = (int)skinny_chunk(a.s, a.l);
  a.nchunks = (int)ceil_div(a.s, a.chunk);
  const int64_t items = tiles * a.nchunks;
  const unsigned blocks = (unsigned)std::max<int64_t>(std::min<int64_t>(items, kNumSMs),
                                                      std::min<int64_t>(ceil_div(items, 8), (sizeof(T) == 4 ? 4 : 2) * kNumSMs));
  const size_t smem = (size_t)a.K * a.sp * sizeof(T) + (size_t)(a.sp + kSkinnyMaxK) * sizeof(int64_t) +
                      (stage ? (size_t)8 * 32 * 33 * sizeof(T) : 0);
  const auto kernel = stage ? skinny_kernel<T, true> : skinny_kernel<T, false>;
  SCESS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  launch(kernel, blocks, 256, smem, stream, a);
  SCESS_CHECK_LAUNCH();
}
}  // namespace

void skinny_table(const TableGemm &g, bool small_is_a, bool stage, bool fp64, cudaStream_t stream) {
  SkinnyArgs a;
  a.Sm = (small_is_a ? g.A + g.baseA : g.B + g.baseB);
  a.Lg = (small_is_a ? g.B + g.baseB : g.A + g.baseA);
  a.C = g.C + g.baseC;
  a.sR = small_is_a ? g.rowA : g.colB;
  a.sK = small_is_a ? g.kA : g.kB;
  a.lR = small_is_a ? g.colB : g.rowA;
  a.lK = small_is_a ? g.kB : g.kA;
  a.cS = small_is_a ? g.rowC : g.colC;
  a.cL = small_is_a ? g.colC : g.rowC;
  const int64_t s = small_is_a ? g.M : g.N, l = small_is_a ? g.N : g.M;
  if (s < 1 || s > kSkinnyMaxS || g.K < 1 || g.K > kSkinnyMaxK || l < 1)
    throw Error(SCESS_ERR_INVALID, "skinny contraction out of range");
  a.s = (int)s;
  a.sp = (int)round_up(s, 4);
  a.K = (int)g.K;
  a.l = l;
  a.alpha = g.alpha;
  a.beta = g.beta;
  if (fp64) skinny_launch<double>(a, stage, stream);
  else skinny_launch<float>(a, stage, stream);
}

double skinny64_us(const TableGemm &g) {
  const int64_t s = std::min(g.M, g.N), l = std::max(g.M, g.N);
  if (g.K < 1 || g.K > kSkinnyMaxK || s < 1 || s > kSkinnyMaxS) return 1e30;
  // 6 us of latency, then the FP64 units of the SM with the most items, or C written and read
  const int64_t chunk = skinny_chunk(s, l), items = ceil_div(l, 32) * ceil_div(s, chunk);
  const double fma = (double)ceil_div(items, kNumSMs) * 32.0 * (double)chunk * (double)(g.K + 2);
  return 6.0 + std::max(fma / (2.0 * 1900.0), (double)s * (double)l * 16.0 / 5.0e6);
}

void dgemv_table(const TableGemm &g, cudaStream_t stream) {
  if (g.M <= 0) return;
  if (g.M < 8 * kNumSMs && g.K >= 512)  // too few rows for a warp each to fill the device
    launch(dgemv_table_kernel<true>, (unsigned)std::min<int64_t>(g.M, 8 * kNumSMs), 256, 0, stream, g);
  else
    launch(dgemv_table_kernel<false>, (unsigned)std::min<int64_t>(ceil_div(g.M * 32, 256), 16 * kNumSMs), 256,
           0, stream, g);
  SCESS_CHECK_LAUNCH();
}

int64_t dgemm_table_workspace(const TableGemm &g) {
  const int s = choose_splits(g);
  return s > 1 ? s * g.M * g.N : 0;
}

void dgemm_table(const TableGemm &g, double *workspace, cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0) return;
  if (g.K <= 0) {
    // C = beta * C
    TableGemm h = g;
    h.alpha = 0.0;
    launch(splitk_reduce_kernel, (unsigned)std::min<int64_t>(ceil_div(g.M * g.N, 256), 4096), 256, 0, stream,
           h, 0, nullptr);
    SCESS_CHECK_LAUNCH();
    return;
  }
  const int splits = choose_splits(g);
  const int64_t kChunk = round_up(ceil_div(g.K, splits), BK);
  const int nz = (int)ceil_div(g.K, kChunk);
  dim3 grid((unsigned)ceil_div(g.M, BM), (unsigned)ceil_div(g.N, BN), (unsigned)nz);
  if (nz > 1) {
    if (!workspace) throw Error(SCESS_ERR_INVALID, "dgemm_table: split-K needs a workspace");
    launch(dgemm_table_kernel, grid, 256, 0, stream, g, kChunk, workspace);
    SCESS_CHECK_LAUNCH();
    launch(splitk_reduce_kernel, (unsigned)std::min<int64_t>(ceil_div(g.M * g.N, 256), 4096), 256, 0, stream,
           g, nz, workspace);
  } else {
    launch(dgemm_table_kernel, grid, 256, 0, stream, g, kChunk, nullptr);
  }
  SCESS_CHECK_LAUNCH();
}

void dgemm_table_bounded(const TableGemm &g, double *workspace, int64_t ws_doubles,
                         cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0) return;
  const unsigned rblocks = (unsigned)std::min<int64_t>(ceil_div(g.M * g.N, 256), 4096);
  if (g.K <= 0) {
    TableGemm h = g;
    h.alpha = 0.0;
    launch(splitk_reduce_kernel, rblocks, 256, 0, stream, h, 0, nullptr);
    SCESS_CHECK_LAUNCH();
    return;
  }
  int splits = choose_splits(g);
  while (splits > 1 && (int64_t)splits * g.M * g.N > ws_doubles) splits--;
  const int64_t kChunk = round_up(ceil_div(g.K, splits), BK);
  const int nz = (int)ceil_div(g.K, kChunk);
  dim3 grid((unsigned)ceil_div(g.M, BM), (unsigned)ceil_div(g.N, BN), (unsigned)nz);
  if (nz > 1) {
    launch(dgemm_table_kernel, grid, 256, 0, stream, g, kChunk, workspace);
    SCESS_CHECK_LAUNCH();
    launch(splitk_reduce_kernel, rblocks, 256, 0, stream, g, nz, workspace);
  } else {
    launch(dgemm_table_kernel, grid, 256, 0, stream, g, kChunk, nullptr);
  }
  SCESS_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------------------------

namespace {

__global__ void permute_add_kernel(PermDesc d, double alpha, const double *__restrict__ X,
                                   double beta, double *__restrict__ Y, int64_t n) {
  chain();
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = e, xo = 0, yo = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      if (k < d.nd) {
        const int64_t i = r % d.ext[k];
        r /= d.ext[k];
        xo += i * d.xs[k];
        yo += i * d.ys[k];
      }
    }
    double val = alpha * X[xo];
    if (beta != 0.0) val += beta * Y[yo];
    Y[yo] = val;
  }
}

unsigned grid_for(int64_t n, int threads = 256) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, threads), 16 * kNumSMs * 8));
}

__global__ void tau_kernel(int64_t o, int64_t v, const double *__restrict__ t1,
                           const double *__restrict__ t2, double s, double *__restrict__ tau) {
  chain();
  const int64_t n = o * o * v * v;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % o, j = (e / o) % o, a = (e / (o * o)) % v, b = e / (o * o * v);
    tau[e] = t2[e] + s * t1[i + o * a] * t1[j + o * b];
  }
}

// dtau = tau(t1_0 + dt1, t2_0 + dt2) - tau(t1_0, t2_0)
//      = dt2 + dt1(i,a) t1_1(j,b) + t1_0(i,a) dt1(j,b),  t1_1 = t1_0 + dt1
__global__ void tau_delta_kernel(int64_t o, int64_t v, const double *__restrict__ t1_0,
                                 const double *__restrict__ dt1, const double *__restrict__ dt2,
                                 double *__restrict__ dtau) {
  chain();
  const int64_t n = o * o * v * v;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % o, j = (e / o) % o, a = (e / (o * o)) % v, b = e / (o * o * v);
    const int64_t ia = i + o * a, jb = j + o * b;
    dtau[e] = dt2[e] + dt1[ia] * (t1_0[jb] + dt1[jb]) + t1_0[ia] * dt1[jb];
  }
}

// Pairs of the particle ladder's symmetric / antisymmetric form: upper pairs
// p <= q of n labels at u(p, q) = q (q + 1) / 2 + p, strict pairs p < q at
// s(p, q) = q (q - 1) / 2 + p; pu / ps list each pair's (p, q).
__device__ __forceinline__ int64_t upair(int64_t p, int64_t q) { return q * (q + 1) / 2 + p; }
__device__ __forceinline__ int64_t spair(int64_t p, int64_t q) { return q * (q - 1) / 2 + p; }

// Vp(x, k) = V(a,b,c,d) + V(a,b,d,c) (c < d) or V(a,b,c,c) (c = d) for upper
// pairs x = (a,b), k = (c,d); Vm(x, k) = V(a,b,c,d) - V(a,b,d,c) for strict
// pairs.  V(a,b,c,d) = V[a s0 + b s1 + c s2 + d s3].
__global__ void ladder_vpm_kernel(const double *__restrict__ V, int64_t s0, int64_t s1, int64_t s2,
                                  int64_t s3, const int2 *__restrict__ pu, int64_t nu,
                                  const int2 *__restrict__ ps, int64_t ns, double *__restrict__ Vp,
                                  double *__restrict__ Vm) {
  chain();
  const int64_t total = nu * nu + ns * ns;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    if (e < nu * nu) {
      const int2 ab = pu[e % nu], cd = pu[e / nu];
      const int64_t base = ab.x * s0 + ab.y * s1;
      const double v1 = V[base + cd.x * s2 + cd.y * s3];
      Vp[e] = cd.x < cd.y ? v1 + V[base + cd.y * s2 + cd.x * s3] : v1;
    } else {
      const int64_t f = e - nu * nu;
      const int2 ab = ps[f % ns], cd = ps[f / ns];
      const int64_t base = ab.x * s0 + ab.y * s1;
      Vm[f] = V[base + cd.x * s2 + cd.y * s3] - V[base + cd.y * s2 + cd.x * s3];
    }
  }
}

// Tp(y, k) = (tau(i,j,c,d) + tau(i,j,d,c)) / 2 over upper pairs y = (i,j),
// k = (c,d); Tm(y, k) = (tau(i,j,c,d) - tau(i,j,d,c)) / 2 over strict pairs.
__global__ void ladder_tpm_kernel(int64_t o, int64_t v, const double *__restrict__ tau,
                                  const int2 *__restrict__ puo, int64_t nuo,
                                  const int2 *__restrict__ pso, int64_t nso,
                                  const int2 *__restrict__ puv, int64_t nuv,
                                  const int2 *__restrict__ psv, int64_t nsv,
                                  double *__restrict__ Tp, double *__restrict__ Tm) {
  chain();
  const int64_t total = nuo * nuv + nso * nsv, o2 = o * o, o2v = o2 * v;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    if (e < nuo * nuv) {
      const int2 ij = puo[e % nuo], cd = puv[e / nuo];
      const int64_t b = ij.x + o * ij.y;
      Tp[e] = 0.5 * (tau[b + o2 * cd.x + o2v * cd.y] + tau[b + o2 * cd.y + o2v * cd.x]);
    } else {
      const int64_t f = e - nuo * nuv;
      const int2 ij = pso[f % nso], cd = psv[f / nso];
      const int64_t b = ij.x + o * ij.y;
      Tm[f] = 0.5 * (tau[b + o2 * cd.x + o2v * cd.y] - tau[b + o2 * cd.y + o2v * cd.x]);
    }
  }
}

// R2(i,j,a,b) += Sp(u(i,j), u(a,b)) + sgn Sm(s(i,j), s(a,b)) with the pairs
// sorted and sgn = +1 when (i < j) == (a < b), -1 otherwise (0 when i = j or
// a = b): Sp is symmetric and Sm antisymmetric in each pair.  Sp is
// nuo x nuv, Sm nso x nsv, both column-major.
__global__ void ladder_unpack_kernel(int64_t o, int64_t v, const double *__restrict__ Sp,
                                     const double *__restrict__ Sm, double *__restrict__ R2) {
  chain();
  const int64_t n = o * o * v * v, nuo = o * (o + 1) / 2, nso = o * (o - 1) / 2;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % o, j = (e / o) % o, a = (e / (o * o)) % v, b = e / (o * o * v);
    const int64_t i0 = i < j ? i : j, j0 = i < j ? j : i, a0 = a < b ? a : b, b0 = a < b ? b : a;
    double s = Sp[upair(i0, j0) + nuo * upair(a0, b0)];
    if (i != j && a != b) {
      const double m = Sm[spair(i0, j0) + nso * spair(a0, b0)];
      s += ((i < j) == (a < b)) ? m : -m;
    }
    R2[e] += s;
  }
}

__global__ void denom_kernel(int64_t o, int64_t v, const double *__restrict__ eps,
                             const double *__restrict__ R1, const double *__restrict__ R2,
                             double *__restrict__ t1, double *__restrict__ t2) {
  chain();
  const int64_t n1 = o * v, n2 = o * o * v * v;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n1 + n2;
       e += (int64_t)gridDim.x * blockDim.x) {
    if (e < n1) {
      const int64_t i = e % o, a = e / o;
      t1[e] = R1[e] / (eps[i] - eps[o + a]);
    } else {
      const int64_t x = e - n1;
      const int64_t i = x % o, j = (x / o) % o, a = (x / (o * o)) % v, b = x / (o * o * v);
      // eijab = eia(i,a) + eia(j,b), the reference's association (RCCSD.cpp:331)
      const double d = (eps[i] - eps[o + a]) + (eps[j] - eps[o + b]);
      t2[x] = R2[x] / d;
    }
  }
}

__global__ void plus_transpose_kernel(int64_t o, int64_t v, double alpha,
                                      const double *__restrict__ X, double *__restrict__ out) {
  chain();
  const int64_t n = o * o * v * v;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % o, j = (e / o) % o, a = (e / (o * o)) % v, b = e / (o * o * v);
    const int64_t et = j + o * i + o * o * b + o * o * v * a;
    out[e] += alpha * (X[e] + X[et]);
  }
}

__global__ void axpby_kernel(int64_t n, double a, const double *__restrict__ x, double b,
                             double *__restrict__ y) {
  chain();
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    y[e] = a * x[e] + (b == 0.0 ? 0.0 : b * y[e]);
}

__device__ double block_sum(double v) {
  __shared__ double sh[32];
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (w == 0) {
    r = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) r += __shfl_down_sync(0xffffffffu, r, off);
  }
  __syncthreads();
  return r;  // valid in thread 0
}

__global__ void dot_partial_kernel(int64_t n, const double *__restrict__ x,
                                   const double *__restrict__ y, double *__restrict__ partials) {
  chain();
  double s = 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    s = fma(x[e], y[e], s);
  s = block_sum(s);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// Dots of nv vectors xs[q] with y, one per blockIdx.y: each is dot_partial_kernel's sum.
__global__ void dots_partial_kernel(int64_t n, DotVectors xs, const double *__restrict__ y,
                                    double *__restrict__ partials) {
  chain();
  const double *__restrict__ x = xs.p[blockIdx.y];
  double s = 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    s = fma(x[e], y[e], s);
  s = block_sum(s);
  if (threadIdx.x == 0) partials[blockIdx.y * gridDim.x + blockIdx.x] = s;
}

__global__ void sum_partials_kernel(int np, const double *__restrict__ partials,
                                    double *__restrict__ result) {
  chain();
  double s = 0.0;
  for (int e = threadIdx.x; e < np; e += blockDim.x) s += partials[(int64_t)blockIdx.x * np + e];
  s = block_sum(s);
  if (threadIdx.x == 0) result[blockIdx.x] = s;
}

__global__ void tau_energy_partial_kernel(int64_t o, int64_t v, const double *__restrict__ L,
                                          const double *__restrict__ t1,
                                          const double *__restrict__ t2,
                                          double *__restrict__ partials) {
  chain();
  const int64_t n = o * o * v * v;
  double s = 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % o, j = (e / o) % o, a = (e / (o * o)) % v, b = e / (o * o * v);
    const double tau = t2[e] + t1[i + o * a] * t1[j + o * b];
    s = fma(L[e], tau, s);
  }
  s = block_sum(s);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// MP2 (RHF.cpp:289-296, 324-340): x = (ia|jb) = g[i si + a sa + j sj + b sb],
// y = (ib|ja) (a and b swapped), eps occupied first.
__global__ void mp2_partial_kernel(int64_t o, int64_t v, const double *__restrict__ g, int64_t si,
                                   int64_t sa, int64_t sj, int64_t sb,
                                   const double *__restrict__ eps, double *__restrict__ partials) {
  chain();
  const int64_t n = o * v * o * v;
  double s = 0.0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e % o, a = (e / o) % v, j = (e / (o * v)) % o, b = e / (o * v * o);
    const double x = g[i * si + a * sa + j * sj + b * sb];
    const double y = g[i * si + b * sa + j * sj + a * sb];
    s -= x * (2.0 * x - y) / (eps[o + a] + eps[o + b] - eps[i] - eps[j]);
  }
  s = block_sum(s);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// Non-negative doubles order like their bits; a NaN (sign cleared) is above all of them.
__global__ void pair_asymmetry_kernel(const double *__restrict__ x, Ext4 n, Ext4 st, double *__restrict__ out) {
  chain();
  const int64_t total = n.e[0] * n.e[1] * n.e[2] * n.e[3];
  unsigned long long d = 0, m = 0;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = e % n.e[0], q = (e / n.e[0]) % n.e[1], rs = e / (n.e[0] * n.e[1]), r = rs % n.e[2], s = rs / n.e[2];
    if (s < r || (s == r && q < p)) continue;  // each pair once
    const double a = x[p * st.e[0] + q * st.e[1] + r * st.e[2] + s * st.e[3]];
    const double b = x[q * st.e[0] + p * st.e[1] + s * st.e[2] + r * st.e[3]];
    d = max(d, (unsigned long long)__double_as_longlong(fabs(a - b)));
    m = max(m, (unsigned long long)__double_as_longlong(fabs(a)));
  }
  for (int off = 16; off > 0; off >>= 1) {
    d = max(d, __shfl_down_sync(0xffffffffu, d, off));
    m = max(m, __shfl_down_sync(0xffffffffu, m, off));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(reinterpret_cast<unsigned long long *>(out), d);
    atomicMax(reinterpret_cast<unsigned long long *>(out) + 1, m);
  }
}

__global__ void lincomb_kernel(int64_t n, int nv, LinComb lc, bool first, double *__restrict__ out) {
  chain();
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    double s = first ? 0.0 : out[e];
    for (int c = 0; c < nv; c++) s += lc.coef[c] * lc.p[c][e];
    out[e] = s;
  }
}

__global__ void finite_kernel(int64_t n, const double *__restrict__ x, int *flag) {
  chain();
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x)
    if (!isfinite(x[e])) *flag = 1;
}

}  // namespace

void permute_add(const PermDesc &d, double alpha, const double *X, double beta, double *Y,
                 cudaStream_t stream) {
  int64_t n = 1;
  for (int k = 0; k < d.nd; k++) n *= d.ext[k];
  if (n == 0) return;
  launch(permute_add_kernel, grid_for(n), 256, 0, stream, d, alpha, X, beta, Y, n);
  SCESS_CHECK_LAUNCH();
}

void make_tau(int64_t o, int64_t v, const double *t1, const double *t2, double s, double *tau,
              cudaStream_t stream) {
  launch(tau_kernel, grid_for(o * o * v * v), 256, 0, stream, o, v, t1, t2, s, tau);
  SCESS_CHECK_LAUNCH();
}

void make_tau_delta(int64_t o, int64_t v, const double *t1_0, const double *dt1,
                    const double *dt2, double *dtau, cudaStream_t stream) {
  launch(tau_delta_kernel, grid_for(o * o * v * v), 256, 0, stream, o, v, t1_0, dt1, dt2, dtau);
  SCESS_CHECK_LAUNCH();
}

void ladder_vpm(const double *V, int64_t s0, int64_t s1, int64_t s2, int64_t s3, const int2 *pu,
                int64_t nu, const int2 *ps, int64_t ns, double *Vp, double *Vm,
                cudaStream_t stream) {
  launch(ladder_vpm_kernel, grid_for(nu * nu + ns * ns), 256, 0, stream, V, s0, s1, s2, s3, pu, nu, ps, ns, Vp,
         Vm);
  SCESS_CHECK_LAUNCH();
}

void ladder_tpm(int64_t o, int64_t v, const double *tau, const int2 *puo, int64_t nuo,
                const int2 *pso, int64_t nso, const int2 *puv, int64_t nuv, const int2 *psv,
                int64_t nsv, double *Tp, double *Tm, cudaStream_t stream) {
  launch(ladder_tpm_kernel, grid_for(nuo * nuv + nso * nsv), 256, 0, stream, o, v, tau, puo, nuo, pso, nso,
         puv, nuv, psv, nsv, Tp, Tm);
  SCESS_CHECK_LAUNCH();
}

void ladder_unpack(int64_t o, int64_t v, const double *Sp, const double *Sm, double *R2,
                   cudaStream_t stream) {
  launch(ladder_unpack_kernel, grid_for(o * o * v * v), 256, 0, stream, o, v, Sp, Sm, R2);
  SCESS_CHECK_LAUNCH();
}

void divide_denominators(int64_t o, int64_t v, const double *eps, const double *R1,
                         const double *R2, double *t1, double *t2, cudaStream_t stream) {
  launch(denom_kernel, grid_for(o * v + o * o * v * v), 256, 0, stream, o, v, eps, R1, R2, t1, t2);
  SCESS_CHECK_LAUNCH();
}

void plus_transpose(int64_t o, int64_t v, double alpha, const double *X, double *out,
                    cudaStream_t stream) {
  launch(plus_transpose_kernel, grid_for(o * o * v * v), 256, 0, stream, o, v, alpha, X, out);
  SCESS_CHECK_LAUNCH();
}

void axpby(int64_t n, double a, const double *x, double b, double *y, cudaStream_t stream) {
  if (n == 0) return;
  launch(axpby_kernel, grid_for(n), 256, 0, stream, n, a, x, b, y);
  SCESS_CHECK_LAUNCH();
}

void dot(int64_t n, const double *x, const double *y, double *partials, double *result,
         cudaStream_t stream) {
  launch(dot_partial_kernel, kDotBlocks, 256, 0, stream, n, x, y, partials);
  SCESS_CHECK_LAUNCH();
  launch(sum_partials_kernel, 1, 1024, 0, stream, kDotBlocks, partials, result);
  SCESS_CHECK_LAUNCH();
}

void dots(int64_t n, const double *const *xs, int nv, const double *y, double *partials, double *result,
          cudaStream_t stream) {
  for (int q0 = 0; q0 < nv; q0 += kDotVectors) {
    DotVectors v{};
    const int m = std::min(kDotVectors, nv - q0);
    for (int q = 0; q < m; q++) v.p[q] = xs[q0 + q];
    launch(dots_partial_kernel, dim3(kDotBlocks, (unsigned)m), 256, 0, stream, n, v, y, partials);
    SCESS_CHECK_LAUNCH();
    launch(sum_partials_kernel, (unsigned)m, 1024, 0, stream, kDotBlocks, partials, result + q0);
    SCESS_CHECK_LAUNCH();
  }
}

void linear_combination(int64_t n, int nv, const double *const *vecs, const double *coef,
                        double *out, cudaStream_t stream) {
  for (int c0 = 0; c0 < nv; c0 += kDotVectors) {
    LinComb lc{};
    const int m = std::min(kDotVectors, nv - c0);
    for (int c = 0; c < m; c++) {
      lc.p[c] = vecs[c0 + c];
      lc.coef[c] = coef[c0 + c];
    }
    launch(lincomb_kernel, grid_for(n), 256, 0, stream, n, m, lc, c0 == 0, out);
    SCESS_CHECK_LAUNCH();
  }
}

void tau_energy(int64_t o, int64_t v, const double *L, const double *t1, const double *t2,
                double *partials, double *result, cudaStream_t stream) {
  launch(tau_energy_partial_kernel, kDotBlocks, 256, 0, stream, o, v, L, t1, t2, partials);
  SCESS_CHECK_LAUNCH();
  launch(sum_partials_kernel, 1, 1024, 0, stream, kDotBlocks, partials, result);
  SCESS_CHECK_LAUNCH();
}

void mp2_energy(int64_t o, int64_t v, const double *g, int64_t si, int64_t sa, int64_t sj,
                int64_t sb, const double *eps, double *partials, double *result,
                cudaStream_t stream) {
  launch(mp2_partial_kernel, kDotBlocks, 256, 0, stream, o, v, g, si, sa, sj, sb, eps, partials);
  SCESS_CHECK_LAUNCH();
  launch(sum_partials_kernel, 1, 1024, 0, stream, kDotBlocks, partials, result);
  SCESS_CHECK_LAUNCH();
}

void pair_asymmetry(const double *x, Ext4 ext, Ext4 str, double *out, cudaStream_t stream) {
  const int64_t n = ext.e[0] * ext.e[1] * ext.e[2] * ext.e[3];
  launch(pair_asymmetry_kernel, (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256),
         8 * kNumSMs)), 256, 0, stream, x, ext, str, out);
  SCESS_CHECK_LAUNCH();
}

void check_finite(int64_t n, const double *x, int *flag, cudaStream_t stream) {
  if (n == 0) return;
  launch(finite_kernel, grid_for(n), 256, 0, stream, n, x, flag);
  SCESS_CHECK_LAUNCH();
}

}  // namespace scess
