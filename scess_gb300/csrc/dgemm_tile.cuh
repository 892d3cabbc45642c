// One 64 x 64 tile of the FP64 (DFMA) table GEMM: 256 threads, 4 x 4 register
// blocking, operands gathered through the offset tables.  Shared by the plain
// kernel and by the one that completes outputs of non-finite operands.
#pragma once
#include "kernels.h"

namespace scess {

constexpr int kDgemmTile = 64, kDgemmBK = 16;

struct DgemmShared {
  double As[kDgemmBK][kDgemmTile], Bs[kDgemmBK][kDgemmTile];
  int64_t sRowA[kDgemmTile], sColB[kDgemmTile], sKA[kDgemmBK], sKB[kDgemmBK];
};

// sum_(kb <= k < ke) A(m, k) B(k, n) of the tile at (m0, n0), each result handed
// to store(m, n, sum).
template <class Store>
__device__ __forceinline__ void dgemm_tile(DgemmShared &sh, const TableGemm &g, int64_t m0, int64_t n0, int64_t kb,
                                           int64_t ke, Store store) {
  constexpr int BM = kDgemmTile, BN = kDgemmTile, BK = kDgemmBK;
  auto &As = sh.As, &Bs = sh.Bs;
  auto &sRowA = sh.sRowA, &sColB = sh.sColB;
  auto &sKA = sh.sKA, &sKB = sh.sKB;
  const int t = threadIdx.x;
  if (t < BM) {
    const int64_t m = m0 + t;
    sRowA[t] = m < g.M ? g.baseA + g.rowA[m] : -1;
  } else if (t < BM + BN) {
    const int64_t n = n0 + (t - BM);
    sColB[t - BM] = n < g.N ? g.baseB + g.colB[n] : -1;
  }
  double acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.0;
  const int tx = t & 15, ty = t >> 4;
  for (int64_t k0 = kb; k0 < ke; k0 += BK) {
    __syncthreads();
    if (t < BK) {
      const int64_t k = k0 + t;
      sKA[t] = k < ke ? g.kA[k] : -1;
    } else if (t >= 32 && t < 32 + BK) {
      const int64_t k = k0 + (t - 32);
      sKB[t - 32] = k < ke ? g.kB[k] : -1;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int idx = t + 256 * r;
      int mm, kk;
      if (g.aUnitM) { mm = idx & (BM - 1); kk = idx / BM; }
      else { kk = idx & (BK - 1); mm = idx / BK; }
      const int64_t ro = sRowA[mm], ko = sKA[kk];
      As[kk][mm] = (ro >= 0 && ko >= 0) ? g.A[ro + ko] : 0.0;
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int idx = t + 256 * r;
      int nn, kk;
      if (g.bUnitN) { nn = idx & (BN - 1); kk = idx / BN; }
      else { kk = idx & (BK - 1); nn = idx / BK; }
      const int64_t co = sColB[nn], ko = sKB[kk];
      Bs[kk][nn] = (co >= 0 && ko >= 0) ? g.B[co + ko] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      double a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = As[kk][tx + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = Bs[kk][ty + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int64_t m = m0 + tx + 16 * i;
    if (m >= g.M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int64_t n = n0 + ty + 16 * j;
      if (n < g.N) store(m, n, acc[i][j]);
    }
  }
}

}  // namespace scess
