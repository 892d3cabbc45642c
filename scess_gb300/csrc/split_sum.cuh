// Sums over the K ranges of a split product, shared by the reductions of both
// tensor-core engines: load(z, e), z in a fixed order, added as V.
#pragma once
#include <cstdint>

namespace scess {

// Outputs of a block: ZG = 1, one per thread (grid stride); ZG = 8, 32 per block whose
// eight warps take every eighth z.  With one thread per output, a small product cut into
// 150 ranges (10 x 90 x 9000) ran four blocks for 36 us; eight warps take 7.
constexpr int kSplitGroups = 8;
inline bool split_groups(int64_t MN, int splits) { return splits >= 16 && MN <= 32 * 1024; }
inline unsigned split_blocks(int64_t MN, bool groups) {
  const int64_t per = groups ? 32 : 256, n = (MN + per - 1) / per;
  return (unsigned)(groups || n < 2048 ? n : 2048);
}

// finish(m, n, sum) for every output e = m + M n.
template <int ZG, typename V, typename L, typename F>
__device__ __forceinline__ void split_sum(int64_t M, int64_t N, int splits, const L &load, const F &finish) {
  const int64_t MN = M * N;
  auto indices = [&](int64_t e, int64_t &m, int64_t &n) {
    if (MN <= UINT32_MAX) {
      const unsigned q = (unsigned)e / (unsigned)M;
      n = q;
      m = (unsigned)e - q * (unsigned)M;
    } else {
      n = e / M;
      m = e - n * M;
    }
  };
  if constexpr (ZG == 1) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < MN; e += (int64_t)gridDim.x * blockDim.x) {
      V s{};
#pragma unroll 4
      for (int z = 0; z < splits; z++) s += load(z, e);
      int64_t m, n;
      indices(e, m, n);
      finish(m, n, s);
    }
  } else {
    __shared__ __align__(16) unsigned char raw[ZG * 32 * sizeof(V)];
    V(*red)[32] = reinterpret_cast<V(*)[32]>(raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t e = blockIdx.x * (int64_t)32 + lane;
    V s{};
    if (e < MN) {
#pragma unroll 4
      for (int z = w; z < splits; z += ZG) s += load(z, e);
    }
    red[w][lane] = s;
    __syncthreads();
    if (w == 0 && e < MN) {
      s = red[0][lane];
      for (int z = 1; z < ZG; z++) s += red[z][lane];
      int64_t m, n;
      indices(e, m, n);
      finish(m, n, s);
    }
  }
}

}  // namespace scess
