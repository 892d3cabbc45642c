// Row tiling shared by the pack kernels of the tensor-core GEMMs.
#pragma once
#include <algorithm>
#include <cstdint>

namespace scess {

// Row tiles of 32 rows along a group's smallest-stride label: row tile x holds
// rows r = pre + P (32 ft + t + E post), t < 32 (-1 past the label's extent),
// so that a tile's source values are contiguous when that stride is 1.
struct RowTiles {
  int64_t P = 1, E = 1, nft = 1, count = 0;
  static RowTiles make(int64_t rows, int64_t P, int64_t E) {
    RowTiles r;
    if (P < 1 || E < 1 || rows % (P * E) != 0) {  // not a product grouping: plain tiles
      P = 1;
      E = std::max<int64_t>(rows, 1);
    }
    r.P = P;
    r.E = E;
    r.nft = (E + 31) / 32;
    r.count = P * r.nft * (std::max<int64_t>(rows, 1) / (P * E));
    return r;
  }
  __device__ int64_t row(int64_t x, int t) const {
    const int64_t pre = x % P, rem = x / P, ft = rem % nft, post = rem / nft;
    const int64_t f = ft * 32 + t;
    return f < E ? pre + P * (f + E * post) : -1;
  }
};

}  // namespace scess
