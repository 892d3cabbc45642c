// Row order of the pack kernels of the tensor-core GEMMs.
#pragma once
#include <algorithm>
#include <cstdint>

namespace scess {

// A pack walks an operand's rows along its smallest-stride row label first, so that
// the source values of consecutive rows lie together.  Rows r = pre + P (f + E post) with
// f < E that label's index, P the product of the extents before it; the q-th row of
// the order has f = q mod E, then pre, then post.  Tiles are cut from this order, so
// that a label shorter than a tile leaves no rows of it empty (with one label per tile
// the packs of o = 10 filled 10 rows of 32).
struct RowTiles {
  int64_t P = 1, E = 1, rows = 0, count = 0;  // count: tiles of T rows
  static RowTiles make(int64_t rows, int64_t P, int64_t E, int T = 32) {
    RowTiles r;
    if (P < 1 || E < 1 || rows % (P * E) != 0) {  // not a product grouping: consecutive rows
      P = 1;
      E = std::max<int64_t>(rows, 1);
    }
    r.P = P;
    r.E = E;
    r.rows = rows;
    r.count = (std::max<int64_t>(rows, 1) + T - 1) / T;
    return r;
  }
  // The q-th row, -1 past the last.
  __device__ int64_t row(int64_t q) const {
    if (q >= rows) return -1;
    if (P == 1) return q;
    const int64_t f = q % E, rest = q / E;
    return rest % P + P * (f + E * (rest / P));
  }
};

}  // namespace scess
