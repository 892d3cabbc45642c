// FP64 contractions on the tensor cores: operands cut into BF16 slices.
//
// GB300's FP64 units run at about 1 TFLOP/s, 1/1900 of its BF16 tensor rate.  An
// FP64 value is therefore cut into kSlices = 7 signed base-512 digits of a fixed
// point number scaled to its row's largest exponent (error-free splitting in
// the manner of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012; on
// tensor cores Mukunoki et al., ISC 2020):
//   x = 2^(E - 6) sum_p d_p 2^(-9 p),  |d_0| <= 64, |d_p| <= 256,
// E the row's exponent, the last digit rounded: 60 bits below the row's largest
// value.  Digits d_p 2^(-9 p) are exact in BF16.  A product of two rows is
//   sum_d 2^(-9 d) S_d,  S_d = sum_k sum_(p + q = d) a_p b_q,
// and as long as an S_d stays within 2^24 (64 values of k at least, for d <= 4) its
// FP32 sum inside the tensor core is exact.  The kernel drains S_0 .. S_4 in time
// into one 64-bit integer per output (exact), lets S_5 (weight 2^-45) and, apart from
// it, S_6 + S_7 (2^-54, 2^-63; the six products of S_7 that the digits have) add up in
// FP32 in tensor memory over the whole K range, and rounds integer + tails to FP64 once:
// 34 products.  The tensor core truncates its sums, so S_5 has an accumulator of its own,
// where its integers stay exact up to 2^24.
// Per output the error is about 2^-61 |row max| |column max| sqrt(K) and one
// rounding to 53 bits, where a chain of K fused multiply-adds rounds K times.  Measured
// against exact sums, relative rms over 200 outputs, here and on the FP64 units (64-wide
// tiles, K in sequence): Gaussian K = 900 1.5e-16, 3.1e-16; K = 9870 1.7e-16, 7.7e-16; ring
// products (kc|ld) t2 of the iterations o5 v19 .1e-16, 1.5e-16; o8 v47 .9e-16, 1.6e-16;
// o10 v90 .7e-16, 4.5e-16; o16 v140 .8e-16, 12e-16.  (With S_5 + S_6 in one accumulator and
// S_7 dropped, 28 products: 1.4, 2.6, 4.8 and 9.6e-16.)  Values far below their row's
// largest are held to that row's 60 bits, not to 53 of their own: where they decide an
// output, sum_k |a_k b_k| is small beside |row max| |column max|.  An eighth plane of the packs
// holds the values' magnitudes, whose product tells that sum for every output (two MMAs for
// the digits' 68).  Outputs that are short of the rule at slice_left, and those of rows and
// columns with Inf or NaN, are left to the FP64 units (slice_left_kernel, behind every GEMM; it
// returns at once where nothing is left).  So an output's error is of the size of a chain of
// FP64 multiply-adds', relative to sum_k |a_k b_k|, whatever the values.  The grouped launches of
// (T) do without (see triples_slices_hold).
#pragma once
#include <cuda.h>

#include <algorithm>
#include <map>
#include <memory>
#include <set>
#include <string>
#include <tuple>
#include <vector>

#include "engine.h"

namespace scess {

constexpr int kSlices = 7, kPlanes = kSlices + 1;  // digits, magnitudes
constexpr int kSliceBK = 32;        // K block of the kernel: 32 x 16 bit = 64 B rows, SWIZZLE_64B
constexpr int kRowNonFinite = 2047;  // row exponent of a row that holds Inf or NaN

// rows x [kPlanes][Kpad] BF16 values, Kpad a multiple of 32, and per row one biased FP64
// exponent (0: all values zero; kRowNonFinite: Inf or NaN); behind the exponents, for products
// that stand alone, the rows' sums of squares relative to their largest value (in units of
// square_unit), and then their numbers of values that are not zero.
struct SlicedPack {
  DevMem mem, exps;
  DevMem part;  // partial row exponents of long rows
  int64_t rows = 0, K = 0, Kpad = 0;
  const int *e() const { return exps.as<int>(); }
};

// One K segment of a grouped launch (see TcSegment, gemm_tc.h).
struct SliceSegment {
  int mapA = 0, mapB = 1;
  int64_t Kpad = 0;
  int64_t rowA0[3] = {0, 0, 0}, rowAy[3] = {0, 0, 0}, rowAz[3] = {0, 0, 0};
  int64_t rowB0[3] = {0, 0, 0}, rowBy[3] = {0, 0, 0}, rowBz[3] = {0, 0, 0};
};
struct SliceProblemSet {
  CUtensorMap maps[6];
  int nmaps = 0;
  int64_t M = 0, N = 0;
  int ny = 1, nz = 1, ng = 1, nseg = 1;
  SliceSegment seg[4];
  bool tri[3] = {false, false, false};  // group g keeps its problems with y >= z
  // exponents of output row m / column n of group g: expA[expA0[g] + m], expB[n]
  const int *expA = nullptr, *expB = nullptr;
  int64_t expA0[3] = {0, 0, 0};
  // outputs left to the FP64 units (see SliceArgs)
  int est = 0;
  float sq_unit = 0.0f;
  uint32_t *left = nullptr;
  uint8_t *flags = nullptr;
  // output element (m, n) of problem (y, z, g): C[baseC + y cy + z cz + cg + rowC[m] + colC[n]]
  double *C = nullptr;
  int64_t baseC = 0, cy[3] = {0, 0, 0}, cz[3] = {0, 0, 0}, cg[3] = {0, 0, 0};
  const int64_t *rowC[3] = {nullptr, nullptr, nullptr}, *colC[3] = {nullptr, nullptr, nullptr};
  double alpha = 1.0, beta = 0.0;
};

class SliceEngine {
 public:
  explicit SliceEngine(Ctx &ctx);
  // The device runs the kernel and the sizes are within its coordinates.
  bool usable(int64_t M, int64_t N, int64_t K) const;
  // Whether an M x N product is launched with its sides exchanged (as N x M): lanes of the
  // epilogue walk the GEMM rows, so C's unit-stride index (cUnitM, cUnitN, if known) is put there,
  // unless a side is short: rows come in tiles of 128, columns in steps of 16.
  static bool exchanges(int64_t M, int64_t N, bool cUnitM, bool cUnitN) {
    return std::min(M, N) <= 64 ? M < N : (!cUnitM && cUnitN);
  }
  // Estimated time of a product with its packs, in us, in the orientation it is launched in.
  static double estimate_us(int64_t M, int64_t N, int64_t K, bool cUnitM, bool cUnitN);
  // C = alpha A.B + beta C through the tables of g (the FP64 engine's GEMM).
  // False when the packs do not fit into device memory: nothing was launched
  // and the caller uses the DFMA kernel.
  bool table_gemm(const TableGemm &g, const char *name);
  bool contract(const EinsumPlan &pl, double alpha, const double *A, const double *B, double beta,
                double *C, bool constA, bool constB);
  void gemm_grouped(const SliceProblemSet &ps, double flops, const char *name);

  // Largest biased exponent of every row of the gather src[rowOff[r] + kOff[k]],
  // folded into exps[expIdx[r]] (atomic max; the caller clears exps first).
  void row_exps(const double *src, const int64_t *rowOff, int64_t rows, const int64_t *kOff,
                int64_t K, bool unitK, int *exps, const int64_t *expIdx);
  // Digits of the gather relative to the given exponents exps[expIdx[r]] (no smaller
  // than the row's own), optionally negated.
  void pack_with_exps(const double *src, const int64_t *rowOff, int64_t rows, const int64_t *kOff,
                      int64_t K, bool unitK, const int *exps, const int64_t *expIdx, bool negate,
                      SlicedPack &out);
  static CUtensorMap map_of(const SlicedPack &p, int box_rows);
  // Column-tile width of an N-column product: the box rows of its B-side map
  // (its A-side map has boxes of 128 rows).
  static int tile_n(int64_t N);

  // Packs of constant operands, kept for the owner of their source (see TcEngine).
  void set_cache_owner(const void *o) { owner_ = o; }
  void clear_cache(const void *owner);
  // Gives back what it keeps (packs, workspaces) unless a contraction is being set up:
  // called when an allocation fails.
  void reclaim();
  // A tensor that stays unchanged until clear_stable(): einsums that gather it
  // through equal tables share one pack.
  void add_stable(const double *p) { stable_.insert(p); }
  void clear_stable();
  int64_t workspace_bytes() const { return (int64_t)(tmpA_.mem.bytes() + tmpB_.mem.bytes() + partial_.bytes() + left_.bytes()); }
  // Throws SCESS_ERR_CUDA if a bounded wait of a launch since the last check expired.
  void check_error();
  void clear_error();

 private:
  struct Gather {  // an operand seen through its tables
    const double *src = nullptr;
    const int64_t *row = nullptr;
    int64_t rows = 0;
    const int64_t *k = nullptr;
    int64_t K = 0;
    bool unitK = false;
    int64_t rs = -1, ks = -1, P = 1, E = 0;
  };
  // Packs of up to two operands in one launch (two where K is long).
  void pack(const Gather *g, SlicedPack *const *out, int n);
  void alloc(SlicedPack &out, int64_t rows, int64_t K);
  // The product of g's operands, packed as A and B.
  void product(const TableGemm &g, const SlicedPack &A, const SlicedPack &B, const char *name);
  void launch(const SliceProblemSet &ps, int splits, double *partial);

  Ctx &ctx_;
  struct Key {  // a gather: source, content hash of its tables, sizes; owner of a kept pack
    const double *src;
    uint64_t hash;
    int64_t rows, K;
    const void *owner;
    bool operator<(const Key &o) const {
      return std::tie(src, hash, rows, K, owner) < std::tie(o.src, o.hash, o.rows, o.K, o.owner);
    }
  };
  std::map<Key, std::unique_ptr<SlicedPack>> cache_, reuse_;
  static constexpr int kSpare = 12;
  std::vector<std::unique_ptr<SlicedPack>> spare_;  // packs of stable tensors, done with
  std::set<const double *> stable_;
  const void *owner_ = nullptr;
  // Workspaces of products: kept between calls up to this size.
  static constexpr int64_t kKeptBytes = int64_t(256) << 20;
  void release_workspaces();
  SlicedPack tmpA_, tmpB_;
  DevMem err_, partial_, left_;
  bool launched_ = false, busy_ = false, kernel_ok_ = false;
};

}  // namespace scess
