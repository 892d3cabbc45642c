// Host-side engine: context, device memory, tensor views and the einsum compiler.
#pragma once
#include <chrono>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "common.cuh"
#include "host_pages.h"
#include "kernels.h"

namespace scess {

// Owning device allocation (freed on destruction).
struct Ctx;

// Device blocks released while an API call of their context runs are
// kept by that context (exact sizes, multiples of 512 bytes) instead of going back
// through cudaFree, which synchronises the whole device (a small call's dozens of small
// blocks too: a residual gradient at o = 8 v = 47 took 10.7 ms instead of 6.7 in a process
// with a history of allocations); later allocations of the same size in the same
// context reuse them.  All of a context's kernels run on its one
// stream, so a reused block's earlier work precedes its new work.  When the cache is full the
// oldest blocks make room: a cache full of another size's blocks left every call its cudaFree
// ((T) o5 v19 0.86 ms instead of 0.42 in a process that had run the large sizes).  The cache
// is emptied when an allocation fails and with the context.
class BlockCache {
 public:
  static constexpr size_t kMinBytes = 512;
  static constexpr size_t kMaxCached = size_t(96) << 30;
  void *take(size_t bytes);
  // false: the caller frees it; evicted: bytes of blocks freed to make room
  bool give(void *p, size_t bytes, size_t &evicted);
  size_t flush();  // frees every cached block; returns the bytes freed
  size_t bytes() const { return total_; }

 private:
  struct Block {
    void *p;
    uint64_t stamp;
  };
  std::multimap<size_t, Block> free_;
  std::map<uint64_t, std::multimap<size_t, Block>::iterator> age_;  // oldest first
  uint64_t clock_ = 0;
  size_t total_ = 0;
};

// Internal tuning switches, for tests and tuning runs only: the environment
// variable SCESS_TUNE holds "key=value" pairs separated by commas, read at
// every call.  Keys: t_nb (virtual block size of (T), both forms; default: the
// size chosen from o and v), t_kbd (K blocks of 64 per TMEM drain in the
// mixed (T) launch: 1, 2 or 4), t_wbuf (W buffers of the mixed (T): 1 or 3) and f64
// (FP64 products: 1 on the tensor cores' slices, 2 on the FP64 units, there with the 12
// products a block triple of (T)).
// Returns `def` for an unset key.
int64_t tune_value(const char *key, int64_t def);
// TMEM drain cadence of the mixed (T) launch (K blocks of 64 per drain).
constexpr int kTriplesKbd = 4;
// W buffers of the mixed (T): 1 (the groups add into one with L2 reductions) or
// 3 (one per group, plain stores).
constexpr int kTriplesWBuffers = 1;

// The context whose API call runs on this thread (null outside calls).
Ctx *current_ctx();
struct CurrentCtx {
  Ctx *prev;
  explicit CurrentCtx(Ctx *c);
  ~CurrentCtx();
};

class DevMem {
 public:
  DevMem() = default;
  explicit DevMem(size_t bytes) { alloc(bytes); }
  ~DevMem() { release(); }
  DevMem(const DevMem &) = delete;
  DevMem &operator=(const DevMem &) = delete;
  DevMem(DevMem &&o) noexcept : p_(o.p_), bytes_(o.bytes_), owner_(o.owner_) {
    o.p_ = nullptr;
    o.bytes_ = 0;
    o.owner_ = nullptr;
  }
  DevMem &operator=(DevMem &&o) noexcept {
    if (this != &o) {
      release();
      p_ = o.p_;
      bytes_ = o.bytes_;
      owner_ = o.owner_;
      o.p_ = nullptr;
      o.bytes_ = 0;
      o.owner_ = nullptr;
    }
    return *this;
  }
  void alloc(size_t bytes);
  void release();
  template <class T> T *as() const { return static_cast<T *>(p_); }
  double *d() const { return static_cast<double *>(p_); }
  size_t bytes() const { return bytes_; }

 private:
  void *p_ = nullptr;
  size_t bytes_ = 0;
  Ctx *owner_ = nullptr;  // context whose API call allocated it
};

// Strided view of an FP64 tensor in device memory: element (i_0, ..., i_{nd-1})
// lives at p[sum_d i_d * str[d]].
struct TV {
  double *p = nullptr;
  int nd = 0;
  int64_t ext[6] = {1, 1, 1, 1, 1, 1};
  int64_t str[6] = {0, 0, 0, 0, 0, 0};
  int64_t size() const {
    int64_t n = 1;
    for (int d = 0; d < nd; d++) n *= ext[d];
    return n;
  }
};
// Column-major (first index fastest) dense view.
TV cm(double *p, std::initializer_list<int64_t> ext);
// A dense column-major tensor that owns its memory.
struct DTensor {
  DevMem mem;
  TV v;
  DTensor() = default;
  DTensor(std::initializer_list<int64_t> ext);
  double *p() const { return v.p; }
  int64_t size() const { return v.size(); }
};

// Geometry of an einsum (label groups and offset tables), shared by backends.
struct EinsumPlan {
  int64_t M = 1, N = 1, K = 1;
  std::vector<int64_t> rowA, kA, colB, kB, rowC, colC;  // host copies
  std::shared_ptr<DevMem> dev;  // rowA | kA | colB | kB | rowC | colC on the device
  const int64_t *d_rowA = nullptr, *d_kA = nullptr, *d_colB = nullptr, *d_kB = nullptr;
  const int64_t *d_rowC = nullptr, *d_colC = nullptr;
  bool aUnitM = false, bUnitN = false, aUnitK = false, bUnitK = false;
  bool cUnitM = false, cUnitN = false;  // C's unit-stride label leads the M / N group
  // the operand offset tables as plain strides (offset = index * stride), or -1
  int64_t aRowStride = -1, aKStride = -1, bColStride = -1, bKStride = -1;
  // packing hints: rows r = pre + P (f + E post), f along the operand's
  // smallest-stride row label; dense: the gather is a permutation of src[0, n)
  int64_t aRowP = 1, aRowE = 1, bColP = 1, bColE = 1;
  bool aDense = false, bDense = false;
  std::string key;
  std::string spec;
  // content hashes of (rowA, kA) and (colB, kB), computed on first use: two
  // plans that gather an operand through equal tables pack it identically
  mutable uint64_t hashA = 0, hashB = 0;
};
// Content hash of an operand's two offset tables (never 0).
uint64_t table_hash(const std::vector<int64_t> &r, const std::vector<int64_t> &k);
class TcEngine;     // tensor-core (mixed precision) backend, gemm_tc.cu
class SliceEngine;  // FP64 contractions on tensor-core slices, gemm_slice.cu

// Forward-op record for the hand-written adjoint: every einsum / permute (and
// the residual's tau and PlusTranspose steps) issued while Ctx::tape is set is
// appended with its operand views; adjoint.cu sweeps the list in reverse.
struct TapeOp {
  enum Kind { EINSUM = 0, PERMUTE = 1, TAU = 2, PLUS_T = 3 } kind = EINSUM;
  std::string spec;
  double alpha = 1.0, beta = 0.0;
  TV A, B, C;
  int64_t o = 0, v = 0;
};
struct Tape {
  std::vector<TapeOp> ops;
};

// Per-call control: cancellation and the time limit.
struct Control {
  scess_cancel_fn cancel = nullptr;
  void *user = nullptr;
  double time_limit_s = 0.0;
  std::chrono::steady_clock::time_point start = std::chrono::steady_clock::now();
  void poll() const;
};

// Optional per-kernel timing: CUDA events recorded on the launching stream
// around each instrumented launch, aggregated per kernel name (launches,
// device milliseconds, algorithmic FLOPs and bytes).
class KernelTimer {
 public:
  struct Agg {
    int64_t launches = 0;
    double ms = 0.0, flops = 0.0, bytes = 0.0;
  };
  bool on = false;
  ~KernelTimer();
  void begin(const char *name, double flops, double bytes, cudaStream_t s);
  void end(cudaStream_t s);
  void collect();  // waits for the recorded events and folds them into agg
  // host-side phase (wall clock, ms), reported beside the kernels as "host:<name>"
  void host(const char *name, double ms);
  void reset();
  std::map<std::string, Agg> agg;

 private:
  struct Rec {
    std::string name;
    cudaEvent_t a, b;
    double flops, bytes;
  };
  cudaEvent_t get();
  std::vector<Rec> recs_;
  std::vector<size_t> open_;  // records whose end() is pending (scopes nest)
  std::vector<cudaEvent_t> pool_;
};

// RAII helper: times the launches issued in its scope when the timer is on.
struct TimedScope {
  KernelTimer &t;
  cudaStream_t s;
  bool active;
  TimedScope(KernelTimer &tm, const char *name, double flops, double bytes, cudaStream_t st)
      : t(tm), s(st), active(tm.on) {
    if (active) t.begin(name, flops, bytes, s);
  }
  ~TimedScope() {
    if (active) t.end(s);
  }
};

// Bounds of the tensor-core kernels' pipeline waits.  The defaults are the production
// ones; the diagnostics entry point arms a short bound and a withheld first
// stage for one launch, to exercise the expiry path.
struct WaitDiag {
  long long wait_cycles = 1ll << 32;
  bool withhold_first = false;
};

struct Ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string last_error;
  scess_cancel_fn cancel = nullptr;
  scess_log_fn log = nullptr;
  void *user = nullptr;

  // einsum plans (offset tables), keyed by spec + operand geometry
  std::map<std::string, std::unique_ptr<EinsumPlan>> plans;
  DevMem workspace;          // split-K partials
  DevMem scratch;            // partial sums of reductions + device scalars
  DevMem counters;           // dgemm_small's tile counters (zero between launches)
  double *partials = nullptr;
  double *dscalars = nullptr;  // 64 device doubles
  double *hscalars = nullptr;  // 64 pinned host doubles
  std::unique_ptr<TcEngine> tc;
  std::unique_ptr<SliceEngine> slices;
  KernelTimer timer;
  Tape *tape = nullptr;  // recording target while an adjoint forward pass runs
  BlockCache blocks;     // released large device blocks (see BlockCache)
  // Device memory held by this context's calls (live blocks and the block
  // cache) and its cap (0 = none): an allocation beyond the cap fails with
  // SCESS_ERR_OOM as if the device were full (scess_ctx_set_memory_limit).
  size_t mem_held = 0, mem_limit = 0;

  explicit Ctx(int dev);
  ~Ctx();
  void sync() const { SCESS_CUDA(cudaStreamSynchronize(stream)); }
  double *ensure_workspace(int64_t doubles);
  void logf(int level, const char *fmt, ...) const;
  TcEngine &tensor_cores();
  SliceEngine *slice_engine();  // null: no room for it
  WaitDiag wait_diag;  // of the next tensor-core launch (either engine's)
  WaitDiag take_wait_diag() {
    const WaitDiag d = wait_diag;
    wait_diag = WaitDiag();
    return d;
  }
};

// C = alpha A.B + beta C in FP64 through the tables of g: small products on the
// FP64 units, the others on the tensor cores' slices (gemm_slice.h).
void fp64_table_gemm(Ctx &ctx, const TableGemm &g, const char *name);

// FP64: FP64 units and slices.  MIXED: tensor cores for contractions large enough to pay
// for packing, FP64 for the rest.  TENSOR: tensor cores for every contraction.
enum class Backend { FP64 = 0, MIXED = 1, TENSOR = 2 };

// C[labels] = alpha * A[labels] B[labels] + beta * C   (spec "kcld,ilcd->ki").
// Backend::MIXED routes large contractions to the tcgen05 engine and keeps
// small ones in FP64.  `constA`/`constB` mark operands whose contents do not
// change during the call so that their tensor-core packing can be reused.
void einsum(Ctx &ctx, const char *spec, double alpha, const TV &A, const TV &B, double beta,
            const TV &C, Backend be = Backend::FP64, bool constA = false, bool constB = false);
// Y[out labels] = alpha * X[in labels] + beta * Y   (spec "kcai->akic").
void permute(Ctx &ctx, const char *spec, double alpha, const TV &X, double beta, const TV &Y);

const EinsumPlan &plan_einsum(Ctx &ctx, const char *spec, const TV &A, const TV &B, const TV &C);

// xs[q] . y for nv vectors (host array of device pointers), on the host.  Any nv: the context's
// device and pinned scalars hold 64 at a time.
std::vector<double> dots_on_host(Ctx &ctx, int64_t n, const double *const *xs, int nv, const double *y);

// Upload helpers (synchronous w.r.t. the host buffer).
void upload(Ctx &ctx, double *dst, const double *src, int64_t n);
void download(Ctx &ctx, double *dst, const double *src, int64_t n);

}  // namespace scess
