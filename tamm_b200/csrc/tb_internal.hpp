// Internal declarations shared by the host (C++) and device (CUDA) sources of
// libtamm_b200.so.  Nothing here is part of the public C ABI (include/tamm_b200.h).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <memory>
#include <mutex>
#include <set>
#include <stdexcept>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/tamm_b200.h"

namespace tb {

constexpr int kMaxModes = 8; // modes per tensor
constexpr int kMaxClass = 4; // labels per label class in a contraction

// Status-carrying exception used inside the library; converted to a status code
// and tb_last_error() message at the C-ABI boundary.
struct Error: std::runtime_error {
  int code;
  Error(int c, const std::string& m): std::runtime_error(m), code(c) {}
};

[[noreturn]] void fail(int code, const std::string& msg);
void              set_last_error(const std::string& msg);

#define TB_EXPECTS(cond, msg)                                                          \
  do {                                                                                 \
    if(!(cond)) ::tb::fail(TB_ERR_INVALID, std::string("EXPECTS failed: ") + (msg));   \
  } while(0)

#define TB_CUDA(call)                                                                  \
  do {                                                                                 \
    cudaError_t e_ = (call);                                                           \
    if(e_ != cudaSuccess)                                                              \
      ::tb::fail(e_ == cudaErrorMemoryAllocation ? TB_ERR_NO_MEMORY : TB_ERR_CUDA,      \
                 std::string(#call) + ": " + cudaGetErrorString(e_));                  \
  } while(0)

// Label classes of one contraction C(cl) += A(al) * B(bl), following
// kernels::block_multiply (src/tamm/kernels/multiply.hpp:237-330):
//   batch  : in C, A and B          (mode positions in C, A, B)
//   m      : in C and A only        (A-outer; C order)
//   n      : in C and B only        (B-outer; C order)
//   k      : in A and B only        (inner; A order)
//   ar, br : only in A / only in B  (reduced by beta-chained GEMM steps)
struct LabelClasses {
  int    nc = 0, na = 0, nb = 0;
  int    nbatch = 0, nm = 0, nn = 0, nk = 0, nar = 0, nbr = 0;
  int8_t batch_c[kMaxClass], batch_a[kMaxClass], batch_b[kMaxClass];
  int8_t m_c[kMaxClass], m_a[kMaxClass];
  int8_t n_c[kMaxClass], n_b[kMaxClass];
  int8_t k_a[kMaxClass], k_b[kMaxClass];
  int8_t ar_a[kMaxClass], br_b[kMaxClass];
  // which class holds the stride-1 (last) mode of A and of B: 0 m/n, 1 k, 2 other
  int8_t a_contig = 0, b_contig = 0;
};

LabelClasses classify(const int* cl, int nc, const int* al, int na, const int* bl, int nb);

// Device work-list records.
struct DevGroup {
  int64_t c_off;
  int32_t task_begin, task_end;
  int32_t cdims[kMaxModes];
};
struct DevTask {
  int64_t a_off, b_off;
  int32_t adims[kMaxModes];
  int32_t bdims[kMaxModes];
  int32_t pos, pad; // K chunks of the group's admitted tasks before this one, run or skipped
};
constexpr int kChunkK = 32; // K elements per chunk of the FP64 kernel
// One CTA's work in the FP64 kernel: an output tile (group, batch index, first row /
// column) run whole (nparts = 1), or one segment of its K: `nchunks` chunks from chunk
// `chunk0` of task `task0` on, the `part`th nonempty one of `nparts`, whose accumulators
// go to slot ws + part of the workspace.  `tile` numbers the tiles of the launch; a whole
// tile of nseg > 1 segments over `total` chunk positions closes a partial sum at each.
struct DevItem {
  int32_t group, batch, m0, n0;
  int32_t task0, chunk0, nchunks;
  int32_t tile, part, nparts, ws;
  int32_t total, nseg;
};

// Where the small device tables of a context (work lists, layouts, item and block lists)
// come from.  A plan or scheduler object is often used once, as a user's loop makes a new
// one per step, and cudaMalloc and cudaFree per table held the host for 25 us and until the
// device was idle: 93 and 123 of them per three streaming steps of the triples.  Tables
// come from the device's stream-ordered pool instead, in the order of the context's stream,
// on which alone they are used, and are filled through a pinned buffer, so that neither
// making nor dropping one waits for the device.  While the stream is being captured (memory
// of the pool would become part of the graph) and without a home, cudaMalloc serves.
class TableHome {
public:
  TableHome(int device, cudaStream_t stream): device_(device), stream_(stream) {}
  ~TableHome();
  struct Piece {
    const void* src; // host data (null: left as it is)
    size_t      bytes, off;
  };
  void* make(const std::vector<Piece>& pieces, size_t bytes);
  void  drop(void* p);
  void  close(); // the stream is about to go, and is idle

private:
  bool               capturing() const;
  std::mutex         mu_;
  int                device_ = 0;
  cudaStream_t       stream_ = nullptr;
  char*              pinned_ = nullptr; // kPinned bytes, the first used_ of them in copies under way
  size_t             used_   = 0;
  std::set<void*>    direct_; // tables from cudaMalloc
  std::vector<void*> late_;   // dropped during a capture
};

// One device allocation holding several tables.  add() notes a table, make() allocates the
// block, fills it and sets the tables' pointers; the block goes with the object.
class Tables {
public:
  Tables() = default;
  Tables(const Tables&) = delete;
  Tables& operator=(const Tables&) = delete;
  ~Tables();
  template<typename T>
  void add(T*& p, const std::vector<T>& v) {
    if(!v.empty()) note(reinterpret_cast<void**>(&p), v.data(), sizeof(T) * v.size());
  }
  template<typename T>
  void room(T*& p, size_t n) { // not filled
    note(reinterpret_cast<void**>(&p), nullptr, sizeof(T) * std::max<size_t>(n, 1));
  }
  void make(const std::shared_ptr<TableHome>& home); // on the current device

private:
  void note(void** p, const void* src, size_t bytes);
  std::vector<TableHome::Piece> pieces_;
  std::vector<void**>           ptrs_;
  size_t                        bytes_ = 0;
  std::shared_ptr<TableHome>    home_;
  void*                         base_   = nullptr;
  int                           device_ = -1;
};

// Error word of the FP64 contraction's device-side waits, in host memory mapped to the GPU,
// so that the host reads it without a copy once the launches that may set it have finished.
// A context has one, and so has each call of the block entry and each work list of a caller's
// own: a wait that gave up is reported where that work is waited for, and nowhere else.
class WaitWord {
public:
  WaitWord(); // on the current device
  WaitWord(const WaitWord&) = delete;
  WaitWord& operator=(const WaitWord&) = delete;
  ~WaitWord();
  int* device() const { return device_; }
  void check(); // throws TB_ERR_TIMEOUT if a wait gave up since the last check, and clears the word

private:
  int *host_ = nullptr, *device_ = nullptr;
};

// Host mirror of a work list plus its device copies.
struct WorkList {
  std::vector<DevGroup> groups;
  std::vector<DevTask>  tasks;
  std::vector<int32_t>  group_chunks;      // K chunks of each group's admitted tasks, run or skipped
  int64_t               out_tiles = 0;     // 128 x 64 tiles of the whole contraction's output blocks: of all
                                           // ranks and batches, whatever part of them this list holds
  double                flops = 0;         // admitted FP64 FLOPs (tasks that run + skipped tasks)
  double                flops_run = 0;     // FP64 FLOPs of the tasks in the list
  double                flops_skipped = 0; // admitted tasks left out: an exactly-zero block of a read-only operand
  int64_t               ntasks_skipped = 0;
  DevGroup*             d_groups = nullptr;
  DevTask*              d_tasks  = nullptr;
  mutable std::unique_ptr<WaitWord> waits; // of FP64 launches without a context
  std::shared_ptr<TableHome> home; // of the scheduler whose stream runs the list (null: any stream)
  Tables                tables;
  int                   device   = -1;
  // tile items of the FP64 kernel, built (and uploaded) on its first launch over this
  // work list: contractions that run split-INT8 or BF16x3 never need them
  mutable std::vector<DevItem> items_fp64;
  mutable DevItem*             d_items     = nullptr;
  mutable char *               d_group_recs = nullptr, *d_task_recs = nullptr;
  mutable Tables               tables_fp64;
  mutable bool                 items_built = false;
  mutable int                  items_shape = 64; // tile shape of those items, by its width
  mutable int64_t              ntiles_fp64 = 0;  // output tiles
  mutable int64_t              split_parts = 0;  // segments that run as items of their own
  mutable bool                 multi_segment = false; // a tile of several segments runs whole
  ~WorkList();
};

class Arena;
struct Tensor;

// Energy epilogue of a contraction (tb_sched_mult_energy): instead of C (+)= alpha * A * B
// the kernels add sum (C + alpha * A * B)^2 / D over the elements of the output groups
// with tasks and leave C unchanged; D = sum_m sg[m] * eps[estart[group * nc + m] + x_m]
// is the orbital-energy denominator of element (x_0, ..., x_(nc-1)) of the group's
// block.  Each warp of a tile writes one partial sum into `part` (tile index x warps).
struct EnergyArgs {
  const double*  eps    = nullptr;
  const int32_t* estart = nullptr;
  double*        part   = nullptr;
  double         sg[kMaxModes] = {0, 0, 0, 0, 0, 0, 0, 0};
};

#ifdef __CUDACC__
// 1 / D for a normal, nonzero double: two Newton-Raphson steps x' = x + x (1 - D x)
// from the hardware's approximate reciprocal (rcp.approx.ftz.f64); the denominator
// kernels and the energy epilogues share it, so their sums see the same 1 / D.
__device__ __forceinline__ double recip_nr(double D) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(D));
  double e = fma(-D, x, 1.0);
  x        = fma(x, e, x);
  e        = fma(-D, x, 1.0);
  return fma(x, e, x);
}

// The part of D over `n` modes of a C block: x decomposed over dims[0..n) (last
// fastest), sum_j sg[cm[j]] * eps[start[cm[j]] + x_j].
__device__ __forceinline__ double energy_part(int32_t x, int n, const int32_t* dims, const int8_t* cm,
                                              const EnergyArgs& en, const int32_t* start) {
  double d = 0.0;
  for(int j = n - 1; j >= 0; j--) {
    const int32_t q = x / dims[j];
    const int     c = cm[j];
    d += en.sg[c] * __ldg(en.eps + start[c] + (x - q * dims[j]));
    x = q;
  }
  return d;
}
#endif

// Scratch of a captured CUDA graph: buffers stay allocated for the graph's lifetime;
// ops of the graph run in stream order, so a buffer returned by one op can serve the
// next.  The graph holds the largest scratch of one op, not the sum.
struct CapturePool {
  Arena*                                    arena = nullptr;
  std::vector<std::tuple<void*, int64_t, bool>> bufs; // pointer, bytes, in use
  void*                                     get(int64_t bytes);
  void                                      put(void* p);
  void                                      release(); // back to the arena
};

struct Plan {
  LabelClasses lc;
  int          mode       = TB_MODE_FP64;
  double       err_target = 1e-11;
  int          nslices    = 0;
  tb_stats     last{};
  Arena*       arena        = nullptr; // scratch source (null: cudaMallocAsync)
  int          tile_n       = 0;       // split-INT8 output tile width (0: default for S)
  bool         few_uses     = false;   // split-INT8 requested, but FP64 is faster (see few_uses)
  bool         check_errors = true;    // read the device error word after a launch
  int*         wait_err     = nullptr; // error word of FP64 launches (null: the work list's)
  // while a CUDA graph is being captured: scratch comes from (and returns to) this
  // pool, which keeps it allocated for the graph's replays
  struct CapturePool* pinned = nullptr;
  bool         profile      = false;   // time the phases with CUDA events (synchronises)
  // C = alpha * A * B instead of C += alpha * A * B on the output blocks of groups with
  // tasks: the FP64 kernel stores its result without reading C (each element of C
  // belongs to exactly one output tile); blocks of groups without tasks are left
  // untouched
  bool         store        = false;
  // energy epilogue (EnergyArgs): *energy_out += energy_scale * the kernels' partial
  // sums; null for a plain contraction
  const EnergyArgs* energy       = nullptr;
  double*           energy_out   = nullptr;
  double            energy_scale = 1.0;
  // read-only operands whose split digits may be kept (tb_ctx_set_digit_cache), and the
  // context's cache account
  const Tensor* cache_a = nullptr;
  const Tensor* cache_b = nullptr;
  int64_t       cache_limit = 0;
  int64_t*      cache_used  = nullptr;
};

void forget_int8_layout(const WorkList* wl);
// FP64 FLOPs of one task of a group (2 * |C block| * K, times the one-sided steps).
double task_flops(const LabelClasses& lc, const DevGroup& g, const DevTask& t);
// 128 x 64 tiles of one output block, over its batch labels.
int64_t block_tiles(const LabelClasses& lc, const int32_t* cdims);
// K chunks of one task, over all its one-sided reduction steps.
int64_t task_chunks(const LabelClasses& lc, const DevTask& t);
// Largest split-INT8 slice count the error target needs (3..8).
int int8_slices_for(double err_target);

// ---- launchers (device code in *.cu) ----
void launch_contract_fp64(const Plan& plan, const WorkList& wl, double alpha, double beta,
                          int is_assign, const double* A, const double* B, double* C,
                          cudaStream_t stream);
// The same for one block triple, without a work list in device memory.
void launch_block_fp64(const LabelClasses& lc, const DevGroup& g, const DevTask& t, double alpha, double beta,
                       int is_assign, const double* A, const double* B, double* C, int* err, cudaStream_t stream);
void contract_int8(Plan& plan, const WorkList& wl, double alpha, const double* A,
                   const double* B, double* C, cudaStream_t stream);
void contract_bf16x3(Plan& plan, const WorkList& wl, double alpha, const double* A,
                     const double* B, double* C, cudaStream_t stream);

struct AssignLoop {
  int     nd = 0;
  int64_t dims[4];
  int64_t dld[4];
  int64_t sld[4];
};
AssignLoop plan_assign(const int64_t* ddims, const int* dlabels, int nd, const int64_t* sdims,
                       const int* slabels, int ns);
void launch_assign(const AssignLoop& lp, double* dst, double scale, const double* src,
                   int is_assign, cudaStream_t stream);
// One block pair of a permuted AddOp: offsets and the loop of plan_assign, with the
// position of the source's stride-1 loop mode when the pair goes through the
// shared-memory transpose (-1: streamed by rows of the destination's last mode).  The
// pair's work is cut into `units` work units of at most 2048 elements, numbered from
// `first` across the launch: `per_unit` sub-tiles of tq x tp (q: the destination's
// last mode, tq <= 64; p: the source's stride-1 mode, tp <= 32) of the transposed
// plane, or `per_unit` rows of tq elements when streamed (`upr` > 1: a row longer
// than a unit, cut into upr units).
// Counts, strides and offsets within one pair are below 2^31; `mag` holds the 64-bit
// multipliers of the divisions the kernel makes (x / d = umul64hi(x, mag) for d >= 2).
struct BlockAssign {
  int64_t  dst_off, src_off;
  int64_t  first;
  int32_t  nd, p;
  int32_t  dims[4], dld[4], sld[4];
  int32_t  units, per_unit;
  int32_t  tq, tp, upr;
  int32_t  nsub;     // sub-tiles (transposed) or rows (streamed) of the pair
  int32_t  nbq, nbp; // sub-tiles along q and p
  uint64_t mag[6];   // multipliers for dims[0..3], nbq, nbp (0: divisor 1)
};
// `first` is the number of work units of the pairs before this one in the launch.
BlockAssign make_block_assign(const AssignLoop& lp, int64_t dst_off, int64_t src_off, int64_t first);
// All block pairs of an AddOp in one launch (device array of nblocks BlockAssign
// holding nunits work units in all).
void launch_assign_blocks(double* dst, double scale, const double* src, const BlockAssign* blocks, int nblocks,
                          int64_t nunits, int is_assign, cudaStream_t stream);
// Consecutive AddOps dst (=|+=) alpha_k * src(permuted labels) of one destination and one
// source, run in one pass: the destination's blocks, each with the source block and strides
// of every op that applies to it (`present`; `staged`: through the shared-memory transpose,
// whose plane's other mode is `p` for all of them).  Units as in BlockAssign, always
// sub-tiles of the (q, p) plane.
constexpr int kFuseOps = 4;
struct FusedBlock {
  int64_t  dst_off, first;
  int32_t  nd, p;
  int32_t  dims[4], dld[4];
  int32_t  units, per_unit, tq, tp, nsub, nbq, nbp;
  int32_t  present, staged;
  int64_t  src_off[kFuseOps];
  int32_t  sld[kFuseOps][4];
  uint64_t mag[6]; // multipliers for dims[0..3], nbq, nbp
};
struct FusedOps {
  int32_t n, assign;       // ops; the first one assigns
  int32_t flat;            // ops of equal layout (bit per op): one fused multiply-add, as the flat add
  double  alpha[kFuseOps];
};
// False where the ops cannot share a pass over this block (more than one transposing mode,
// 2^31 elements and more); `units` counts the launch's work units.
bool make_fused_block(const AssignLoop* loops, const int64_t* src_off, int present, int n, int64_t dst_off,
                      int64_t units, FusedBlock& out);
void launch_fused_adds(double* dst, const double* src, const FusedBlock* blocks, int nblocks, int64_t nunits,
                       int staged, const FusedOps& ops, cudaStream_t stream);
void launch_fill(double* x, int64_t n, double value, int is_assign, cudaStream_t stream);
// Segment lists of the block-wise fill and map: per run of blocks (dst offset, src
// offset or -1, n, first), `first` the sum of n over the runs before it.
// seg_list merges blocks that are adjacent on both sides into one run.
std::vector<int64_t> seg_list(const std::vector<int64_t>& triples);
// x[off .. off + n) (=|+=) value for each run of a device segment list holding
// `total` elements
void launch_fill_blocks(double* x, const int64_t* segs, int nseg, int64_t total, double value, int is_assign,
                        cudaStream_t stream);
void launch_axpby(double alpha, const double* x, double beta, double* y, int64_t n,
                  cudaStream_t stream);
// For each run (dst offset, src offset or -1, n, first) of a device segment list
// holding `total` elements: dst[0:n) = f(src[0:n)) with f = TB_MAP_* and parameter p
// (src -1: zeros).
void launch_map_blocks(double* dst, const double* src, const int64_t* segs, int nseg, int64_t total, int fn,
                       double p, cudaStream_t stream);
double reduce_dot(const double* x, const double* y, int64_t n, cudaStream_t stream);
// *out = scale * x.y (root: scale * sqrt(x.x)), staying on the device; part holds
// 1024 doubles of scratch.  y == nullptr means x.x.
void launch_dot_to(const double* x, const double* y, int64_t n, double scale, int root, double* out, double* part,
                   cudaStream_t stream);
// One admitted block of a denominator update: packed offset, dims, and the root
// orbital index of each mode's first element.
struct DenomBlock {
  int64_t off;
  int64_t dims[kMaxModes];
  int64_t first[kMaxModes];
};
struct DenomSigns {
  double s[kMaxModes];
};
// A unit of denominator work: `rows` consecutive rows (all modes but the last) of one
// block, from row r0.
struct DenomUnit {
  int32_t block, rows;
  int64_t r0;
};
constexpr int kDenomUnitRows  = 2048;  // at most, so that the row parts fit in shared memory
constexpr int kDenomUnitElems = 16384; // about, per unit
// Scalar products taken along with a denominator update over one store: operands a[n] and
// b[n] are 0 for t as it was before the update, 1 for r, 2 for x; *out[n] = scale[n] * sum
// (root: of the sum's square root).
struct DenomDots {
  const double* x = nullptr;
  int           n = 0;
  int8_t        a[2] = {0, 0}, b[2] = {0, 0};
  int           root[2]  = {0, 0};
  double        scale[2] = {0, 0};
  double*       out[2]   = {nullptr, nullptr};
};
// (part: 2 nunits doubles of scratch; nunits > 0)
void launch_denom_dots(double* t, const double* r, double scale, const DenomBlock* blocks, const DenomUnit* units,
                       int nunits, int nmodes, const double* eps, DenomSigns signs, const DenomDots& dots,
                       double* part, cudaStream_t stream);
void launch_denom(double* t, const double* r, double scale, const DenomBlock* blocks, const DenomUnit* units,
                  int nunits, int nmodes, const double* eps, DenomSigns signs, cudaStream_t stream);
// *out += scale * sum w^2 / D over the blocks (part: nunits doubles of scratch).
void launch_denom_energy(const double* w, double scale, const DenomBlock* blocks, const DenomUnit* units,
                         int nunits, int nmodes, const double* eps, DenomSigns signs, double* part, double* out,
                         cudaStream_t stream);
void launch_set_scalar(double* out, double v, cudaStream_t stream);
// *out += scale * sum part[0 .. np), summed in a fixed order (deterministic).
void launch_energy_final(const double* part, int64_t np, double scale, double* out, cudaStream_t stream);
// nonzero[b] = 1 if x[off_b, off_b + n_b) holds an element other than +0.0 / -0.0, else
// 0, for the (off, n) pairs of a device array (the launcher clears nonzero first).
void launch_block_nonzero(const double* x, const int64_t* pairs, int nblocks, uint32_t* nonzero,
                          cudaStream_t stream);
// Reads and clears the device error word of the split-INT8 launches of a work list;
// throws TB_ERR_TIMEOUT if a device-side wait gave up.
void check_int8_errors(const WorkList& wl, cudaStream_t stream);
// The split layout that the last split launch over a work list used (null: none), to keep
// its device tables and to check the error word of its launches.
std::shared_ptr<void> int8_layout(const WorkList& wl);
void check_int8_errors(const std::shared_ptr<void>& layout, cudaStream_t stream);
void   launch_fill_random(double* x, int64_t n, uint64_t seed, uint64_t first, int dist, double p0,
                          double p1, cudaStream_t stream);

// Build the work list for one block triple (the single-block entry point).
WorkList* single_block_worklist(const LabelClasses& lc, const int64_t* adims, const int64_t* bdims,
                                const int64_t* cdims);
void finalize_worklist(const LabelClasses& lc, WorkList& wl, bool upload = true); // items + device copy

} // namespace tb
