// Grouped FP64 block contraction on the FP64 tensor cores (DMMA, mma.sync m16n8k8 f64).
//
// One launch runs a whole MultOp::execute_bufacc (src/tamm/multop.hpp:576-893): a CTA
// owns one tile of one output block (a "group") and loops over the group's (A block, B
// block) tasks — the admitted reduction tiles — and, inside each task, over the A-only x
// B-only reduction steps and the K chunks, accumulating in registers.  Operands are
// gathered straight from the block store with the label permutation folded into per-row
// / per-k offset tables (no Ainter/Binter copies as in kernels::block_multiply's
// transpose_inputs, multiply.hpp:159-194), staged through a cp.async pipeline, and the
// result is written once into C in C's own label order (transpose_output,
// multiply.hpp:196-210, fused into the epilogue).
//
// The kernel is bound by the FP64 tensor pipe (64 multiply-adds per SM and clock), so
// what counts is that every SM holds work until the end.  A group's K is therefore cut
// into segments of at most kSegment chunks, and C's element is the sum of its segments'
// sums, in order.  A tile runs whole, in one CTA that closes a partial sum at each
// segment's end, or spread over the SMs (split reduction): each segment in a CTA of its
// own leaves its accumulators in a workspace, and the one that arrives last sums them all
// in order and writes C.  Both give the same bits, and the cuts follow the group's own
// admitted tasks alone, whether they run or are skipped as exact zeros: a result depends
// neither on the other blocks of the launch nor on how its work was spread.  Two exceptions,
// within the rounding of the sums: one block triple through the block entry is cut into as
// many parts as its extents and the GPU's SMs ask for, and where not even the closed sums'
// 82 KB per CTA can be had the segments are not closed.
//
// Measured on one B200 (cuBLAS DGEMM: 35.4 TFLOP/s): full 128 x 80 tiles 28 TFLOP/s; the
// O = 30, V = 180 ladder 7.25 ms (8.19 with one whole 128 x 80 tile per CTA, the gather in
// the computing warps), a small doubles iteration (O = 20, V = 100) 2.60 ms (10.0).
#include "tb_internal.hpp"
#include "tb_runtime.hpp"
#include "tb_sm100.cuh"

#include <algorithm>
#include <cmath>

namespace tb {
namespace {
using namespace sm100;

constexpr int BK = kChunkK;

// Shared-memory tiles are stored unpadded with the column XOR-swizzled by the row's four
// low bits, two by two exchanged: the DMMA fragment loads (4 rows x 4 columns per half
// warp) and the stores of 16 consecutive rows in one column hit 16 distinct bank pairs.
__device__ __forceinline__ int swz(int row, int col) { return col ^ (((row & 3) << 2) | ((row >> 2) & 3)); }

// An output tile of BM x BN on WM x WN consumer warps (2 m16 x NJ n8 DMMA tiles each) and
// NP producer warps, ST chunks staged, CTAS per SM.
//   Wide (128 x 80 or 64): the least operand traffic per multiply-add; one CTA per SM.
//   Narrow (64 x 32): a fifth of the work per chunk, for contractions with too few wide
//   tiles to fill the SMs and for output blocks that would leave most of a wide tile empty.
// RP, RC: registers of a producer and a consumer thread, out of those the CTA is launched
// with (0: as launched).
template<int BM_, int BN_, int WM_, int WN_, int NP_, int ST_, int CTAS_, int RP_ = 0, int RC_ = 0>
struct Shape {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, ST = ST_, CTAS = CTAS_, RP = RP_, RC = RC_;
  static constexpr int NC = WM * WN, PT = 32 * NP_;      // consumer warps, producer threads
  static constexpr int CT = 32 * NC, NTHREADS = CT + PT; // consumer threads, all threads
  static constexpr int NJ = BN / WN / 8;                 // n8 fragments of a warp
  static_assert(BM == 32 * WM && BN % (8 * WN) == 0 && BM % 16 == 0 && BN % 16 == 0 && BK * 16 % PT == 0, "tile shape");
  static_assert(RP == 0 || (NC % 4 == 0 && NP_ % 4 == 0), "whole warpgroups");
};
using Wide80 = Shape<128, 80, 4, 2, 8, 4, 1, 88, 168>;
using Wide64 = Shape<128, 64, 4, 2, 8, 4, 1, 88, 168>;
using Narrow = Shape<64, 32, 2, 2, 4, 4, 2>;
// the register shares add up to no more than the launch's (128 each)
static_assert(Wide80::PT * Wide80::RP + Wide80::CT * Wide80::RC <= 128 * Wide80::NTHREADS, "register shares");
static_assert(Wide64::PT * Wide64::RP + Wide64::CT * Wide64::RC <= 128 * Wide64::NTHREADS, "register shares");


// A list of labels as the kernel walks it: extents and the multipliers of the divisions by
// them: x / d = umulhi(x, ceil(2^32 / d)) for x d < 2^32 and d >= 2 (Granlund and Montgomery,
// division by invariant integers using multiplication); 0 for d = 1, or 1 where the list's
// indices are too large for that (plain division).
struct Labels {
  uint32_t mag[kMaxClass];
  int32_t  dim[kMaxClass];
};

// Output block of a group: worked out on the host, so that a CTA starts on one record
// instead of a chain of loads and products.
struct alignas(16) GroupRec {
  Labels  m, n;
  int32_t mstr[kMaxClass], nstr[kMaxClass]; // C strides
  int32_t bdim[kMaxClass], bstr[kMaxClass]; // batch labels: extents and C strides
  int64_t c_off;
  int32_t M, N, task_end, pad;
};

// One (A block, B block) task, likewise.
struct alignas(16) TaskRec {
  Labels  k;
  int64_t a_off, b_off;
  int32_t kstrA[kMaxClass], kstrB[kMaxClass], mstrA[kMaxClass], nstrB[kMaxClass];
  int32_t bstrA[kMaxClass], bstrB[kMaxClass]; // batch labels
  int32_t ardim[kMaxClass], arstrA[kMaxClass], brdim[kMaxClass], brstrB[kMaxClass];
  int32_t K, ARBR, BR, pos;
};
static_assert(sizeof(GroupRec) % 16 == 0 && sizeof(TaskRec) % 16 == 0 && sizeof(TaskRec) / 16 <= 64, "record sizes");

// What the consumers need to know of a staged chunk.
struct StageInfo {
  int32_t kvalid;     // K elements of the chunk; -1: no more items
  int32_t last;       // the item's last chunk
  int32_t close;      // a new segment begins with this chunk
  int32_t first_step; // a one-sided reduction step begins with it
};

// An item's output tile as the producers hand it to the consumers.
template<class T>
struct TileGeo {
  double  rowD[T::BM], colD[T::BN]; // energy epilogue: the rows' and columns' parts of the denominators
  int32_t rowC[T::BM], colC[T::BN];
  int64_t c_base;
  int32_t m_lim, n_lim; // rows / columns of the tile within the output block
  int32_t tile, part, nparts, ws;
};

template<class T>
struct Smem {
  double    As[T::ST][T::BM][BK]; // [m][k ^ swz]
  double    Bs[T::ST][BK][T::BN]; // [k][n ^ swz]
  uint64_t  full[T::ST], empty[T::ST], gempty[2];
  TileGeo<T> geo[2];
  int32_t   rowA[2][T::BM], colB[2][T::BN]; // by task parity
  GroupRec  group;
  TaskRec   task[2]; // by task parity
  StageInfo sd[T::ST];
  int32_t   next; // next item of a persistent CTA
};

// (228 KB of shared memory per SM, 1 KB of it reserved per CTA)
template<class T>
constexpr bool fits = T::CTAS * (sizeof(Smem<T>) + 1024) <= 228 * 1024 && sizeof(Smem<T>) <= 227 * 1024;
static_assert(fits<Wide80> && fits<Wide64> && fits<Narrow>, "resident FP64 CTAs per SM");

struct Params {
  LabelClasses    lc;
  const double*   A;
  const double*   B;
  double*         C;
  const GroupRec* groups;
  const TaskRec*  tasks;
  const DevItem*  items;
  double          alpha, beta;
  int             is_assign;
  int             energy = 0; // sum (C + alpha * acc)^2 / D into en.part, C unchanged
  EnergyArgs      en;
  int*            err;    // set by a wait that gave up
  int             nitems = 0;
  double*         ws  = nullptr; // accumulators of split tiles' segments (null: each tile's first item runs it whole)
  int32_t*        cnt = nullptr; // arrivals per split tile and warp, from its first part's slot on (zero at launch)
  double*         sum = nullptr; // sums of a whole tile's closed segments, one tile per CTA (null: not closed)
  int32_t*        ctr = nullptr; // items handed out beyond the grid's (zero at launch; null: one per CTA)
  // one block triple without a work list in memory: the group and task travel with the
  // launch, the items are numbered by the grid
  int             single = 0, mtiles = 0, ntiles = 0, nparts = 1, nchunks = 0;
  GroupRec        g1{};
  TaskRec         t1{};
};

// A load that is issued where it stands (a plain one would be moved down to its first use,
// behind the wait for a free stage, one round trip after the other).
__device__ __forceinline__ double load_now(const double* p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];\n" : "=d"(v) : "l"(p));
  return v;
}

// Barrier of the producer warps; true if `failed` holds for any of their threads.  The
// barrier counts warps: a warp whose lanes left a wait or a loop one by one has to be
// together again before it arrives.
template<int PT>
__device__ __forceinline__ bool producers_any(bool failed) {
  uint32_t any;
  __syncwarp();
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
               "bar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
               : "=r"(any)
               : "r"((uint32_t) failed), "n"(PT)
               : "memory");
  return any != 0;
}

// D(16x8) += A(16x8) * B(8x8) in FP64.  Fragments (g = lane / 4, t = lane % 4):
// a = {A[g][t], A[g+8][t], A[g][t+4], A[g+8][t+4]}, b = {B[t][g], B[t+4][g]},
// c = {C[g][2t], C[g][2t+1], C[g+8][2t], C[g+8][2t+1]}.
__device__ __forceinline__ void dmma16(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// Offsets of linear index x decomposed over the n labels l (last fastest) with two sets of
// strides.
__device__ __forceinline__ int2 decompose2(uint32_t x, int n, const Labels& l, const int32_t* s1, const int32_t* s2) {
  int2 off = make_int2(0, 0);
#pragma unroll
  for(int j = kMaxClass - 1; j >= 0; j--) {
    if(j >= n) continue;
    const uint32_t mag = l.mag[j], d = l.dim[j];
    const uint32_t q = mag == 0 ? x : mag == 1 ? x / d : __umulhi(x, mag);
    const int32_t  r = (int32_t) (x - q * d);
    off.x += r * s1[j];
    off.y += r * s2[j];
    x = q;
  }
  return off;
}
__device__ __forceinline__ int32_t decompose(uint32_t x, int n, const Labels& l, const int32_t* str) {
  return decompose2(x, n, l, str, str).x;
}

// The same over a few labels with plain divisions (rare: batch and one-sided reduction labels).
__device__ __forceinline__ int64_t decompose_div(int32_t x, int n, const int32_t* dims, const int32_t* str) {
  int64_t off = 0;
  for(int j = n - 1; j >= 0; j--) {
    const int32_t q = x / dims[j];
    off += (int64_t) (x - q * dims[j]) * str[j];
    x = q;
  }
  return off;
}

// A record of 16-byte words to shared memory by the first threads of the producers.
template<class R>
__device__ __forceinline__ void copy_record(R& dst, const R& src, int pt) {
  if(pt < (int) (sizeof(R) / 16)) reinterpret_cast<uint4*>(&dst)[pt] = reinterpret_cast<const uint4*>(&src)[pt];
}

// The producer warps: item by item, task by task, chunk by chunk they bring the elements
// through registers into the next free stage, up to ST chunks (and into the next item)
// ahead of the consumers.  What they do per chunk has to fit beside the consumers' issue
// slots and into the chunk's tensor time (2.7 us for 128 x 80), so: records instead of
// geometry worked out here; the chunk's K offsets in the lanes of every warp, so that the
// producers meet only where a task or an item begins; all loads of a chunk in flight
// together, their offsets fetched ahead of them; no bounds tests (rows and columns past
// the block repeat its last one and reach no stored element, K past the task's is zeroed
// in its last chunk); shared-memory addresses that differ by constants.  (8-byte cp.async
// copies with tables in shared memory and a barrier per chunk took 4.9 us per chunk.)
template<class T>
__device__ __forceinline__ void produce(const Params& p, Smem<T>& s) {
  constexpr int       BM = T::BM, BN = T::BN, PT = T::PT;
  const LabelClasses& lc = p.lc;
  const int           pt = threadIdx.x - T::CT, lane = pt & 31;
  int                 stage = 0, tslot = 0;
  uint32_t            phase = 0;
  bool                bad   = false; // a wait of this thread gave up
  // With K contiguous in an operand a warp reads 32 k of one row (column) at a time;
  // otherwise half a warp reads 16 consecutive rows (columns) of one k.
  const bool a_kfast = lc.a_contig == 1, b_kfast = lc.b_contig == 1;
  const int  pw = pt >> 5, p16 = pt & 15, k16 = pt >> 4; // row of the kfast walk; row and k of the other
  int        x       = blockIdx.x;
  for(int n = 0;; n++) {
    if(!p.single && x >= p.nitems) break;
    DevItem it;
    if(p.single) { // tile-major: the parts of a tile are neighbours
      int y      = x;
      it.part    = y % p.nparts;
      it.tile    = y / p.nparts;
      y          = it.tile;
      it.n0      = y % p.ntiles * BN;
      y /= p.ntiles;
      it.m0      = y % p.mtiles * BM;
      it.batch   = y / p.mtiles;
      it.group   = it.task0 = 0;
      it.nparts  = p.nparts;
      it.ws      = it.tile * p.nparts;
      it.chunk0  = (int) ((int64_t) p.nchunks * it.part / p.nparts);
      it.nchunks = (int) ((int64_t) p.nchunks * (it.part + 1) / p.nparts) - it.chunk0;
      it.total   = p.nchunks;
      it.nseg    = 1;
    }
    else it = p.items[x];
    bool skip = false;
    if(it.nparts > 1 && p.ws == nullptr) { // no workspace: the first part runs the whole tile
      skip       = it.part > 0;
      it.nparts  = 1;
      it.nchunks = 0x7fffffff;
    }
    if(!skip) {
      // ---- the output tile's and the first task's records ----
      TileGeo<T>& geo = s.geo[n & 1];
      copy_record(s.group, p.single ? p.g1 : p.groups[it.group], pt);
      copy_record(s.task[tslot], p.single ? p.t1 : p.tasks[it.task0], pt);
      bad |= !mbar_wait(&s.gempty[n & 1], ((n >> 1) & 1) ^ 1, p.err, 31);
      if(producers_any<PT>(bad)) goto failed;
      const GroupRec& g     = s.group;
      const int       m_lim = min(g.M - it.m0, BM), n_lim = min(g.N - it.n0, BN), te = g.task_end;
      if(pt == 0) {
        geo.c_base = g.c_off + decompose_div(it.batch, lc.nbatch, g.bdim, g.bstr);
        geo.m_lim  = m_lim;
        geo.n_lim  = n_lim;
        geo.tile   = it.tile;
        geo.part   = it.part;
        geo.nparts = it.nparts;
        geo.ws     = it.ws;
      }
      for(int m = pt; m < m_lim; m += PT) geo.rowC[m] = decompose(it.m0 + m, lc.nm, g.m, g.mstr);
      for(int c = pt; c < n_lim; c += PT) geo.colC[c] = decompose(it.n0 + c, lc.nn, g.n, g.nstr);
      if(p.energy) { // batch labels' part folded into the rows'
        const int32_t* es = p.en.estart + (int64_t) it.group * lc.nc;
        const double   db = energy_part(it.batch, lc.nbatch, g.bdim, lc.batch_c, p.en, es);
        for(int m = pt; m < m_lim; m += PT)
          geo.rowD[m] = db + energy_part(it.m0 + m, lc.nm, g.m.dim, lc.m_c, p.en, es);
        for(int c = pt; c < n_lim; c += PT) geo.colD[c] = energy_part(it.n0 + c, lc.nn, g.n.dim, lc.n_c, p.en, es);
      }
      // ---- chunks over (task, reduction step, k0), uniform across the producers ----
      int           t = it.task0, st = 0, k0 = 0, K = 0, ARBR = 0, pos = 0;
      const int     nseg = it.nparts > 1 ? 1 : it.nseg; // (a part is one segment)
      int           seg = 0, seg_end = nseg > 1 ? (int) ((int64_t) it.total / nseg) : 0x7fffffff;
      int32_t       kA = 0, kB = 0; // this lane's K element of the chunk: its offsets in the blocks
      const double *a = nullptr, *b = nullptr;
      bool          fresh = true; // a new task begins
      auto          chunk_offsets = [&] {
        const TaskRec& tk = s.task[tslot];
        const int2     o  = decompose2(min(k0 + lane, K - 1), lc.nk, tk.k, tk.kstrA, tk.kstrB);
        kA = o.x;
        kB = o.y;
      };
      for(int c = 0; c < it.nchunks && t < te; c++) {
        if(fresh) {
          if(c > 0) {
            copy_record(s.task[tslot], p.tasks[t], pt);
            if(producers_any<PT>(bad)) goto failed;
          }
          const TaskRec& tk = s.task[tslot];
          K    = tk.K;
          ARBR = tk.ARBR;
          pos  = tk.pos;
          if(c == 0) { // the item's first chunk, within its first task
            const int nck = (K + BK - 1) / BK;
            st            = it.chunk0 / nck;
            k0            = (it.chunk0 - st * nck) * BK;
            pos += it.chunk0;
          }
          for(int m = pt; m < BM; m += PT)
            s.rowA[tslot][m] = decompose(it.m0 + min(m, m_lim - 1), lc.nm, g.m, tk.mstrA);
          for(int y = pt; y < BN; y += PT)
            s.colB[tslot][y] = decompose(it.n0 + min(y, n_lim - 1), lc.nn, g.n, tk.nstrB);
          a = p.A + tk.a_off + decompose_div(it.batch, lc.nbatch, g.bdim, tk.bstrA);
          b = p.B + tk.b_off + decompose_div(it.batch, lc.nbatch, g.bdim, tk.bstrB);
          chunk_offsets();
          if(producers_any<PT>(bad)) goto failed; // (the tables are complete)
        }
        bool close = false;
        while(pos >= seg_end) { // (segments whose tasks are all skipped are passed over)
          seg++;
          seg_end = seg + 1 < nseg ? (int) ((int64_t) it.total * (seg + 1) / nseg) : 0x7fffffff;
          close   = c > 0;
        }
        const int      kvalid = min(BK, K - k0);
        const int32_t *rowA = s.rowA[tslot], *colB = s.colB[tslot];
        const double * as = a, *bs = b;
        if(ARBR > 1) { // one-sided reduction step
          const TaskRec& tk = s.task[tslot];
          const int      ar = st / tk.BR;
          as += decompose_div(ar, lc.nar, tk.ardim, tk.arstrA);
          bs += decompose_div(st - ar * tk.BR, lc.nbr, tk.brdim, tk.brstrB);
        }
        constexpr int EA = BM * BK / PT, EB = BN * BK / PT; // elements per thread
        constexpr int GA = BM / 16, GB = BN / 16;           // groups of 16 rows, columns
        constexpr int PW = PT / 32, KS = PT / 16, NI = BK / KS; // warps; k steps of the other walk
        double        va[EA], vb[EB];
        if(a_kfast) { // element e: row pw + PW e, k = lane
          const double* src = as + kA;
          constexpr int U   = EA < 16 ? EA : 16;
#pragma unroll
          for(int e0 = 0; e0 < EA; e0 += U) {
            int32_t off[U];
#pragma unroll
            for(int e = 0; e < U; e++) off[e] = rowA[pw + PW * (e0 + e)];
#pragma unroll
            for(int e = 0; e < U; e++) va[e0 + e] = load_now(src + off[e]);
          }
        }
        else { // element NI g + i: row p16 + 16 g, k = k16 + KS i
          int32_t ko[NI], off[GA];
#pragma unroll
          for(int i = 0; i < NI; i++) ko[i] = __shfl_sync(0xffffffffu, kA, k16 + KS * i);
#pragma unroll
          for(int g2 = 0; g2 < GA; g2++) off[g2] = rowA[p16 + 16 * g2];
#pragma unroll
          for(int i = 0; i < NI; i++) {
            const double* src = as + ko[i];
#pragma unroll
            for(int g2 = 0; g2 < GA; g2++) va[NI * g2 + i] = load_now(src + off[g2]);
          }
        }
        if(b_kfast) { // element e: column pw + PW e, k = lane
          const double* src = bs + kB;
          int32_t       off[EB];
#pragma unroll
          for(int e = 0; e < EB; e++) off[e] = colB[pw + PW * e];
#pragma unroll
          for(int e = 0; e < EB; e++) vb[e] = load_now(src + off[e]);
        }
        else { // element NI g + i: column p16 + 16 g, k = k16 + KS i
          int32_t ko[NI], off[GB];
#pragma unroll
          for(int i = 0; i < NI; i++) ko[i] = __shfl_sync(0xffffffffu, kB, k16 + KS * i);
#pragma unroll
          for(int g2 = 0; g2 < GB; g2++) off[g2] = colB[p16 + 16 * g2];
#pragma unroll
          for(int i = 0; i < NI; i++) {
            const double* src = bs + ko[i];
#pragma unroll
            for(int g2 = 0; g2 < GB; g2++) vb[NI * g2 + i] = load_now(src + off[g2]);
          }
        }
        // on to the next chunk while the loads are on their way
        const int first_step = st > 0 && k0 == 0;
        pos++;
        k0 += BK;
        fresh = false;
        if(k0 >= K) {
          k0 = 0;
          if(++st >= ARBR) {
            st = 0;
            t++;
            fresh = true;
            tslot ^= 1;
          }
        }
        if(!fresh) chunk_offsets();
        bad |= !mbar_wait(&s.empty[stage], phase ^ 1, p.err, 32); // (agreed on at the next barrier)
        if(kvalid < BK) { // the task's last chunk
#pragma unroll
          for(int e = 0; e < EA; e++)
            if((a_kfast ? lane : k16 + KS * (e % NI)) >= kvalid) va[e] = 0.0;
#pragma unroll
          for(int e = 0; e < EB; e++)
            if((b_kfast ? lane : k16 + KS * (e % NI)) >= kvalid) vb[e] = 0.0;
        }
        if(a_kfast) {
#pragma unroll
          for(int e = 0; e < EA; e++) s.As[stage][pw + PW * e][swz(pw + PW * e, lane)] = va[e];
        }
        else {
#pragma unroll
          for(int e = 0; e < EA; e++) s.As[stage][p16 + 16 * (e / NI)][swz(p16, k16 + KS * (e % NI))] = va[e];
        }
        if(b_kfast) {
#pragma unroll
          for(int e = 0; e < EB; e++) s.Bs[stage][lane][swz(lane, pw + PW * e)] = vb[e];
        }
        else {
#pragma unroll
          for(int e = 0; e < EB; e++)
            s.Bs[stage][k16 + KS * (e % NI)][swz(k16 + KS * (e % NI), p16) + 16 * (e / NI)] = vb[e];
        }
        if(pt == 0)
          s.sd[stage] = StageInfo{kvalid, c + 1 >= it.nchunks || t >= te, close && p.sum != nullptr, first_step};
        mbar_arrive(&s.full[stage]); // (release: this thread's elements, the chunk's record, the tile's geometry)
        if(++stage == T::ST) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    else n--; // (the geometry slot stays free)
    if(p.ctr == nullptr) break;
    if(pt == 0) {
      int next = (int) gridDim.x + atomicAdd(p.ctr, 1);
      if(p.ws == nullptr) // (so that only a CTA's first item can be one to skip: s.next is not written twice between barriers)
        while(next < p.nitems && p.items[next].part > 0) next = (int) gridDim.x + atomicAdd(p.ctr, 1);
      s.next = next;
    }
    if(producers_any<PT>(bad)) goto failed;
    x = s.next;
  }
  // no more items
  if(!bad && mbar_wait(&s.empty[stage], phase ^ 1, p.err, 33)) {
    if(pt == 0) s.sd[stage] = StageInfo{-1, 1, 0, 0};
    mbar_arrive(&s.full[stage]);
  }
failed:;
}

// The consumer warps: DMMA over the staged chunks, then the tile's epilogue.  A warp's two
// m16 fragments lie 16 * WM rows apart, so that a tile with half its rows takes half the
// time on every tensor pipe.  Warps never wait for each other: each closes, sums and
// writes its own piece of the tile.
template<class T>
__device__ __forceinline__ void consume(const Params& p, Smem<T>& s) {
  constexpr int BM = T::BM, BN = T::BN, NJ = T::NJ, CT = T::CT;
  const int     tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lg = lane >> 2, lt = lane & 3;
  const int     wr = (warp % T::WM) * 16, wn = (warp / T::WM) * (BN / T::WN);
  int           stage = 0;
  uint32_t      phase = 0;
  auto          mrow  = [&](int i) { return wr + i * 16 * T::WM; }; // first row of fragment i
  for(int n = 0;; n++) {
    if(!mbar_wait_warp(&s.full[stage], phase, p.err, 34) || s.sd[stage].kvalid < 0) return;
    const TileGeo<T>& geo   = s.geo[n & 1];
    const int         m_lim = geo.m_lim, n_lim = geo.n_lim;
    const int  nj    = m_lim > wr ? max(0, min(NJ, (n_lim - wn + 7) >> 3)) : 0;
    const bool two   = mrow(1) < m_lim;
    const bool whole = two && 5 * nj >= 4 * NJ; // (computed in full: its empty columns cost less than tests)
    bool       closed = false; // segments before the current one are summed up in p.sum
    double     acc[2][NJ][4];
#pragma unroll
    for(int i = 0; i < 2; i++)
#pragma unroll
      for(int j = 0; j < NJ; j++)
#pragma unroll
        for(int h = 0; h < 4; h++) acc[i][j][h] = 0.0;
    auto reg = [&](int i, int j, int h) { return ((i * NJ + j) * 4 + h) * CT; }; // slot of an accumulator
    auto has = [&](int i, int j) { return j < nj && (i == 0 || two); };
    for(bool last = false, first = true; !last; first = false) {
      if(!first && !mbar_wait_warp(&s.full[stage], phase, p.err, 35)) return;
      const StageInfo d = s.sd[stage];
      last              = d.last != 0;
      if(d.first_step) { // beta chaining of A-only x B-only reduction steps (gemm_wrapper)
#pragma unroll
        for(int i = 0; i < 2; i++)
#pragma unroll
          for(int j = 0; j < NJ; j++)
#pragma unroll
            for(int h = 0; h < 4; h++) acc[i][j][h] *= p.beta;
      }
      if(d.close) { // the sums of the segments so far, in this CTA's part of p.sum
        double* const w = p.sum + (int64_t) blockIdx.x * (BM * BN) + tid;
#pragma unroll
        for(int i = 0; i < 2; i++)
#pragma unroll
          for(int j = 0; j < NJ; j++)
#pragma unroll
            for(int h = 0; h < 4; h++) {
              if(has(i, j)) __stcg(w + reg(i, j, h), closed ? __ldcg(w + reg(i, j, h)) + acc[i][j][h] : acc[i][j][h]);
              acc[i][j][h] = 0.0;
            }
        closed = true;
      }
      auto load_a = [&](int i, int k8, double (&a)[4]) {
        const int r = mrow(i) + lg;
        a[0]        = s.As[stage][r][swz(r, k8 + lt)];
        a[1]        = s.As[stage][r + 8][swz(r + 8, k8 + lt)];
        a[2]        = s.As[stage][r][swz(r, k8 + lt + 4)];
        a[3]        = s.As[stage][r + 8][swz(r + 8, k8 + lt + 4)];
      };
      auto load_b = [&](int j, int k8, double (&b)[2]) {
        b[0] = s.Bs[stage][k8 + lt][swz(k8 + lt, wn + 8 * j + lg)];
        b[1] = s.Bs[stage][k8 + lt + 4][swz(k8 + lt + 4, wn + 8 * j + lg)];
      };
      if(whole && d.kvalid > BK - 8) { // the next step's fragments load while this one's products run
        double a[2][2][4], b[2][NJ][2];
        auto   load = [&](int k8, int buf) {
#pragma unroll
          for(int i = 0; i < 2; i++) load_a(i, k8, a[buf][i]);
#pragma unroll
          for(int j = 0; j < NJ; j++) load_b(j, k8, b[buf][j]);
        };
        load(0, 0);
#pragma unroll
        for(int k8 = 0; k8 < BK; k8 += 8) {
          const int buf = (k8 >> 3) & 1;
          if(k8 + 8 < BK) load(k8 + 8, buf ^ 1);
#pragma unroll
          for(int j = 0; j < NJ; j++) {
            dmma16(acc[0][j], a[buf][0], b[buf][j]);
            dmma16(acc[1][j], a[buf][1], b[buf][j]);
          }
        }
      }
      else if(nj > 0) { // only the fragments that reach into the output block, the K steps that reach into the task
#pragma unroll 1
        for(int k8 = 0; k8 < d.kvalid; k8 += 8) {
          double a[2][4];
          load_a(0, k8, a[0]);
          if(two) load_a(1, k8, a[1]);
#pragma unroll
          for(int j = 0; j < NJ; j++)
            if(j < nj) {
              double b[2];
              load_b(j, k8, b);
              dmma16(acc[0][j], a[0], b);
              if(two) dmma16(acc[1][j], a[1], b);
            }
        }
      }
      __syncwarp();
      if(lane == 0) mbar_arrive(&s.empty[stage]);
      if(++stage == T::ST) {
        stage = 0;
        phase ^= 1;
      }
    }
    if(closed) {
      const double* w = p.sum + (int64_t) blockIdx.x * (BM * BN) + tid;
#pragma unroll
      for(int i = 0; i < 2; i++)
#pragma unroll
        for(int j = 0; j < NJ; j++)
#pragma unroll
          for(int h = 0; h < 4; h++)
            if(has(i, j)) acc[i][j][h] = __ldcg(w + reg(i, j, h)) + acc[i][j][h];
    }
    bool write = true;
    if(geo.nparts > 1) {
      // split reduction: this segment's accumulators to the workspace, one slot per thread
      // and register so that every access is a full line; of the tile's CTAs, the one
      // whose warp arrives last sums this warp's piece over the segments, in order
      double* const w0 = p.ws + (int64_t) geo.ws * (BM * BN) + tid;
      double* const w  = w0 + (int64_t) geo.part * (BM * BN);
#pragma unroll
      for(int i = 0; i < 2; i++)
#pragma unroll
        for(int j = 0; j < NJ; j++)
#pragma unroll
          for(int h = 0; h < 4; h++)
            if(has(i, j)) __stcg(w + reg(i, j, h), acc[i][j][h]);
      write = warp_arrives_last(p.cnt + (int64_t) geo.ws * T::NC + warp, geo.nparts, lane);
      if(write) {
        for(int part = 0; part < geo.nparts; part++) {
          const double* r = w0 + (int64_t) part * (BM * BN);
#pragma unroll
          for(int i = 0; i < 2; i++)
#pragma unroll
            for(int j = 0; j < NJ; j++)
#pragma unroll
              for(int h = 0; h < 4; h++)
                if(has(i, j)) {
                  const double v = __ldcg(r + reg(i, j, h));
                  acc[i][j][h]   = part == 0 ? v : acc[i][j][h] + v;
                }
        }
      }
    }
    if(write && p.energy) { // sum (C + alpha * acc)^2 / D over the piece, C unchanged; a partial per warp
      double e = 0.0;
#pragma unroll
      for(int i = 0; i < 2; i++) {
#pragma unroll
        for(int hr = 0; hr < 2; hr++) {
          const int m = mrow(i) + 8 * hr + lg;
          if(m >= m_lim) continue;
          const double* crow = p.C + geo.c_base + geo.rowC[m];
          const double  dr   = geo.rowD[m];
#pragma unroll
          for(int j = 0; j < NJ; j++) {
#pragma unroll
            for(int h = 0; h < 2; h++) {
              const int c = wn + 8 * j + 2 * lt + h;
              if(c >= n_lim) continue;
              const double w = __ldcs(crow + geo.colC[c]) + p.alpha * acc[i][j][2 * hr + h];
              e              = fma(w * w, recip_nr(dr + geo.colD[c]), e);
            }
          }
        }
      }
#pragma unroll
      for(int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
      if(lane == 0) p.en.part[(int64_t) geo.tile * T::NC + warp] = e;
    }
    else if(write && nj > 0) { // C (=|+=) alpha * acc in C's own layout, a row's old values in flight together
#pragma unroll
      for(int i = 0; i < 2; i++) {
#pragma unroll
        for(int hr = 0; hr < 2; hr++) {
          const int m = mrow(i) + 8 * hr + lg;
          if(m >= m_lim) continue;
          double* const crow = p.C + geo.c_base + geo.rowC[m];
          double        old[NJ][2];
#pragma unroll
          for(int j = 0; j < NJ; j++)
#pragma unroll
            for(int h = 0; h < 2; h++) {
              const int c = wn + 8 * j + 2 * lt + h;
              old[j][h]   = (!p.is_assign && c < n_lim) ? crow[geo.colC[c]] : 0.0;
            }
#pragma unroll
          for(int j = 0; j < NJ; j++)
#pragma unroll
            for(int h = 0; h < 2; h++) {
              const int c = wn + 8 * j + 2 * lt + h;
              if(c >= n_lim) continue;
              const double v    = p.alpha * acc[i][j][2 * hr + h];
              crow[geo.colC[c]] = p.is_assign ? v : old[j][h] + v;
            }
        }
      }
    }
    __syncwarp();
    if(lane == 0) mbar_arrive(&s.gempty[n & 1]);
  }
}

template<class T>
__global__ void __launch_bounds__(T::NTHREADS, T::CTAS) k_contract_fp64(const __grid_constant__ Params p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem<T>&                                      s = *reinterpret_cast<Smem<T>*>(smem_raw);
  if(threadIdx.x == 0) {
    for(int x = 0; x < T::ST; x++) {
      mbar_init(&s.full[x], T::PT);
      mbar_init(&s.empty[x], T::NC);
    }
    for(int x = 0; x < 2; x++) mbar_init(&s.gempty[x], T::NC);
    fence_mbarrier_init();
  }
  __syncthreads();
  __syncwarp(); // (setmaxnreg is warp-wide)
  if(threadIdx.x < T::CT) {
    if constexpr(T::RC > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(T::RC));
    consume<T>(p, s);
  }
  else {
    if constexpr(T::RP > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(T::RP));
    produce<T>(p, s);
  }
}

// SMs of the current device.
int sm_count() {
  int dev = 0, n = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

template<class T>
void launch_k(const Params& p, int64_t nitems, cudaStream_t stream) {
  TB_EXPECTS(nitems < (1ll << 31), "work list too large");
  const size_t smem = sizeof(Smem<T>);
  static bool  configured[64] = {false};
  int          dev            = 0;
  TB_CUDA(cudaGetDevice(&dev));
  if(dev < 64 && !configured[dev]) {
    TB_CUDA(cudaFuncSetAttribute(k_contract_fp64<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    configured[dev] = true;
  }
  k_contract_fp64<T><<<(unsigned) nitems, T::NTHREADS, smem, stream>>>(p);
  TB_CUDA(cudaGetLastError());
}

void launch_shape(const Params& p, int shape, int64_t nitems, cudaStream_t stream) {
  if(shape == 80) launch_k<Wide80>(p, nitems, stream);
  else if(shape == 64) launch_k<Wide64>(p, nitems, stream);
  else launch_k<Narrow>(p, nitems, stream);
}

// Tile extents and warps by the shape's code (its width).
struct Geo {
  int bm, bn, warps, ctas;
};
template<class T>
constexpr Geo geo_of() {
  return Geo{T::BM, T::BN, T::NC, T::CTAS};
}
Geo geo(int shape) { return shape == 80 ? geo_of<Wide80>() : shape == 64 ? geo_of<Wide64>() : geo_of<Narrow>(); }

// Sets the launch up in workspace: the item counter and the split tiles' arrival counters
// (cleared here), then a tile of accumulators per part and, for tiles of several segments
// that run whole, per CTA.  Where the arena has no room for the parts (up to 128 MB) all tiles
// run whole, closing their segments: the same bits.  Where there is no memory at all for those
// sums (82 KB per CTA) they run without closing them: the same sums in another order.
void split_space(Params& p, Workspace& w, int64_t parts, int64_t sums, int64_t grid, bool counter, const Geo& g,
                 cudaStream_t stream) {
  const int64_t tile_elems = (int64_t) g.bm * g.bn;
  for(;;) {
    if(parts == 0 && sums == 0 && !counter) return;
    const int64_t ncnt = 1 + parts * g.warps, head = (4 * ncnt + 255) / 256 * 256;
    if(void* const mem = w.get(head + 8 * (parts + sums) * tile_elems, parts == 0)) {
      double* const t = reinterpret_cast<double*>(static_cast<char*>(mem) + head);
      if(counter) p.ctr = static_cast<int32_t*>(mem);
      p.cnt = static_cast<int32_t*>(mem) + 1;
      p.ws  = parts ? t : nullptr;
      p.sum = sums ? t + parts * tile_elems : nullptr;
      if(parts || counter) TB_CUDA(cudaMemsetAsync(mem, 0, 4 * ncnt, stream));
      return;
    }
    if(parts == 0) return;
    parts = 0;
    sums  = grid;
  }
}

int64_t ceil_div(int64_t x, int64_t d) { return (x + d - 1) / d; }

void extents(const LabelClasses& lc, const DevGroup& g, int64_t& nbatch, int64_t& M, int64_t& N) {
  nbatch = M = N = 1;
  for(int j = 0; j < lc.nbatch; j++) nbatch *= g.cdims[lc.batch_c[j]];
  for(int j = 0; j < lc.nm; j++) M *= g.cdims[lc.m_c[j]];
  for(int j = 0; j < lc.nn; j++) N *= g.cdims[lc.n_c[j]];
}

// (see Labels) of indices below `count`
void set_magic(Labels& l, int n, int64_t count) {
  for(int j = 0; j < n; j++)
    l.mag[j] = l.dim[j] <= 1 ? 0 : count * l.dim[j] < (1ll << 32) ? 0xffffffffu / (uint32_t) l.dim[j] + 1 : 1;
}

void block_strides(const int32_t* dims, int n, int64_t* str) { // row-major
  int64_t s = 1;
  for(int i = n - 1; i >= 0; i--) {
    str[i] = s;
    s *= dims[i];
  }
}

GroupRec group_rec(const LabelClasses& lc, const DevGroup& g) {
  int64_t cstr[kMaxModes];
  block_strides(g.cdims, lc.nc, cstr);
  GroupRec r{};
  r.c_off    = g.c_off;
  r.task_end = g.task_end;
  r.M = r.N = 1;
  for(int j = 0; j < lc.nm; j++) {
    r.m.dim[j] = g.cdims[lc.m_c[j]];
    r.mstr[j]  = (int32_t) cstr[lc.m_c[j]];
    r.M *= r.m.dim[j];
  }
  for(int j = 0; j < lc.nn; j++) {
    r.n.dim[j] = g.cdims[lc.n_c[j]];
    r.nstr[j]  = (int32_t) cstr[lc.n_c[j]];
    r.N *= r.n.dim[j];
  }
  set_magic(r.m, lc.nm, r.M);
  set_magic(r.n, lc.nn, r.N);
  for(int j = 0; j < lc.nbatch; j++) {
    r.bdim[j] = g.cdims[lc.batch_c[j]];
    r.bstr[j] = (int32_t) cstr[lc.batch_c[j]];
  }
  return r;
}

TaskRec task_rec(const LabelClasses& lc, const DevTask& t) {
  int64_t astr[kMaxModes], bstr[kMaxModes];
  block_strides(t.adims, lc.na, astr);
  block_strides(t.bdims, lc.nb, bstr);
  TaskRec r{};
  r.a_off = t.a_off;
  r.b_off = t.b_off;
  r.pos   = t.pos;
  r.K     = 1;
  for(int j = 0; j < lc.nk; j++) {
    r.k.dim[j] = t.adims[lc.k_a[j]];
    r.kstrA[j] = (int32_t) astr[lc.k_a[j]];
    r.kstrB[j] = (int32_t) bstr[lc.k_b[j]];
    r.K *= r.k.dim[j];
  }
  set_magic(r.k, lc.nk, r.K);
  r.ARBR = r.BR = 1;
  for(int j = 0; j < lc.nar; j++) {
    r.ardim[j]  = t.adims[lc.ar_a[j]];
    r.arstrA[j] = (int32_t) astr[lc.ar_a[j]];
    r.ARBR *= r.ardim[j];
  }
  for(int j = 0; j < lc.nbr; j++) {
    r.brdim[j]  = t.bdims[lc.br_b[j]];
    r.brstrB[j] = (int32_t) bstr[lc.br_b[j]];
    r.BR *= r.brdim[j];
  }
  r.ARBR *= r.BR;
  for(int j = 0; j < lc.nm; j++) r.mstrA[j] = (int32_t) astr[lc.m_a[j]];
  for(int j = 0; j < lc.nn; j++) r.nstrB[j] = (int32_t) bstr[lc.n_b[j]];
  for(int j = 0; j < lc.nbatch; j++) {
    r.bstrA[j] = (int32_t) astr[lc.batch_a[j]];
    r.bstrB[j] = (int32_t) bstr[lc.batch_b[j]];
  }
  return r;
}

// Segments of at most this many chunks (K of 2048): long enough that closing one (a tile
// of accumulators to L2 and back, about 2 us) stays near 1 % of its time (170 us for a
// wide tile), short enough that the tiles of a contraction with few of them cover the SMs
// (a 10 x 10 output over K = 370000 ran 5.5 ms in two CTAs, 0.09 ms as segments).
constexpr int kSegment = 64;
// Bytes of workspace for split tiles, at most.
constexpr int64_t kSplitBytes = int64_t(128) << 20;

struct Extent {
  int64_t nbatch, M, N, chunks;
};

// Clocks of one chunk of a tile on an SM of its own share of the tensor pipe: the DMMA
// steps that reach into the output block and what the shape loses around them (measured
// on full tiles).
double chunk_clocks(const Geo& g, double rows, double cols) {
  return std::max(rows * cols * BK / 64.0, (double) (g.bm + g.bn) * BK / 16.0) + (g.bn == Narrow::BN ? 500.0 : 400.0);
}

// Tile shape with the shortest estimated run: the items (segments of tiles) come in waves
// of one per SM, and the run is no shorter than its longest item.  Wide tiles (80 columns,
// or 64, whichever pads the output less) take less per multiply-add, narrow ones spread
// small contractions over more SMs and waste less of a small output block.
int pick_shape(const std::vector<Extent>& ext, int sms) {
  double best = 1e300;
  int    pick = 64;
  for(int shape: {64, 80, (int) Narrow::BN}) {
    const Geo g     = geo(shape);
    double    total = 0, longest = 0, items = 0;
    for(const auto& e: ext) {
      const int64_t mt = ceil_div(e.M, g.bm), nt = ceil_div(e.N, g.bn), segs = ceil_div(e.chunks, kSegment);
      const double  c  = chunk_clocks(g, (double) ceil_div(e.M, 16) * 16 / mt, (double) ceil_div(e.N, 8) * 8 / nt);
      const double  n  = (double) e.nbatch * mt * nt;
      total += c * e.chunks * n;
      items += n * segs;
      longest = std::max(longest, c * e.chunks / segs);
    }
    const double est = std::max(std::ceil(items / sms) * (total / items), longest);
    if(est < best) {
      best = est;
      pick = shape;
    }
  }
  return pick;
}

} // namespace

static void build_items_fp64(const LabelClasses& lc, const WorkList& wl);

void launch_contract_fp64(const Plan& plan, const WorkList& wl, double alpha, double beta,
                          int is_assign, const double* A, const double* B, double* C,
                          cudaStream_t stream) {
  if(!wl.items_built) build_items_fp64(plan.lc, wl);
  if(wl.items_fp64.empty()) return;
  Params p;
  p.lc        = plan.lc;
  p.A         = A;
  p.B         = B;
  p.C         = C;
  p.groups    = reinterpret_cast<const GroupRec*>(wl.d_group_recs);
  p.tasks     = reinterpret_cast<const TaskRec*>(wl.d_task_recs);
  p.items     = wl.d_items;
  if(plan.wait_err == nullptr && !wl.waits) wl.waits = std::make_unique<WaitWord>();
  p.err       = plan.wait_err ? plan.wait_err : wl.waits->device();
  p.alpha     = alpha;
  p.beta      = beta;
  p.is_assign = is_assign;
  if(plan.energy) {
    TB_EXPECTS(!is_assign && beta == 1.0, "energy epilogue of an assignment");
    p.energy = 1;
    p.en     = *plan.energy;
  }
  TB_EXPECTS(beta == 1.0, "work lists accumulate with beta 1"); // (segments are summed)
  const Geo     g      = geo(wl.items_shape);
  const int64_t nitems = (int64_t) wl.items_fp64.size(), slots = (int64_t) sm_count() * g.ctas;
  const int64_t grid   = std::min(nitems, slots);
  Workspace     ws(plan.arena, plan.pinned, stream);
  split_space(p, ws, wl.split_parts, wl.multi_segment ? grid : 0, grid, nitems > grid, g, stream);
  p.nitems = (int) nitems;
  launch_shape(p, wl.items_shape, p.ctr ? grid : nitems, stream);
  ws.put();
  if(plan.energy) launch_energy_final(p.en.part, wl.ntiles_fp64 * g.warps, plan.energy_scale, plan.energy_out, stream);
}

// One block triple (the block kernel entry point): group and task travel in the launch's
// parameters, so that the call needs no device memory for a work list.  The tiles' K
// chunks are cut into equal parts, as many as fill the SMs.  A 744 x 400 block over K =
// 1073: 78 us per call; 826 us with a work list uploaded per call and 30 whole tiles (the
// kernel 188 us).
void launch_block_fp64(const LabelClasses& lc, const DevGroup& g1, const DevTask& t1, double alpha, double beta,
                       int is_assign, const double* A, const double* B, double* C, int* err, cudaStream_t stream) {
  Params p;
  p.lc        = lc;
  p.A         = A;
  p.B         = B;
  p.C         = C;
  p.groups    = nullptr;
  p.tasks     = nullptr;
  p.items     = nullptr;
  p.err       = err;
  p.alpha     = alpha;
  p.beta      = beta;
  p.is_assign = is_assign;
  p.single    = 1;
  p.g1        = group_rec(lc, g1);
  p.t1        = task_rec(lc, t1);
  Extent e;
  extents(lc, g1, e.nbatch, e.M, e.N);
  e.chunks = task_chunks(lc, t1);
  TB_EXPECTS(e.chunks < (1ll << 31), "contraction too long");
  const int     sms   = sm_count();
  const int     shape = pick_shape({e}, sms);
  const Geo     g     = geo(shape);
  constexpr int64_t kMinPart = 4; // chunks; below, a part's start costs more than an idle SM
  const int64_t mt = ceil_div(e.M, g.bm), nt = ceil_div(e.N, g.bn), tiles = e.nbatch * mt * nt;
  const int64_t slots = (int64_t) sms * g.ctas;
  // the number of parts whose last wave is the fullest, the fewest of equals
  int64_t nparts = 1;
  if(beta == 1.0 || (lc.nar == 0 && lc.nbr == 0)) {
    double best = 1e300;
    for(int64_t n = 1; n <= 16 && n * kMinPart <= std::max(e.chunks, kMinPart) && tiles * n <= 8 * slots; n++) {
      const double cost = (double) ceil_div(tiles * n, slots) * (double) (ceil_div(e.chunks, n) + 10); // + its start
      if(cost < best) {
        best   = cost;
        nparts = n;
      }
    }
  }
  p.mtiles  = (int) mt;
  p.ntiles  = (int) nt;
  p.nparts  = (int) nparts;
  p.nchunks = (int) e.chunks;
  TB_EXPECTS(tiles * nparts < (1ll << 31), "work list too large");
  Workspace ws(nullptr, nullptr, stream);
  split_space(p, ws, nparts > 1 ? tiles * nparts : 0, 0, 0, false, g, stream);
  launch_shape(p, shape, tiles * nparts, stream);
  ws.put();
}

// Work items of the FP64 kernel: one per (group, batch index, tile), longest group first
// so that handing them out in order balances uneven groups, and the tiles that would
// start when less than twice their own length is left per CTA slot as their segments
// (within kSplitBytes of workspace), so that all SMs finish together.  A contraction with
// few tiles and a long K (a Fock-like intermediate: 4 tiles of thousands of chunks) is
// spread over the SMs the same way.
static void build_items_fp64(const LabelClasses& lc, const WorkList& wl) {
  struct Ord {
    int64_t chunks; // of the tasks that run
    int32_t group, total, nseg;
    Extent  e;
  };
  std::vector<Ord>    order;
  std::vector<Extent> ext;
  order.reserve(wl.groups.size());
  for(size_t gi = 0; gi < wl.groups.size(); gi++) {
    const DevGroup& g = wl.groups[gi];
    if(g.task_begin == g.task_end) continue;
    Ord o{0, (int32_t) gi, wl.group_chunks[gi], 0, {}};
    for(int t = g.task_begin; t < g.task_end; t++) o.chunks += task_chunks(lc, wl.tasks[t]);
    o.nseg = (int32_t) ceil_div(o.total, kSegment);
    extents(lc, g, o.e.nbatch, o.e.M, o.e.N);
    o.e.chunks = o.chunks;
    order.push_back(o);
    ext.push_back(o.e);
  }
  std::stable_sort(order.begin(), order.end(), [](const Ord& a, const Ord& b) { return a.chunks > b.chunks; });
  const int     sms       = sm_count();
  const int     shape     = pick_shape(ext, sms);
  const Geo     gm        = geo(shape);
  const double  slots     = (double) sms * gm.ctas;
  const int64_t max_parts = kSplitBytes / (8 * gm.bm * gm.bn);
  double        left      = 0; // chunks of the tiles not handed out yet
  int64_t       ntiles    = 0;
  for(const auto& o: order) {
    const int64_t n = o.e.nbatch * ceil_div(o.e.M, gm.bm) * ceil_div(o.e.N, gm.bn);
    ntiles += n;
    left += (double) n * o.chunks;
  }
  TB_EXPECTS(ntiles < (1ll << 31), "work list too large");
  int64_t tile = 0, parts = 0;
  wl.items_fp64.clear();
  wl.items_fp64.reserve((size_t) ntiles);
  wl.multi_segment = false;
  std::vector<DevItem> segs; // the group's nonempty segments
  for(const auto& o: order) {
    const DevGroup& g = wl.groups[o.group];
    segs.clear();
    if(o.nseg > 1) {
      int32_t seg = -1;
      for(int t = g.task_begin; t < g.task_end; t++) {
        const int64_t p0 = wl.tasks[t].pos, n = task_chunks(lc, wl.tasks[t]);
        for(int64_t c = 0; c < n;) { // the task's chunks, segment by segment
          int32_t s = (int32_t) ((p0 + c) * o.nseg / o.total);
          while((int64_t) o.total * (s + 1) / o.nseg <= p0 + c) s++;
          const int64_t end = std::min(n, (int64_t) o.total * (s + 1) / o.nseg - p0);
          if(s != seg) {
            DevItem it{};
            it.task0  = t;
            it.chunk0 = (int32_t) c;
            segs.push_back(it);
            seg = s;
          }
          segs.back().nchunks += (int32_t) (end - c);
          c = end;
        }
      }
    }
    for(int64_t b = 0; b < o.e.nbatch; b++)
      for(int64_t m0 = 0; m0 < o.e.M; m0 += gm.bm)
        for(int64_t n0 = 0; n0 < o.e.N; n0 += gm.bn, tile++) {
          DevItem    it{o.group, (int32_t) b, (int32_t) m0, (int32_t) n0, g.task_begin, 0, (int32_t) o.chunks,
                     (int32_t) tile, 0, 1, 0, o.total, o.nseg};
          const bool split = segs.size() > 1 && (double) o.chunks > 0.5 * left / slots &&
                             parts + (int64_t) segs.size() <= max_parts;
          left -= (double) o.chunks;
          if(!split) {
            wl.items_fp64.push_back(it);
            wl.multi_segment |= segs.size() > 1;
            continue;
          }
          it.nparts = (int32_t) segs.size();
          it.ws     = (int32_t) parts;
          parts += it.nparts;
          for(const auto& sg: segs) {
            it.task0   = sg.task0;
            it.chunk0  = sg.chunk0;
            it.nchunks = sg.nchunks;
            wl.items_fp64.push_back(it);
            it.part++;
          }
        }
  }
  TB_EXPECTS(wl.items_fp64.size() < (1ull << 31), "work list too large");
  if(!wl.items_fp64.empty()) { // items, group and task records in one device block
    std::vector<GroupRec> gr;
    std::vector<TaskRec>  tr;
    gr.reserve(wl.groups.size());
    tr.reserve(wl.tasks.size());
    for(const auto& g: wl.groups) gr.push_back(group_rec(lc, g));
    for(const auto& t: wl.tasks) tr.push_back(task_rec(lc, t));
    GroupRec* dg = nullptr;
    TaskRec*  dt = nullptr;
    wl.tables_fp64.add(dg, gr);
    wl.tables_fp64.add(dt, tr);
    wl.tables_fp64.add(wl.d_items, wl.items_fp64);
    wl.tables_fp64.make(wl.home);
    wl.d_group_recs = reinterpret_cast<char*>(dg);
    wl.d_task_recs  = reinterpret_cast<char*>(dt);
  }
  wl.ntiles_fp64 = tile;
  wl.split_parts = parts;
  wl.items_shape = shape;
  wl.items_built = true;
}

} // namespace tb
