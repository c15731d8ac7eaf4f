// Digit split kernels (see tb_split.hpp): the staged kernel for operand blocks whose rows lie
// one after another in memory, the general kernel for all others.  Both are bound by HBM:
// 8 bytes read and S (bf16: 4) written per element.
#include "tb_split.hpp"
#include "tb_sm100.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace tb {
namespace {
using namespace sm100;

int sm_count() {
  int dev = 0, n = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

constexpr int kPadRow = -0x7fffffff; // shift marker of a padding row (no digits)

// Row exponent e with |x| * 2^-e <= 127/128 for every x of the row, so that
// round(x * 2^(8S-1-e)) has a leading balanced digit within [-127, 127].
__device__ __forceinline__ int row_exponent(double mx) {
  int e = 0;
  if(mx > 0.0) {
    const double f = frexp(mx, &e); // mx = f * 2^e, f in [0.5, 1)
    if(f > 127.0 / 128.0) e += 1;
  }
  return e;
}


// round(x * 2^sh) + bias as a 64-bit word whose bytes are the balanced digits + 128.
// For S <= 6 (|X| < 2^47) one FMA against 1.5 * 2^52 leaves the integer, rounded to
// nearest even, in the low mantissa bits (2^52 + 2^51 + X); larger S convert directly.
template<int S>
__device__ __forceinline__ uint64_t digit_word(double x, double f, uint64_t bias) {
  if constexpr(S <= 6) {
    const uint64_t t = (uint64_t) __double_as_longlong(fma(x, f, 6755399441055744.0));
    return t + (bias - ((uint64_t) 1075 << 52) - ((uint64_t) 1 << 51));
  }
  else return (uint64_t) __double2ll_rn(x * f) + bias;
}

// The two bf16 pieces of y as bit patterns: hi = bf16(y), lo = bf16(y - hi), to nearest.
__device__ __forceinline__ void bf16_pieces(double y, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat16 h = __double2bfloat16(y);
  const __nv_bfloat16 l = __double2bfloat16(y - (double) __bfloat162float(h));
  hi                    = __bfloat16_as_ushort(h);
  lo                    = __bfloat16_as_ushort(l);
}

// Staged split for operand blocks whose rows lie one after another in memory (K
// contiguous and row r at element offset r * K: e.g. v(a,b,c,d) split as rows (a,b) by
// K = (c,d)).  The unit of work is a pair of rows, one contiguous range of 2K doubles,
// brought into shared memory by one bulk copy; every element is read from HBM once, and
// both the row maxima and the digit conversion read shared memory.
//   Producer (warp 0): resolves 32 units at a time, one per lane (block by binary
// search over the per-block chunk prefix, then the unit's copy range and the fields the
// consumers need), and issues their copies in order into the stage of the group that
// takes each unit.  A CTA owns whole 8-row chunks: the four units of a chunk fill the
// same 128-byte lines of every digit plane, and lines completed by one SM within a
// short time leave L2 whole (units spread over SMs measured 1.4x slower at the size
// of the O=40/V=360 ladder's v, while as fast on a quarter of it).  The unit records
// travel in shared memory beside the stages, so a consumer reads no block record from
// global memory.
//   Consumers: independent groups of kSplitGroup warps, each group with two stages of
// its own, so a group's only synchronisation is a named barrier of its own warps.
// Warp h of a group takes the h-th K range of the row maxima and every kSplitGroup-th
// group of four 16-k chunks of the digits.  Lane (row, chunk c, quad q) reads its four
// values in an order rotated by (q + c) mod 4, so that the 16 lanes of a row hit 16
// distinct bank pairs, and the final byte permute puts the digits back in k order;
// each warp store covers the two rows of 32-byte sectors.
//   The copy covers the 16-byte aligned interior [floor16(start), floor16(end)) of the
// pair; a last element past floor16(end) is loaded with a plain load.  Units made of
// padding rows only write their exponents.  Waits are bounded: a timeout records
// `code` in *err and the warps of a group agree (bar.red) to leave together.
struct UnitMeta {
  int64_t tail_src; // element index of the unit's last element (the tail load)
  int64_t dst_off;  // byte offset of the block's digits
  int32_t exp_base; // exponent index of the unit's first row
  int32_t id, K, K_pad, tile_rows, row0, nlive, delta, tail;
  int32_t pad[3];
};
static_assert(sizeof(UnitMeta) == 64, "unit record size");

constexpr int     kSplitGroup     = 4;            // consumer warps per group
constexpr int     kSplitMaxGroups = 4;            // groups per CTA, at most
constexpr int64_t kStagedSmem     = 227 * 1024;   // dynamic shared memory of one CTA, at most
constexpr int64_t kStagedHead     = 2048;         // barriers, unit records, partial maxima
// bytes of one stage of 2 rows of K doubles (+16 for the aligned start), 128-byte multiple
__host__ __device__ constexpr int64_t staged_stage_bytes(int64_t K) {
  return (2 * K * 8 + 16 + 127) / 128 * 128;
}

// BF: two bf16 pieces, hi = bf16(x 2^-e) and lo = bf16(x 2^-e - hi), in the same layout with
// 2-byte elements: a lane's four values fill half of a 16-byte row of each piece.
// O=30/V=200 ladder, v of 4 GB: 1.11 ms (1.41 in two passes over the rows).
//
// TR: rows per operand tile (128 for A; 0 = read from the unit record).
template<int S, int TR, bool BF>
__global__ void __launch_bounds__(32 * (1 + kSplitMaxGroups * kSplitGroup), 1)
  k_split_staged(const SplitBlock* __restrict__ blocks, const int32_t* __restrict__ chunk_begin, int nblocks,
                 int nchunks, int ngroups, uint32_t stage_bytes, const double* __restrict__ src,
                 uint8_t* __restrict__ dst, int32_t* __restrict__ exps, int32_t* __restrict__ blockmax, int* err) {
  constexpr int G = kSplitGroup;
  extern __shared__ __align__(128) uint8_t sm[];
  uint64_t*     full  = reinterpret_cast<uint64_t*>(sm);           // [2 per group]
  uint64_t*     empty = full + 2 * kSplitMaxGroups;                // [2 per group]
  UnitMeta*     meta  = reinterpret_cast<UnitMeta*>(sm + 256);     // [2 per group]
  double*       part  = reinterpret_cast<double*>(sm + 1280);      // [group][parity][warp][row]
  uint8_t*      ring  = sm + kStagedHead;
  static_assert(4 * kSplitMaxGroups * 8 <= 256 && 256 + 2 * kSplitMaxGroups * 64 <= 1280, "stage records");
  static_assert(1280 + 2 * kSplitMaxGroups * G * 2 * 8 <= kStagedHead, "partial maxima");
  const int     warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int     nunits = nchunks * 4; // two rows per unit, four units per 8-row chunk
  // units of this CTA: the four of each of its chunks
  const int     myunits = ((nchunks - (int) blockIdx.x + (int) gridDim.x - 1) / (int) gridDim.x) * 4;
  if(threadIdx.x == 0) {
    for(int x = 0; x < 2 * ngroups; x++) {
      mbar_init(&full[x], 1);
      mbar_init(&empty[x], G); // one arrival per warp of the group
    }
    fence_mbarrier_init();
  }
  __syncthreads();
  if(warp == 0) {
    // ---------------- producer: 32 unit records at a time, copies in unit order -------
    // The CTA's j-th unit is unit j mod 4 of 8-row chunk blockIdx.x + (j / 4) * gridDim.x
    // (the four units of a chunk, whose digits share every 128-byte line, are written
    // by one SM close together in time); it goes to group j mod ngroups, that group's
    // stage (j / ngroups) mod 2.
    for(int jb = 0; jb < myunits; jb += 32) {
      const int jl = jb + lane;
      const int u  = jl < myunits ? ((int) blockIdx.x + (jl >> 2) * (int) gridDim.x) * 4 + (jl & 3) : nunits;
      UnitMeta  mine{};
      uintptr_t a16   = 0;
      uint32_t  bytes = 0;
      if(u < nunits) {
        const int c = u >> 2;
        int       lo = 0, hi = nblocks - 1; // last block whose first chunk is <= c
        while(lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if(__ldg(chunk_begin + mid) <= c) lo = mid;
          else hi = mid - 1;
        }
        const SplitBlock& b    = blocks[lo];
        const int         row0 = 8 * (c - __ldg(chunk_begin + lo)) + (u & 3) * 2;
        const int         K    = b.K;
        const int         nl   = max(0, min(2, b.rows - row0));
        mine.dst_off   = b.dst_off;
        mine.exp_base  = b.exp_off + row0;
        mine.id        = b.id;
        mine.K         = K;
        mine.K_pad     = b.K_pad;
        mine.tile_rows = b.tile_rows;
        mine.row0      = row0;
        mine.nlive     = nl;
        mine.tail_src  = b.src_off + (int64_t) (row0 + nl) * K - 1;
        if(nl > 0) {
          const uintptr_t start = reinterpret_cast<uintptr_t>(src + b.src_off + (int64_t) row0 * K);
          const uintptr_t end   = start + (uintptr_t) nl * K * 8;
          a16                   = start & ~uintptr_t(15);
          bytes                 = (uint32_t) ((end & ~uintptr_t(15)) - a16);
          mine.delta            = (int32_t) (start - a16);
          mine.tail             = (end & 15) ? 1 : 0;
        }
      }
      for(int t = 0; t < 32; t++) {
        if(jb + t >= myunits) break;
        const int      j     = jb + t;
        const int      x     = 2 * (j % ngroups) + ((j / ngroups) & 1);
        const uint32_t round = (uint32_t) (j / (2 * ngroups));
        if(!mbar_wait(&empty[x], (round & 1) ^ 1, err, 21)) return; // (every lane polls; all agree)
        if(lane == t) {
          meta[x] = mine;
          mbar_arrive_expect_tx(&full[x], bytes);
          if(bytes > 0)
            bulk_g2s(ring + (size_t) x * stage_bytes, reinterpret_cast<const void*>(a16), bytes, &full[x]);
        }
        __syncwarp();
      }
    }
    return;
  }
  // ---------------- consumers: groups of G warps ----------------
  const int cw = warp - 1, grp = cw / G, h = cw % G;
  if(grp >= ngroups) return;
  const int      barid = 1 + grp; // named barrier of the group (0 is __syncthreads)
  const uint64_t bias  = S >= 8 ? 0x8080808080808080ull : ((1ull << (8 * S)) - 1) / 255 * 128;
  const int      rr = lane >> 4, c = (lane >> 2) & 3, q = lane & 3; // row of the pair, chunk, quad
  const int      rot = (q + c) & 3;
  uint32_t       sel2 = 0; // byte permute taking the rotated values back to k order
#pragma unroll
  for(int pos = 0; pos < 4; pos++) {
    const int t = (pos - rot) & 3;
    sel2 |= (uint32_t) (t < 2 ? t : t + 2) << (4 * pos);
  }
  for(int j = grp; j < myunits; j += ngroups) {
    const int      par   = (j / ngroups) & 1, x = 2 * grp + par;
    const uint32_t round = (uint32_t) (j / (2 * ngroups));
    {
      const bool got = mbar_wait(&full[x], round & 1, err, 22);
      uint32_t   anyfail;
      __syncwarp(); // (the barrier counts warps)
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.eq.u32 p, %1, 0;\n\t"
                   "bar.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
                   : "=r"(anyfail)
                   : "r"((uint32_t) got), "r"(barid), "n"(32 * G)
                   : "memory");
      if(anyfail) return;
    }
    const UnitMeta m       = meta[x];
    const int      K       = m.K;
    const int      tr      = TR > 0 ? TR : m.tile_rows;
    double*        rowbase = reinterpret_cast<double*>(ring + (size_t) x * stage_bytes + m.delta);
    if(m.tail) { // the last element, past the copy's 16-byte aligned end
      if(h == 0 && lane == 0) {
        rowbase[(int64_t) m.nlive * K - 1] = __ldg(src + m.tail_src);
        // ordered before the bulk copy that later refills this stage
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      }
      asm volatile("bar.sync %0, %1;\n" ::"r"(barid), "n"(32 * G) : "memory");
    }
    // row maxima: 16 lanes per row over this warp's K range, then over the group
    const double* xr   = rowbase + (int64_t) rr * K;
    const bool    live = rr < m.nlive;
    double        mx   = 0.0;
    if(live) {
      const int span = (K + G - 1) / G, kb = h * span, ke = min(K, kb + span);
      double    m0 = 0.0, m1 = 0.0, m2 = 0.0, m3 = 0.0;
      int       k = kb + (lane & 15);
      for(; k + 48 < ke; k += 64) {
        m0 = fmax(m0, fabs(xr[k]));
        m1 = fmax(m1, fabs(xr[k + 16]));
        m2 = fmax(m2, fabs(xr[k + 32]));
        m3 = fmax(m3, fabs(xr[k + 48]));
      }
      for(; k < ke; k += 16) m0 = fmax(m0, fabs(xr[k]));
      mx = fmax(fmax(m0, m1), fmax(m2, m3));
    }
#pragma unroll
    for(int o = 8; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    // partials alternate between two buffers by unit parity: a warp writes this buffer
    // again only after the group's next barrier, which every reader of it has passed
    double* pp = part + (grp * 2 + par) * G * 2;
    if((lane & 15) == 0) pp[h * 2 + rr] = mx;
    asm volatile("bar.sync %0, %1;\n" ::"r"(barid), "n"(32 * G) : "memory");
    mx = 0.0;
#pragma unroll
    for(int w = 0; w < G; w++) mx = fmax(mx, pp[w * 2 + rr]);
    const int e = row_exponent(mx);
    if(h == 0 && (lane & 15) == 0) {
      exps[m.exp_base + rr] = e;
      if(mx > 0.0) atomicMax(blockmax + m.id, e);
    }
    if(m.nlive > 0) {
      // digits: 2^sh in one factor where it is a normal double, else as two (tiny rows)
      const int     sh   = !live ? 0 : BF ? -e : 8 * S - 1 - e;
      const bool    wide = sh > 1000 || sh < -1000;
      const double  f1 = ldexp(1.0, wide ? sh / 2 : sh), f2 = ldexp(1.0, wide ? sh - sh / 2 : 0);
      const int     row   = m.row0 + rr;
      const int     nkc   = m.K_pad * (BF ? 2 : 1) / KC;
      const int64_t dstep = (int64_t) S * tr * 16 * (BF ? 2 : 1); // 16 K elements
      uint8_t*      o = dst + m.dst_off + (int64_t) (row / tr) * nkc * S * tr * KC + ((row % tr) >> 3) * 128 +
                   (row & 7) * 16 + (BF ? (q >> 1) * S * tr * 16 + (q & 1) * 8 : q * 4) + (c + (int64_t) h * 4) * dstep;
      const int     n16     = m.K_pad / 16;
      const bool    anywide = __any_sync(0xffffffffu, wide && live);
      for(int k16 = 4 * h + c; k16 < n16; k16 += 4 * G, o += 4 * G * dstep) {
        const int k0 = k16 * 16 + q * 4;
        double    v[4];
#pragma unroll
        for(int t = 0; t < 4; t++) {
          const int kk = k0 + ((t + rot) & 3);
          v[t]         = (live && kk < K) ? xr[kk] : 0.0;
        }
        if(anywide)
#pragma unroll
          for(int t = 0; t < 4; t++) v[t] *= f2;
        if constexpr(BF) {
          uint64_t hw = 0, lw = 0;
#pragma unroll
          for(int t = 0; t < 4; t++) {
            uint32_t hb, lb;
            bf16_pieces(v[t] * f1, hb, lb);
            hw |= (uint64_t) hb << (16 * ((t + rot) & 3));
            lw |= (uint64_t) lb << (16 * ((t + rot) & 3));
          }
          __stcs(reinterpret_cast<unsigned long long*>(o), (unsigned long long) hw);
          __stcs(reinterpret_cast<unsigned long long*>(o + tr * 16), (unsigned long long) lw);
        }
        else {
          uint32_t lo[4], hi[4];
#pragma unroll
          for(int t = 0; t < 4; t++) {
            const uint64_t Y = digit_word<S>(v[t], f1, bias);
            lo[t]            = (uint32_t) Y;
            hi[t]            = (uint32_t) (Y >> 32);
          }
#pragma unroll
          for(int i = 0; i < S; i++) {
            const int p = S - 1 - i; // byte of Y holding digit i
            uint32_t  t0, t1;
            if(p < 4) {
              t0 = __byte_perm(lo[0], lo[1], p | ((p + 4) << 4));
              t1 = __byte_perm(lo[2], lo[3], p | ((p + 4) << 4));
            }
            else {
              t0 = __byte_perm(hi[0], hi[1], (p - 4) | (p << 4));
              t1 = __byte_perm(hi[2], hi[3], (p - 4) | (p << 4));
            }
            __stcs(reinterpret_cast<unsigned int*>(o + (int64_t) i * tr * 16), __byte_perm(t0, t1, sel2) ^ 0x80808080u);
          }
        }
      }
    }
    __syncwarp();
    if(lane == 0) mbar_arrive(&empty[x]); // this warp is done with the stage
  }
}

// The general split, for every block the staged kernel cannot take (permuted K, strided
// rows, rows that do not follow each other).  A work unit is a few whole rows, as many as
// keep three CTAs on an SM: their elements come in one coalesced pass - lanes along K where
// the block's stride-1 mode is a K label, else along the rows, which are then contiguous -
// into shared memory, where the row maxima and the digits are taken from them, so every
// element is read from HBM once.  Rows longer than a unit holds are read twice in segments
// (the second time from L2).  The pitch is 1 beyond a multiple of 16 doubles: stores along
// rows or along K and the digits' reads (4 rows x 4 quads of a half warp) hit 16 distinct
// bank pairs.  A warp turns the 8 rows x 16 k of a core matrix at a time: thread (row r,
// quad q) turns k = 4q..4q+3 into Y = round(x * 2^(8S-1-e)) + 0x80..80, whose plain
// base-256 bytes are the balanced digits + 128; the bytes of the 4 values are gathered per
// digit with PRMT, flipped back with one XOR and stored as one 4-byte word, so every warp
// store is a contiguous 128-byte core matrix.
// Slice layout per 32-byte K chunk of a tile: [K half (16 bytes)][digit][row][16 bytes],
// i.e. the S digits' core matrices of one K half follow each other, so that the digits
// j0..j1 of a B tile form one UMMA operand of (j1 - j0 + 1) x NT rows.
// Measured: the splits of the doubles iteration at O=40/V=160 11.3 -> 4.4 ms, t2 of the
// O=30/V=240 ladder (155 MB, rows contiguous) 277 -> 154 us, against a kernel that gathered
// 8 rows twice with a warp per row (32 sectors per load where the rows, not K, are
// contiguous) and an integer division per label and element.  The copies are 8-byte
// cp.async: loads through registers, 8 per thread in flight, took 1.7x as long.
constexpr int     kSplitThreads = 256;
constexpr int64_t kUnitBytes    = 70 * 1024;  // shared memory of a unit that leaves room for three CTAs
constexpr int64_t kUnitMax      = 200 * 1024; // of any unit: 8 rows longer than that are read in segments
// Shorter rows go to the general kernel, many to a unit: pairs of rows of K = 20 (t2 against
// an occupied-occupied intermediate, O=40/V=160) took the staged kernel 1.0 ms, it 0.1.
constexpr int     kStagedMinK   = 128;
constexpr int     kUnitRows     = 128;        // rows of a unit, at most

__host__ __device__ constexpr int64_t unit_smem(int rows, int K) { // tile and K offsets
  return (int64_t) rows * ((K + 31) / 32 * 32 + 1) * 8 + (int64_t) K * 4;
}

__device__ __forceinline__ void copy8(uint32_t dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src));
}

// x / d for 0 <= x < count: umulhi(x, mag); mag 0 for d = 1, 1 where x d may reach 2^32.
__device__ __forceinline__ int32_t decomp_mag(uint32_t x, int n, const int32_t* dims, const uint32_t* mag,
                                              const int32_t* str) {
  int32_t off = 0;
#pragma unroll
  for(int j = kMaxClass - 1; j >= 0; j--) {
    if(j >= n) continue;
    const uint32_t m = mag[j], d = dims[j];
    const uint32_t q = m == 0 ? x : m == 1 ? x / d : __umulhi(x, m);
    off += (int32_t) (x - q * d) * str[j];
    x = q;
  }
  return off;
}

template<int S, bool BF>
__global__ void __launch_bounds__(kSplitThreads, 3)
  k_split_tile(const SplitBlock* __restrict__ blocks, const int32_t* __restrict__ unit_begin, int nblocks, int nunits,
               int64_t cap, const double* __restrict__ src, uint8_t* __restrict__ dst, int32_t* __restrict__ exps,
               int32_t* __restrict__ blockmax) {
  extern __shared__ __align__(128) uint8_t sm[];
  __shared__ SplitBlock                   b; // (per-thread copies indexed by label would live in local memory)
  __shared__ int32_t                      s_row[kUnitRows], s_sh[kUnitRows];
  __shared__ double                       s_mx[kUnitRows];
  constexpr int                           NW = kSplitThreads / 32;
  double* const  tile = reinterpret_cast<double*>(sm);
  const int      tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint64_t bias = S >= 8 ? 0x8080808080808080ull : ((1ull << (8 * S)) - 1) / 255 * 128;
  // Block of unit u: the last block whose first unit is <= u (empty blocks skipped).  The
  // next unit of a CTA is usually a few blocks on, so each lane holds the first unit of one
  // of the 32 blocks after the current one, loaded one unit ahead; past them, a 32-way
  // search with one ballot per step keeps unit_begin[lo] <= u < unit_begin[hi].
  auto probe = [&](int from) {
    return from + 1 + lane < nblocks ? __ldg(unit_begin + from + 1 + lane) : 0x7fffffff;
  };
  int lo = 0, next_first = probe(0);
  for(int u = blockIdx.x; u < nunits; u += gridDim.x) {
    int hi;
    {
      const int cnt = __popc(__ballot_sync(0xffffffffu, next_first <= u));
      lo += cnt;
      hi = cnt < 32 ? lo + 1 : nblocks; // a failed probe at lo + 1 bounds the block
    }
    while(hi - lo > 1) {
      const int      step = (hi - lo + 31) >> 5, idx = lo + (lane + 1) * step;
      const unsigned le   = __ballot_sync(0xffffffffu, idx < hi && __ldg(unit_begin + idx) <= u);
      const int      cnt  = __popc(le);
      hi                  = min(hi, lo + (cnt + 1) * step);
      lo += cnt * step;
    }
    if(tid < (int) (sizeof(SplitBlock) / 4))
      reinterpret_cast<uint32_t*>(&b)[tid] = __ldg(reinterpret_cast<const uint32_t*>(blocks + lo) + tid);
    const int unit = u - __ldg(unit_begin + lo);
    next_first     = probe(lo);
    __syncthreads();
    const int rb = b.unit_rows, row0 = unit * rb, nlive = max(0, min(rb, b.rows - row0)), K = b.K;
    if(nlive == 0) { // padding rows: exponents only
      if(tid < rb) exps[b.exp_off + row0 + tid] = 0;
      __syncthreads();
      continue;
    }
    if(tid < nlive) s_row[tid] = decomp_mag(row0 + tid, b.nr, b.rdim, b.rmag, b.rstr);
    if(tid < rb) s_mx[tid] = 0.0;
    // segments of whole 64-element steps that fit the shared memory
    int kseg = K;
    if(unit_smem(rb, K) > cap) kseg = (int) ((cap / (rb * 8 + 4) - 17) / 64 * 64);
    const int  nseg  = (K + kseg - 1) / kseg;
    const int  pitch = (kseg + 31) / 32 * 32 + 1;
    int32_t*   koff  = reinterpret_cast<int32_t*>(tile + (int64_t) rb * pitch);
    const bool kfast = b.kfast != 0;
    const double* const s0 = src + b.src_off;
    for(int pass = nseg > 1 ? 0 : 1; pass < 2; pass++) { // pass 0: row maxima only
      for(int g0 = 0; g0 < K; g0 += kseg) {
        const int kn = min(kseg, K - g0), kpad = g0 + kseg < K ? kseg : b.K_pad - g0; // elements, with the zeros behind
        for(int k = tid; k < kn; k += kSplitThreads) koff[k] = decomp_mag(g0 + k, b.nk, b.kdim, b.kmag, b.kstr);
        __syncthreads();
        // all copies in flight at once, 8 bytes each (blocks start on any element)
        const uint32_t t0 = smem_u32(tile);
        if(kfast && kn >= 64) { // a warp per row, lanes along K
          for(int r = warp; r < nlive; r += NW) {
            const double*  s = s0 + s_row[r];
            const uint32_t t = t0 + r * pitch * 8;
#pragma unroll 4
            for(int k = lane; k < kn; k += 32) copy8(t + k * 8, s + koff[k]);
          }
        }
        else if(kfast) { // consecutive threads along K, wrapping to the next row
          const int dk = kSplitThreads % kn, dr = kSplitThreads / kn;
          int       k = tid % kn, r = tid / kn;
#pragma unroll 4
          while(r < nlive) {
            copy8(t0 + (r * pitch + k) * 8, s0 + s_row[r] + koff[k]);
            k += dk;
            r += dr;
            if(k >= kn) {
              k -= kn;
              r++;
            }
          }
        }
        else { // consecutive threads along the rows, wrapping to the next k
          const int dr = kSplitThreads % nlive, dk = kSplitThreads / nlive;
          int       r = tid % nlive, k = tid / nlive;
#pragma unroll 4
          while(k < kn) {
            copy8(t0 + (r * pitch + k) * 8, s0 + s_row[r] + koff[k]);
            r += dr;
            k += dk;
            if(r >= nlive) {
              r -= nlive;
              k++;
            }
          }
        }
        if(kpad > kn)
          for(int x = tid; x < nlive * (kpad - kn); x += kSplitThreads)
            tile[(x / (kpad - kn)) * pitch + kn + x % (kpad - kn)] = 0.0;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if(pass == 0 || nseg == 1) { // row maxima, a warp per row
          for(int r = warp; r < nlive; r += NW) {
            const double* t = tile + (int64_t) r * pitch;
            double        m0 = 0.0, m1 = 0.0;
            int           k = lane;
            for(; k + 32 < kn; k += 64) {
              m0 = fmax(m0, fabs(t[k]));
              m1 = fmax(m1, fabs(t[k + 32]));
            }
            if(k < kn) m0 = fmax(m0, fabs(t[k]));
            m0 = fmax(m0, m1);
#pragma unroll
            for(int o = 16; o > 0; o >>= 1) m0 = fmax(m0, __shfl_xor_sync(0xffffffffu, m0, o));
            if(lane == 0) s_mx[r] = fmax(s_mx[r], m0);
          }
        }
        __syncthreads();
        if(pass == 0) continue; // (the tile and the offsets are free again)
        if(g0 == 0 && tid < rb) {
          const double mx = s_mx[tid];
          const int    e  = row_exponent(mx);
          s_sh[tid]       = tid < nlive ? (BF ? -e : 8 * S - 1 - e) : kPadRow;
          exps[b.exp_off + row0 + tid] = e;
          if(mx > 0.0) atomicMax(blockmax + b.id, e);
        }
        __syncthreads();
        // ---- digits of the segment: core matrices of 8 rows, one per warp and step ----
        const int     r = lane >> 2, q = lane & 3, ng = (nlive + 7) >> 3;
        const int     nkc = b.K_pad * (BF ? 2 : 1) / KC, tr = b.tile_rows;
        constexpr int W = BF ? 8 : 16; // K elements of a core matrix
        const int     nw = (kpad + W - 1) / W;
        int           grp = 0, kw = warp;
        while(kw >= nw && grp < ng) { // (fewer core matrices along K than warps)
          kw -= nw;
          grp++;
        }
        while(grp < ng) {
          const int    rr = grp * 8 + r, row = row0 + grp * 8; // this lane's row in the unit, the group's first row
          const int    sh = s_sh[rr];
          const bool   live = sh != kPadRow;
          const double* t = tile + (int64_t) rr * pitch + kw * W;
          uint8_t*      o = dst + b.dst_off + (int64_t) (row / tr) * nkc * S * tr * KC + ((row % tr) >> 3) * 128 + r * 16 +
                       q * 4 + (int64_t) (g0 / W + kw) * S * tr * 16;
          // 2^sh in one factor where it is a normal double, else as two
          const bool   wide = live && (sh > 1000 || sh < -1000);
          const int    h = wide ? sh / 2 : 0;
          const double f1 = ldexp(1.0, live ? sh - h : 0), f2 = ldexp(1.0, h);
          if constexpr(BF) {
            uint32_t hi2 = 0, lo2 = 0;
#pragma unroll
            for(int x = 0; x < 2; x++) {
              double v = live ? t[2 * q + x] : 0.0;
              if(wide) v *= f2;
              uint32_t hb, lb;
              bf16_pieces(v * f1, hb, lb);
              hi2 |= hb << (16 * x);
              lo2 |= lb << (16 * x);
            }
            __stcs(reinterpret_cast<unsigned int*>(o), hi2);
            __stcs(reinterpret_cast<unsigned int*>(o + tr * 16), lo2);
          }
          else {
            uint32_t l4[4], h4[4];
#pragma unroll
            for(int x = 0; x < 4; x++) {
              double v = live ? t[4 * q + x] : 0.0;
              if(wide) v *= f2;
              const uint64_t Y = digit_word<S>(v, f1, bias);
              l4[x]            = (uint32_t) Y;
              h4[x]            = (uint32_t) (Y >> 32);
            }
#pragma unroll
            for(int i = 0; i < S; i++) {
              const int p = S - 1 - i; // byte of Y holding digit i
              uint32_t  w;
              if(p < 4) {
                const uint32_t t0 = __byte_perm(l4[0], l4[1], p | ((p + 4) << 4));
                const uint32_t t1 = __byte_perm(l4[2], l4[3], p | ((p + 4) << 4));
                w                 = __byte_perm(t0, t1, 0x5410);
              }
              else {
                const uint32_t t0 = __byte_perm(h4[0], h4[1], (p - 4) | (p << 4));
                const uint32_t t1 = __byte_perm(h4[2], h4[3], (p - 4) | (p << 4));
                w                 = __byte_perm(t0, t1, 0x5410);
              }
              __stcs(reinterpret_cast<unsigned int*>(o + (int64_t) i * tr * 16), w ^ 0x80808080u);
            }
          }
          kw += NW;
          while(kw >= nw && grp < ng) {
            kw -= nw;
            grp++;
          }
        }
        __syncthreads(); // the tile, the offsets and the unit's records are free
      }
    }
  }
}

} // namespace

// The GEMM view of one operand block: rows = the outer labels (positions rpos, in C's
// order), K = the inner labels (positions kpos, in A's order), element strides of the
// block's row-major layout; tile_rows / kstep set the padding.
static void split_magic(uint32_t* mag, const int32_t* dim, int n, int64_t count) {
  for(int j = 0; j < n; j++)
    mag[j] = dim[j] <= 1 ? 0 : count * dim[j] < (1ll << 32) ? 0xffffffffu / (uint32_t) dim[j] + 1 : 1;
}

// The rows of a general unit: the most that divide the tile's rows into whole 8-row groups
// and leave room for three CTAs on an SM (at least 8).
static int rows_per_unit(int tile_rows, int K) {
  for(int n = 1; n <= tile_rows / 8; n++) {
    const int rows = tile_rows / n;
    if(tile_rows % n == 0 && rows % 8 == 0 && rows <= kUnitRows && unit_smem(rows, K) <= kUnitBytes) return rows;
  }
  return 8;
}

SplitBlock view_block(const int32_t* dims, int nmodes, const int8_t* rpos, int nr, const int8_t* kpos, int nk,
                      int tile_rows, int kstep) {
  int64_t str[kMaxModes];
  int64_t st = 1;
  for(int i = nmodes - 1; i >= 0; i--) {
    str[i] = st;
    st *= dims[i];
  }
  SplitBlock b{};
  b.nr   = nr;
  b.nk   = nk;
  b.rows = 1;
  for(int j = 0; j < nr; j++) {
    b.rdim[j] = dims[rpos[j]];
    b.rstr[j] = (int32_t) str[rpos[j]];
    b.rows *= b.rdim[j];
  }
  b.K = 1;
  for(int j = 0; j < nk; j++) {
    b.kdim[j] = dims[kpos[j]];
    b.kstr[j] = (int32_t) str[kpos[j]];
    b.K *= b.kdim[j];
  }
  b.kfast = 0;
  for(int j = 0; j < nk; j++) b.kfast |= b.kstr[j] == 1 && b.kdim[j] > 1;
  split_magic(b.rmag, b.rdim, nr, b.rows);
  split_magic(b.kmag, b.kdim, nk, b.K);
  b.kcontig = 1;
  for(int j = 0; j < nk; j++) b.kcontig &= (kpos[j] == nmodes - nk + j) ? 1 : 0;
  b.tile_rows = tile_rows;
  b.unit_rows = rows_per_unit(tile_rows, b.K);
  b.rows_pad  = (int32_t) ((b.rows + tile_rows - 1) / tile_rows * tile_rows);
  b.K_pad     = (int32_t) ((b.K + kstep - 1) / kstep * kstep);
  return b;
}

// Staged-kernel eligibility: K contiguous, row r at element offset r * K, and the two
// stages of one warp group (two rows each) fit in shared memory.
static bool staged_ok(const SplitBlock& b) {
  if(!b.kcontig || b.K < kStagedMinK) return false;
  int64_t st = b.K;
  for(int j = b.nr - 1; j >= 0; j--) {
    if(b.rstr[j] != st) return false;
    st *= b.rdim[j];
  }
  return staged_stage_bytes(b.K) * 2 + kStagedHead <= kStagedSmem;
}

int64_t split_units(const SplitBlock& b) { return b.rows_pad / b.unit_rows; }

static void unit_table(SplitSet& x, bool staged) {
  x.cbegin.resize(x.blocks.size() + 1);
  int64_t n = 0;
  for(size_t i = 0; i < x.blocks.size(); i++) {
    const SplitBlock& b = x.blocks[i];
    x.cbegin[i]         = (int32_t) n;
    n += staged ? b.rows_pad / 8 : split_units(b);
    if(!staged) x.smem = std::max(x.smem, std::min(unit_smem(b.unit_rows, b.K), kUnitMax));
    TB_EXPECTS(n < (1ll << 31), "too many split row groups");
  }
  x.cbegin[x.blocks.size()] = (int32_t) n;
}

void partition_sets(const std::vector<SplitBlock>& all, SplitSet& st, SplitSet& ge) {
  for(const auto& b: all) {
    SplitSet& x = staged_ok(b) ? st : ge;
    x.blocks.push_back(b);
    x.kmax = std::max(x.kmax, b.K);
  }
  unit_table(st, true);
  unit_table(ge, false);
}

namespace {
template<int S, int TR, bool BF>
void launch_staged(const SplitSet& x, const double* src, uint8_t* slices, int32_t* exps,
                   int32_t* blockmax, int* err, cudaStream_t st) {
  const int      nblocks = (int) x.cbegin.size() - 1, nchunks = x.cbegin.back();
  const uint32_t sb      = (uint32_t) staged_stage_bytes(x.kmax);
  const int      ngroups = (int) std::min<int64_t>(kSplitMaxGroups, (kStagedSmem - kStagedHead) / (2 * (int64_t) sb));
  TB_EXPECTS(ngroups >= 1, "staged split: one group's stages must fit in shared memory");
  const size_t   smem    = kStagedHead + (size_t) 2 * ngroups * sb;
  static bool    configured[64] = {false};
  int            dev            = 0;
  TB_CUDA(cudaGetDevice(&dev));
  if(dev < 64 && !configured[dev]) {
    TB_CUDA(cudaFuncSetAttribute(k_split_staged<S, TR, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStagedSmem));
    configured[dev] = true;
  }
  const int grid = (int) std::min<int64_t>((int64_t) nchunks, sm_count()); // whole chunks per CTA
  k_split_staged<S, TR, BF><<<grid, 32 * (1 + ngroups * kSplitGroup), smem, st>>>(
    x.d_blocks, x.d_cbegin, nblocks, nchunks, ngroups, sb, src, slices, exps, blockmax, err);
}

template<int S, bool BF>
void launch_tile(const SplitBlock* d_blocks, const int32_t* d_cbegin, int nblocks, int nunits, int64_t smem,
                 const double* src, uint8_t* slices, int32_t* exps, int32_t* blockmax, cudaStream_t st) {
  static bool configured[64] = {false};
  int         dev            = 0;
  TB_CUDA(cudaGetDevice(&dev));
  if(dev < 64 && !configured[dev]) {
    TB_CUDA(cudaFuncSetAttribute(k_split_tile<S, BF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kUnitMax));
    configured[dev] = true;
  }
  const int64_t resident = std::max<int64_t>(1, std::min<int64_t>(4, 220 * 1024 / (smem + 4096)));
  const int     grid     = (int) std::min<int64_t>(nunits, sm_count() * resident);
  k_split_tile<S, BF><<<grid, kSplitThreads, (size_t) smem, st>>>(d_blocks, d_cbegin, nblocks, nunits, smem, src, slices,
                                                                  exps, blockmax);
}

template<int S, bool BF>
void split_sets_s(const SplitSet& staged, const SplitSet& general, const double* src, uint8_t* slices, int32_t* exps,
                  int32_t* blockmax, int* err, cudaStream_t st) {
  if(!general.blocks.empty() && general.cbegin.back() > 0)
    launch_tile<S, BF>(general.d_blocks, general.d_cbegin, (int) general.blocks.size(), general.cbegin.back(),
                       general.smem, src, slices, exps, blockmax, st);
  if(!staged.blocks.empty() && staged.cbegin.back() > 0) {
    // A tiles (128 rows) with the row count fixed at compile time, B tiles read it
    if(staged.blocks.front().tile_rows == MT) launch_staged<S, MT, BF>(staged, src, slices, exps, blockmax, err, st);
    else launch_staged<S, 0, BF>(staged, src, slices, exps, blockmax, err, st);
  }
  TB_CUDA(cudaGetLastError());
}
} // namespace

void split_sets(int S, bool bf, const SplitSet& staged, const SplitSet& general, const double* src, uint8_t* slices,
                int32_t* exps, int32_t* blockmax, int* err, cudaStream_t st) {
  if(bf) return split_sets_s<2, true>(staged, general, src, slices, exps, blockmax, err, st);
  switch(S) {
    case 3: return split_sets_s<3, false>(staged, general, src, slices, exps, blockmax, err, st);
    case 4: return split_sets_s<4, false>(staged, general, src, slices, exps, blockmax, err, st);
    case 5: return split_sets_s<5, false>(staged, general, src, slices, exps, blockmax, err, st);
    case 6: return split_sets_s<6, false>(staged, general, src, slices, exps, blockmax, err, st);
    case 7: return split_sets_s<7, false>(staged, general, src, slices, exps, blockmax, err, st);
    default: return split_sets_s<8, false>(staged, general, src, slices, exps, blockmax, err, st);
  }
}

void split_one(int S, const SplitBlock& b, const SplitBlock* d_block, const int32_t* d_cbegin, const double* src,
               uint8_t* slices, int32_t* exps, int32_t* blockmax, cudaStream_t st) {
  const int     n    = (int) split_units(b);
  const int64_t smem = std::min(unit_smem(b.unit_rows, b.K), kUnitMax);
  switch(S) {
    case 3: return launch_tile<3, false>(d_block, d_cbegin, 1, n, smem, src, slices, exps, blockmax, st);
    case 4: return launch_tile<4, false>(d_block, d_cbegin, 1, n, smem, src, slices, exps, blockmax, st);
    case 5: return launch_tile<5, false>(d_block, d_cbegin, 1, n, smem, src, slices, exps, blockmax, st);
    case 6: return launch_tile<6, false>(d_block, d_cbegin, 1, n, smem, src, slices, exps, blockmax, st);
    case 7: return launch_tile<7, false>(d_block, d_cbegin, 1, n, smem, src, slices, exps, blockmax, st);
    default: return launch_tile<8, false>(d_block, d_cbegin, 1, n, smem, src, slices, exps, blockmax, st);
  }
}

} // namespace tb
