// Digit split of contraction operands: FP64 blocks to balanced INT8 digit slices (S digits)
// or to two bf16 pieces, in the layout the tcgen05 contraction kernel reads.
#pragma once

#include "tb_internal.hpp"

namespace tb {

constexpr int MT = 128; // UMMA M: output rows of a tile
constexpr int KC = 32;  // bytes of K per pipeline stage (one INT8 MMA k-step)

// One operand block to split into digit slices.
struct SplitBlock {
  int64_t  src_off; // element offset in the FP64 arena
  int64_t  dst_off; // byte offset of the block's slices in the scratch
  int32_t  exp_off; // first exponent (int32 per padded row)
  int32_t  id;      // index into the per-block max-exponent array
  int32_t  rows, K, rows_pad, K_pad, tile_rows;
  int32_t  nr, nk, kcontig;
  int32_t  kfast;     // the block's stride-1 mode is one of the K labels
  int32_t  unit_rows; // general kernel: rows of a work unit
  int32_t  rdim[kMaxClass], rstr[kMaxClass];
  int32_t  kdim[kMaxClass], kstr[kMaxClass];
  uint32_t rmag[kMaxClass], kmag[kMaxClass]; // multipliers of the divisions by rdim, kdim (split_magic)
};

// Blocks split by one kernel: the staged kernel (rows contiguous) or the general one, with
// the first work unit of each block (staged: an 8-row chunk), then the total.
struct SplitSet {
  std::vector<SplitBlock> blocks;
  std::vector<int32_t>    cbegin;
  SplitBlock*             d_blocks = nullptr;
  int32_t*                d_cbegin = nullptr;
  int                     kmax     = 0;
  int64_t                 smem     = 0; // general: dynamic shared memory of the largest unit
};

SplitBlock view_block(const int32_t* dims, int nmodes, const int8_t* rpos, int nr, const int8_t* kpos, int nk,
                      int tile_rows, int kstep);
void       partition_sets(const std::vector<SplitBlock>& all, SplitSet& st, SplitSet& ge);
// Splits the blocks of one operand (bf: two bf16 pieces, S = 2): the staged kernel for the
// blocks with contiguous rows, the general kernel for the rest.
void split_sets(int S, bool bf, const SplitSet& staged, const SplitSet& general, const double* src, uint8_t* slices,
                int32_t* exps, int32_t* blockmax, int* err, cudaStream_t st);
// One block through the general kernel, its descriptor and unit table already on the device.
void    split_one(int S, const SplitBlock& b, const SplitBlock* d_block, const int32_t* d_cbegin, const double* src,
                  uint8_t* slices, int32_t* exps, int32_t* blockmax, cudaStream_t st);
int64_t split_units(const SplitBlock& b); // work units of a block in the general kernel

} // namespace tb
