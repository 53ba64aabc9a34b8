// Tables of the pack kernels (dgf_jk_pack.cuh), of the kernels that build
// their pair fragments, and of the row kernels' stored form, filled by
// generated units (dgf_jk_inst_pack.cuh, dgf_jk_inst_row.cuh).
#pragma once

#include "dgf_internal.h"

namespace dgf {

// Pair fragments of the bra and ket lists of a launch.
struct PackArgs {
  const double *bra_frag, *ket_frag;
};

struct PackEntry {
  void (*launch)(const JKArgs &, const PackArgs &, int grid, cudaStream_t);  // null: the class has no pack kernel
  cudaError_t (*prepare)();
  int wpb, blocks;   // warps per block, resident blocks per SM
  bool preferred;    // the default over the row and warp kernels
};
extern PackEntry g_pack_table[kNumPairClass][kNumPairClass];

struct FragEntry {
  void (*launch)(const PairRec *, const PrimPair *, int npair, const double *sph, double *out, int grid, cudaStream_t);
  int doubles;  // per pair
};
extern FragEntry g_frag_table[kNumPairClass];

extern ClassKernel g_row_stored[kNumPairClass][kNumPairClass];  // launch null: none
extern ClassKernel g_row_batch[kNumPairClass][kNumPairClass];   // the batches' form

constexpr int kPackVariant = -6;
constexpr int kKindPack = 10;  // ClassKernel::kind
// Bound of the pair fragments a context keeps.
constexpr size_t kFragMaxBytes = (size_t)16 << 30;

}  // namespace dgf
