// Instantiation of part 3 of the quartet-class kernel table (see
// dgf_jk_inst.cuh): the row kernels.
#pragma once

#include "dgf_jk_inst.cuh"
#include "dgf_jk_row.cuh"
#include "dgf_pack.h"

namespace dgf {
namespace jkinst {

// Classes with a row kernel, and their A-chunk counts.
constexpr int row_chunks(int LA, int LB, int LC, int LD) {
  const int L = LA + LB + LC + LD;
  if (L > 5) return 0;
  const int rest = (2 * LB + 1) * (2 * LC + 1) * (2 * LD + 1);
  for (int ca = 1; ca <= 2 * LA + 1; ++ca) {
    if (LA == 2 && ca > 2 && ca < 5) continue;
    if (row::chunk_most(LA, ca) * rest <= 27) return ca;
  }
  return 2 * LA + 1;
}

constexpr int kRowCarveoutPercent = 60;

template <int LA, int LB, int LC, int LD, int CA, bool BT>
void launch_row(const JKArgs &a, int grid, int block, size_t smem, cudaStream_t s) {
  jk_row_kernel<LA, LB, LC, LD, CA, BT><<<dim3(grid, CA), block, smem, s>>>(a);
}

template <int LA, int LB, int LC, int LD, int CA>
void launch_row_stored(const JKArgs &a, int grid, int block, size_t smem, cudaStream_t s) {
  jk_row_stored_kernel<LA, LB, LC, LD, CA><<<dim3(grid, CA), block, smem, s>>>(a);
}
template <int LA, int LB, int LC, int LD, int CA>
constexpr size_t row_stored_smem() {
  return (size_t)(kRowStoredBlock / 32) * row::Shape<LA, LB, LC, LD, CA>::kPerWarp * 8;
}

template <int X, int Y>
cudaError_t prepare_row() {
  constexpr int LA = cls_la(X), LB = cls_lb(X), LC = cls_la(Y), LD = cls_lb(Y), CA = row_chunks(LA, LB, LC, LD);
  if constexpr (CA > 0) {
    using S = row::Shape<LA, LB, LC, LD, CA>;
    static_assert(S::kR == row_max_bras(X) && CA <= kRowChunksMax && S::L <= kFineMaxM, "row kernel limits");
    // One carveout for all of them (it fits their resident blocks, and the
    // rest stays L1 cache for the density gathers): an SM that changes it
    // between two kernels drains first.
    static_assert((S::smem() + 1024) * S::kMinBlocks <= (size_t)kRowCarveoutPercent * 228 * 1024 / 100, "row carveout");
    cudaError_t e = cudaSuccess;
    auto prepare = [&](auto *f) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem());
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, kRowCarveoutPercent);
    };
    prepare(jk_row_kernel<LA, LB, LC, LD, CA, false>);
    prepare(jk_row_kernel<LA, LB, LC, LD, CA, true>);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(jk_row_stored_kernel<LA, LB, LC, LD, CA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)row_stored_smem<LA, LB, LC, LD, CA>());
    return e;
  }
  return cudaSuccess;
}

template <int X, int Y>
void fill_row() {
  constexpr int LA = cls_la(X), LB = cls_lb(X), LC = cls_la(Y), LD = cls_lb(Y), CA = row_chunks(LA, LB, LC, LD);
  JKEntry &e = g_jk_table[X][Y];
  e.prepare[3] = &prepare_row<X, Y>;
  if constexpr (CA > 0) {
    using S = row::Shape<LA, LB, LC, LD, CA>;
    e.row = ClassKernel{&launch_row<LA, LB, LC, LD, CA, false>, S::kBlock, S::smem(), CA, S::kMinBlocks, kKindRow};
    g_row_batch[X][Y] = ClassKernel{&launch_row<LA, LB, LC, LD, CA, true>, S::kBlock, S::smem(), CA, S::kMinBlocks, kKindRow};
    g_row_stored[X][Y] = ClassKernel{&launch_row_stored<LA, LB, LC, LD, CA>, kRowStoredBlock,
                                     row_stored_smem<LA, LB, LC, LD, CA>(), CA, 2, kKindRow};
  }
}

}  // namespace jkinst
}  // namespace dgf

// Static initialiser filling part 3 of entry (X, Y).
#define DGF_JK_ROW_CLASS(X, Y)                                                                \
  namespace dgf {                                                                             \
  namespace {                                                                                 \
  struct RowInit_##X##_##Y {                                                                  \
    RowInit_##X##_##Y() { jkinst::fill_row<X, Y>(); }                                         \
  } g_row_init_##X##_##Y;                                                                     \
  }                                                                                           \
  }
