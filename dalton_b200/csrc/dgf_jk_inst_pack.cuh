// Instantiation of the pack kernels, one class pair per generated unit.
#pragma once

#include "dgf_jk_inst.cuh"
#include "dgf_jk_pack.cuh"

namespace dgf {
namespace jkinst {

// Classes with a pack kernel: bras with a d or f shell and kets of at least
// five functions (three for f bras), from L = 4.
constexpr bool pack_eligible(int LA, int LB, int LC, int LD) {
  return LA >= 2 && LA + LB + LC + LD >= 4 && (2 * LC + 1) * (2 * LD + 1) >= (LA == 3 ? 3 : 5);
}
// The default among them: L > 5, where the row kernel has no form.  Every such
// class is faster than with the warp kernel (team kernel: *); ms per class on
// C5H12 / cc-pVTZ: (fd|ps) 1.77 against 3.44, (dp|dp) 1.63 / 2.21, (fs|dp)
// 1.46 / 1.80, (fp|ds) 1.39 / 2.77, (fd|dp) 1.00 / 3.32, (ff|ps) 0.35 / 1.85,
// (ff|fd) 0.19 / 2.97*; on (H2O)32 / cc-pVDZ: (dd|pp) 2.01 / 2.09, (dp|dp)
// 1.72 / 2.78, (dd|ds) 1.46 / 1.51, (dd|dp) 0.60 / 1.01, (dd|dd) 0.07 / 0.25.
constexpr bool pack_preferred(int LA, int LB, int LC, int LD) { return LA + LB + LC + LD > 5; }

template <int LA, int LB, int LC, int LD>
void launch_pack(const JKArgs &a, const PackArgs &pk, int grid, cudaStream_t s) {
  using S = pack::Shape<LA, LB, LC, LD>;
  jk_pack_kernel<LA, LB, LC, LD><<<grid, 32 * S::WPB, S::smem(S::WPB), s>>>(a, pk);
}

template <int LA, int LB, int LC, int LD>
cudaError_t prepare_pack() {
  using S = pack::Shape<LA, LB, LC, LD>;
  return cudaFuncSetAttribute(jk_pack_kernel<LA, LB, LC, LD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)S::smem(S::WPB));
}

template <int LA, int LB>
void launch_frag(const PairRec *pairs, const PrimPair *pp, int npair, const double *sph, double *out, int grid,
                 cudaStream_t s) {
  pair_frag_kernel<LA, LB><<<grid, 128, 0, s>>>(pairs, pp, npair, sph, out);
}

template <int X, int Y>
void fill_pack() {
  constexpr int LA = cls_la(X), LB = cls_lb(X), LC = cls_la(Y), LD = cls_lb(Y);
  if constexpr (X == Y && X > 0) g_frag_table[X] = FragEntry{&launch_frag<LA, LB>, pack::frag_doubles(LA, LB)};
  if constexpr (pack_eligible(LA, LB, LC, LD)) {
    using S = pack::Shape<LA, LB, LC, LD>;
    g_pack_table[X][Y] = PackEntry{&launch_pack<LA, LB, LC, LD>, &prepare_pack<LA, LB, LC, LD>, S::WPB, S::kBlocks,
                                   pack_preferred(LA, LB, LC, LD)};
  }
}

}  // namespace jkinst
}  // namespace dgf

// Static initialiser of the pack tables' entry (X, Y).
#define DGF_JK_PACK_CLASS(X, Y)                                                               \
  namespace dgf {                                                                             \
  namespace {                                                                                 \
  struct PackInit_##X##_##Y {                                                                 \
    PackInit_##X##_##Y() { jkinst::fill_pack<X, Y>(); }                                       \
  } g_pack_init_##X##_##Y;                                                                    \
  }                                                                                           \
  }
