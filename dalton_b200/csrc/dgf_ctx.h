// Context of libdgfock (the opaque dgf_ctx of the C ABI): device-resident
// shell-pair data and the per-call scratch of one molecule/basis.
#pragma once

#include <memory>

#include "../../include/dgfock.h"
#include "dgf_internal.h"
#include "dgf_work.h"

#define DGF_CUDA_CHECK(expr)                                                   \
  do {                                                                         \
    cudaError_t _e = (expr);                                                   \
    if (_e != cudaSuccess) {                                                   \
      ::dgf::set_error(__FILE__, __LINE__, std::string(#expr) + ": " + cudaGetErrorString(_e)); \
      return DGF_ERR_CUDA;                                                     \
    }                                                                          \
  } while (0)


constexpr int kCounterSlots = 256;

struct ClassPlan {
  int X, Y;
  int bucket;         // primitive-count bucket of the kets (0: one primitive pair each)
  int kb0, kb1;       // ket range of this entry: one primitive-count bucket of class Y (relative to its start)
  int64_t off;        // offset of this entry's qoff array in the plan buffer
  int64_t nquartet;
  // row kernels, Fock and gradient (row_ntask 0: none): their tasks in d_row_tasks
  int64_t row_off = 0;
  int row_ntask = 0;
};
// Task counters of the row launches of a call (kRowChunksMax each): at most 55
// plan entries, eight density slots, two operators.
constexpr int kRowSlots = 1024;

// Map between the AO basis (Dalton's contracted functions) and the
// two-electron working basis, as sparse rows: wr_* gives, for every working
// function, the AO functions it contributes to with the contraction
// coefficient (D_w = C D C^T); ac_* gives, for every AO function, the working
// functions it is made of (F = C^T F_w C).  Device copies in one allocation.
struct WorkMapHost {
  std::vector<int> wr_off, wr_idx, ac_off, ac_idx;
  std::vector<double> wr_c, ac_c;
};

// Streams the class launches of a build are spread over (the caller's is the
// first), so that the tail of one launch, or a launch too small to fill the
// GPU, runs beside others.
constexpr int kForkStreams = 8;

// A build captured as a graph (fock_impl): its options, the executable graph
// (null before the second call), kernel launches in it, calls seen.
struct dgf_graph {
  std::string key;
  cudaGraphExec_t exec;
  int64_t launches;
  int64_t seen;
};

// Kernel choices kept for a resolved context that is not made yet.
struct dgf_tuning {
  int choice[dgf::kNumPairClass][dgf::kNumPairClass][2];
  int split_ok[dgf::kNumPairClass][dgf::kNumPairClass];
};

struct dgf_ctx {
  int device = 0, nbf = 0, natom = 0, nshell = 0, spherical = 1, maxl = 0, nsm = 148;
  std::vector<double> xyz, charge;
  // AO shells: one per contracted function of a Dalton block (one-electron
  // integrals and gradients work on these)
  std::vector<int> sh_l, sh_atom, sh_ao, sh_nprim, sh_p0;
  std::vector<double> sh_a, sh_c;
  // Two-electron working basis: a block whose contracted functions share
  // primitives (a general contraction) is resolved into one shell per
  // primitive; every other block keeps one shell per contracted function.
  // nwf functions in nwshell shells; w_identity when no block was resolved
  // (the working basis is then the AO basis, function for function).
  // A context whose blocks are segmented contractions (several primitives,
  // none shared) keeps them contracted; `prim` is then a second context with
  // every contracted shell resolved into its primitives, which direct Fock
  // builds and gradients use (direct_ctx).  It is made by the first of them
  // from the copy of the basis kept here.
  bool resolve_all = false;   // this is such a second context
  bool prim_fits = false;     // the basis has a resolved form that fits every entry point
  bool prim_failed = false;   // it could not be made here (no memory): this context serves the whole builds
  bool user_tuned = false;    // a kernel was pinned on this context: it serves all calls itself, shards excepted
  dgf_ctx *prim = nullptr;
  std::unique_ptr<dgf_tuning> prim_tuning;  // copied choices `prim` starts with (null: the defaults)
  dgf_basis basis_copy = {};
  std::vector<dgf_int> basis_i;
  std::vector<double> basis_d;
  int nwf = 0, nwshell = 0, w_identity = 1;
  std::vector<int> ws_l, ws_atom, ws_ao, ws_nprim, ws_p0;
  std::vector<double> ws_a, ws_c;
  WorkMapHost wmap;
  int *d_wmap_i = nullptr;      // wr_off | wr_idx | ac_off | ac_idx
  double *d_wmap_c = nullptr;   // wr_c | ac_c
  int64_t *d_wmeta = nullptr;   // {0, nwf^2} {0, nbf^2} element offsets of the single-molecule form
  int *d_wdims = nullptr;       // {nwf, nbf, 0, 0}
  double *d_one = nullptr;      // scratch of the one-electron calls (dgf_grad.cu), made by the first of them
  // their primitive pairs beyond the two-electron lists, by class (far_pairs)
  bool far_made = false;
  int far_off[dgf::kNumPairClass + 1] = {0};
  dgf::PairRec *d_far = nullptr;
  dgf::PrimPair *d_far_pp = nullptr;
  double *d_pg = nullptr;       // two-electron gradient: derivatives per pair (6 each), then task counters
  double *d_gw = nullptr;       // working-basis densities of the two-electron gradient (2 nwf^2)
  int *d_shinfo = nullptr;      // per working shell: first function | function count (density bounds)
  // conventional form: the integral store (dgf_store_integrals) for the plan
  // of store_thrs, one block of store_nint(X, Y) values per quartet, plan
  // entry e starting at store_off[e]
  double *d_store = nullptr;
  int64_t store_doubles = 0;
  double store_thrs = -1.0;
  std::vector<int64_t> store_off;
  std::vector<dgf::PairRec> pairs;  // class-major, Schwarz-descending inside a class
  int cls_off[dgf::kNumPairClass + 1] = {0};
  // per class: bucket boundaries (relative to the class start), pairs sorted by (bucket, -Schwarz bin, shells)
  int bkt_off[dgf::kNumPairClass][dgf::kNumBuckets + 1] = {};
  double cls_avg_npp[dgf::kNumPairClass] = {};  // mean primitive pairs of a class's pairs (shard cost model)
  int cls_max_npp[dgf::kNumPairClass] = {};     // most primitive pairs of a class's pairs
  std::vector<dgf::PrimPair> pp;
  dgf::PairRec *d_pairs = nullptr;
  // ket table of single-primitive kets (JKArgs::ks_*), one entry per pair of
  // d_pairs; null when a shell index does not fit 16 bits
  int4 *d_ks_i = nullptr;
  double *d_ks_q = nullptr, *d_ks_pp = nullptr;
  dgf::PrimPair *d_pp = nullptr;
  double *d_boys = nullptr, *d_sph = nullptr;
  // row kernels: fine Boys tables, bra pairs in row order (by class, A shell,
  // primitive-count bucket, Schwarz factor descending; positions within the
  // class), the plan's tasks and the launches' task counters
  double *d_fine = nullptr;
  std::vector<int> row_bra;
  int *d_row_bra = nullptr;
  int4 *d_row_tasks = nullptr;
  size_t row_tasks_cap = 0;
  double *d_frag[dgf::kNumPairClass] = {};  // pack kernels: the classes' pair fragments, made with the first plan that uses them
  bool pack_on = false;     // the plan's fragments stay within their bound
  bool frag_short = false;  // ... but there was no memory for some of them
  unsigned *d_row_work = nullptr;
  int row_slot = 0;  // next free slot of d_row_work in the running call
  // per-call buffers
  int cap_slots = 0, cap_io = 0;
  double *d_D = nullptr, *d_Ds = nullptr, *d_Fh = nullptr, *d_io = nullptr;
  float *d_dmax = nullptr;
  // Dalton blocks and the density screen on them: block of each AO shell
  // and working shell (ws_blk_flag with kWholeBlock where the shell is its
  // whole block), each block's first AO function and function count; device
  // block Schwarz factors (nblk^2, built at the first screened call), block
  // info (ao0 | nf) and block density maxima ((1 + cap_blk_slots) x nblk^2)
  int nblk = 0;
  std::vector<int> sh_blk, ws_blk, ws_blk_flag, blk_ao0, blk_nf;
  double *d_blk_gab = nullptr;
  int *d_blk_info = nullptr;
  float *d_blk_dmax = nullptr;
  int cap_blk_slots = 0;
  unsigned long long *d_cnt = nullptr;  // kCounterSlots x 4 per-launch counters
  // quartet plan, cached by Schwarz threshold
  double plan_thrs = -1.0;
  std::vector<ClassPlan> plan;
  int64_t *d_qoff = nullptr;
  size_t qoff_cap = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaStream_t fork[kForkStreams] = {};
  cudaEvent_t ev_fork = nullptr, ev_join[kForkStreams] = {};
  std::vector<dgf_graph> graphs;
  int64_t gen = 0, graph_gen = 0;  // counts changes of plan, buffers and kernel choices; of the kept graphs
  // kernel choice per class pair and precision (-6 = pack kernel, -5 = row
  // kernel, -4 and -3 = warp kernels, -2 and -1 = team kernels, >= 0 =
  // thread-kernel variant), set by the autotuner;
  // kDefaultVariant by default
  int choice[dgf::kNumPairClass][dgf::kNumPairClass][2] = {};
  // mixed form: whether a class pair is split into FP64 and FP32 launches
  // (1: by default, where the class has no row kernel; set by the autotuner
  // to 2 where the FP32 half pays for the second pass over the class's
  // quartets, to 0 elsewhere)
  int split_ok[dgf::kNumPairClass][dgf::kNumPairClass];
  // per-class launch profiling (dgf_set_profiling)
  int profiling = 0;
  std::vector<cudaEvent_t> prof_ev;
  std::vector<dgf_class_time> prof;
};

// Bra pairs of one molecule and class for row_tasks: their row order (class
// positions), the class list, the plan's prefix sums by class position, the
// place of the first one in the launch's row_bra list, and their kets.
struct RowSource {
  const int *order;
  int n;
  const dgf::PairRec *pairs;
  const int64_t *qoff;
  int bra0, ket0, ket_end;
};
// Makes the far pairs of a context's one-electron calls (dgf_api.cu).
int far_pairs(dgf_ctx *c);

// Appends the row tasks of a launch (dgf_api.cu).
void row_tasks(const std::vector<RowSource> &src, int max_bras, int min_width, std::vector<int4> &tasks);

// Schwarz threshold of a resolved context for the caller's threshold: a
// contracted integral is a sum of primitive ones, so the primitives are
// screened more tightly than the contracted quartet would be.  At the same
// threshold the Fock matrix of H2O / 6-31G* was 2e-13 from the unscreened
// one (relative), where the contracted form drops nothing.
constexpr double kPrimThrs = 1e-3;
// The context a direct build or gradient of `c` runs in (dgf_api.cu): its
// resolved form when it has one, can be made, and no kernel was pinned on `c`;
// else itself.  A shard's context depends on the basis alone, as all ranks
// must cut the same queue: pins do not count, and where the resolved form
// cannot be made the call fails.
int direct_ctx(dgf_ctx *c, bool sharded, dgf_ctx **out);

// The single-molecule form of the AO <-> working-basis maps of a context.
inline dgf::WorkMaps ctx_maps(const dgf_ctx *c) {
  dgf::WorkMaps m;
  const size_t nr = c->wmap.wr_idx.size();
  m.nmol = 1;
  m.w_elem = c->d_wmeta;
  m.a_elem = c->d_wmeta + 2;
  m.nw = c->d_wdims;
  m.na = c->d_wdims + 1;
  m.wf_base = c->d_wdims + 2;
  m.af_base = c->d_wdims + 3;
  m.wr_off = c->d_wmap_i;
  m.wr_idx = c->d_wmap_i + (c->nwf + 1);
  m.ac_off = c->d_wmap_i + (c->nwf + 1) + nr;
  m.ac_idx = c->d_wmap_i + (c->nwf + 1) + nr + (c->nbf + 1);
  m.wr_c = c->d_wmap_c;
  m.ac_c = c->d_wmap_c + nr;
  return m;
}

// A copy to the device on one of the library's streams.  Work on other streams
// may use it once that stream has been waited for: every function that uploads
// ends with that wait, except for what only the same stream reads before.
// cudaMemcpy does not do: it may return with the data still on its way (staged
// from pageable memory, or device to device), and only the legacy stream and
// those that wait for it run after it, while the library's streams are
// non-blocking, and so may the caller's be.
inline cudaError_t upload(cudaStream_t st, void *dst, const void *src, size_t bytes,
                          cudaMemcpyKind kind = cudaMemcpyHostToDevice) {
  return cudaMemcpyAsync(dst, src, bytes, kind, st);
}

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

