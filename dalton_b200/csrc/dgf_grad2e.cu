// Two-electron part of the RHF nuclear gradient (pattern 3, the backward
// kernel): for every canonical shell quartet the derivative integrals are
// recomputed (never stored) and contracted with the symmetrised density
// product
//   G_abcd = w [2 (D1_ab D2_cd + D2_ab D1_cd)
//             - hfx/2 (D1_ac D2_bd + D2_ac D1_bd + D1_ad D2_bc + D2_ad D1_bc)],
// so that with D1 = D2 = D the sum is d/dx of 1/2 sum (pq|rs)[D_pq D_rs -
// hfx/2 D_pr D_qs] (TWOEXP -> INTEX1 -> DEROUT, DALTON/abacus/aba2tex.F:242,
// her2ave.F:91-830), and for D1 = C (a cotangent) it is half the derivative
// of <C, G(D)>.
//
// Quartets come from the Fock build's Schwarz-screened class plan; the class
// launches run beside each other on the context's forked streams.
//
// Host side; the kernels are in dgf_grad_row.cuh (dgf_grad_kernel.cuh for
// contracted bras with (ss) and (ps) kets), instantiated one class pair per
// translation unit (DGF_GRAD_CLASS, generated by the build).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dgf_ctx.h"
#include "dgf_grad_row.cuh"

using namespace dgf;
using namespace dgf::grad;

namespace dgf {
namespace grad {
GradLauncher g_grad_table[kGradClasses][kGradClasses];
GradEntry g_grad_entry[kGradClasses][kGradClasses];
}  // namespace grad
}  // namespace dgf

int dgf_plan_for(dgf_ctx *c, double thrs);         // dgf_api.cu
int dgf_finish_profile(dgf_ctx *c, cudaStream_t st);  // dgf_api.cu

namespace {

// Sums the pairs' derivatives over the atoms: a warp loads five pairs at a
// time, six lanes on a pair's values, and adds them one pair after the other
// to its own sums in shared memory (smem_acc; with more atoms than fit,
// straight to grad).
constexpr int kPairGradWarps = 4;
__global__ void __launch_bounds__(32 * kPairGradWarps)
    grad_pairs_kernel(const PairRec *__restrict__ pairs, const double *__restrict__ pg, int npair, int natom,
                      int smem_acc, double *__restrict__ grad) {
  extern __shared__ double sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n3a = 3 * natom;
  double *acc = sm + warp * n3a;
  if (smem_acc)
    for (int i = lane; i < n3a; i += 32) acc[i] = 0.0;
  __syncwarp();
  const int stride = gridDim.x * kPairGradWarps * 5;
  for (int e0 = (blockIdx.x * kPairGradWarps + warp) * 5; e0 < npair; e0 += stride) {
    const int e = e0 + lane / 6, k = lane % 6;
    const bool on = lane < 30 && e < npair;
    int at = 0;
    double v = 0.0;
    if (on) {
      at = k < 3 ? pairs[e].atA : pairs[e].atB;
      v = pg[6 * (size_t)e + k];
    }
    if (smem_acc) {
      // pair by pair, centre A before B (they may be one atom)
#pragma unroll
      for (int j = 0; j < 10; ++j) {
        if (on && lane / 3 == j) acc[3 * at + k % 3] += v;
        __syncwarp();
      }
    } else if (on && v != 0.0) {
      atomicAdd(grad + 3 * at + k % 3, v);
    }
  }
  if (smem_acc) {
    __syncthreads();
    for (int i = threadIdx.x; i < n3a; i += blockDim.x) {
      double v = 0.0;
      for (int w = 0; w < kPairGradWarps; ++w) v += sm[w * n3a + i];
      if (v != 0.0) atomicAdd(grad + i, v);
    }
  }
}

}  // namespace

static int grad_impl(dgf_ctx *c, const double *d1, const double *d2, double hfx, double thrs, double *grad,
                     cudaStream_t st) {
  if (c->maxl > 2) {
    dgf::set_error(__FILE__, __LINE__, "the two-electron gradient covers s, p and d shells");
    return DGF_ERR_UNSUPPORTED;
  }
  int r = dgf_plan_for(c, thrs);
  if (r) return r;
  cudaError_t e = cudaMemsetAsync(grad, 0, 3 * (size_t)c->natom * sizeof(double), st);
  if (e != cudaSuccess) {
    dgf::set_error(__FILE__, __LINE__, cudaGetErrorString(e));
    return DGF_ERR_CUDA;
  }
  // The densities in the working basis (D_w = C D C^T; the derivative
  // integrals do not act on the contraction coefficients).
  const size_t n2w = (size_t)c->nwf * c->nwf;
  if (!c->d_gw) {
    if (cudaMalloc(&c->d_gw, 2 * n2w * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      c->d_gw = nullptr;
      dgf::set_error(__FILE__, __LINE__, "device allocation of the working-basis densities failed");
      return DGF_ERR_NOMEM;
    }
  }
  const WorkMaps maps = ctx_maps(c);
  const bool same = (d2 == d1);
  launch_work_prep(maps, d1, c->d_gw, nullptr, 0, (int64_t)n2w, c->nsm, st);
  if (!same) launch_work_prep(maps, d2, c->d_gw + n2w, nullptr, 0, (int64_t)n2w, c->nsm, st);
  d1 = c->d_gw;
  d2 = same ? c->d_gw : c->d_gw + n2w;
  JKArgs a;
  memset(&a, 0, sizeof(a));
  a.pp = c->d_pp;
  a.sph = c->d_sph;
  a.spherical = c->spherical;
  a.nbf = c->nwf;
  a.G1 = d1;
  a.G2 = d2;
  a.grad = grad;
  a.hfx = hfx;
  a.natom = c->natom;
  a.schwarz_thr = thrs;
  a.ket_pp0 = -1;
  // Per-launch profile (dgf_set_profiling): one record per class launch,
  // kernel 5 = gradient; quartets are the plan's, primitive quartets from the
  // classes' mean primitive-pair counts.
  if (c->profiling) {
    for (cudaEvent_t ev : c->prof_ev) cudaEventDestroy(ev);
    c->prof_ev.clear();
    c->prof.clear();
  }
  // Per-pair sums, cleared with the row kernels' task counters behind them.
  const size_t npair = c->pairs.size();
  const size_t pg_bytes = 6 * npair * sizeof(double) + kRowSlots * sizeof(unsigned);
  if (!c->d_pg) {
    for (int X = 0; X < kGradClasses; ++X)
      for (int Y = 0; Y <= X; ++Y)
        if ((e = g_grad_entry[X][Y].prepare()) != cudaSuccess) {
          dgf::set_error(__FILE__, __LINE__, cudaGetErrorString(e));
          return DGF_ERR_CUDA;
        }
    if (cudaMalloc(&c->d_pg, pg_bytes) != cudaSuccess) {
      cudaGetLastError();
      c->d_pg = nullptr;
      dgf::set_error(__FILE__, __LINE__, "device allocation of the pair derivatives failed");
      return DGF_ERR_NOMEM;
    }
  }
  PairGrad pg;
  pg.out = c->d_pg;
  unsigned *work = reinterpret_cast<unsigned *>(c->d_pg + 6 * npair);
  e = cudaMemsetAsync(c->d_pg, 0, pg_bytes, st);
  static const double kBucketPrims[kNumBuckets] = {1, 2, 4, 8, 16, 32, 64};
  // Longest first over the forked streams: model operations at 3 TFLOP/s,
  // plus the time one quartet takes alone.
  struct Item {
    const ClassPlan *cp;
    double s;
  };
  std::vector<Item> items;
  for (const ClassPlan &cp : c->plan) {
    const int L = cls_la(cp.X) + cls_lb(cp.X) + cls_la(cp.Y) + cls_lb(cp.Y);
    const double nab = ncart(cls_la(cp.X)) * ncart(cls_lb(cp.X)), ncd = ncart(cls_la(cp.Y)) * ncart(cls_lb(cp.Y));
    const double prims = std::max(1.0, c->cls_avg_npp[cp.X]) * kBucketPrims[cp.bucket];
    items.push_back({&cp, (double)cp.nquartet * prims * (100.0 + 6.0 * n3(L + 1) + 30.0 * nab * ncd) / 3e12 + 1e-5 + 5e-7 * n3(L)});
  }
  std::stable_sort(items.begin(), items.end(), [](const Item &u, const Item &v) { return u.s > v.s; });
  const int nf = c->profiling ? 1 : (int)std::min<size_t>(kForkStreams, items.size());
  double load[kForkStreams] = {};
  if (e == cudaSuccess && nf > 1) e = cudaEventRecord(c->ev_fork, st);
  for (int k = 1; k < nf && e == cudaSuccess; ++k) e = cudaStreamWaitEvent(c->fork[k], c->ev_fork, 0);
  if (e != cudaSuccess) {
    dgf::set_error(__FILE__, __LINE__, cudaGetErrorString(e));
    return DGF_ERR_CUDA;
  }
  int nrow = 0;
  for (const Item &it : items) {
    const ClassPlan &cp = *it.cp;
    const int k = (int)(std::min_element(load, load + nf) - load);
    load[k] += it.s;
    cudaStream_t ls = k == 0 ? st : c->fork[k];
    a.bra = c->d_pairs + c->cls_off[cp.X];
    a.ket = c->d_pairs + c->cls_off[cp.Y] + cp.kb0;
    a.ket_off = cp.kb0;
    a.nbra = c->cls_off[cp.X + 1] - c->cls_off[cp.X];
    a.same_class = (cp.X == cp.Y);
    a.qoff = c->d_qoff + cp.off;
    a.q_begin = 0;
    a.nquartet = cp.nquartet;
    pg.bra = c->cls_off[cp.X];
    pg.ket = c->cls_off[cp.Y] + cp.kb0;
    const int L = cls_la(cp.X) + cls_lb(cp.X) + cls_la(cp.Y) + cls_lb(cp.Y);
    a.boys = c->d_boys + (size_t)(L + 1) * kBoysTableDoubles;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (c->profiling) {
      cudaEventCreate(&e0);
      cudaEventCreate(&e1);
      c->prof_ev.push_back(e0);
      c->prof_ev.push_back(e1);
      cudaEventRecord(e0, ls);
    }
    const GradEntry &g = g_grad_entry[cp.X][cp.Y];
    if (g.row && (a.spherical || g.row_cart) && cp.row_ntask > 0 && nrow < kRowSlots) {
      a.row_bra = c->d_row_bra + c->cls_off[cp.X];
      a.row_tasks = c->d_row_tasks + cp.row_off;
      a.row_task0 = 0;
      a.row_task1 = cp.row_ntask;
      a.row_work = work + nrow++;
      g.row(a, pg, std::max(1, std::min((cp.row_ntask + g.row_warps - 1) / g.row_warps, c->nsm * g.row_blocks)), ls);
    } else if (g.warp) {
      g.warp(a, pg,
             (int)std::max<int64_t>(1, std::min<int64_t>((cp.nquartet + g.warp_warps - 1) / g.warp_warps, c->nsm * 16)),
             ls);
    } else {  // contracted pairs: one thread per quartet, straight into the gradient
      g_grad_table[cp.X][cp.Y](
          a, (int)std::max<int64_t>(1, std::min<int64_t>((cp.nquartet + kGradBlock - 1) / kGradBlock, c->nsm * 8)),
          kGradBlock, ls);
    }
    if (c->profiling) {
      cudaEventRecord(e1, ls);
      dgf_class_time r;
      r.la = cls_la(cp.X);
      r.lb = cls_lb(cp.X);
      r.lc = cls_la(cp.Y);
      r.ld = cls_lb(cp.Y);
      r.precision = 64;
      r.kernel = 5;
      r.quartets = r.evaluated = cp.nquartet;
      const double bra = c->cls_avg_npp[cp.X] > 0 ? c->cls_avg_npp[cp.X] : 1.0;
      r.prim_quartets = (int64_t)std::llround((double)cp.nquartet * bra * kBucketPrims[cp.bucket]);
      r.ms = 0.0;
      c->prof.push_back(r);
    }
  }
  e = cudaGetLastError();
  for (int k = 1; k < nf; ++k) {
    cudaError_t e2 = cudaEventRecord(c->ev_join[k], c->fork[k]);
    if (e2 == cudaSuccess) e2 = cudaStreamWaitEvent(st, c->ev_join[k], 0);
    if (e == cudaSuccess) e = e2;
  }
  if (e == cudaSuccess && npair) {
    const size_t smem = (size_t)kPairGradWarps * 3 * c->natom * sizeof(double);
    const bool fits = smem <= 48 * 1024;
    const int per_block = 5 * kPairGradWarps;
    grad_pairs_kernel<<<(int)std::min<size_t>((npair + per_block - 1) / per_block, c->nsm * 2), 32 * kPairGradWarps,
                        fits ? smem : 0, st>>>(c->d_pairs, c->d_pg, (int)npair, c->natom, fits ? 1 : 0, grad);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    dgf::set_error(__FILE__, __LINE__, cudaGetErrorString(e));
    return DGF_ERR_CUDA;
  }
  if (c->profiling) return dgf_finish_profile(c, st);
  return DGF_OK;
}

// The gradient in the resolved context of c where there is one.
static int grad_direct(dgf_ctx *c, const double *d1, const double *d2, double hfx, double thrs, double *grad,
                       cudaStream_t st) {
  dgf_ctx *d = nullptr;
  if (const int r = direct_ctx(c, false, &d)) return r;
  if (d == c) return grad_impl(c, d1, d2, hfx, thrs, grad, st);
  d->profiling = c->profiling;
  const int r = grad_impl(d, d1, d2, hfx, thrs * kPrimThrs, grad, st);
  if (c->profiling) c->prof = d->prof;
  return r;
}

extern "C" int dgf_grad2e_bilinear_device(dgf_ctx *c, const double *d1, const double *d2, double hfxfac, double thrs,
                                          double *grad_device, void *stream) {
  if (!c || !d1 || !d2 || !grad_device) {
    dgf::set_error(__FILE__, __LINE__, "NULL argument");
    return DGF_ERR_ARG;
  }
  DeviceGuard g(c->device);
  return grad_direct(c, d1, d2, hfxfac, thrs, grad_device, (cudaStream_t)stream);
}

extern "C" int dgf_grad2e_device(dgf_ctx *c, const double *dmat_device, double hfxfac, double thrs,
                                 double *grad_device, void *stream) {
  return dgf_grad2e_bilinear_device(c, dmat_device, dmat_device, hfxfac, thrs, grad_device, stream);
}

extern "C" int dgf_grad2e(dgf_ctx *c, const double *dmat, double hfxfac, double thrs, double *grad) {
  if (!c || !dmat || !grad) {
    dgf::set_error(__FILE__, __LINE__, "NULL argument");
    return DGF_ERR_ARG;
  }
  DeviceGuard g(c->device);
  const size_t n2 = (size_t)c->nbf * c->nbf;
  double *d = nullptr;
  if (cudaMalloc(&d, (n2 + 3 * (size_t)c->natom) * sizeof(double)) != cudaSuccess) {
    cudaGetLastError();
    dgf::set_error(__FILE__, __LINE__, "device allocation failed");
    return DGF_ERR_NOMEM;
  }
  cudaError_t e = cudaMemcpyAsync(d, dmat, n2 * 8, cudaMemcpyHostToDevice, c->stream);
  int r = (e == cudaSuccess) ? grad_direct(c, d, d, hfxfac, thrs, d + n2, c->stream) : DGF_ERR_CUDA;
  if (r == DGF_OK) {
    e = cudaMemcpyAsync(grad, d + n2, 3 * (size_t)c->natom * 8, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
      dgf::set_error(__FILE__, __LINE__, cudaGetErrorString(e));
      r = DGF_ERR_CUDA;
    }
  }
  cudaFree(d);
  return r;
}
