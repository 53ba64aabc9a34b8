// One-electron integrals (S, T, V) and the one-electron part of the RHF
// gradient: the HER1 pieces the SCF host needs next to the Fock build
// (HER1INT, DALTON/abacus/her1drv.F; the operators' derivative integrals,
// DALTON/abacus/aba1mat.F).
//
// Both work on the shell pairs of the two-electron working basis and on the
// primitive pairs that its lists leave out (far_pairs), class by class with
// compile-time angular momenta: one thread per pair, everything in registers for s, p and d
// shells, so that no index arithmetic or local memory stands between the Boys
// functions.  A general contraction's primitives are evaluated once and mapped
// to the AO basis afterwards (S = C^T S_w C; D_w = C D C^T).  The nuclear
// attraction sums R_tuv over the nuclei before it is contracted with the
// Hermite coefficients; its gradient contracts the density with the
// differentiated coefficients first, so that a nucleus costs one R_tuv and
// three short dot products, and the force on it is summed over the warp before
// it is added.  Bound by FP64 arithmetic and the latency of the Boys function.
// Measured on (H2O)16 / cc-pVDZ (384 functions, 48 nuclei), both calls with
// their host copies: 76.4 ms with one thread per ordered pair of contracted
// shells and run-time angular momenta, 2.6 ms so.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dgf_ctx.h"
#include "dgf_grad_kernel.cuh"
#include "dgf_jk_row.cuh"

using namespace dgf;

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr double kInvR2Pi52 = 0.16906264579104438;  // 1 / sqrt(2 pi^(5/2))
constexpr int kOneBlock = 128;

struct OneArgs {
  // one class: its two-electron list, then its far pairs (far_pairs); a
  // contracted pair may be in both
  const PairRec *pairs, *far;
  const PrimPair *pp, *far_pp;
  int nnear, npair;
  const double *xyz, *charge;  // nuclei
  int natom, nwf;
  const double *boys;    // table of the order this launch needs
  double *S, *T, *V;     // half matrices in the working basis, or null
  const double *D, *W;   // gradient: working-basis weights
  double *grad;          // (natom, 3)
  int smem_acc;          // forces on the nuclei collect in shared memory
};

// f(i, j) over the component pairs of two shells: unrolled with constant
// indices, or rolled (large shells: code size).
template <bool ROLL, int NI, int NJ, typename F>
__device__ __forceinline__ void comp_loop(F &&f) {
  if constexpr (ROLL) {
#pragma unroll 1
    for (int i = 0; i < NI; ++i)
#pragma unroll 1
      for (int j = 0; j < NJ; ++j) f(i, j);
  } else {
    static_for<NI>([&](auto i) { static_for<NJ>([&](auto j) { f(i, j); }); });
  }
}

// One-dimensional overlaps S_ij = E^ij_0 for i <= I, j <= J, layout [i*(J+1)+j].
template <int I, int J>
__device__ __forceinline__ void overlap_1d(double h, double pa, double pb, double *s) {
  s[0] = 1.0;
#pragma unroll
  for (int i = 0; i <= I; ++i)
#pragma unroll
    for (int j = 0; j <= J; ++j) {
      if (i == 0 && j == 0) continue;
      double v;
      if (i > 0) {  // raise i from (i-1, j)
        v = pa * s[(i - 1) * (J + 1) + j];
        if (i > 1) v += h * (i - 1) * s[(i - 2) * (J + 1) + j];
        if (j > 0) v += h * j * s[(i - 1) * (J + 1) + j - 1];
      } else {
        v = pb * s[j - 1];
        if (j > 1) v += h * (j - 1) * s[j - 2];
      }
      s[i * (J + 1) + j] = v;
    }
}

// Kinetic energy factor of one direction, -1/2 <i| d^2/dx^2 |j> over the
// overlaps s[i][j <= J + 2].
template <int J>
__device__ __forceinline__ double kin_1d(const double *s, int i, int j, double eb) {
  const double *r = s + i * (J + 3);
  double v = eb * (2 * j + 1) * r[j] - 2.0 * eb * eb * r[j + 2];
  if (j > 1) v -= 0.5 * j * (j - 1) * r[j - 2];
  return v;
}

// The same as 1/2 <i'|j'>, over the overlaps s[i <= I + 1][j <= J + 1]: without
// kin_1d's difference of terms as large as the exponent, which for a tight
// function beside a diffuse one leaves the rounding of the tight exponent.
template <int J>
__device__ __forceinline__ double kin_sym_1d(const double *s, int i, int j, double ea, double eb) {
  constexpr int ST = J + 2;
  double v = 2.0 * ea * eb * s[(i + 1) * ST + j + 1];
  if (j > 0) v -= ea * j * s[(i + 1) * ST + j - 1];
  if (i > 0) v -= eb * i * s[(i - 1) * ST + j + 1];
  if (i > 0 && j > 0) v += 0.5 * i * j * s[(i - 1) * ST + j - 1];
  return v;
}

template <int LA, int LB, bool SPH>
__global__ void __launch_bounds__(kOneBlock) oneint_kernel(const OneArgs a) {
  constexpr int NA = ncart(LA), NB = ncart(LB), LAB = LA + LB, NH = n3(LAB);
  constexpr bool ROLL = LAB >= 3;  // component loops stay rolled (code size; tables in local memory)
  constexpr int FA = SPH && LA >= 2 ? 2 * LA + 1 : NA, FB = SPH && LB >= 2 ? 2 * LB + 1 : NB;
  __shared__ double tab[kBoysTableDoubles];
  for (int i = threadIdx.x; i < kBoysTableDoubles; i += blockDim.x) tab[i] = a.boys[i];
  __syncthreads();
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < a.npair; e += gridDim.x * blockDim.x) {
    const bool far = e >= a.nnear;
    const PairRec pr = load_pair(far ? a.far + (e - a.nnear) : a.pairs + e);
    const PrimPair *pp = (far ? a.far_pp : a.pp) + pr.pp0;
    double S[NA * NB], T[NA * NB], V[NA * NB];
#pragma unroll
    for (int k = 0; k < NA * NB; ++k) S[k] = T[k] = V[k] = 0.0;
    for (int m = 0; m < pr.npp; ++m) {
      const PrimPair P = load_prim<true>(pp + m);
      const double eb = P.p - P.ea, h = 0.5 / P.p, kab = P.K * P.p * kInvR2Pi52;
      {
        constexpr int ST = LB + 2;
        double sx[(LA + 2) * ST], sy[(LA + 2) * ST], sz[(LA + 2) * ST];
        overlap_1d<LA + 1, LB + 1>(h, P.PAx, P.PBx, sx);
        overlap_1d<LA + 1, LB + 1>(h, P.PAy, P.PBy, sy);
        overlap_1d<LA + 1, LB + 1>(h, P.PAz, P.PBz, sz);
        const double r = kPi / P.p, s0 = r * sqrt(r) * kab;
        comp_loop<ROLL, NA, NB>([&](auto ia, auto ib) {
            const int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
            const int bx = cart_x(LB, ib), by = cart_y(LB, ib), bz = cart_z(LB, ib);
            const double x = sx[ax * ST + bx], y = sy[ay * ST + by], z = sz[az * ST + bz];
            S[ia * NB + ib] += s0 * (x * y * z);
            T[ia * NB + ib] += s0 * (kin_sym_1d<LB>(sx, ax, bx, P.ea, eb) * y * z +
                                     x * kin_sym_1d<LB>(sy, ay, by, P.ea, eb) * z +
                                     x * y * kin_sym_1d<LB>(sz, az, bz, P.ea, eb));
          });
      }
      if (a.V) {
        double Rs[NH];
#pragma unroll
        for (int k = 0; k < NH; ++k) Rs[k] = 0.0;
        for (int c = 0; c < a.natom; ++c) {
          const double x = P.Px - __ldg(a.xyz + 3 * c), y = P.Py - __ldg(a.xyz + 3 * c + 1),
                       z = P.Pz - __ldg(a.xyz + 3 * c + 2);
          double F[LAB + 1], R[NH];
          boys_eval<LAB>(P.p * (x * x + y * y + z * z), tab, F);
          double s = -__ldg(a.charge + c);
#pragma unroll
          for (int n = 0; n <= LAB; ++n) {
            F[n] *= s;
            s *= -2.0 * P.p;
          }
          hermite_r_inplace<LAB, double>(F, x, y, z, R);
#pragma unroll
          for (int k = 0; k < NH; ++k) Rs[k] += R[k];
        }
        constexpr int EN = (LA + 1) * (LB + 1) * (LAB + 1);
        double ex[EN], ey[EN], ez[EN];
        herm_e<LA, LB, 1, double>(h, P.PAx, P.PBx, ex);
        herm_e<LA, LB, 1, double>(h, P.PAy, P.PBy, ey);
        herm_e<LA, LB, 1, double>(h, P.PAz, P.PBz, ez);
        const double v0 = 2.0 * kPi / P.p * kab;
        comp_loop<ROLL, NA, NB>([&](auto ia, auto ib) {
            const int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
            const int bx = cart_x(LB, ib), by = cart_y(LB, ib), bz = cart_z(LB, ib);
            double s = 0.0;
#pragma unroll (ROLL ? 1 : 16)
            for (int t = 0; t <= ax + bx; ++t)
#pragma unroll (ROLL ? 1 : 16)
              for (int u = 0; u <= ay + by; ++u) {
                double r = 0.0;
#pragma unroll (ROLL ? 1 : 16)
                for (int v = 0; v <= az + bz; ++v)
                  r += ez[(az * (LB + 1) + bz) * (LAB + 1) + v] * Rs[tuv_index(t, u, v)];
                s += ex[(ax * (LB + 1) + bx) * (LAB + 1) + t] * ey[(ay * (LB + 1) + by) * (LAB + 1) + u] * r;
              }
            V[ia * NB + ib] += v0 * s;
          });
      }
    }
    // half matrices: the epilogue adds the transpose
    const double w = pr.same ? 0.5 : 1.0;
    auto put = [&](double *M, const double *c) {
      if (!M) return;
      double f[FA * FB];
      if constexpr (SPH) {
        sph_pair<LA, LB>(c, f);
      } else {
#pragma unroll
        for (int k = 0; k < FA * FB; ++k) f[k] = c[k];
      }
#pragma unroll
      for (int k = 0; k < FA * FB; ++k) atomicAdd(M + (size_t)(pr.aoA + k / FB) * a.nwf + pr.aoB + k % FB, w * f[k]);
    };
    put(a.S, S);
    put(a.T, T);
    put(a.V, V);
  }
}

// Derivatives with respect to the centre of the bra function i of S (weight
// -W), T and V (weight D), doubled for the equal ket term; the operator term
// of V by translational invariance (the force on a nucleus is minus the two
// functions' forces).  SWAP: i is the pair's B shell (LI its momentum).
template <int LI, int LJ, bool SPH, bool SWAP>
__global__ void __launch_bounds__(kOneBlock) grad1e_kernel(const OneArgs a) {
  constexpr int NI = ncart(LI), NJ = ncart(LJ), LIJ = LI + LJ, NH = n3(LIJ + 1);
  constexpr bool ROLL = LIJ >= 3;  // component loops stay rolled (code size; tables in local memory)
  extern __shared__ double sm[];
  double *tab = sm, *acc = sm + kBoysTableDoubles;  // acc: 3 natom sums per warp
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int n3a = 3 * a.natom;
  for (int i = threadIdx.x; i < kBoysTableDoubles; i += blockDim.x) tab[i] = a.boys[i];
  if (a.smem_acc)
    for (int i = threadIdx.x; i < nwarp * n3a; i += blockDim.x) acc[i] = 0.0;
  __syncthreads();
  double *wacc = acc + warp * n3a;
  const int slot = row::warp_slot<3>(lane);
  const int stride = gridDim.x * blockDim.x;
  for (int e0 = blockIdx.x * blockDim.x + warp * 32; e0 < a.npair; e0 += stride) {
    const bool in = e0 + lane < a.npair;
    const int e = in ? e0 + lane : a.npair - 1;
    const bool far = e >= a.nnear;
    const PairRec pr = load_pair(far ? a.far + (e - a.nnear) : a.pairs + e);
    const PrimPair *pp = (far ? a.far_pp : a.pp) + pr.pp0;
    const bool work = in && !(SWAP && pr.same);
    double D[NI * NJ], W[NI * NJ];
    grad::cart_block<LI, LJ, SPH>(a.D, a.nwf, SWAP ? pr.aoB : pr.aoA, SWAP ? pr.aoA : pr.aoB, D);
    grad::cart_block<LI, LJ, SPH>(a.W, a.nwf, SWAP ? pr.aoB : pr.aoA, SWAP ? pr.aoA : pr.aoB, W);
    double gi[3] = {0.0, 0.0, 0.0};
    const int nmax = __reduce_max_sync(0xffffffffu, work ? pr.npp : 0);
    for (int m = 0; m < nmax; ++m) {
      const bool on = work && m < pr.npp;
      const PrimPair P = load_prim<true>(pp + (on ? m : 0));
      const double ea = SWAP ? P.p - P.ea : P.ea, eb = P.p - ea, h = 0.5 / P.p;
      const double kab = on ? 2.0 * P.K * P.p * kInvR2Pi52 : 0.0;
      const double PI[3] = {SWAP ? P.PBx : P.PAx, SWAP ? P.PBy : P.PAy, SWAP ? P.PBz : P.PAz};
      const double PJ[3] = {SWAP ? P.PAx : P.PBx, SWAP ? P.PAy : P.PBy, SWAP ? P.PAz : P.PBz};
      {  // overlap and kinetic energy
        constexpr int ST = LJ + 3;
        double s[3][(LI + 2) * ST];
#pragma unroll
        for (int k = 0; k < 3; ++k) overlap_1d<LI + 1, LJ + 2>(h, PI[k], PJ[k], s[k]);
        const double r = kPi / P.p, s0 = r * sqrt(r) * kab;
        double g[3] = {0.0, 0.0, 0.0};
        comp_loop<ROLL, NI, NJ>([&](auto i, auto j) {
            const int ci[3] = {cart_x(LI, i), cart_y(LI, i), cart_z(LI, i)};
            const int cj[3] = {cart_x(LJ, j), cart_y(LJ, j), cart_z(LJ, j)};
            double o[3], t[3], od[3], td[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              o[k] = s[k][ci[k] * ST + cj[k]];
              t[k] = kin_1d<LJ>(s[k], ci[k], cj[k], eb);
              od[k] = 2.0 * ea * s[k][(ci[k] + 1) * ST + cj[k]];
              td[k] = 2.0 * ea * kin_1d<LJ>(s[k], ci[k] + 1, cj[k], eb);
              if (ci[k] > 0) {
                od[k] -= ci[k] * s[k][(ci[k] - 1) * ST + cj[k]];
                td[k] -= ci[k] * kin_1d<LJ>(s[k], ci[k] - 1, cj[k], eb);
              }
            }
            const double d = D[i * NJ + j], w = W[i * NJ + j];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const int u = (k + 1) % 3, v = (k + 2) % 3;
              const double ov = od[k] * o[u] * o[v];
              const double ke = td[k] * o[u] * o[v] + od[k] * (t[u] * o[v] + o[u] * t[v]);
              g[k] += d * ke - w * ov;
            }
          });
#pragma unroll
        for (int k = 0; k < 3; ++k) gi[k] += s0 * g[k];
      }
      // nuclear attraction: H^k_tuv = sum_ij D_ij dE^ij_tuv / dI_k
      double H[3][NH];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int q = 0; q < NH; ++q) H[k][q] = 0.0;
      {
        constexpr int TT = LIJ + 2, EN = (LI + 2) * (LJ + 1) * TT;
        double E[3][EN];
#pragma unroll
        for (int k = 0; k < 3; ++k) herm_e<LI + 1, LJ, 1, double>(h, PI[k], PJ[k], E[k]);
        comp_loop<ROLL, NI, NJ>([&](auto i, auto j) {
            const int ci[3] = {cart_x(LI, i), cart_y(LI, i), cart_z(LI, i)};
            const int cj[3] = {cart_x(LJ, j), cart_y(LJ, j), cart_z(LJ, j)};
            const double d = D[i * NJ + j];
            auto ev = [&](int k, int t) -> double {
              return t <= ci[k] + cj[k] ? E[k][(ci[k] * (LJ + 1) + cj[k]) * TT + t] : 0.0;
            };
            auto dv = [&](int k, int t) -> double {
              double r = 2.0 * ea * E[k][((ci[k] + 1) * (LJ + 1) + cj[k]) * TT + t];
              if (ci[k] > 0 && t <= ci[k] - 1 + cj[k]) r -= ci[k] * E[k][((ci[k] - 1) * (LJ + 1) + cj[k]) * TT + t];
              return r;
            };
#pragma unroll (ROLL ? 1 : 16)
            for (int t = 0; t <= ci[0] + cj[0] + 1; ++t)
#pragma unroll (ROLL ? 1 : 16)
              for (int u = 0; u <= ci[1] + cj[1] + 1; ++u)
#pragma unroll (ROLL ? 1 : 16)
                for (int v = 0; v <= ci[2] + cj[2] + 1; ++v) {
                  // at most one index past the plain range (the raised one)
                  const int over = (t > ci[0] + cj[0]) + (u > ci[1] + cj[1]) + (v > ci[2] + cj[2]);
                  if (over > 1) continue;
                  const double e0 = ev(0, t), e1 = ev(1, u), e2 = ev(2, v);
                  H[0][tuv_index(t, u, v)] += d * dv(0, t) * e1 * e2;
                  H[1][tuv_index(t, u, v)] += d * e0 * dv(1, u) * e2;
                  H[2][tuv_index(t, u, v)] += d * e0 * e1 * dv(2, v);
                }
          });
      }
      const double v0 = 2.0 * kPi / P.p * kab;
      for (int c = 0; c < a.natom; ++c) {
        const double x = P.Px - __ldg(a.xyz + 3 * c), y = P.Py - __ldg(a.xyz + 3 * c + 1),
                     z = P.Pz - __ldg(a.xyz + 3 * c + 2);
        double F[LIJ + 2], R[NH];
        boys_eval<LIJ + 1>(P.p * (x * x + y * y + z * z), tab, F);
        double s = -v0 * __ldg(a.charge + c);
#pragma unroll
        for (int n = 0; n <= LIJ + 1; ++n) {
          F[n] *= s;
          s *= -2.0 * P.p;
        }
        hermite_r_inplace<LIJ + 1, double>(F, x, y, z, R);
        double f[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double q = 0.0;
#pragma unroll
          for (int n = 0; n < NH; ++n) q += H[k][n] * R[n];
          gi[k] += q;
          f[k] = -q;
        }
        const double tot = row::warp_sums<3>(f, lane);
        if (slot >= 0) {
          if (a.smem_acc)
            wacc[3 * c + slot] += tot;
          else
            atomicAdd(a.grad + 3 * c + slot, tot);
        }
      }
    }
    if (work) {
      const int at = SWAP ? pr.atB : pr.atA;
#pragma unroll
      for (int k = 0; k < 3; ++k) atomicAdd(a.grad + 3 * at + k, gi[k]);
    }
  }
  if (a.smem_acc) {
    __syncthreads();
    for (int i = threadIdx.x; i < n3a; i += blockDim.x) {
      double v = 0.0;
      for (int w = 0; w < nwarp; ++w) v += acc[w * n3a + i];
      if (v != 0.0) atomicAdd(a.grad + i, v);
    }
  }
}

template <int LA, int LB>
void launch_oneint(const OneArgs &a, bool sph, int nsm) {
  const int grid = std::min((a.npair + kOneBlock - 1) / kOneBlock, nsm * 8);
  if (sph)
    oneint_kernel<LA, LB, true><<<grid, kOneBlock>>>(a);
  else
    oneint_kernel<LA, LB, false><<<grid, kOneBlock>>>(a);
}

// Both functions of the pairs as bra, one launch each.
template <int LA, int LB>
void launch_grad1e(const OneArgs &a, bool sph, int nsm) {
  const int grid = std::min((a.npair + kOneBlock - 1) / kOneBlock, nsm * 4);
  const size_t smem = (kBoysTableDoubles + (a.smem_acc ? (size_t)(kOneBlock / 32) * 3 * a.natom : 0)) * 8;
  if (sph) {
    grad1e_kernel<LA, LB, true, false><<<grid, kOneBlock, smem>>>(a);
    grad1e_kernel<LB, LA, true, true><<<grid, kOneBlock, smem>>>(a);
  } else {
    grad1e_kernel<LA, LB, false, false><<<grid, kOneBlock, smem>>>(a);
    grad1e_kernel<LB, LA, false, true><<<grid, kOneBlock, smem>>>(a);
  }
}

typedef void (*OneLauncher)(const OneArgs &, bool, int);
const OneLauncher kOneint[kNumPairClass] = {
    launch_oneint<0, 0>, launch_oneint<1, 0>, launch_oneint<1, 1>, launch_oneint<2, 0>, launch_oneint<2, 1>,
    launch_oneint<2, 2>, launch_oneint<3, 0>, launch_oneint<3, 1>, launch_oneint<3, 2>, launch_oneint<3, 3>};
const OneLauncher kGrad1e[kNumPairClass] = {
    launch_grad1e<0, 0>, launch_grad1e<1, 0>, launch_grad1e<1, 1>, launch_grad1e<2, 0>, launch_grad1e<2, 1>,
    launch_grad1e<2, 2>, launch_grad1e<3, 0>, launch_grad1e<3, 1>, launch_grad1e<3, 2>, launch_grad1e<3, 3>};
constexpr int kPairClassL[kNumPairClass] = {0, 1, 2, 2, 3, 4, 3, 4, 5, 6};

// Atoms whose force sums of a block fit the 48 KB every launch may ask for.
constexpr int kOneSmemAtoms = 384;
// The scratch of these calls stays with the context up to this size.
constexpr size_t kOneKeepBytes = (size_t)256 << 20;

// Scratch: three working-basis matrices, three AO-basis ones, nuclei and
// charges (uploaded here), the gradient.
struct OneScratch {
  dgf_ctx *c;
  double *w = nullptr, *ao = nullptr, *xyz = nullptr, *charge = nullptr, *grad = nullptr;
  size_t n2w, n2, doubles;
  explicit OneScratch(dgf_ctx *ctx) : c(ctx) {
    n2w = (size_t)c->nwf * c->nwf;
    n2 = (size_t)c->nbf * c->nbf;
    doubles = 3 * n2w + 3 * n2 + 7 * (size_t)c->natom;
  }
  int open() {
    if (!c->d_one) {
      double *p = nullptr;
      if (cudaMalloc(&p, doubles * 8) != cudaSuccess) {
        cudaGetLastError();
        dgf::set_error(__FILE__, __LINE__, "device allocation of the one-electron scratch failed");
        return DGF_ERR_NOMEM;
      }
      c->d_one = p;
      cudaError_t e = cudaMemcpy(p + 3 * n2w + 3 * n2, c->xyz.data(), 24 * (size_t)c->natom, cudaMemcpyHostToDevice);
      if (e == cudaSuccess)
        e = cudaMemcpy(p + 3 * n2w + 3 * n2 + 3 * (size_t)c->natom, c->charge.data(), 8 * (size_t)c->natom,
                       cudaMemcpyHostToDevice);
      if (e != cudaSuccess) {
        cudaFree(p);
        c->d_one = nullptr;
        dgf::set_error(__FILE__, __LINE__, cudaGetErrorString(e));
        return DGF_ERR_CUDA;
      }
    }
    w = c->d_one;
    ao = w + 3 * n2w;
    xyz = ao + 3 * n2;
    charge = xyz + 3 * (size_t)c->natom;
    grad = charge + c->natom;
    return DGF_OK;
  }
  ~OneScratch() {
    if (c->d_one && doubles * 8 > kOneKeepBytes) {
      cudaFree(c->d_one);
      c->d_one = nullptr;
    }
  }
};

OneArgs one_args(const dgf_ctx *c, const OneScratch &s) {
  OneArgs a;
  memset(&a, 0, sizeof(a));
  a.pp = c->d_pp;
  a.far_pp = c->d_far_pp;
  a.xyz = s.xyz;
  a.charge = s.charge;
  a.natom = c->natom;
  a.nwf = c->nwf;
  return a;
}

// The pairs of class X; false: none.
bool class_pairs(const dgf_ctx *c, int X, OneArgs &a) {
  a.nnear = c->cls_off[X + 1] - c->cls_off[X];
  a.npair = a.nnear + c->far_off[X + 1] - c->far_off[X];
  a.pairs = c->d_pairs + c->cls_off[X];
  a.far = c->d_far + c->far_off[X];
  return a.npair > 0;
}

}  // namespace

extern "C" int dgf_oneint(dgf_ctx *c, double *S, double *T, double *V) {
  if (!c) {
    dgf::set_error(__FILE__, __LINE__, "ctx is NULL");
    return DGF_ERR_ARG;
  }
  DeviceGuard g(c->device);
  OneScratch s(c);
  int r = s.open();
  if (!r) r = far_pairs(c);
  if (r) return r;
  OneArgs a = one_args(c, s);
  a.S = S ? s.w : nullptr;
  a.T = T ? s.w + s.n2w : nullptr;
  a.V = V ? s.w + 2 * s.n2w : nullptr;
  cudaError_t e = cudaMemsetAsync(s.w, 0, 3 * s.n2w * 8);
  for (int X = 0; X < kNumPairClass && e == cudaSuccess; ++X) {
    if (!class_pairs(c, X, a)) continue;
    a.boys = c->d_boys + (size_t)kPairClassL[X] * kBoysTableDoubles;
    kOneint[X](a, c->spherical != 0, c->nsm);
    e = cudaGetLastError();
  }
  double *outs[3] = {S, T, V};
  const WorkMaps maps = ctx_maps(c);
  for (int k = 0; k < 3; ++k)
    if (outs[k])
      launch_work_combine(maps, s.w + k * s.n2w, s.w + k * s.n2w, s.ao + k * s.n2, 1.0, (int64_t)s.n2, c->nsm, nullptr);
  if (e == cudaSuccess) e = cudaGetLastError();
  for (int k = 0; k < 3 && e == cudaSuccess; ++k)
    if (outs[k]) e = cudaMemcpy(outs[k], s.ao + k * s.n2, s.n2 * 8, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    dgf::set_error(__FILE__, __LINE__, std::string("oneint: ") + cudaGetErrorString(e));
    return DGF_ERR_CUDA;
  }
  return DGF_OK;
}

extern "C" int dgf_grad1e(dgf_ctx *c, const double *dmat, const double *wmat, double *grad) {
  if (!c || !dmat || !wmat || !grad) {
    dgf::set_error(__FILE__, __LINE__, "NULL argument");
    return DGF_ERR_ARG;
  }
  DeviceGuard g(c->device);
  OneScratch s(c);
  int r = s.open();
  if (!r) r = far_pairs(c);
  if (r) return r;
  OneArgs a = one_args(c, s);
  cudaError_t e = cudaMemcpy(s.ao, dmat, s.n2 * 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(s.ao + s.n2, wmat, s.n2 * 8, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemsetAsync(s.grad, 0, 24 * (size_t)c->natom);
  const WorkMaps maps = ctx_maps(c);
  launch_work_prep(maps, s.ao, s.w, nullptr, 0, (int64_t)s.n2w, c->nsm, nullptr);
  launch_work_prep(maps, s.ao + s.n2, s.w + s.n2w, nullptr, 0, (int64_t)s.n2w, c->nsm, nullptr);
  a.D = s.w;
  a.W = s.w + s.n2w;
  a.grad = s.grad;
  a.smem_acc = c->natom <= kOneSmemAtoms;
  if (e == cudaSuccess) e = cudaGetLastError();
  for (int X = 0; X < kNumPairClass && e == cudaSuccess; ++X) {
    if (!class_pairs(c, X, a)) continue;
    a.boys = c->d_boys + (size_t)(kPairClassL[X] + 1) * kBoysTableDoubles;
    kGrad1e[X](a, c->spherical != 0, c->nsm);
    e = cudaGetLastError();
  }
  std::vector<double> gr(3 * (size_t)c->natom);
  if (e == cudaSuccess) e = cudaMemcpy(gr.data(), s.grad, gr.size() * 8, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    dgf::set_error(__FILE__, __LINE__, std::string("grad1e: ") + cudaGetErrorString(e));
    return DGF_ERR_CUDA;
  }
  // nuclear repulsion gradient
  for (int i = 0; i < c->natom; ++i)
    for (int j = 0; j < c->natom; ++j) {
      if (i == j) continue;
      double dx[3], r2 = 0.0;
      for (int k = 0; k < 3; ++k) {
        dx[k] = c->xyz[3 * i + k] - c->xyz[3 * j + k];
        r2 += dx[k] * dx[k];
      }
      const double r3 = r2 * std::sqrt(r2);
      for (int k = 0; k < 3; ++k) gr[3 * i + k] -= c->charge[i] * c->charge[j] * dx[k] / r3;
    }
  memcpy(grad, gr.data(), gr.size() * 8);
  return DGF_OK;
}
