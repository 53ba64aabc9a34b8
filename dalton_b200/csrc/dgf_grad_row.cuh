// Two-electron gradient kernels in relative coordinates.
//
// With P the bra's product centre and X = A - B (Q and Y = C - D on the ket),
// (ab|cd) depends on P - Q through R_tuv and on X and Y through the Hermite
// coefficients and e^{-mu X^2}, so that (Helgaker and Taylor, Theor. Chim.
// Acta 83, 177 (1992))
//   dE/dA = (a/p) dE/dP + dE/dX,   dE/dB = (b/p) dE/dP - dE/dX,
//   dE/dC = -(c/q) dE/dP + dE/dY,  dE/dD = -(d/q) dE/dP - dE/dY.
// dE/dP raises an index of R_tuv; dE^{ij}_t/dX = -2 mu X E^{ij}_t
// - (b/p) i E^{i-1,j}_t + (a/p) j E^{i,j-1}_t, whose first term is -2 mu X
// times the energy itself.  The density product G_abcd is contracted with the
// bra coefficients first (W_tuv), so that per ket component the raised and
// plain sums share one ket transform, where differentiating every integral
// block costs nine bra contractions per component pair.
//
// Each pair collects its two centres' derivatives in pair_grad[pair][6]
// (A then B), which grad_pairs_kernel sums over the atoms: neighbouring lanes
// add to different addresses, where the molecule's few atoms would be hot.
//
// grad_row_kernel: small kets, single-primitive pairs; the row kernels' tiles
// (dgf_jk_row.cuh): a warp on the bras of one A shell, one ket per lane.
// grad_warp_kernel: the other kets; one warp per quartet, a lane on each ket
// component, R_tuv in shared memory.
#pragma once

#include "dgf_grad_kernel.cuh"
#include "dgf_jk_row.cuh"
#include "dgf_jk_warp.cuh"

namespace dgf {
namespace grad {

// Where a launch's pairs collect their derivatives: six values per pair, the
// launch's bra and ket lists starting at pairs `bra` and `ket`.
struct PairGrad {
  double *out;
  int bra, ket;
};

// Exponent of direction k of Cartesian component i of shell l.
__host__ __device__ constexpr int cart_e(int l, int i, int k) {
  return k == 0 ? cart_x(l, i) : k == 1 ? cart_y(l, i) : cart_z(l, i);
}

// Lowered coefficients of one direction, t <= i + j - 1: -(b/p) i E^{i-1,j}_t
// + (a/p) j E^{i,j-1}_t (f1 = -b/p, f2 = a/p), from the tables of herm_e<LA, LB>.
template <int LA, int LB>
__device__ __forceinline__ double lowered(const double *E, int i, int j, int t, double f1, double f2) {
  constexpr int NT = LA + LB + 1;
  double v = 0.0;
  if (i > 0 && t <= i - 1 + j) v += f1 * i * E[((i - 1) * (LB + 1) + j) * NT + t];
  if (j > 0 && t <= i + j - 1) v += f2 * j * E[(i * (LB + 1) + j - 1) * NT + t];
  return v;
}

// ---------------------------------------------------------------- row kernel
template <int LA, int LB>
struct RowGrad {
  static constexpr int NA = ncart(LA), NB = ncart(LB);
  static constexpr int kR = row_max_bras(pair_class(LA, LB));
  // a bra's staged doubles: p, P, K, Q, {aoB, position}, {same, atom B},
  // a, P-A, P-B, two densities' AB blocks
  static constexpr int kPA = 10, kPB = 13, kAB = 16, kRow = kAB + 2 * NA * NB;
  static constexpr int kPerWarp = kR * (kRow + 3);  // then the bras' dE/dB sums
  static constexpr int kBlock = 128, kWarps = kBlock / 32;
  static constexpr size_t smem() { return (size_t)(kBoysTableDoubles + kWarps * kPerWarp) * 8; }
};

template <int LA, int LB, int LC, int LD, bool SPH>
__global__ void __launch_bounds__(128, (LA + LB + LC + LD <= 1) ? 4 : (LA + LB + LC + LD <= 2) ? 3 : 2)
    grad_row_kernel(const __grid_constant__ JKArgs a, const PairGrad pg) {
  using S = RowGrad<LA, LB>;
  constexpr int L = LA + LB + LC + LD, LAB = LA + LB, LCD = LC + LD;
  constexpr int NA = S::NA, NB = S::NB, NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
  constexpr int EA = (LA + 1) * (LB + 1) * (LAB + 1), EC = (LC + 1) * (LD + 1) * (LCD + 1);
  constexpr unsigned full = 0xffffffffu;
  extern __shared__ double sm[];
  for (int i = threadIdx.x; i < kBoysTableDoubles; i += blockDim.x) sm[i] = a.boys[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  double *wsm = sm + kBoysTableDoubles + (size_t)(threadIdx.x >> 5) * S::kPerWarp;
  double *gb = wsm + S::kR * S::kRow;
  const int slot = row::warp_slot<3>(lane);
  const int N = a.nbf;
  const double h = 0.5 * a.hfx;
  int seg = -1, nb = 0, aoA = 0;
  double gA[3] = {0.0, 0.0, 0.0};
  auto flush = [&]() {  // the segment's sums to its pairs
    const double tot = row::warp_sums<3>(gA, lane);
    const int ib0 = __double2hiint(wsm[6]);
    if (slot >= 0) atomicAdd(pg.out + 6 * (size_t)(pg.bra + ib0) + slot, tot);
    __syncwarp();
    for (int e = lane; e < 3 * nb; e += 32) {
      const int ib = __double2hiint(wsm[(e / 3) * S::kRow + 6]);
      atomicAdd(pg.out + 6 * (size_t)(pg.bra + ib) + 3 + e % 3, gb[e]);
    }
    __syncwarp();
    gA[0] = gA[1] = gA[2] = 0.0;
  };
  for (;;) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(a.row_work, 1u);
    t = __shfl_sync(full, t, 0) + a.row_task0;
    if (t >= a.row_task1) break;
    const int4 tk = __ldg(a.row_tasks + t);
    if (tk.x != seg) {
      if (seg >= 0) flush();
      seg = tk.x;
      nb = tk.y & 0xffff;
      if (lane < nb) {
        const int ib = __ldg(a.row_bra + seg + lane);
        const PairRec br = load_pair(a.bra + ib);
        const PrimPair P = load_prim<true>(a.pp + br.pp0);
        double *w = wsm + lane * S::kRow;
        w[0] = P.p;
        w[1] = P.Px;
        w[2] = P.Py;
        w[3] = P.Pz;
        w[4] = P.K;
        w[5] = br.Q;
        w[6] = __hiloint2double(ib, br.aoB);
        w[7] = __hiloint2double(br.atB, br.same);
        w[8] = P.ea;
        w[S::kPA] = P.PAx;
        w[S::kPA + 1] = P.PAy;
        w[S::kPA + 2] = P.PAz;
        w[S::kPB] = P.PBx;
        w[S::kPB + 1] = P.PBy;
        w[S::kPB + 2] = P.PBz;
        aoA = br.aoA;
        double blk[NA * NB];
        cart_block<LA, LB, SPH>(a.G1, N, br.aoA, br.aoB, blk);
#pragma unroll
        for (int k = 0; k < NA * NB; ++k) w[S::kAB + k] = blk[k];
        cart_block<LA, LB, SPH>(a.G2, N, br.aoA, br.aoB, blk);
#pragma unroll
        for (int k = 0; k < NA * NB; ++k) w[S::kAB + NA * NB + k] = blk[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) gb[3 * lane + k] = 0.0;
      }
      aoA = __shfl_sync(full, aoA, 0);
      __syncwarp();
    }
    const int kend = min(tk.w, tk.z + 32 * (tk.y >> 16));
    for (int ic0 = tk.z; ic0 < kend; ic0 += 32) {
      const int ic = ic0 + lane;
      const bool valid = ic < kend;
      const PairRec kt = load_pair(a.ket + (valid ? ic : kend - 1));
      const double Qk = valid ? kt.Q : 0.0;
      unsigned todo;
      {
        const unsigned qm = __reduce_max_sync(full, __float_as_uint(__double2float_ru(Qk)));
        bool on = false;
        if (lane < nb) {
          const double *w = wsm + lane * S::kRow;
          on = w[5] * (double)__uint_as_float(qm) >= a.schwarz_thr &&
               (!a.same_class || __double2hiint(w[6]) >= ic0 + a.ket_off);
        }
        todo = __ballot_sync(full, on);
      }
      if (!todo) continue;
      const PrimPair P2 = load_prim<true>(a.pp + kt.pp0);
      const double q = P2.p, f2c = P2.ea / q;  // c/q
      double e2[3][EC];
      herm_e<LC, LD, -1, double>(0.5 / q, P2.PAx, P2.PBx, e2[0]);
      herm_e<LC, LD, -1, double>(0.5 / q, P2.PAy, P2.PBy, e2[1]);
      herm_e<LC, LD, -1, double>(0.5 / q, P2.PAz, P2.PBz, e2[2]);
      double cd1[NCD], cd2[NCD], ac1[NA * NC], ac2[NA * NC], ad1[NA * ND], ad2[NA * ND];
      cart_block<LC, LD, SPH>(a.G1, N, kt.aoA, kt.aoB, cd1);
      cart_block<LC, LD, SPH>(a.G2, N, kt.aoA, kt.aoB, cd2);
      cart_block<LA, LC, SPH>(a.G1, N, aoA, kt.aoA, ac1);
      cart_block<LA, LC, SPH>(a.G2, N, aoA, kt.aoA, ac2);
      cart_block<LA, LD, SPH>(a.G1, N, aoA, kt.aoB, ad1);
      cart_block<LA, LD, SPH>(a.G2, N, aoA, kt.aoB, ad2);
      const double wk = kt.same ? 0.5 : 1.0;
      double gQ[3] = {0.0, 0.0, 0.0}, gY[3] = {0.0, 0.0, 0.0}, en = 0.0;
      while (todo) {
        const int r = __ffs(todo) - 1;
        todo &= todo - 1;
        const double *w = wsm + r * S::kRow;
        const int ib = __double2hiint(w[6]), aoB = __double2loint(w[6]);
        const bool work = valid && w[5] * Qk >= a.schwarz_thr && (!a.same_class || ic + a.ket_off <= ib);
        if (!__any_sync(full, work)) continue;
        double wgt = work ? wk : 0.0;
        if (__double2loint(w[7])) wgt *= 0.5;
        if (a.same_class && ib == ic + a.ket_off) wgt *= 0.5;
        double bc1[NB * NC], bc2[NB * NC], bd1[NB * ND], bd2[NB * ND];
        cart_block<LB, LC, SPH>(a.G1, N, aoB, kt.aoA, bc1);
        cart_block<LB, LC, SPH>(a.G2, N, aoB, kt.aoA, bc2);
        cart_block<LB, LD, SPH>(a.G1, N, aoB, kt.aoB, bd1);
        cart_block<LB, LD, SPH>(a.G2, N, aoB, kt.aoB, bd2);
        const double p = w[0], ea = w[8];
        const double fb = (ea - p) / p, fa = ea / p;  // -b/p, a/p
        double R[n3(L + 1)];
        {
          const double rs = rsqrt(p + q), alpha = p * q * rs * rs;
          const double x = w[1] - P2.Px, y = w[2] - P2.Py, z = w[3] - P2.Pz;
          double F[L + 2];
          boys_eval<L + 1>(alpha * (x * x + y * y + z * z), sm, F);
          double s = w[4] * P2.K * rs * wgt;
#pragma unroll
          for (int n = 0; n <= L + 1; ++n) {
            F[n] *= s;
            s *= -2.0 * alpha;
          }
          hermite_r_inplace<L + 1, double>(F, x, y, z, R);
        }
        double e1[3][EA];
#pragma unroll
        for (int k = 0; k < 3; ++k) herm_e<LA, LB, 1, double>(0.5 / p, w[S::kPA + k], w[S::kPB + k], e1[k]);
        double gP[3] = {0.0, 0.0, 0.0}, gX[3] = {0.0, 0.0, 0.0}, e0 = 0.0;
        static_for<NCD>([&](auto CD_) {
          constexpr int c = decltype(CD_)::value / ND, d = decltype(CD_)::value % ND;
          constexpr int k0 = cart_e(LC, c, 0), k1 = cart_e(LC, c, 1), k2 = cart_e(LC, c, 2);
          constexpr int l0 = cart_e(LD, d, 0), l1 = cart_e(LD, d, 1), l2 = cart_e(LD, d, 2);
          auto K = [&](int k, int tt) {
            return e2[k][(cart_e(LC, c, k) * (LD + 1) + cart_e(LD, d, k)) * (LCD + 1) + tt];
          };
          // ket transform, one index past the bra's range
          double xk[n3(LAB + 1)];
#pragma unroll
          for (int e = 0; e < n3(LAB + 1); ++e) xk[e] = 0.0;
#pragma unroll
          for (int ta = 0; ta <= k0 + l0; ++ta)
#pragma unroll
            for (int na = 0; na <= k1 + l1; ++na)
#pragma unroll
              for (int fa2 = 0; fa2 <= k2 + l2; ++fa2) {
                const double e3 = K(0, ta) * K(1, na) * K(2, fa2);
#pragma unroll
                for (int tt = 0; tt <= LAB + 1; ++tt)
#pragma unroll
                  for (int u = 0; u <= LAB + 1 - tt; ++u)
#pragma unroll
                    for (int v = 0; v <= LAB + 1 - tt - u; ++v)
                      xk[tuv_index(tt, u, v)] += e3 * R[tuv_index(tt + ta, u + na, v + fa2)];
              }
          // W: the density product contracted with the bra coefficients; the
          // lowered bra coefficients go straight into dE/dX
          double W[n3(LAB)];
#pragma unroll
          for (int e = 0; e < n3(LAB); ++e) W[e] = 0.0;
          static_for<NA * NB>([&](auto AB_) {
            constexpr int ab = decltype(AB_)::value, ia = ab / NB, jb = ab % NB;
            const double g = 2.0 * (w[S::kAB + ab] * cd2[c * ND + d] + w[S::kAB + NA * NB + ab] * cd1[c * ND + d]) -
                             h * (ac1[ia * NC + c] * bd2[jb * ND + d] + ac2[ia * NC + c] * bd1[jb * ND + d] +
                                  ad1[ia * ND + d] * bc2[jb * NC + c] + ad2[ia * ND + d] * bc1[jb * NC + c]);
            auto E = [&](int k, int tt) {
              return e1[k][(cart_e(LA, ia, k) * (LB + 1) + cart_e(LB, jb, k)) * (LAB + 1) + tt];
            };
            constexpr int s0 = cart_e(LA, ia, 0) + cart_e(LB, jb, 0), s1 = cart_e(LA, ia, 1) + cart_e(LB, jb, 1),
                          s2 = cart_e(LA, ia, 2) + cart_e(LB, jb, 2);
#pragma unroll
            for (int tt = 0; tt <= s0; ++tt)
#pragma unroll
              for (int u = 0; u <= s1; ++u) {
                const double gxy = g * (E(0, tt) * E(1, u));
#pragma unroll
                for (int v = 0; v <= s2; ++v) W[tuv_index(tt, u, v)] += gxy * E(2, v);
              }
            static_for<3>([&](auto K_) {
              constexpr int k = decltype(K_)::value;
              constexpr int ck = cart_e(LA, ia, k), dk = cart_e(LB, jb, k);
              if constexpr (ck + dk > 0) {
                constexpr int m0 = s0 - (k == 0), m1 = s1 - (k == 1), m2 = s2 - (k == 2);
                double s = 0.0;
#pragma unroll
                for (int tt = 0; tt <= m0; ++tt)
#pragma unroll
                  for (int u = 0; u <= m1; ++u)
#pragma unroll
                    for (int v = 0; v <= m2; ++v) {
                      const double x0 = k == 0 ? lowered<LA, LB>(e1[0], ck, dk, tt, fb, fa) : E(0, tt);
                      const double x1 = k == 1 ? lowered<LA, LB>(e1[1], ck, dk, u, fb, fa) : E(1, u);
                      const double x2 = k == 2 ? lowered<LA, LB>(e1[2], ck, dk, v, fb, fa) : E(2, v);
                      s += x0 * x1 * x2 * xk[tuv_index(tt, u, v)];
                    }
                gX[k] += g * s;
              }
            });
          });
          double s = 0.0;
#pragma unroll
          for (int tt = 0; tt <= LAB; ++tt)
#pragma unroll
            for (int u = 0; u <= LAB - tt; ++u)
#pragma unroll
              for (int v = 0; v <= LAB - tt - u; ++v) {
                const double we = W[tuv_index(tt, u, v)];
                s += we * xk[tuv_index(tt, u, v)];
                gP[0] += we * xk[tuv_index(tt + 1, u, v)];
                gP[1] += we * xk[tuv_index(tt, u + 1, v)];
                gP[2] += we * xk[tuv_index(tt, u, v + 1)];
              }
          e0 += s;
          // lowered ket coefficients: dE/dY
          static_for<3>([&](auto K_) {
            constexpr int k = decltype(K_)::value, ck = cart_e(LC, c, k), dk = cart_e(LD, d, k);
            if constexpr (ck + dk > 0) {
              constexpr int m0 = k0 + l0 - (k == 0), m1 = k1 + l1 - (k == 1), m2 = k2 + l2 - (k == 2);
#pragma unroll
              for (int ta = 0; ta <= m0; ++ta)
#pragma unroll
                for (int na = 0; na <= m1; ++na)
#pragma unroll
                  for (int fa2 = 0; fa2 <= m2; ++fa2) {
                    const double x0 = k == 0 ? lowered<LC, LD>(e2[0], ck, dk, ta, f2c - 1.0, f2c) : K(0, ta);
                    const double x1 = k == 1 ? lowered<LC, LD>(e2[1], ck, dk, na, f2c - 1.0, f2c) : K(1, na);
                    const double x2 = k == 2 ? lowered<LC, LD>(e2[2], ck, dk, fa2, f2c - 1.0, f2c) : K(2, fa2);
                    double y = 0.0;
#pragma unroll
                    for (int tt = 0; tt <= LAB; ++tt)
#pragma unroll
                      for (int u = 0; u <= LAB - tt; ++u)
#pragma unroll
                        for (int v = 0; v <= LAB - tt - u; ++v)
                          y += W[tuv_index(tt, u, v)] * R[tuv_index(tt + ta, u + na, v + fa2)];
                    gY[k] += x0 * x1 * x2 * y;
                  }
            }
          });
        });
        // X = A - B = (P - B) - (P - A)
        double fB[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double X = w[S::kPB + k] - w[S::kPA + k];
          const double gx = gX[k] + 2.0 * ea * fb * X * e0;  // -2 mu X, mu = a b / p
          gA[k] += fa * gP[k] + gx;
          fB[k] = -fb * gP[k] - gx;
          gQ[k] += gP[k];
        }
        en += e0;
        const double tot = row::warp_sums<3>(fB, lane);
        if (slot >= 0) gb[3 * r + slot] += tot;
      }
      if (valid) {
        double *o = pg.out + 6 * (size_t)(pg.ket + ic);
        const double Y[3] = {P2.PBx - P2.PAx, P2.PBy - P2.PAy, P2.PBz - P2.PAz};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double gy = gY[k] + 2.0 * P2.ea * (f2c - 1.0) * Y[k] * en;  // -2 nu Y, nu = c d / q
          atomicAdd(o + k, -f2c * gQ[k] + gy);
          atomicAdd(o + 3 + k, (f2c - 1.0) * gQ[k] - gy);
        }
      }
    }
  }
  if (seg >= 0) flush();
}

// --------------------------------------------------------------- warp kernel
// Compact lowered-product tables of a shell pair: for direction k, component
// pair ij with ix + jx > 0 in that direction, terms t, u, v with the range of
// direction k one shorter.
constexpr int low_n(int la, int lb, int ij, int k, int d) {
  const int i = ij / ncart(lb), j = ij % ncart(lb);
  const int s = d == 0 ? cart_x(la, i) + cart_x(lb, j) : d == 1 ? cart_y(la, i) + cart_y(lb, j) : cart_z(la, i) + cart_z(lb, j);
  return s + 1 - (k == d ? 1 : 0);  // 0 for the lowered direction without a function to lower
}
constexpr int low_terms(int la, int lb, int ij, int k) {
  return low_n(la, lb, ij, k, 0) * low_n(la, lb, ij, k, 1) * low_n(la, lb, ij, k, 2);
}
constexpr int low_off(int la, int lb, int ij, int k) {
  int off = 0;
  for (int m = 0; m < ij; ++m)
    for (int d = 0; d < 3; ++d) off += low_terms(la, lb, m, d);
  for (int d = 0; d < k; ++d) off += low_terms(la, lb, ij, d);
  return off;
}

template <int LA, int LB, int LC, int LD>
struct WarpGrad {
  static constexpr int L = LA + LB + LC + LD, LAB = LA + LB, LCD = LC + LD, BOX = L + 2;  // R to L + 1
  static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD), NAB = NA * NB, NCD = NC * ND;
  static constexpr int SB = BOX | 1, SA = (SB * BOX) | 1, RBOX = SA * (L + 1) + 1;
  static constexpr int NT1 = LAB + 1, NT2 = LCD + 1;
  static constexpr int EA = (LA + 1) * (LB + 1) * NT1, EC = (LC + 1) * (LD + 1) * NT2;
  static constexpr int TAB = wq::nterm_all(LA, LB), TLO = low_off(LA, LB, NAB, 0);
  static constexpr int BLK = NAB + NCD + NA * NC + NA * ND + NB * NC + NB * ND;  // Cartesian density blocks
  // per warp: R boxes; 1D tables of bra and ket, plain then lowered; products
  // of the bra, plain then lowered; density blocks of two densities
  static constexpr int PER_WARP = 2 * RBOX + 6 * EA + 6 * EC + TAB + TLO + 2 * BLK;
  static constexpr int NR = n3(L + 1);
  // block-wide: Boys and spherical tables, (t,u,v) positions, term indices
  static constexpr int COMMON = kBoysTableDoubles + kSphTableDoubles + (NR + TAB + TLO + 1) / 2;
  static constexpr size_t smem(int warps) { return (size_t)(COMMON + warps * PER_WARP) * 8; }
  static constexpr int WPB = smem(4) <= 100 * 1024 ? 4 : 2;
};

// The (lx, ly) block of D in Cartesian components, one element per lane.
template <int LX, int LY, bool SPH>
__device__ __forceinline__ void cart_block_warp(const double *__restrict__ D, int N, int p0, int q0, const double *sph,
                                                double *out, int lane) {
  constexpr int NX = ncart(LX), NY = ncart(LY);
  constexpr bool TX = SPH && LX >= 2, TY = SPH && LY >= 2;
  constexpr int FX = TX ? 2 * LX + 1 : NX, FY = TY ? 2 * LY + 1 : NY;
  const double *cx = sph + sph_offset(LX), *cy = sph + sph_offset(LY);
  for (int e = lane; e < NX * NY; e += 32) {
    const int i = e / NY, j = e % NY;
    double s = 0.0;
#pragma unroll 1
    for (int x = TX ? 0 : i; x < (TX ? FX : i + 1); ++x) {
      const double fx = TX ? cx[x * NX + i] : 1.0;
      if (TX && fx == 0.0) continue;
      double r = 0.0;
      if (TY) {
#pragma unroll
        for (int y = 0; y < FY; ++y) r += cy[y * NY + j] * __ldg(D + (size_t)(p0 + x) * N + q0 + y);
      } else {
        r = __ldg(D + (size_t)(p0 + x) * N + q0 + j);
      }
      s += fx * r;
    }
    out[e] = s;
  }
}

template <int LA, int LB, int LC, int LD, bool SPH>
__global__ void __launch_bounds__(128) grad_warp_kernel(const __grid_constant__ JKArgs a, const PairGrad pg) {
  using S = WarpGrad<LA, LB, LC, LD>;
  constexpr int L = S::L, LAB = S::LAB, SA = S::SA, SB = S::SB, NA = S::NA, NB = S::NB, NC = S::NC, ND = S::ND,
                NAB = S::NAB, NCD = S::NCD, EA = S::EA, EC = S::EC, TAB = S::TAB, TLO = S::TLO;
  constexpr unsigned full = 0xffffffffu;
  extern __shared__ double sm[];
  double *tab = sm, *sph = tab + kBoysTableDoubles;
  int *pos = (int *)(sph + kSphTableDoubles), *idx = pos + S::NR, *idl = idx + TAB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  double *R0 = sm + S::COMMON + (size_t)warp * S::PER_WARP, *R1 = R0 + S::RBOX, *Eb = R1 + S::RBOX, *Lb = Eb + 3 * EA,
         *Ek = Lb + 3 * EA, *Lk = Ek + 3 * EC, *Tb = Lk + 3 * EC, *Tl = Tb + TAB, *B1 = Tl + TLO, *B2 = B1 + S::BLK;
  for (int i = threadIdx.x; i < kBoysTableDoubles; i += blockDim.x) tab[i] = a.boys[i];
  for (int i = threadIdx.x; i < kSphTableDoubles; i += blockDim.x) sph[i] = a.sph[i];
  for (int e = threadIdx.x; e < S::NR; e += blockDim.x) {
    int t, u, v;
    tuv_decode(e, t, u, v);
    pos[e] = t * SA + u * SB + v;
  }
  wq_term_index<LA, LB>(idx, threadIdx.x, blockDim.x);
  // lowered terms: positions in Eb (0 .. 3 EA) and Lb (3 EA .. 6 EA), 10 bits each
  for (int ij = threadIdx.x; ij < NAB; ij += blockDim.x) {
    int ci[3], cj[3], off = 0;
    cart_decode(LA, ij / NB, ci[0], ci[1], ci[2]);
    cart_decode(LB, ij % NB, cj[0], cj[1], cj[2]);
    for (int m = 0; m < ij; ++m)
      for (int k = 0; k < 3; ++k) off += low_terms(LA, LB, m, k);
    for (int k = 0; k < 3; ++k) {
      int b[3];
      for (int d = 0; d < 3; ++d)
        b[d] = (d == k ? 3 * EA : 0) + d * EA + (ci[d] * (LB + 1) + cj[d]) * S::NT1;
      for (int t = 0; t < ci[0] + cj[0] + (k != 0); ++t)
        for (int u = 0; u < ci[1] + cj[1] + (k != 1); ++u)
          for (int v = 0; v < ci[2] + cj[2] + (k != 2); ++v) idl[off++] = (b[0] + t) | ((b[1] + u) << 10) | ((b[2] + v) << 20);
    }
  }
  __syncthreads();
  const int N = a.nbf;
  const double h = 0.5 * a.hfx;
  const int slot = row::warp_slot<12>(lane);
  const int64_t nteam = (int64_t)gridDim.x * nw, team = (int64_t)blockIdx.x * nw + warp;
  const int64_t span = (a.nquartet - a.q_begin + nteam - 1) / nteam;
  const int64_t qbeg = a.q_begin + team * span, qend = min(qbeg + span, a.nquartet);
  int ibw = -1, tb = -1;
  for (int64_t qq = qbeg; qq < qend; ++qq) {
    if (lane == 0) {
      if (ibw < 0) {
        ibw = find_bra(a.qoff, a.nbra, qq);
      } else {
        int steps = 0;
        while (qq >= a.qoff[ibw + 1] && steps < 32) {
          ++ibw;
          ++steps;
        }
        if (qq >= a.qoff[ibw + 1]) ibw = find_bra(a.qoff, a.nbra, qq);
      }
    }
    ibw = __shfl_sync(full, ibw, 0);
    const int ib = ibw, ic = (int)(qq - a.qoff[ib]);
    const PairRec br = load_pair(a.bra + ib), kt = load_pair(a.ket + ic);
    if (br.Q * kt.Q < a.schwarz_thr) continue;  // the plan's last Schwarz bin
    double wgt = 1.0;
    if (br.same) wgt *= 0.5;
    if (kt.same) wgt *= 0.5;
    if (a.same_class && ib == ic + a.ket_off) wgt *= 0.5;
    __syncwarp();
    for (int s = 0; s < 2; ++s) {
      const double *D = s ? a.G2 : a.G1;
      double *o = s ? B2 : B1;
      cart_block_warp<LA, LB, SPH>(D, N, br.aoA, br.aoB, sph, o, lane);
      cart_block_warp<LC, LD, SPH>(D, N, kt.aoA, kt.aoB, sph, o + NAB, lane);
      cart_block_warp<LA, LC, SPH>(D, N, br.aoA, kt.aoA, sph, o + NAB + NCD, lane);
      cart_block_warp<LA, LD, SPH>(D, N, br.aoA, kt.aoB, sph, o + NAB + NCD + NA * NC, lane);
      cart_block_warp<LB, LC, SPH>(D, N, br.aoB, kt.aoA, sph, o + NAB + NCD + NA * (NC + ND), lane);
      cart_block_warp<LB, LD, SPH>(D, N, br.aoB, kt.aoB, sph, o + NAB + NCD + NA * (NC + ND) + NB * NC, lane);
    }
    double out[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) out[k] = 0.0;
    for (int i = 0; i < br.npp; ++i) {
      const PrimPair P1 = load_prim<true>(a.pp + br.pp0 + i);
      const double fb = (P1.ea - P1.p) / P1.p, fa = P1.ea / P1.p;
      __syncwarp();
      if (br.npp > 1 || tb != ib) {
        if (lane < 3) {
          const double pa = lane == 0 ? P1.PAx : lane == 1 ? P1.PAy : P1.PAz;
          const double pb = lane == 0 ? P1.PBx : lane == 1 ? P1.PBy : P1.PBz;
          herm_e<LA, LB, 1, double>(0.5 / P1.p, pa, pb, Eb + lane * EA);
        }
        __syncwarp();
        for (int e = lane; e < 3 * EA; e += 32) {
          const int d = e / EA, r = e % EA, t = r % S::NT1, ij = r / S::NT1;
          Lb[e] = lowered<LA, LB>(Eb + d * EA, ij / (LB + 1), ij % (LB + 1), t, fb, fa);
        }
        __syncwarp();
        wq_product_table<TAB, double>(Eb, idx, Tb, lane);
        wq_product_table<TLO, double>(Eb, idl, Tl, lane);
        tb = br.npp == 1 ? ib : -1;
      }
      for (int j = 0; j < kt.npp; ++j) {
        const PrimPair P2 = load_prim<true>(a.pp + kt.pp0 + j);
        const double gc = (P2.ea - P2.p) / P2.p, gd = P2.ea / P2.p;  // -d/q, c/q
        __syncwarp();
        if (lane < 3) {
          const double pa = lane == 0 ? P2.PAx : lane == 1 ? P2.PAy : P2.PAz;
          const double pb = lane == 0 ? P2.PBx : lane == 1 ? P2.PBy : P2.PBz;
          herm_e<LC, LD, -1, double>(0.5 / P2.p, pa, pb, Ek + lane * EC);
        }
        __syncwarp();
        for (int e = lane; e < 3 * EC; e += 32) {
          const int d = e / EC, r = e % EC, t = r % S::NT2, ij = r / S::NT2;
          Lk[e] = lowered<LC, LD>(Ek + d * EC, ij / (LD + 1), ij % (LD + 1), t, gc, gd);
        }
        const double rs = rsqrt(P1.p + P2.p), alpha = P1.p * P2.p * rs * rs;
        const double x = P1.Px - P2.Px, y = P1.Py - P2.Py, z = P1.Pz - P2.Pz;
        double Fs[L + 2];
        boys_eval<L + 1>(alpha * (x * x + y * y + z * z), tab, Fs);
        {
          double s = P1.K * P2.K * rs * wgt;
#pragma unroll
          for (int n = 0; n <= L + 1; ++n) {
            Fs[n] *= s;
            s *= -2.0 * alpha;
          }
        }
        double *prev = R0, *cur = R1;
        if (lane == 0) prev[0] = Fs[L + 1];
        __syncwarp();
#pragma unroll 1
        for (int n = L; n >= 0; --n) {
          const int cnt = n3(L + 1 - n);
          double f0 = 0.0;
#pragma unroll
          for (int m = 0; m <= L; ++m)
            if (m == n) f0 = Fs[m];
          for (int e = lane; e < cnt; e += 32) {
            const int ps = pos[e], t = ps / SA, u = (ps % SA) / SB, v = (ps % SA) % SB;
            double val;
            if (e == 0) {
              val = f0;
            } else if (t > 0) {
              val = x * prev[ps - SA];
              if (t > 1) val += (t - 1) * prev[ps - 2 * SA];
            } else if (u > 0) {
              val = y * prev[ps - SB];
              if (u > 1) val += (u - 1) * prev[ps - 2 * SB];
            } else {
              val = z * prev[ps - 1];
              if (v > 1) val += (v - 1) * prev[ps - 2];
            }
            cur[ps] = val;
          }
          __syncwarp();
          double *sw = prev;
          prev = cur;
          cur = sw;
        }
        const double *R = prev;
        double gP[3] = {0.0, 0.0, 0.0}, gX[3] = {0.0, 0.0, 0.0}, gY[3] = {0.0, 0.0, 0.0}, e0 = 0.0;
#pragma unroll 1
        for (int cd = lane; cd < NCD; cd += 32) {
          // an offset of zero that the compiler does not see through: it
          // would lift the bra tables' loads out of the loop, and spill them
          int z0;
          asm volatile("mov.u32 %0, 0;" : "=r"(z0));
          const double *Tbz = Tb + z0, *Tlz = Tl + z0;
          const int c = cd / ND, d = cd % ND;
          int cc[3], dd[3];
          cart_decode(LC, c, cc[0], cc[1], cc[2]);
          cart_decode(LD, d, dd[0], dd[1], dd[2]);
          const double *K0 = Ek + (cc[0] * (LD + 1) + dd[0]) * S::NT2, *K1 = Ek + EC + (cc[1] * (LD + 1) + dd[1]) * S::NT2,
                       *K2 = Ek + 2 * EC + (cc[2] * (LD + 1) + dd[2]) * S::NT2;
          // ket transform
          double xk[n3(LAB + 1)];
#pragma unroll
          for (int e = 0; e < n3(LAB + 1); ++e) xk[e] = 0.0;
#pragma unroll 1
          for (int t = 0; t <= cc[0] + dd[0]; ++t)
#pragma unroll 1
            for (int u = 0; u <= cc[1] + dd[1]; ++u)
#pragma unroll 1
              for (int v = 0; v <= cc[2] + dd[2]; ++v) {
                const double ck = K0[t] * K1[u] * K2[v];
                const double *Rf = R + t * SA + u * SB + v;
                static_for<n3(LAB + 1)>([&](auto E_) {
                  constexpr int e = decltype(E_)::value;
                  xk[e] += ck * Rf[wq::tuv_t(e) * SA + wq::tuv_u(e) * SB + wq::tuv_v(e)];
                });
              }
          // density product over the bra components
          const double *ac1 = B1 + NAB + NCD + c, *ad1 = B1 + NAB + NCD + NA * NC + d,
                       *bc1 = B1 + NAB + NCD + NA * (NC + ND) + c, *bd1 = bc1 - c + NB * NC + d;
          const double *ac2 = ac1 + S::BLK, *ad2 = ad1 + S::BLK, *bc2 = bc1 + S::BLK, *bd2 = bd1 + S::BLK;
          const double cd1 = B1[NAB + cd], cd2 = B2[NAB + cd];
          double W[n3(LAB)];
#pragma unroll
          for (int e = 0; e < n3(LAB); ++e) W[e] = 0.0;
          static_for<NAB>([&](auto AB_) {
            constexpr int ab = decltype(AB_)::value, ia = ab / NB, jb = ab % NB;
            const double g = 2.0 * (B1[ab] * cd2 + B2[ab] * cd1) -
                             h * (ac1[ia * NC] * bd2[jb * ND] + ac2[ia * NC] * bd1[jb * ND] + ad1[ia * ND] * bc2[jb * NC] +
                                  ad2[ia * ND] * bc1[jb * NC]);
            static_for<n3(LAB)>([&](auto E_) {
              constexpr int e = decltype(E_)::value, et = wq::tuv_t(e), eu = wq::tuv_u(e), ev = wq::tuv_v(e);
              if constexpr (wq::uses(LA, LB, ab, et, eu, ev)) W[e] += g * Tbz[wq::term_at(LA, LB, ab, et, eu, ev)];
            });
            static_for<3>([&](auto K_) {
              constexpr int k = decltype(K_)::value;
              constexpr int n0 = low_n(LA, LB, ab, k, 0), n1 = low_n(LA, LB, ab, k, 1), n2 = low_n(LA, LB, ab, k, 2);
              if constexpr (n0 * n1 * n2 > 0) {
                constexpr int o = low_off(LA, LB, ab, k);
                double s = 0.0;
                static_for<n0 * n1 * n2>([&](auto T_) {
                  constexpr int m = decltype(T_)::value;
                  s += Tlz[o + m] * xk[tuv_index(m / (n1 * n2), (m / n2) % n1, m % n2)];
                });
                gX[k] += g * s;
              }
            });
          });
          static_for<n3(LAB)>([&](auto E_) {
            constexpr int e = decltype(E_)::value, et = wq::tuv_t(e), eu = wq::tuv_u(e), ev = wq::tuv_v(e);
            e0 += W[e] * xk[e];
            gP[0] += W[e] * xk[tuv_index(et + 1, eu, ev)];
            gP[1] += W[e] * xk[tuv_index(et, eu + 1, ev)];
            gP[2] += W[e] * xk[tuv_index(et, eu, ev + 1)];
          });
          // lowered ket coefficients
          const double *G0 = Lk + (K0 - Ek), *G1 = Lk + (K1 - Ek), *G2 = Lk + (K2 - Ek);
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int m0 = cc[0] + dd[0] - (k == 0), m1 = cc[1] + dd[1] - (k == 1), m2 = cc[2] + dd[2] - (k == 2);
#pragma unroll 1
            for (int t = 0; t <= m0; ++t)
#pragma unroll 1
              for (int u = 0; u <= m1; ++u)
#pragma unroll 1
                for (int v = 0; v <= m2; ++v) {
                  const double ck = (k == 0 ? G0 : K0)[t] * (k == 1 ? G1 : K1)[u] * (k == 2 ? G2 : K2)[v];
                  const double *Rf = R + t * SA + u * SB + v;
                  double s = 0.0;
                  static_for<n3(LAB)>([&](auto E_) {
                    constexpr int e = decltype(E_)::value;
                    s += W[e] * Rf[wq::tuv_t(e) * SA + wq::tuv_u(e) * SB + wq::tuv_v(e)];
                  });
                  gY[k] += ck * s;
                }
          }
        }
        const double X[3] = {P1.PBx - P1.PAx, P1.PBy - P1.PAy, P1.PBz - P1.PAz};
        const double Y[3] = {P2.PBx - P2.PAx, P2.PBy - P2.PAy, P2.PBz - P2.PAz};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double gx = gX[k] + 2.0 * P1.ea * fb * X[k] * e0, gy = gY[k] + 2.0 * P2.ea * gc * Y[k] * e0;
          out[k] += fa * gP[k] + gx;
          out[3 + k] += -fb * gP[k] - gx;
          out[6 + k] += -gd * gP[k] + gy;
          out[9 + k] += gc * gP[k] - gy;
        }
        __syncwarp();
      }
    }
    const double tot = row::warp_sums<12>(out, lane);
    if (slot >= 0)
      atomicAdd(pg.out + 6 * (size_t)(slot < 6 ? pg.bra + ib : pg.ket + ic) + slot % 6, tot);
  }
}

// Kernels of a class pair (null: none): the row kernel takes plan entries
// with row tasks; the warp kernel any; the thread kernel (dgf_grad_kernel.cuh)
// the contracted pairs of classes without a warp kernel.
typedef void (*PairGradLauncher)(const JKArgs &, const PairGrad &, int grid, cudaStream_t);
struct GradEntry {
  PairGradLauncher row, warp;
  bool row_cart;              // the row kernel also takes Cartesian functions
  int row_warps, row_blocks;  // warps per block, resident blocks per SM
  int warp_warps;
  cudaError_t (*prepare)();
};
extern GradEntry g_grad_entry[kGradClasses][kGradClasses];  // dgf_grad2e.cu; filled by DGF_GRAD_CLASS units

// Classes with the row kernel: kets (ss) and (ps), where the warp kernel
// would leave most lanes without a ket component, and (pp) and (ds) kets up to
// L = 5 (their larger ones spill R_tuv and take minutes to compile; Cartesian
// functions stop at L = 4). On (H2O)9 / cc-pVDZ, warp then row kernel: (ds|pp)
// 2.88 and 0.15 ms, (pp|pp) 1.45 and 0.17, (ds|ds) 1.00 and 0.08, (dp|pp) 1.85
// and 1.01, (dp|ds) 1.55 and 0.36.
constexpr bool grad_by_row(int LA, int LB, int LC, int LD) {
  return ncart(LC) * ncart(LD) <= 3 || LA + LB + LC + LD <= 5;
}
constexpr bool grad_by_row_cart(int LA, int LB, int LC, int LD) {
  return ncart(LC) * ncart(LD) <= 3 || LA + LB + LC + LD <= 4;
}
// Classes with the warp kernel: the other kets; it also serves the contracted
// pairs of the row kernel's classes with more than three ket components.
constexpr bool grad_by_warp(int LC, int LD) { return ncart(LC) * ncart(LD) > 3; }

template <int LA, int LB, int LC, int LD>
void launch_grad_row(const JKArgs &a, const PairGrad &pg, int grid, cudaStream_t s) {
  using R = RowGrad<LA, LB>;
  if constexpr (grad_by_row_cart(LA, LB, LC, LD)) {
    if (!a.spherical) {
      grad_row_kernel<LA, LB, LC, LD, false><<<grid, R::kBlock, R::smem(), s>>>(a, pg);
      return;
    }
  }
  grad_row_kernel<LA, LB, LC, LD, true><<<grid, R::kBlock, R::smem(), s>>>(a, pg);
}

template <int LA, int LB, int LC, int LD>
void launch_grad_warp(const JKArgs &a, const PairGrad &pg, int grid, cudaStream_t s) {
  using W = WarpGrad<LA, LB, LC, LD>;
  if (a.spherical)
    grad_warp_kernel<LA, LB, LC, LD, true><<<grid, 32 * W::WPB, W::smem(W::WPB), s>>>(a, pg);
  else
    grad_warp_kernel<LA, LB, LC, LD, false><<<grid, 32 * W::WPB, W::smem(W::WPB), s>>>(a, pg);
}

template <int LA, int LB, int LC, int LD>
cudaError_t prepare_grad() {
  cudaError_t e = cudaSuccess;
  auto allow = [&](auto *f, size_t smem) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  };
  if constexpr (grad_by_row(LA, LB, LC, LD)) {
    allow(grad_row_kernel<LA, LB, LC, LD, true>, RowGrad<LA, LB>::smem());
    if constexpr (grad_by_row_cart(LA, LB, LC, LD))
      allow(grad_row_kernel<LA, LB, LC, LD, false>, RowGrad<LA, LB>::smem());
  }
  if constexpr (grad_by_warp(LC, LD)) {
    using W = WarpGrad<LA, LB, LC, LD>;
    allow(grad_warp_kernel<LA, LB, LC, LD, true>, W::smem(W::WPB));
    allow(grad_warp_kernel<LA, LB, LC, LD, false>, W::smem(W::WPB));
  }
  return e;
}

template <int X, int Y>
void fill_grad() {
  constexpr int LA = cls_la(X), LB = cls_lb(X), LC = cls_la(Y), LD = cls_lb(Y);
  GradEntry &e = g_grad_entry[X][Y];
  e.prepare = &prepare_grad<LA, LB, LC, LD>;
  if constexpr (grad_by_row(LA, LB, LC, LD)) {
    e.row = &launch_grad_row<LA, LB, LC, LD>;
    e.row_cart = grad_by_row_cart(LA, LB, LC, LD);
    e.row_warps = RowGrad<LA, LB>::kWarps;
    e.row_blocks = LA + LB + LC + LD <= 1 ? 4 : LA + LB + LC + LD <= 2 ? 3 : 2;
  }
  if constexpr (grad_by_warp(LC, LD)) {
    e.warp = &launch_grad_warp<LA, LB, LC, LD>;
    e.warp_warps = WarpGrad<LA, LB, LC, LD>::WPB;
  } else {
    g_grad_table[X][Y] = &launch_grad<LA, LB, LC, LD>;
  }
}

}  // namespace grad
}  // namespace dgf

// Defines the static initialiser that fills entry (X, Y) of the gradient
// tables (one generated translation unit per class pair).
#define DGF_GRAD_CLASS(X, Y)                                        \
  namespace dgf {                                                   \
  namespace grad {                                                  \
  namespace {                                                       \
  struct GradClassInit_##X##_##Y {                                  \
    GradClassInit_##X##_##Y() { fill_grad<X, Y>(); }                \
  } g_grad_class_init_##X##_##Y;                                    \
  }                                                                 \
  }                                                                 \
  }
