// Row kernel: McMurchie-Davidson J/K quartets of single-primitive pairs, a
// warp on a tile of bra pairs that share their A shell times 32 ket pairs.
//
// Each lane keeps one ket pair for all bra pairs of its tile, so that per
// tile instead of per quartet
//   - the ket's primitive data and Hermite tables are loaded and formed,
//   - D_ac, D_ad and Ds_cd are gathered,
//   - K_ac, K_ad and J_cd, which the tile's quartets share, are added to the
//     half Fock matrix (they accumulate in registers over the bras).
// What is left per quartet is two density gathers (D_bc, D_bd) and the
// atomics of K_bc and K_bd; for a p or d shell A these are the small blocks.
// J_ab is summed across the lanes by a transposing butterfly (all FA FB
// values together) into the warp's shared memory, and added to the matrix
// when the warp leaves the tile row.  The bras' primitive data, Ds_ab and
// screening data are staged in shared memory once per row.
//
// Rows: the bra pairs of one class sorted by (A shell, primitive-count
// bucket, Schwarz factor descending), cut into segments of at most `R`; a
// task is a segment times some 32-ket chunks of its ket prefix (in a batch,
// of its molecule's kets).  Warps
// take tasks from a counter, so that the staircase of the Schwarz prefixes
// balances itself.
//
// Boys function: F_L from a table of degree-7 polynomials on intervals of
// 1/8 (Chebyshev interpolants), e^-T by its Taylor series about the
// interval's midpoint from the same table row; above T = 40 the asymptotic
// F_0 and upward recursion (boys_scaled).
#pragma once

#include "dgf_select.cuh"

namespace dgf {
namespace row {

// The scaled R^n_000 = K (-2 alpha)^n F_n(alpha r2) / sqrt(B), n = 0 .. M, for
// alpha = A / B (plain operator: A = p q, B = p + q; the attenuated one has
// A = p q mu^2, B = (p + q) mu^2 + p q, K times mu).  One reciprocal square
// root serves both ranges: of B below T = alpha r2 = 40, of A r2 above it,
// where R^0 = K sqrt(pi / (A r2)) / 2 and each higher order divides by r2;
// the lanes of a warp usually fall on both sides.
// Below, F_M comes from the fine table (rows of kFineStride doubles: 8
// coefficients in x in [-1, 1], e^-mid, unused).
template <int M>
__device__ __forceinline__ void boys_scaled(double A, double B, double r2, double K, const double *__restrict__ tab,
                                            double *F) {
  const double ar = A * r2;
  const bool large = ar >= kBoysTmax * B;
  const double y = rsqrt(large ? ar : B), y2 = y * y;
  double s = K * y;
  if (!large) {
    const double alpha = A * y2, T = fmin(alpha * r2, kBoysTmax * (1.0 - 1e-15));
    const int i = (int)(T * kFinePerUnit);
    const double u = T - ((double)i + 0.5) * (1.0 / kFinePerUnit);  // |u| <= 1/16
    const double x = u * (2.0 * kFinePerUnit);
    const double2 *c = reinterpret_cast<const double2 *>(tab + i * kFineStride);
    const double2 c01 = c[0], c23 = c[1], c45 = c[2], c67 = c[3];
    const double x2 = x * x;
    const double p01 = fma(c01.y, x, c01.x), p23 = fma(c23.y, x, c23.x), p45 = fma(c45.y, x, c45.x),
                 p67 = fma(c67.y, x, c67.x);
    F[M] = fma(fma(p67, x2, p45), x2 * x2, fma(p23, x2, p01));
    if (M > 0) {
      // e^-T = e^-mid e^-u, the Taylor series to u^9 / 9! (|u|^10 / 10! < 3e-19)
      const double u2 = u * u;
      const double e01 = 1.0 - u, e23 = fma(u, -1.0 / 6.0, 0.5), e45 = fma(u, -1.0 / 120.0, 1.0 / 24.0),
                   e67 = fma(u, -1.0 / 5040.0, 1.0 / 720.0), e89 = fma(u, -1.0 / 362880.0, 1.0 / 40320.0);
      const double u4 = u2 * u2;
      const double et = c[4].x * fma(fma(e89, u4, fma(e67, u2, e45)), u4, fma(e23, u2, e01));
      const double t2 = 2.0 * T;
#pragma unroll
      for (int m = M - 1; m >= 0; --m) F[m] = fma(t2, F[m + 1], et) * (1.0 / (2 * m + 1));
    }
#pragma unroll
    for (int n = 0; n <= M; ++n) {
      F[n] *= s;
      s *= -2.0 * alpha;
    }
  } else {
    F[0] = 0.88622692545275801364908374167057 * s;
    if (M > 0) {
      const double ir = -(A * y2);  // -1 / r2
      // e^-T in F_{m+1} = ((2m+1) F_m - e^-T) / (2T): at T >= 40 it is 3e-17
      // of F_0, and at most 1e-11 of (2m+1) F_m up to the order of these
      // kernels; its single-precision value, 7e-6 off with its argument's
      // rounding, moves F_{m+1} by less than 1e-16.  (4e5 random exponents
      // and distances with T from 40: largest and mean error against extended
      // precision equal to those with a double-precision e^-T.)
      float ef = 0.f, af = 0.f;
      if (M > 1) {
        const float bf = (float)B;
        af = -2.f * ((float)A / bf);
        ef = expf(-((float)ar / bf)) * (float)K * rsqrtf(bf) * af;
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
        double v = (double)(2 * m + 1) * F[m];
        if (m > 0) {
          v -= (double)ef;
          ef *= af;
        }
        F[m + 1] = v * ir;
      }
    }
  }
}

// Sums of V values over the warp by a transposing butterfly: after the call
// the lane whose slot() is v holds the total of value v.
template <int V>
__device__ __forceinline__ double warp_sums(double (&v)[V], int lane) {
  constexpr unsigned full = 0xffffffffu;
  static_for<5>([&](auto S_) {
    constexpr int s = decltype(S_)::value;
    constexpr int off = 16 >> s;
    constexpr int n = ((V + (1 << s) - 1) >> s);  // values left before this step
    if constexpr (n > 1) {
      constexpr int m = (n + 1) / 2;
      const bool up = lane & off;
#pragma unroll
      for (int i = 0; i < m; ++i) {
        const double lo = v[i], hi = (i + m < n) ? v[i + m < V ? i + m : 0] : 0.0;
        v[i] = (up ? hi : lo) + __shfl_xor_sync(full, up ? lo : hi, off);
      }
    } else {
      v[0] += __shfl_xor_sync(full, v[0], off);
    }
  });
  return v[0];
}
// The value a lane holds after warp_sums<V>, or -1 (padding, or a copy of a
// lower lane's total): the lane's position in the last split, taken back
// through the splits.
template <int V>
__device__ __forceinline__ int warp_slot(int lane) {
  int local = 0;
  bool ok = true;
#pragma unroll
  for (int s = 4; s >= 0; --s) {
    const int n = (V + (1 << s) - 1) >> s, up = (lane >> (4 - s)) & 1;
    if (n > 1) {
      local += up * ((n + 1) / 2);
      ok = ok && local < n;
    } else {
      ok = ok && !up;
    }
  }
  return ok ? local : -1;
}

// The A functions of chunk CH of CA.  s and p: consecutive components.  d:
// all five, or {xy, yz, xz} and {z2, x2-y2} (three Cartesian components
// each), or one each.  f: consecutive ones.  (Spherical functions in the
// order m = -l..l.)
__host__ __device__ constexpr int chunk_begin(int LA, int CA, int CH) { return CH * (2 * LA + 1) / CA; }
__host__ __device__ constexpr int chunk_size(int LA, int CA, int CH) {
  return (LA == 2 && CA == 2) ? 3 - CH : chunk_begin(LA, CA, CH + 1) - chunk_begin(LA, CA, CH);
}
__host__ __device__ constexpr int chunk_fun(int LA, int CA, int CH, int x) {
  if (LA == 2 && CA == 2) return CH == 0 ? (x == 0 ? 0 : x == 1 ? 1 : 3) : (x == 0 ? 2 : 4);
  return chunk_begin(LA, CA, CH) + x;
}
__host__ __device__ constexpr int chunk_most(int LA, int CA) {
  int m = 0;
  for (int ch = 0; ch < CA; ++ch) m = cmax(m, chunk_size(LA, CA, ch));
  return m;
}
// Coefficient of Cartesian component x in function m of a shell (s, p: the
// components themselves).
template <int L>
__host__ __device__ constexpr double fun_coef(int m, int x) {
  if constexpr (L >= 2)
    return sph::coef<L>(m, x);
  else
    return m == x ? 1.0 : 0.0;
}
// Whether a function of the chunk uses Cartesian component x.
template <int LA>
__host__ __device__ constexpr bool chunk_uses(int CA, int CH, int x) {
  for (int k = 0; k < chunk_size(LA, CA, CH); ++k)
    if (fun_coef<LA>(chunk_fun(LA, CA, CH, k), x) != 0.0) return true;
  return false;
}

// Shape of one class's kernel: block size and resident blocks per SM the
// register allocation is held to, staged bra data, and what lives in
// registers.
template <int LA, int LB, int LC, int LD, int CA>
struct Shape {
  static constexpr int L = LA + LB + LC + LD;
  static constexpr int FB = 2 * LB + 1, FC = 2 * LC + 1, FD = 2 * LD + 1;
  static constexpr int FAx = chunk_most(LA, CA);  // most A functions of a chunk
  // Warps against registers: 16 warps of 128 registers up to L = 1, 12 of 168
  // at L = 2, 8 of 255 above. (H2O)32 / cc-pVDZ with 16 and 12 warps at L = 2
  // and 3: (ps|ps) 5.0 and 4.4 ms, (pp|ps) 6.9 ms with 12 warps (590 bytes
  // spilled) and 4.9 ms with 8, (ds|ps) 2.9 and 2.1.
  static constexpr int kBlock = L <= 1 ? 256 : L == 2 ? 192 : L == 3 ? 128 : 256;
  static constexpr int kMinBlocks = L <= 3 ? 2 : 1;
  static constexpr int kWarps = kBlock / 32;
  static constexpr int kR = row_max_bras(pair_class(LA, LB));  // bras of a segment
  // a bra's staged doubles: p (stored form: its first block), P, K, Q, {aoB, position}, {same, block B},
  // GAB, max |D_AB|, P-A, P-B, Ds_ab
  static constexpr int kPA = 10, kPB = kPA + (LA > 0 ? 3 : 0), kDab = kPB + (LB > 0 ? 3 : 0);
  static constexpr int kRow = (kDab + FAx * FB + 1) & ~1;
  static constexpr int kPerWarp = kR * (kRow + FAx * FB);  // staged bras, then their J_ab sums
  static constexpr size_t smem() { return ((size_t)kFineDoubles + (size_t)kWarps * kPerWarp) * 8; }
};

// What a row kernel runs on: the quartets of one molecule, those of a batch
// (each segment has its own matrices: their size and place take registers,
// 15% of the time of the s kernels, so that the form is its own), or the
// stored integrals of one molecule.
enum { kEval = 0, kBatch = 1, kStored = 2 };

template <int LA, int LB, int LC, int LD, int CA, int CH, int FORM>
__device__ __forceinline__ void row_body(const JKArgs &a, const double *tab, double *wsm, unsigned long long &cnt_q,
                                         unsigned long long &cnt_s) {
  using S = Shape<LA, LB, LC, LD, CA>;
  constexpr int L = S::L, LAB = LA + LB, LCD = LC + LD;
  constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
  constexpr int FA = chunk_size(LA, CA, CH), FB = S::FB, FC = S::FC, FD = S::FD;
  constexpr int EA = (LA + 1) * (LB + 1) * (LAB + 1), EC = (LC + 1) * (LD + 1) * (LCD + 1);
  constexpr unsigned full = 0xffffffffu;
  constexpr bool ST = FORM == kStored, BT = FORM == kBatch;
  const int lane = threadIdx.x & 31;
  double *jab = wsm + S::kR * S::kRow;
  const int jslot = warp_slot<FA * FB>(lane);
  auto afun = [](int x) { return chunk_fun(LA, CA, CH, x); };  // function of A of the chunk's row x
  const double js = a.jscale[0], ks = -a.kscale[0];
  int seg = -1, aoA = 0, nb = 0, blkA = 0;
  int Nb = 0;  // batches: size and place of the segment's matrices
  int64_t db = 0;
#define DGF_ROW_MATRICES                                  \
  const int N = BT ? Nb : a.nbf;                          \
  const double *Dm = BT ? a.D + db : a.D, *Dsm = BT ? a.Ds + db : a.Ds; \
  double *Fm = BT ? a.Fh + db : a.Fh;                     \
  (void)Dm, (void)Dsm, (void)Fm
  // J_ab of the staged bras to the half Fock matrix
  auto flush_jab = [&]() {
    DGF_ROW_MATRICES;
    __syncwarp();
    if (js != 0.0)
      for (int e = lane; e < nb * FA * FB; e += 32) {
        const int r = e / (FA * FB), o = e - r * (FA * FB);
        const double v = jab[e];
        const int aoB = __double2loint(wsm[r * S::kRow + 6]);
        if (v != 0.0) atomicAdd(Fm + (size_t)(aoA + afun(o / FB)) * N + aoB + o % FB, js * v);
      }
    __syncwarp();
  };
  for (;;) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(a.row_work + CH, 1u);
    t = __shfl_sync(full, t, 0) + a.row_task0;
    if (t >= a.row_task1) break;
    const int4 tk = __ldg(a.row_tasks + t);  // first bra (row order), bras | chunks << 16, first ket, end of the kets
    if (tk.x != seg) {
      if (seg >= 0) flush_jab();
      seg = tk.x;
      nb = tk.y & 0xffff;
      if (BT) {
        const PairRec b0 = load_pair_fock(a.bra + __ldg(a.row_bra + seg));
        Nb = b0.nbfm;
        db = b0.dbase;
      }
      DGF_ROW_MATRICES;
      if (lane < nb) {
        const int ib = __ldg(a.row_bra + seg + lane);
        const PairRec br = load_pair_fock(a.bra + ib);
        double *w = wsm + lane * S::kRow;
        if constexpr (ST) {
          w[0] = __longlong_as_double(a.qoff[ib]);  // the bra's first block in the store
        } else {
          const PrimPair P = load_prim<true>(a.pp + br.pp0);
          w[0] = P.p;
          w[1] = P.Px;
          w[2] = P.Py;
          w[3] = P.Pz;
          w[4] = P.K;
          if (LA > 0) {
            w[S::kPA] = P.PAx;
            w[S::kPA + 1] = P.PAy;
            w[S::kPA + 2] = P.PAz;
          }
          if (LB > 0) {
            w[S::kPB] = P.PBx;
            w[S::kPB + 1] = P.PBy;
            w[S::kPB + 2] = P.PBz;
          }
        }
        w[5] = br.Q;
        w[6] = __hiloint2double(ib, br.aoB);
        aoA = br.aoA;
        int blkB = 0;
        double gab = 0.0, dab = 0.0;
        if (a.blk_gab) {
          const int4 bb = block_of_pair(a.bra + ib);
          blkA = bb.x | (bb.z << 30);
          blkB = bb.y | (bb.w << 30);
          gab = a.blk_gab[bb.x * a.nblk + bb.y];
          dab = a.blk_dmax[bb.x * a.nblk + bb.y];
        }
        w[7] = __hiloint2double(blkB, br.same);
        w[8] = gab;
        w[9] = dab;
#pragma unroll
        for (int o = 0; o < FA * FB; ++o) {
          w[S::kDab + o] = __ldg(Dsm + (size_t)(br.aoA + afun(o / FB)) * N + br.aoB + o % FB);
          jab[lane * FA * FB + o] = 0.0;
        }
      }
      aoA = __shfl_sync(full, aoA, 0);
      blkA = __shfl_sync(full, blkA, 0);
      __syncwarp();
    }
    DGF_ROW_MATRICES;
    const int kend = min(tk.w, tk.z + 32 * (tk.y >> 16));
    for (int ic0 = tk.z; ic0 < kend; ic0 += 32) {
      const int ic = ic0 + lane;
      const bool valid = ic < kend;
      const int g0 = a.ks_base + (valid ? ic : kend - 1);
      const double Qk = valid ? __ldg(a.ks_q + g0) : 0.0;
      // bras with a quartet above the threshold in this chunk (and, for a
      // bra class equal to the ket class, at or behind its first ket)
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
      const int4 ki = __ldg(a.ks_i + g0);
      const int aoC = ki.x, aoD = ki.y;
      double q = 1.0, Qx = 0.0, Qy = 0.0, Qz = 0.0, Kk = 0.0;
      double ex2[EC], ey2[EC], ez2[EC];
      if constexpr (!ST) {
        const double *pl = a.ks_pp + g0;
        const int64_t st = a.ks_stride;
        q = __ldg(pl);
        Qx = __ldg(pl + st);
        Qy = __ldg(pl + 2 * st);
        Qz = __ldg(pl + 3 * st);
        Kk = __ldg(pl + 4 * st);
        if constexpr (LCD > 0) {
          const double h2 = 0.5 / q;
          const double cx = __ldg(pl + 5 * st), cy = __ldg(pl + 6 * st), cz = __ldg(pl + 7 * st);
          double dx = 0.0, dy = 0.0, dz = 0.0;
          if constexpr (LD > 0) {
            dx = __ldg(pl + 8 * st);
            dy = __ldg(pl + 9 * st);
            dz = __ldg(pl + 10 * st);
          }
          herm_e<LC, LD, -1, double>(h2, cx, dx, ex2);
          herm_e<LC, LD, -1, double>(h2, cy, dy, ey2);
          herm_e<LC, LD, -1, double>(h2, cz, dz, ez2);
        } else {
          ex2[0] = ey2[0] = ez2[0] = 1.0;
        }
      }
      const double wk = ki.z ? 0.5 : 1.0;
      // density screen: the ket's blocks and the bounds that stay for the tile
      int4 kb = make_int4(0, 0, 0, 0);
      double gcd = 0.0;
      float dcd = 0.f, dacd = 0.f;
      if (a.blk_gab) {
        kb = block_of_pair(a.ket + (valid ? ic : kend - 1));
        const int n = a.nblk, bA = blkA & (kWholeBlock - 1);
        gcd = a.blk_gab[kb.x * n + kb.y];
        dcd = a.blk_dmax[kb.x * n + kb.y];
        dacd = fmaxf(a.blk_dmax[bA * n + kb.x], a.blk_dmax[bA * n + kb.y]);
      }
      double Dac[FA * FC], Dad[FA * FD], Dcd[FC * FD], Kac[FA * FC], Kad[FA * FD], Jcd[FC * FD];
#pragma unroll
      for (int o = 0; o < FA * FC; ++o) {
        Dac[o] = __ldg(Dm + (size_t)(aoA + afun(o / FC)) * N + aoC + o % FC);
        Kac[o] = 0.0;
      }
#pragma unroll
      for (int o = 0; o < FA * FD; ++o) {
        Dad[o] = __ldg(Dm + (size_t)(aoA + afun(o / FD)) * N + aoD + o % FD);
        Kad[o] = 0.0;
      }
#pragma unroll
      for (int o = 0; o < FC * FD; ++o) {
        Dcd[o] = __ldg(Dsm + (size_t)(aoC + o / FD) * N + aoD + o % FD);
        Jcd[o] = 0.0;
      }
      while (todo) {
        const int r = __ffs(todo) - 1;
        todo &= todo - 1;
        const double *w = wsm + r * S::kRow;
        const double2 w01 = *reinterpret_cast<const double2 *>(w), w23 = *reinterpret_cast<const double2 *>(w + 2),
                      w45 = *reinterpret_cast<const double2 *>(w + 4), w67 = *reinterpret_cast<const double2 *>(w + 6);
        const int ib = __double2hiint(w67.x), aoB = __double2loint(w67.x);
        bool work = valid && w45.y * Qk >= a.schwarz_thr && (!a.same_class || ic + a.ket_off <= ib);
        if (a.blk_gab && work) {
          const int n = a.nblk, bB = __double2hiint(w67.y) & (kWholeBlock - 1);
          const float dj = fmaxf((float)w[9], dcd);
          const float dk = fmaxf(dacd, fmaxf(a.blk_dmax[bB * n + kb.x], a.blk_dmax[bB * n + kb.y]));
          if (w[8] * gcd * (double)fmaxf(4.0f * dj, dk) < a.dens_thr) {
            work = false;
            if (CH == 0) ++cnt_s;
          }
        }
        if (!__any_sync(full, work)) continue;
        if (CH == 0) cnt_q += work;
        // the quartet's own density values, fetched ahead of the integrals
        const int rowB = aoB * N;
        double Dbc[FB * FC], Dbd[FB * FD];
#pragma unroll
        for (int o = 0; o < FB * FC; ++o) Dbc[o] = __ldg(Dm + (rowB + (o / FC) * N + aoC + o % FC));
#pragma unroll
        for (int o = 0; o < FB * FD; ++o) Dbd[o] = __ldg(Dm + (rowB + (o / FD) * N + aoD + o % FD));
        double wgt = work ? wk : 0.0;
        if (__double2loint(w67.y)) wgt *= 0.5;
        if (a.same_class && ib == ic + a.ket_off) wgt *= 0.5;
        double g[FA * FB * FC * FD];
        if constexpr (ST) {
          const double *src =
              a.store_in + a.store_base + (__double_as_longlong(w01.x) + (valid ? ic : 0)) * (int64_t)a.store_nint;
#pragma unroll
          for (int xx = 0; xx < FA; ++xx)
#pragma unroll
            for (int o = 0; o < FB * FC * FD; ++o)
              g[xx * FB * FC * FD + o] = work ? wgt * __ldg(src + afun(xx) * FB * FC * FD + o) : 0.0;
        } else {
          // Boys function and R_tuv
          double R[n3(L)], ex1[EA], ey1[EA], ez1[EA];
          {
            const double p = w01.x;
            double A = p * q, B = p + q, K = w45.x * Kk * wgt;
            if (a.erf_mu2 > 0.0) {
              B = fma(B, a.erf_mu2, A);
              A *= a.erf_mu2;
              K *= sqrt(a.erf_mu2);
            }
            const double x = w01.y - Qx, y = w23.x - Qy, z = w23.y - Qz;
            double Fs[L + 1];
            boys_scaled<L>(A, B, x * x + y * y + z * z, K, tab, Fs);
            hermite_r_inplace<L, double>(Fs, x, y, z, R);
            if constexpr (LAB > 0) {
              const double h1 = 0.5 / p;
              herm_e<LA, LB, 1, double>(h1, w[S::kPA], LB > 0 ? w[S::kPB] : 0.0, ex1);
              herm_e<LA, LB, 1, double>(h1, w[S::kPA + 1], LB > 0 ? w[S::kPB + 1] : 0.0, ey1);
              herm_e<LA, LB, 1, double>(h1, w[S::kPA + 2], LB > 0 ? w[S::kPB + 2] : 0.0, ez1);
            } else {
              ex1[0] = ey1[0] = ez1[0] = 1.0;
            }
          }
          // The quartet's integrals, one function pair of the ket at a time:
          // f(cs, ds, g[FA][FB]).  The ket transform sums the Cartesian
          // components of spherical C and D functions, the bra transform those
          // of A.
          auto integrals = [&](auto &&f) {
            static_for<FC>([&](auto CS_) {
              static_for<FD>([&](auto DS_) {
                constexpr int cs = decltype(CS_)::value, ds = decltype(DS_)::value;
                double xk[n3(LAB)];
#pragma unroll
                for (int e = 0; e < n3(LAB); ++e) xk[e] = 0.0;
                static_for<NC>([&](auto C_) {
                  static_for<ND>([&](auto D_) {
                    constexpr int c = decltype(C_)::value, d = decltype(D_)::value;
                    constexpr double cf = fun_coef<LC>(cs, c) * fun_coef<LD>(ds, d);
                    if constexpr (cf != 0.0) {
                      constexpr int cx = cart_x(LC, c), cy = cart_y(LC, c), cz = cart_z(LC, c);
                      constexpr int dx = cart_x(LD, d), dy = cart_y(LD, d), dz = cart_z(LD, d);
#pragma unroll
                      for (int ta = 0; ta <= cx + dx; ++ta)
#pragma unroll
                        for (int na = 0; na <= cy + dy; ++na)
#pragma unroll
                          for (int fa = 0; fa <= cz + dz; ++fa) {
                            const double e3 = cf * (ex2[(cx * (LD + 1) + dx) * (LCD + 1) + ta] *
                                                    ey2[(cy * (LD + 1) + dy) * (LCD + 1) + na] *
                                                    ez2[(cz * (LD + 1) + dz) * (LCD + 1) + fa]);
#pragma unroll
                            for (int tt = 0; tt <= LAB; ++tt)
#pragma unroll
                              for (int u = 0; u <= LAB - tt; ++u)
#pragma unroll
                                for (int v = 0; v <= LAB - tt - u; ++v)
                                  xk[tuv_index(tt, u, v)] += e3 * R[tuv_index(tt + ta, u + na, v + fa)];
                          }
                    }
                  });
                });
                double gc[FA * NB];  // A functions, B components
#pragma unroll
                for (int k = 0; k < FA * NB; ++k) gc[k] = 0.0;
                static_for<NA * NB>([&](auto AB_) {
                  constexpr int ia = decltype(AB_)::value / NB, jb = decltype(AB_)::value % NB;
                  if constexpr (chunk_uses<LA>(CA, CH, ia)) {
                    constexpr int ax = cart_x(LA, ia), ay = cart_y(LA, ia), az = cart_z(LA, ia);
                    constexpr int bx = cart_x(LB, jb), by = cart_y(LB, jb), bz = cart_z(LB, jb);
                    double sum = 0.0;
#pragma unroll
                    for (int tt = 0; tt <= ax + bx; ++tt)
#pragma unroll
                      for (int u = 0; u <= ay + by; ++u) {
                        const double exy = ex1[(ax * (LB + 1) + bx) * (LAB + 1) + tt] *
                                           ey1[(ay * (LB + 1) + by) * (LAB + 1) + u];
#pragma unroll
                        for (int v = 0; v <= az + bz; ++v)
                          sum += exy * ez1[(az * (LB + 1) + bz) * (LAB + 1) + v] * xk[tuv_index(tt, u, v)];
                      }
                    static_for<FA>([&](auto X_) {
                      constexpr int x = decltype(X_)::value;
                      constexpr double ca = fun_coef<LA>(chunk_fun(LA, CA, CH, x), ia);
                      if constexpr (ca != 0.0) gc[x * NB + jb] += ca * sum;
                    });
                  }
                });
                if constexpr (LB >= 2) {
                  double g[FA * FB];
                  sph_index<LB, FA, NB, 0, 1>(gc, g);
                  f(cs, ds, g);
                } else {
                  f(cs, ds, gc);
                }
              });
            });
          };
          integrals([&](int cs, int ds, const double *v) {
#pragma unroll
            for (int k = 0; k < FA * FB; ++k) g[(k * FC + cs) * FD + ds] = v[k];
          });
        }
        bool jw = work, kw = work;
        if (a.ice_thr > 0.0 && work && (blkA & __double2hiint(w67.y) & kWholeBlock) && kb.z && kb.w) {
          // ICEDIF: per-part skips of quartets of whole Dalton blocks, from
          // the largest integral of this chunk's part of the quartet (whose
          // weight, a power of two, is part of g)
          double amax = 0.0;
#pragma unroll
          for (int e = 0; e < FA * FB * FC * FD; ++e) amax = fmax(amax, fabs(g[e]));
          amax /= wgt;
          const float *dm = a.blk_dmax_slot;
          const int n = a.nblk, bA = blkA & (kWholeBlock - 1), bB = __double2hiint(w67.y) & (kWholeBlock - 1);
          const double dj = fmaxf(dm[bA * n + bB], dm[kb.x * n + kb.y]);
          const double dk = fmaxf(fmaxf(dm[bA * n + kb.x], dm[bA * n + kb.y]), fmaxf(dm[bB * n + kb.x], dm[bB * n + kb.y]));
          if ((a.icedif & 1) && dj * amax < a.ice_thr) jw = false;
          if ((a.icedif & 2) && dk * amax < a.ice_thr) kw = false;
        }
        auto G = [&](int xx, int yy, int cc, int dd) -> double { return g[((xx * FB + yy) * FC + cc) * FD + dd]; };
        if (js != 0.0) {
          double jv[FA * FB];
#pragma unroll
          for (int xx = 0; xx < FA; ++xx)
#pragma unroll
            for (int yy = 0; yy < FB; ++yy) {
              const double dab = w[S::kDab + xx * FB + yy];
              double sum = 0.0;
#pragma unroll
              for (int o = 0; o < FC * FD; ++o) {
                const double v = G(xx, yy, o / FD, o % FD);
                sum += v * Dcd[o];
                if (jw) Jcd[o] += v * dab;
              }
              jv[xx * FB + yy] = jw ? sum : 0.0;
            }
          const double tot = warp_sums<FA * FB>(jv, lane);
          if (jslot >= 0) jab[r * FA * FB + jslot] += tot;
        }
        if (kw && ks != 0.0) {
#pragma unroll
          for (int yy = 0; yy < FB; ++yy) {
#pragma unroll
            for (int cc = 0; cc < FC; ++cc) {
              double sum = 0.0;
#pragma unroll
              for (int xx = 0; xx < FA; ++xx)
#pragma unroll
                for (int dd = 0; dd < FD; ++dd) {
                  sum += G(xx, yy, cc, dd) * Dad[xx * FD + dd];
                  Kac[xx * FC + cc] += G(xx, yy, cc, dd) * Dbd[yy * FD + dd];
                }
              atomicAdd(Fm + (rowB + yy * N + aoC + cc), ks * sum);
            }
#pragma unroll
            for (int dd = 0; dd < FD; ++dd) {
              double sum = 0.0;
#pragma unroll
              for (int xx = 0; xx < FA; ++xx)
#pragma unroll
                for (int cc = 0; cc < FC; ++cc) {
                  sum += G(xx, yy, cc, dd) * Dac[xx * FC + cc];
                  Kad[xx * FD + dd] += G(xx, yy, cc, dd) * Dbc[yy * FC + cc];
                }
              atomicAdd(Fm + (rowB + yy * N + aoD + dd), ks * sum);
            }
          }
        }
      }
      // the tile's own blocks
      if (valid) {
        if (ks != 0.0) {
#pragma unroll
          for (int o = 0; o < FA * FC; ++o)
            if (Kac[o] != 0.0) atomicAdd(Fm + (size_t)(aoA + afun(o / FC)) * N + aoC + o % FC, ks * Kac[o]);
#pragma unroll
          for (int o = 0; o < FA * FD; ++o)
            if (Kad[o] != 0.0) atomicAdd(Fm + (size_t)(aoA + afun(o / FD)) * N + aoD + o % FD, ks * Kad[o]);
        }
        if (js != 0.0) {
#pragma unroll
          for (int o = 0; o < FC * FD; ++o)
            if (Jcd[o] != 0.0) atomicAdd(Fm + (size_t)(aoC + o / FD) * N + aoD + o % FD, js * Jcd[o]);
        }
      }
    }
  }
  if (seg >= 0) flush_jab();
}

#undef DGF_ROW_MATRICES

template <int LA, int LB, int LC, int LD, int CA, int CH, int FORM>
__device__ __forceinline__ void row_dispatch(int chunk, const JKArgs &a, const double *tab, double *wsm,
                                             unsigned long long &q, unsigned long long &s) {
  if constexpr (CH < CA) {
    if (chunk == CH)
      row_body<LA, LB, LC, LD, CA, CH, FORM>(a, tab, wsm, q, s);
    else
      row_dispatch<LA, LB, LC, LD, CA, CH + 1, FORM>(chunk, a, tab, wsm, q, s);
  }
}

// Adds a warp's counts of evaluated, primitive and screened quartets.
__device__ __forceinline__ void add_counts(const JKArgs &a, unsigned long long nq, unsigned long long np,
                                           unsigned long long ns) {
  if (!a.counters) return;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    nq += __shfl_xor_sync(0xffffffffu, nq, off);
    np += __shfl_xor_sync(0xffffffffu, np, off);
    ns += __shfl_xor_sync(0xffffffffu, ns, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (nq) atomicAdd(a.counters + 0, nq);
    if (np) atomicAdd(a.counters + 1, np);
    if (ns) atomicAdd(a.counters + 2, ns);
  }
}

}  // namespace row

// CA > 1: blockIdx.y takes one of CA chunks of A's functions, which bounds the
// registers; each chunk forms R_tuv and the ket transform again.
template <int LA, int LB, int LC, int LD, int CA, bool BT>
__global__ void __launch_bounds__(row::Shape<LA, LB, LC, LD, CA>::kBlock, row::Shape<LA, LB, LC, LD, CA>::kMinBlocks)
    jk_row_kernel(const __grid_constant__ JKArgs a) {
  using S = row::Shape<LA, LB, LC, LD, CA>;
  extern __shared__ double sm[];
  for (int i = threadIdx.x; i < kFineDoubles; i += blockDim.x) sm[i] = a.boys_fine[i];
  __syncthreads();
  unsigned long long cnt_q = 0, cnt_s = 0;
  row::row_dispatch<LA, LB, LC, LD, CA, 0, BT ? row::kBatch : row::kEval>(blockIdx.y, a, sm,
                                           sm + kFineDoubles + (size_t)(threadIdx.x >> 5) * S::kPerWarp, cnt_q, cnt_s);
  row::add_counts(a, cnt_q, cnt_q, cnt_s);  // one primitive quartet each
}

// The digestion of stored integral blocks (conventional form) with the same
// tiles: bound by the reads of the store and the two gathers and atomics per
// quartet that are left.
constexpr int kRowStoredBlock = 256;
template <int LA, int LB, int LC, int LD, int CA>
__global__ void __launch_bounds__(kRowStoredBlock, 2) jk_row_stored_kernel(const __grid_constant__ JKArgs a) {
  using S = row::Shape<LA, LB, LC, LD, CA>;
  extern __shared__ double sm[];
  unsigned long long cnt_q = 0, cnt_s = 0;
  row::row_dispatch<LA, LB, LC, LD, CA, 0, row::kStored>(blockIdx.y, a, nullptr, sm + (size_t)(threadIdx.x >> 5) * S::kPerWarp,
                                                 cnt_q, cnt_s);
  row::add_counts(a, cnt_q, 0, cnt_s);
}

}  // namespace dgf
