// Pack kernel: J/K quartets of high angular momentum (single-primitive pairs,
// spherical functions), a warp on one bra pair and several kets at a time,
// both Hermite contractions as dense FP64 tensor-core products (DMMA,
// mma.sync m8n8k4).
//
// A pair's Hermite coefficients with the spherical transforms folded in,
// E[function pair][tuv], do not depend on the partner, so they are formed
// once per context (pair_frag_kernel) in the order the DMMA fragments want
// them: a fragment is one coalesced 256-byte load, and the same table serves
// a pair as bra (rows of A) and as ket (columns of B).  Per ket
//   X[tuv][cd] = sum_f R'[tuv + f] E_cd[f],   R' = R_tuv of Q - P
// with A gathered from R' in shared memory, then for all kets of the pack
//   G[ab][cd] = sum_tuv E_ab[tuv] (-1)^{t+u+v} X[tuv][cd].
// The pack fills the columns of the product and the lanes of the digestion,
// which a single small ket leaves idle: with one quartet per warp, (fd|ps)
// ran its bra transform on 3 of 32 lanes.  Boys functions of 32 kets are
// evaluated together, one per lane.
#pragma once

#include "dgf_jk_row.cuh"
#include "dgf_jk_warp.cuh"
#include "dgf_pack.h"

namespace dgf {

namespace pack {

constexpr int nsph(int l) { return 2 * l + 1; }
// Fragment tiles of a pair class: rows (function pairs) by 8, tuv by 4.
constexpr int frag_mt(int la, int lb) { return (nsph(la) * nsph(lb) + 7) / 8; }
constexpr int frag_kt(int la, int lb) { return (n3(la + lb) + 3) / 4; }
constexpr int frag_doubles(int la, int lb) { return frag_mt(la, lb) * frag_kt(la, lb) * 32; }
// Smallest row length >= n that spreads eight rows of four doubles over all banks.
constexpr int row_stride(int n) {
  while (n % 16 != 4 && n % 16 != 12) ++n;
  return n;
}

template <int LA, int LB, int LC, int LD>
struct Shape {
  static constexpr int L = LA + LB + LC + LD, LAB = LA + LB, LCD = LC + LD;
  static constexpr int FA = nsph(LA), FB = nsph(LB), FC = nsph(LC), FD = nsph(LD), FAB = FA * FB, FCD = FC * FD;
  static constexpr int KE = n3(LAB), KF = n3(LCD), NR = n3(L);
  static constexpr int MT3 = frag_mt(LA, LB), KT3 = frag_kt(LA, LB);
  static constexpr int MT2 = (KE + 7) / 8, NT2 = frag_mt(LC, LD), KT2 = frag_kt(LC, LD);
  // kets of a pack: about 16 columns
  static constexpr int NQ = FCD >= 13 ? 1 : FCD == 9 ? 2 : 16 / FCD;
  static constexpr int COLS = NQ * FCD, NT3 = (COLS + 7) / 8;
  static constexpr int SB = L + 1, SA = SB * SB, RBOX = SA * L + 1;  // R_tuv at SA t + SB u + v
  static constexpr int SX = row_stride(KT3 * 4);                    // X[col][tuv]
  static constexpr int SG = NT3 * 8 + (NT3 % 2 == 0 ? 8 : 0);       // G[ab][col]: rows 64 bytes apart in the banks
  static constexpr int NDQ = FA * FC + FA * FD + FB * FC + FB * FD + FC * FD;  // staged densities of a ket
  static constexpr int PB = RBOX > FAB * SG ? RBOX : FAB * SG;      // R box, later G
  static constexpr int PX = (NT3 * 8) * SX;
  static constexpr int PD = NQ * NDQ + FAB;
  static constexpr int PF = 32 * (L + 4);  // scaled Boys values and Q - P of a chunk's kets
  static constexpr int PER_WARP = ((PB + PX + PD + PF + 1) & ~1) + 32;  // last: {aoC, aoD} of a chunk's kets
  static constexpr int COMMON = kBoysTableDoubles + (NR + 3) / 4 * 2;  // Boys table, element table
  static constexpr size_t smem(int warps) { return (size_t)(COMMON + warps * PER_WARP) * 8; }
  static constexpr int WPB = smem(4) <= 110 * 1024 ? 4 : smem(2) <= 110 * 1024 ? 2 : 1;
  static constexpr int kBlocks = (int)((size_t)220 * 1024 / smem(WPB));  // resident blocks per SM by shared memory
  static constexpr int kMinBlocks = kBlocks * WPB <= 16 ? kBlocks : 16 / WPB;  // registers for up to 16 warps per SM
  static constexpr int MB = MT3 * NT3 <= 16 ? MT3 : (16 / NT3 > 0 ? 16 / NT3 : 1);  // row tiles of G at a time
};

}  // namespace pack

// Fragments of every pair of a class: element (row, k) of tile (mt, kk) at
// lane 4 (row % 8) + k % 4.  A warp per pair.
template <int LA, int LB>
__global__ void __launch_bounds__(128) pair_frag_kernel(const PairRec *pairs, const PrimPair *pp, int npair,
                                                        const double *sph, double *out) {
  constexpr int EA = (LA + 1) * (LB + 1) * (LA + LB + 1), NT = LA + LB + 1;
  constexpr int NA = ncart(LA), NB = ncart(LB), FA = pack::nsph(LA), FB = pack::nsph(LB);
  constexpr int MT = pack::frag_mt(LA, LB), KT = pack::frag_kt(LA, LB), KE = n3(LA + LB);
  __shared__ double E[4][3 * EA];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double *ca = sph + sph_offset(LA), *cb = sph + sph_offset(LB);
  for (int e = blockIdx.x * 4 + warp; e < npair; e += gridDim.x * 4) {
    const PrimPair P = load_prim<true>(pp + pairs[e].pp0);
    __syncwarp();
    if (lane < 3) {
      const double pa = lane == 0 ? P.PAx : lane == 1 ? P.PAy : P.PAz;
      const double pb = lane == 0 ? P.PBx : lane == 1 ? P.PBy : P.PBz;
      herm_e<LA, LB, 1, double>(0.5 / P.p, pa, pb, E[warp] + lane * EA);
    }
    __syncwarp();
    double *o = out + (size_t)e * pack::frag_doubles(LA, LB);
    for (int tile = 0; tile < MT * KT; ++tile) {
      const int row = tile / KT * 8 + (lane >> 2), k = tile % KT * 4 + (lane & 3);
      double v = 0.0;
      if (row < FA * FB && k < KE) {
        const int a = row / FB, b = row % FB;
        int t, u, w;
        tuv_decode(k, t, u, w);
        for (int ia = 0; ia < NA; ++ia) {
          const double fa = ca[a * NA + ia];
          if (fa == 0.0) continue;
          int ax, ay, az;
          cart_decode(LA, ia, ax, ay, az);
          for (int jb = 0; jb < NB; ++jb) {
            const double fb = cb[b * NB + jb];
            if (fb == 0.0) continue;
            int bx, by, bz;
            cart_decode(LB, jb, bx, by, bz);
            if (t > ax + bx || u > ay + by || w > az + bz) continue;
            v += fa * fb * E[warp][(ax * (LB + 1) + bx) * NT + t] * E[warp][EA + (ay * (LB + 1) + by) * NT + u] *
                 E[warp][2 * EA + (az * (LB + 1) + bz) * NT + w];
          }
        }
      }
      o[tile * 32 + lane] = v;
    }
  }
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(32 * pack::Shape<LA, LB, LC, LD>::WPB, pack::Shape<LA, LB, LC, LD>::kMinBlocks)
    jk_pack_kernel(const __grid_constant__ JKArgs a, const PackArgs pk) {
  using S = pack::Shape<LA, LB, LC, LD>;
  constexpr int L = S::L, FA = S::FA, FB = S::FB, FC = S::FC, FD = S::FD, FAB = S::FAB, FCD = S::FCD, KE = S::KE,
                KF = S::KF, NQ = S::NQ, SA = S::SA, SB = S::SB, SX = S::SX, SG = S::SG, NDQ = S::NDQ;
  constexpr int RT = (S::NR + 31) / 32;  // R_tuv elements of a lane
  static_assert(NQ * 5 <= 64, "lanes of a pack are packed in 64 bits");
  constexpr unsigned full = 0xffffffffu;
  extern __shared__ double sm[];
  double *tab = sm;
  int *lev = (int *)(sm + kBoysTableDoubles);  // element: position | direction << 14 | (index - 1) << 16
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  double *box = sm + S::COMMON + (size_t)warp * S::PER_WARP, *X = box + S::PB, *Db = X + S::PX, *Fs = Db + S::PD;
  int2 *ao = (int2 *)(box + ((S::PB + S::PX + S::PD + S::PF + 1) & ~1));
  for (int i = threadIdx.x; i < kBoysTableDoubles; i += blockDim.x) tab[i] = a.boys[i];
  for (int e = threadIdx.x; e < S::NR; e += blockDim.x) {
    int t, u, v;
    tuv_decode(e, t, u, v);
    const int d = t > 0 ? 0 : u > 0 ? 1 : 2, m = t > 0 ? t : u > 0 ? u : v;
    lev[e] = (t * SA + u * SB + v) | (d << 14) | ((m > 0 ? m - 1 : 0) << 16);
  }
  // the products' depth is padded with zero coefficients: their partners must be finite
  for (int c = lane; c < S::NT3 * 8; c += 32)
    for (int k = KE; k < S::KT3 * 4; ++k) X[c * SX + k] = 0.0;
  __syncthreads();
  const int N = a.nbf;
  unsigned long long cnt_q = 0, cnt_s = 0;
  for (;;) {
    int t = 0;
    if (lane == 0) t = (int)atomicAdd(a.row_work, 1u);
    t = __shfl_sync(full, t, 0) + a.row_task0;
    if (t >= a.row_task1) break;
    const int4 tk = __ldg(a.row_tasks + t);
    const int kend = min(tk.w, tk.z + 32 * (tk.y >> 16));
    for (int r0 = 0; r0 < (tk.y & 0xffff); ++r0) {
    const int ib = __ldg(a.row_bra + tk.x + r0);
    const PairRec br = load_pair_fock(a.bra + ib);
    const PrimPair P1 = load_prim<false>(a.pp + br.pp0);
    const double *bf = pk.bra_frag + (size_t)ib * pack::frag_doubles(LA, LB) + lane;
    double jacc[(FAB + 31) / 32];
#pragma unroll
    for (int k = 0; k < (FAB + 31) / 32; ++k) jacc[k] = 0.0;
    const bool jreg = a.nslot == 1;
    for (int ic0 = tk.z; ic0 < kend; ic0 += 32) {
      const int ic = ic0 + lane;
      const bool valid = ic < kend && (!a.same_class || ic + a.ket_off <= ib);
      const PairRec kt = load_pair_fock(a.ket + min(ic, kend - 1));
      bool work = false;
      if (valid) {
        const int sel = quartet_select(a, br, kt, a.bra + ib, a.ket + ic);
        work = sel == 0;
        if (sel == 2) ++cnt_s;
      }
      unsigned todo = __ballot_sync(full, work);
      if (!todo) continue;
      cnt_q += work;
      __syncwarp();
      if (work) {  // one ket per lane: scaled Boys values and Q - P
        const PrimPair P2 = load_prim<false>(a.pp + kt.pp0);
        double w = 1.0;
        if (br.same) w *= 0.5;
        if (kt.same) w *= 0.5;
        if (a.same_class && ib == ic + a.ket_off) w *= 0.5;
        const double rs = rsqrt(P1.p + P2.p);
        double alpha = P1.p * P2.p * rs * rs, s = P1.K * P2.K * rs * w;
        erf_attenuate(a.erf_mu2, alpha, s);
        const double x = P2.Px - P1.Px, y = P2.Py - P1.Py, z = P2.Pz - P1.Pz;
        double F[L + 1];
        boys_eval<L>(alpha * (x * x + y * y + z * z), tab, F);
        double *o = Fs + lane * (L + 4);
#pragma unroll
        for (int n = 0; n <= L; ++n) {
          o[n] = s * F[n];
          s *= -2.0 * alpha;
        }
        o[L + 1] = x;
        o[L + 2] = y;
        o[L + 3] = z;
        ao[lane] = make_int2(kt.aoA, kt.aoB);
      }
      __syncwarp();
      while (todo) {
        // the next kets of the chunk: their lanes, packed 5 bits each
        int nq = 0;
        unsigned long long lanes = 0;
        while (nq < NQ && todo) {
          lanes |= (unsigned long long)(__ffs(todo) - 1) << (5 * nq++);
          todo &= todo - 1;
        }
        for (int q = 0; q < nq; ++q) {
          const int kl = (int)(lanes >> (5 * q)) & 31;
          const double *f = Fs + kl * (L + 4);
          const double xyz[3] = {f[L + 1], f[L + 2], f[L + 3]};
          if (lane == 0) box[0] = f[L];
          __syncwarp();
          // R'_tuv, level n from level n + 1, in place: a lane's elements are
          // read before any is written.  Their places and coefficients are
          // the same at every level.
          const double *src[RT];
          double cx[RT], cm[RT];
          int st[RT];
#pragma unroll
          for (int k = 0; k < RT; ++k) {
            const int e = lane + 32 * k, le = e < S::NR ? lev[e] : 0, d = (le >> 14) & 3;
            st[k] = d == 0 ? SA : d == 1 ? SB : 1;
            cx[k] = d == 0 ? xyz[0] : d == 1 ? xyz[1] : xyz[2];
            cm[k] = (double)(le >> 16);
            src[k] = box + (le & 0x3fff) - (e > 0 ? st[k] : 0);
          }
#pragma unroll 1
          for (int n = L - 1; n >= 0; --n) {
            const int cnt = n3(L - n);
            double val[RT];
#pragma unroll
            for (int k = 0; k < RT; ++k)
              if (lane + 32 * k < cnt) {
                val[k] = cx[k] * src[k][0];
                if (cm[k] > 0.0) val[k] += cm[k] * src[k][-st[k]];
                if (k == 0 && lane == 0) val[0] = f[n];
              }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < RT; ++k)
              if (lane + 32 * k < cnt) box[src[k] - box + (lane + 32 * k > 0 ? st[k] : 0)] = val[k];
            __syncwarp();
          }
          // ket product: rows tuv, columns cd
          const int kc = __shfl_sync(full, ic, kl);
          const double *kf = pk.ket_frag + (size_t)kc * pack::frag_doubles(LC, LD) + lane;
          int pf[S::KT2];
#pragma unroll
          for (int kk = 0; kk < S::KT2; ++kk) {
            const int fi = kk * 4 + t4;
            pf[kk] = fi < KF ? lev[fi] & 0x3fff : 0;
          }
          constexpr bool HOLD = S::NT2 * S::KT2 <= 12;  // the ket's fragments stay in registers
          double bk[HOLD ? S::NT2 * S::KT2 : 1];
          if constexpr (HOLD) {
#pragma unroll
            for (int i = 0; i < S::NT2 * S::KT2; ++i) bk[i] = __ldg(kf + i * 32);
          }
#pragma unroll 1
          for (int mt = 0; mt < S::MT2; ++mt) {
            const int e = mt * 8 + g, le = e < KE ? lev[e] : 0, pe = le & 0x3fff;
            double d0[S::NT2], d1[S::NT2];
#pragma unroll
            for (int nt = 0; nt < S::NT2; ++nt) d0[nt] = d1[nt] = 0.0;
#pragma unroll
            for (int kk = 0; kk < S::KT2; ++kk) {
              const double av = box[pe + pf[kk]];
#pragma unroll
              for (int nt = 0; nt < S::NT2; ++nt)
                wq::dmma(d0[nt], d1[nt], av, HOLD ? bk[HOLD ? nt * S::KT2 + kk : 0] : __ldg(kf + (nt * S::KT2 + kk) * 32));
            }
            if (e < KE) {
              // (-1)^{t+u+v}: the parity of the position's indices
              const int tt = pe / SA, uu = (pe % SA) / SB, vv = pe % SB;
              const double sg = ((tt + uu + vv) & 1) ? -1.0 : 1.0;
#pragma unroll
              for (int nt = 0; nt < S::NT2; ++nt) {
                const int c0 = nt * 8 + 2 * t4;
                if (c0 < FCD) X[(q * FCD + c0) * SX + e] = sg * d0[nt];
                if (c0 + 1 < FCD) X[(q * FCD + c0 + 1) * SX + e] = sg * d1[nt];
              }
            }
          }
          __syncwarp();
        }
        // bra product for the whole pack; G replaces the R box
        double *G = box;
#pragma unroll 1
        for (int m0 = 0; m0 < S::MT3; m0 += S::MB) {
          double acc[S::MB][S::NT3][2];
#pragma unroll
          for (int i = 0; i < S::MB; ++i)
#pragma unroll
            for (int nt = 0; nt < S::NT3; ++nt) acc[i][nt][0] = acc[i][nt][1] = 0.0;
#pragma unroll 2
          for (int kk = 0; kk < S::KT3; ++kk) {
            double bv[S::NT3];
#pragma unroll
            for (int nt = 0; nt < S::NT3; ++nt) bv[nt] = X[(nt * 8 + g) * SX + kk * 4 + t4];
#pragma unroll
            for (int i = 0; i < S::MB; ++i) {
              const double av = m0 + i < S::MT3 ? __ldg(bf + ((m0 + i) * S::KT3 + kk) * 32) : 0.0;
#pragma unroll
              for (int nt = 0; nt < S::NT3; ++nt) wq::dmma(acc[i][nt][0], acc[i][nt][1], av, bv[nt]);
            }
          }
#pragma unroll
          for (int i = 0; i < S::MB; ++i) {
            const int r = (m0 + i) * 8 + g;
            if (r < FAB) {
#pragma unroll
              for (int nt = 0; nt < S::NT3; ++nt)
                *reinterpret_cast<double2 *>(G + r * SG + nt * 8 + 2 * t4) = make_double2(acc[i][nt][0], acc[i][nt][1]);
            }
          }
        }
        __syncwarp();
        // Digestion: every output element of the pack's blocks on a lane.
        unsigned jm = (1u << nq) - 1u, km = jm;
        for (int k = 0; k < a.nslot; ++k) {
          const double *Dk = a.D + k * a.slot_stride, *Dsk = a.Ds + k * a.slot_stride;
          double *Fk = a.Fh + k * a.slot_stride;
          const double js = a.jscale[k], ks = -a.kscale[k];
          if (a.ice_thr > 0.0) {  // ICEDIF: quartets of whole Dalton blocks
            jm = km = (1u << nq) - 1u;
            const int4 bb = block_of_pair(a.bra + ib);
            for (int q = 0; q < nq; ++q) {
              const int kc = __shfl_sync(full, ic, (int)(lanes >> (5 * q)) & 31);
              const int4 kb = block_of_pair(a.ket + kc);
              if (!(bb.z & bb.w & kb.z & kb.w)) continue;
              double am = 0.0;
              for (int e = lane; e < FAB * FCD; e += 32) am = fmax(am, fabs(G[e / FCD * SG + q * FCD + e % FCD]));
#pragma unroll
              for (int off = 16; off > 0; off >>= 1) am = fmax(am, __shfl_xor_sync(full, am, off));
              const PairRec kr = load_pair_fock(a.ket + kc);
              double w = 1.0;  // the weight is part of G
              if (br.same) w *= 0.5;
              if (kr.same) w *= 0.5;
              if (a.same_class && ib == kc + a.ket_off) w *= 0.5;
              am /= w;
              const float *dm = a.blk_dmax_slot + k * a.blk_stride;
              const int n = a.nblk;
              const double dj = fmaxf(dm[bb.x * n + bb.y], dm[kb.x * n + kb.y]);
              const double dk = fmaxf(fmaxf(dm[bb.x * n + kb.x], dm[bb.x * n + kb.y]),
                                      fmaxf(dm[bb.y * n + kb.x], dm[bb.y * n + kb.y]));
              if ((a.icedif & 1) && dj * am < a.ice_thr) jm &= ~(1u << q);
              if ((a.icedif & 2) && dk * am < a.ice_thr) km &= ~(1u << q);
            }
          }
          // density blocks of the pack's kets, and of the bra
          double *Dab = Db + NQ * NDQ;
          for (int e = lane; e < FAB; e += 32) Dab[e] = __ldg(Dsk + (size_t)(br.aoA + e / FB) * N + br.aoB + e % FB);
          for (int i = lane; i < nq * NDQ; i += 32) {
            const int q = i / NDQ, r = i - q * NDQ;
            const int2 cd = ao[(int)(lanes >> (5 * q)) & 31];
            const double *M = Dk;
            int row, col;
            if (r < FA * FC) {
              row = br.aoA + r / FC, col = cd.x + r % FC;
            } else if (r < FA * (FC + FD)) {
              row = br.aoA + (r - FA * FC) / FD, col = cd.y + (r - FA * FC) % FD;
            } else if (r < FA * (FC + FD) + FB * FC) {
              row = br.aoB + (r - FA * (FC + FD)) / FC, col = cd.x + (r - FA * (FC + FD)) % FC;
            } else if (r < (FA + FB) * (FC + FD)) {
              row = br.aoB + (r - FA * (FC + FD) - FB * FC) / FD, col = cd.y + (r - FA * (FC + FD) - FB * FC) % FD;
            } else {
              M = Dsk;
              row = cd.x + (r - (FA + FB) * (FC + FD)) / FD, col = cd.y + (r - (FA + FB) * (FC + FD)) % FD;
            }
            Db[i] = __ldg(M + (size_t)row * N + col);
          }
          __syncwarp();
          constexpr int oAD = FA * FC, oBC = FA * (FC + FD), oBD = oBC + FB * FC, oCD = (FA + FB) * (FC + FD);
          if (js != 0.0) {
#pragma unroll
            for (int i = 0; i < (FAB + 31) / 32; ++i) {  // J_ab
              const int e = lane + 32 * i;
              if (e < FAB) {
                double s = 0.0;
                for (int q = 0; q < nq; ++q)
                  if ((jm >> q) & 1u) {
                    const double *Gr = G + e * SG + q * FCD, *dc = Db + q * NDQ + oCD;
#pragma unroll
                    for (int c = 0; c < FCD; ++c) s += Gr[c] * dc[c];
                  }
                if (jreg)
                  jacc[i] += s;
                else
                  atomicAdd(Fk + (size_t)(br.aoA + e / FB) * N + br.aoB + e % FB, js * s);
              }
            }
            for (int i = lane; i < nq * FCD; i += 32) {  // J_cd
              const int q = i / FCD, c = i - q * FCD;
              if (!((jm >> q) & 1u)) continue;
              double s = 0.0;
#pragma unroll 5
              for (int e = 0; e < FAB; ++e) s += G[e * SG + i] * Dab[e];
              const int2 cd = ao[(int)(lanes >> (5 * q)) & 31];
              atomicAdd(Fk + (size_t)(cd.x + c / FD) * N + cd.y + c % FD, js * s);
            }
          }
          if (ks != 0.0 && km) {
            constexpr int NO = (FA + FB) * (FC + FD);
            for (int i = lane; i < nq * NO; i += 32) {
              const int q = i / NO, r = i - q * NO;
              if (!((km >> q) & 1u)) continue;
              const int2 cd = ao[(int)(lanes >> (5 * q)) & 31];
              const double *Gq = G + q * FCD, *dq = Db + q * NDQ;
              double s = 0.0;
              int row, col;
              if (r < oAD) {  // K_ac = sum_bd g D_bd
                const int x = r / FC, c = r % FC;
#pragma unroll
                for (int y = 0; y < FB; ++y)
#pragma unroll
                  for (int d = 0; d < FD; ++d) s += Gq[(x * FB + y) * SG + c * FD + d] * dq[oBD + y * FD + d];
                row = br.aoA + x, col = cd.x + c;
              } else if (r < oBC) {  // K_ad = sum_bc g D_bc
                const int x = (r - oAD) / FD, d = (r - oAD) % FD;
#pragma unroll
                for (int y = 0; y < FB; ++y)
#pragma unroll
                  for (int c = 0; c < FC; ++c) s += Gq[(x * FB + y) * SG + c * FD + d] * dq[oBC + y * FC + c];
                row = br.aoA + x, col = cd.y + d;
              } else if (r < oBD) {  // K_bc = sum_ad g D_ad
                const int y = (r - oBC) / FC, c = (r - oBC) % FC;
#pragma unroll
                for (int x = 0; x < FA; ++x)
#pragma unroll
                  for (int d = 0; d < FD; ++d) s += Gq[(x * FB + y) * SG + c * FD + d] * dq[oAD + x * FD + d];
                row = br.aoB + y, col = cd.x + c;
              } else {  // K_bd = sum_ac g D_ac
                const int y = (r - oBD) / FD, d = (r - oBD) % FD;
#pragma unroll
                for (int x = 0; x < FA; ++x)
#pragma unroll
                  for (int c = 0; c < FC; ++c) s += Gq[(x * FB + y) * SG + c * FD + d] * dq[x * FC + c];
                row = br.aoB + y, col = cd.y + d;
              }
              atomicAdd(Fk + (size_t)row * N + col, ks * s);
            }
          }
          __syncwarp();
        }
      }
    }
    if (jreg && a.jscale[0] != 0.0) {
#pragma unroll
      for (int i = 0; i < (FAB + 31) / 32; ++i) {
        const int e = lane + 32 * i;
        if (e < FAB && jacc[i] != 0.0)
          atomicAdd(a.Fh + (size_t)(br.aoA + e / FB) * N + br.aoB + e % FB, a.jscale[0] * jacc[i]);
      }
    }
    }
  }
  row::add_counts(a, cnt_q, cnt_q, cnt_s);
}

}  // namespace dgf
