// Adjoint of the DG right-hand side on the FP64 tensor cores (orders 1 to 7):
// the transposes of rhs_fp64.cuh's contraction, batched over elements the same
// way.
//
//   adj_lift_kernel     W[e][p][f] = Fscale s_f sum_i LIFT[i][p] lam_f[i]
//                       (s_f the model's output scale), M = face points;
//   adj_element_kernel  q_bar = [ D_1^T .. D_d^T ] . [ y_1; ..; y_d ] + w at
//                       the face points' nodes, with y_r the transposed chain
//                       rule and volume map of s_f lam_f at the nodes and w
//                       the transposed fluxes of both sides at the face
//                       points (the neighbour's from its W: a gather, no
//                       atomics).  The output pass adds a node's face points
//                       from a list: as one more block of the product, a 0/1
//                       matrix, a w that is not finite would make every node
//                       of the element NaN.
//
// The c gradient of the variable-velocity wave rides along: the face part is
// one more row of w, the volume part sum_f s_f lam_f vol_f(grad q, c = 1) a
// second contraction with the forward derivatives.
//
// Either kernel may also carry one step of the reversed LSRK recurrences
//   lam <- lam + b lq;  lq <- lq + dt (dR/dq)^T lam;  c_bar <- c_bar + dt
//   (dR/dc)^T lam;  lam <- a lam
// (the transpose of hedge/timestep/runge_kutta.py:123-128): the lift kernel
// forms lam in place, the element kernel reads only its own element's and
// writes the rest, so that a stage is two launches and no vector passes.
//
// Bound: launch latency and the point phases.  Both passes, against one block
// per element with the operators read by thread rows: variable-velocity wave
// with the c gradient, 2D, K = 7200, N = 5, 55 -> 20 us, K = 24200 156 -> 79 us; 3D, K =
// 1296, N = 4 77 -> 20 us; 3D Maxwell, K = 6000, N = 4 283 -> 81 us.  8 LSRK4 steps with
// receivers forward and backward at K = 2112, N = 4 take half of the time before.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "dmma.cuh"
#include "models.cuh"
#include "rhs_fp64.cuh"

namespace hb {

// flux at one face point with the given argument vectors (zero when the
// boundary carries no flux)
template <int MODEL, int DIM>
__device__ __forceinline__ void adj_flux_at(const ModelParams& mp, bool bdry, int kind,
                                            const double (&uM)[Args<MODEL, DIM>::N],
                                            const double (&uPin)[Args<MODEL, DIM>::N],
                                            const double (&n)[DIM],
                                            double (&fl)[Traits<MODEL, DIM>::F]) {
  constexpr int NA = Args<MODEL, DIM>::N;
  constexpr int F = Traits<MODEL, DIM>::F;
  double uP[NA];
#pragma unroll
  for (int q = 0; q < NA; ++q) uP[q] = uPin[q];
  if (bdry && !model_bc<MODEL, DIM, double>(mp, kind, uM, n, 0.0, uP)) {
#pragma unroll
    for (int f = 0; f < F; ++f) fl[f] = 0.0;
    return;
  }
  model_flux<MODEL, DIM, double>(mp, bdry, uM, uP, n, fl);
}

template <int MODEL, int DIM, int ORDER, bool WC>
struct AdjShape : F64Shape<MODEL, DIM, ORDER> {
  using B = F64Shape<MODEL, DIM, ORDER>;
  using B::F; using B::C; using B::NP; using B::NFP; using B::NF; using B::NFPT; using B::G;
  using B::KV; using B::MT; using B::RN; using B::NGW; using B::KG; using B::THREADS;
  using B::COLS; using B::LDP;
  // values per face point: the fields, and the c gradient's
  static constexpr int CF = F + (WC ? 1 : 0);
  static constexpr int EB = COLS / CF;
  static constexpr int KP = f64_ru8(KV);
  static constexpr int STEPS = KP / 8;             // of either direction's derivatives
  static constexpr int LDZ = KP % 16 == 8 ? KP : KP + 8;
  static constexpr int ENP = EB * NP;
  static constexpr size_t al(size_t x) { return (x + 15) & ~size_t(15); }
  static constexpr size_t zdoubles =
      COLS * LDZ > KG * COLS * LDP ? COLS * LDZ : KG * COLS * LDP;
  static constexpr size_t oW = al(8 * zdoubles);               // [EB][CF][NFPT] w
  static constexpr size_t oL = al(oW + 8 * EB * CF * NFPT);    // [F][EB][NP] s_f lam_f
  static constexpr size_t oQ = al(oL + 8 * F * ENP);           // [F][EB][NP] state (WC)
  static constexpr size_t oC = al(oQ + (WC ? 8 * F * ENP : 0));   // [EB][NP]
  static constexpr size_t oV = al(oC + 8 * C * ENP);           // [EB][NP] volume c part
  static constexpr size_t oG = al(oV + (WC ? 8 * ENP : 0));
  static constexpr size_t oN = al(oG + 8 * EB * G);
  static constexpr size_t oFm = al(oN + 8 * EB * NF);
  static constexpr size_t oSh = al(oFm + NFPT);                // shuffle
  static constexpr int NLIST = NP + 1 + NFPT;
  static constexpr size_t oNl = al(oSh + 6 * NFP);             // nodes' face points
  static constexpr size_t total = al(oNl + NLIST);
  // lift pass: M = face points, the row tiles split over the warps
  static constexpr int LW = 4;
  static constexpr int LMT = (NFPT + 7) / 8;
  static constexpr int LMW = (LMT + LW - 1) / LW;              // row tiles per warp
  static constexpr int LSTEPS = f64_ru8(NP) / 8;
  static constexpr int LK = LSTEPS * 8;
  static constexpr int LLDZ = LK % 16 == 8 ? LK : LK + 8;
  static constexpr int LRN = 2;
  static constexpr int LCOLS = 32;                             // columns per batch
  static constexpr int LEB = LCOLS / F;
  static constexpr int LLDP = LW * LMW * 8 + 2;
  static constexpr size_t lP = al(8 * LCOLS * LLDZ);
  static constexpr size_t ltotal = al(lP + 8 * LCOLS * LLDP);
};

struct AdjArgs {
  int64_t K, nbatch;
  int E, nperm;
  const double2* lfrag;      // LIFT^T fragments [LSTEPS][LW * LMW][32]
  const double2* afrag;      // [D^T] fragments
  const double2* vfrag;      // [D] fragments (c gradient)
  const uint8_t* nlist;      // [np + 1] begins of the nodes' face points, the face points
  const double* geo;
  const int2* conn;
  const int* fmask;
  const int* shuffle;
  const double* q;
  const double* lam_in;      // the cotangent
  const double* coeff;
  double* work;              // W
  double* q_bar;
  double* c_bar;
  // the recurrence step (fused): lam and lq in place
  int fused;
  double* lam;
  double* lq;
  double ra, rb, dt;
  ModelParams mp;
  int* err;
};

template <int MODEL, int DIM, int ORDER>
__global__ void __launch_bounds__(128) adj_lift_kernel(const AdjArgs a) {
  using S = AdjShape<MODEL, DIM, ORDER, false>;
  constexpr int F = S::F, NP = S::NP, NFP = S::NFP, NFPT = S::NFPT, G = S::G;
  extern __shared__ __align__(16) unsigned char smem[];
  double* sZ = reinterpret_cast<double*>(smem);
  double* sP = reinterpret_cast<double*>(smem + S::lP);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t Knp = a.K * NP;
  double sf[F];
#pragma unroll
  for (int f = 0; f < F; ++f) sf[f] = model_finish<MODEL, DIM, double>(a.mp, f, 1.0, 0.0, 0.0);
  // rows NP .. LK stay zero
  for (int x = tid; x < S::LCOLS * 8; x += 128)
    if (NP + x % 8 < S::LK) sZ[(x / 8) * S::LLDZ + NP + x % 8] = 0.0;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int64_t batch = blockIdx.x; batch < a.nbatch; batch += gridDim.x) {
    const int64_t el0 = batch * a.E;
    const int ne = (int)(a.K - el0 < a.E ? a.K - el0 : a.E);
    for (int x = tid; x < ne * NP; x += 128) {
      const int e = x / NP, j = x - e * NP;
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const int64_t gi = f * Knp + el0 * NP + x;
        double l;
        if (a.fused) {
          l = a.lam[gi] + a.rb * a.lq[gi];
          a.lam[gi] = l;
        } else {
          l = a.lam_in[gi];
        }
        sZ[(e * F + f) * S::LLDZ + j] = sf[f] * l;
      }
    }
    __syncthreads();
    for (int cg = 0; cg * S::LRN * 8 < ne * F; ++cg) {
      double acc[S::LMW][S::LRN][2];
#pragma unroll
      for (int m = 0; m < S::LMW; ++m)
#pragma unroll
        for (int c = 0; c < S::LRN; ++c) acc[m][c][0] = acc[m][c][1] = 0.0;
      dmma_steps<S::LMW, S::LRN, S::LLDZ>(
          acc, a.lfrag + (size_t)warp * S::LSTEPS * S::LMW * 32 + lane,
          sZ + (cg * S::LRN * 8 + (lane >> 2)) * S::LLDZ + 2 * (lane & 3), S::LSTEPS);
      double* P = sP + (cg * S::LRN * 8 + 2 * (lane & 3)) * S::LLDP + warp * S::LMW * 8 + (lane >> 2);
#pragma unroll
      for (int m = 0; m < S::LMW; ++m)
#pragma unroll
        for (int c = 0; c < S::LRN; ++c) {
          P[c * 8 * S::LLDP + m * 8] = acc[m][c][0];
          P[(c * 8 + 1) * S::LLDP + m * 8] = acc[m][c][1];
        }
    }
    __syncthreads();
    for (int x = tid; x < ne * NFPT; x += 128) {
      const int e = x / NFPT, p = x - e * NFPT, fc = p / NFP;
      const double fscale = __ldg(a.geo + (el0 + e) * G + DIM * DIM + fc * (DIM + 1) + DIM);
      double* w = a.work + (el0 * NFPT + x) * F;
#pragma unroll
      for (int f = 0; f < F; ++f) w[f] = fscale * sP[(e * F + f) * S::LLDP + p];
    }
    // the next batch writes Z, which all warps have read, and P only after
    // its own barrier
  }
}

template <int MODEL, int DIM, int ORDER, bool WC>
__global__ void __launch_bounds__(F64Shape<MODEL, DIM, ORDER>::THREADS,
                                  F64Shape<MODEL, DIM, ORDER>::MT <= 5 ? 3 : 1)
    adj_element_kernel(const AdjArgs a) {
  using S = AdjShape<MODEL, DIM, ORDER, WC>;
  constexpr int F = S::F, C = S::C, NP = S::NP, NFP = S::NFP, NF = S::NF, NFPT = S::NFPT;
  constexpr int NA = F + C, CF = S::CF, G = S::G, LDZ = S::LDZ, ENP = S::ENP;
  constexpr int THREADS = S::THREADS, MT = S::MT, RN = S::RN, KG = S::KG, KV = S::KV;
  extern __shared__ __align__(16) unsigned char smem[];
  double* sZ = reinterpret_cast<double*>(smem);
  double* sl = reinterpret_cast<double*>(smem + S::oL);
  double* sq = reinterpret_cast<double*>(smem + S::oQ);
  double* sc = reinterpret_cast<double*>(smem + S::oC);
  double* sv = reinterpret_cast<double*>(smem + S::oV);
  double* sgeo = reinterpret_cast<double*>(smem + S::oG);
  int2* sconn = reinterpret_cast<int2*>(smem + S::oN);
  uint8_t* sfm = smem + S::oFm;
  uint8_t* ssh = smem + S::oSh;
  uint8_t* snl = smem + S::oNl;
  double* sw = reinterpret_cast<double*>(smem + S::oW);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kg = warp % KG, ng = warp / KG;
  const int64_t Knp = a.K * NP;
  for (int x = tid; x < NFPT; x += THREADS) sfm[x] = (uint8_t)a.fmask[x];
  for (int x = tid; x < a.nperm * NFP; x += THREADS) ssh[x] = (uint8_t)a.shuffle[x];
  for (int x = tid; x < S::NLIST; x += THREADS) snl[x] = a.nlist[x];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // product with a derivative operator over the columns [0, cols), partial
  // sums into Z
  auto gemm = [&](const double2* frag, int cols) {
    const bool work = ng * RN * 8 < cols;
    double acc[MT][RN][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int c = 0; c < RN; ++c) acc[m][c][0] = acc[m][c][1] = 0.0;
    if (work) {
      const int s0 = kg * S::STEPS / KG, s1 = (kg + 1) * S::STEPS / KG;
      dmma_steps<MT, RN, LDZ>(
          acc, frag + (size_t)s0 * MT * 32 + lane,
          sZ + (ng * RN * 8 + (lane >> 2)) * LDZ + 2 * (lane & 3) + 8 * s0, s1 - s0);
    }
    __syncthreads();
    if (work) {
      double* P = sZ + (size_t)kg * S::COLS * S::LDP +
                  (ng * RN * 8 + 2 * (lane & 3)) * S::LDP + (lane >> 2);
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int c = 0; c < RN; ++c) {
          P[c * 8 * S::LDP + m * 8] = acc[m][c][0];
          P[(c * 8 + 1) * S::LDP + m * 8] = acc[m][c][1];
        }
    }
    __syncthreads();
  };
  // the rows that pad a column of Z, fewer than 8
  auto zero_rows = [&](int cols) {
    for (int x = tid; x < cols * 8; x += THREADS)
      if (KV + x % 8 < S::KP) sZ[(x / 8) * LDZ + KV + x % 8] = 0.0;
  };
  auto sum = [&](int col, int i) {
    double v = sZ[col * S::LDP + i];
#pragma unroll
    for (int g = 1; g < KG; ++g) v += sZ[(g * S::COLS + col) * S::LDP + i];
    return v;
  };

  for (int64_t batch = blockIdx.x; batch < a.nbatch; batch += gridDim.x) {
    const int64_t el0 = batch * a.E;
    const int ne = (int)(a.K - el0 < a.E ? a.K - el0 : a.E);
    __syncthreads();   // the previous batch is done with shared memory
    for (int x = tid; x < ne * G; x += THREADS) cp_async8(sgeo + x, a.geo + el0 * G + x);
    for (int x = tid; x < ne * NF; x += THREADS) cp_async8(sconn + x, a.conn + el0 * NF + x);
    for (int x = tid; x < ne * NP; x += THREADS) {
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const int64_t gi = f * Knp + el0 * NP + x;
        cp_async8(sl + f * ENP + x, (a.fused ? a.lam : a.lam_in) + gi);
        if constexpr (WC) cp_async8(sq + f * ENP + x, a.q + gi);
      }
      if constexpr (C != 0) cp_async8(sc + x, a.coeff + el0 * NP + x);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();

    if constexpr (WC) {
      // ---- volume part of the c gradient: forward derivatives of q ----
      for (int x = tid; x < ne * NP; x += THREADS) {
        const int e = x / NP, j = x - e * NP;
        const double* ge = sgeo + e * G;
        double* z = sZ + e * F * LDZ + j;
#pragma unroll
        for (int r = 0; r < DIM; ++r) {
          double g[DIM][F], vol[F];
#pragma unroll
          for (int d = 0; d < DIM; ++d)
#pragma unroll
            for (int f = 0; f < F; ++f) g[d][f] = ge[r * DIM + d] * sq[f * ENP + x];
          model_volume<MODEL, DIM, double>(a.mp, g, 1.0, vol);
#pragma unroll
          for (int f = 0; f < F; ++f) z[f * LDZ + r * NP] = vol[f];
        }
      }
      zero_rows(ne * F);
      __syncthreads();
      gemm(a.vfrag, ne * F);
      for (int x = tid; x < ne * NP; x += THREADS) {
        const int e = x / NP, i = x - e * NP;
        double s = 0.0;
#pragma unroll
        for (int f = 0; f < F; ++f)
          s += model_finish<MODEL, DIM, double>(a.mp, f, 1.0, 0.0, 0.0) * sl[f * ENP + x] *
               sum(e * F + f, i);
        sv[x] = s;
      }
      __syncthreads();
    }

    // ---- transposed volume map and chain rule at the nodes ----
    for (int x = tid; x < ne * NP; x += THREADS) {
      const int e = x / NP, i = x - e * NP;
      double l[F], m[DIM][F];
#pragma unroll
      for (int f = 0; f < F; ++f)
        l[f] = model_finish<MODEL, DIM, double>(a.mp, f, 1.0, 0.0, 0.0) * sl[f * ENP + x];
#pragma unroll
      for (int d = 0; d < DIM; ++d)
#pragma unroll
        for (int g = 0; g < F; ++g) {
          double gr[DIM][F];
#pragma unroll
          for (int dd = 0; dd < DIM; ++dd)
#pragma unroll
            for (int gg = 0; gg < F; ++gg) gr[dd][gg] = (dd == d && gg == g) ? 1.0 : 0.0;
          double vol[F];
          model_volume<MODEL, DIM, double>(a.mp, gr, C ? sc[x] : 0.0, vol);
          double s = 0.0;
#pragma unroll
          for (int f = 0; f < F; ++f) s += l[f] * vol[f];
          m[d][g] = s;
        }
      const double* ge = sgeo + e * G;
      double* z = sZ + e * F * LDZ + i;
#pragma unroll
      for (int r = 0; r < DIM; ++r)
#pragma unroll
        for (int g = 0; g < F; ++g) {
          double s = 0.0;
#pragma unroll
          for (int d = 0; d < DIM; ++d) s += ge[r * DIM + d] * m[d][g];
          z[g * LDZ + r * NP] = s;
        }
    }
    zero_rows(ne * F);
    // ---- transposed own-side and neighbour-side fluxes at the face points ----
    for (int it = tid; it < ne * NFPT; it += THREADS) {
      const int e = it / NFPT, p = it - e * NFPT, face = p / NFP, k = p - face * NFP;
      const int lnode = sfm[p];
      const double* ge = sgeo + e * G;
      double n[DIM], nnb[DIM], we[F], wn[F], qn[F];
#pragma unroll
      for (int d = 0; d < DIM; ++d) n[d] = ge[DIM * DIM + face * (DIM + 1) + d];
      const int2 cn = sconn[e * NF + face];
      const bool bdry = cn.x < 0;
      const int kind = bdry ? cn.y : 0;
      // neighbour face point matched to this one
      int64_t nb = -1;
      int pn = 0, nn = 0;
      if (!bdry) {
        const int nface = cn.y & 3, perm = cn.y >> 2;
        if (cn.x < a.K && nface < NF && perm < a.nperm) {
          nb = cn.x;
          pn = nface * NFP + ssh[perm * NFP + k];
          nn = sfm[pn];
        } else {
          atomicCAS(a.err, 0, DEV_BAD_CODE);
        }
      }
#pragma unroll
      for (int f = 0; f < F; ++f) {
        we[f] = a.work[((el0 + e) * NFPT + p) * F + f];
        wn[f] = nb >= 0 ? a.work[(nb * NFPT + pn) * F + f] : 0.0;
        if constexpr (WC) qn[f] = nb >= 0 ? a.q[f * Knp + nb * NP + nn] : 0.0;
      }
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        nnb[d] = nb >= 0 ? __ldg(a.geo + nb * G + DIM * DIM + (cn.y & 3) * (DIM + 1) + d) : 0.0;
      const double cm = C ? sc[e * NP + lnode] : 0.0;
      const double cp = (C && nb >= 0) ? a.coeff[nb * NP + nn] : cm;
      double* w = sw + e * CF * NFPT + p;
#pragma unroll
      for (int g = 0; g < F; ++g) {
        double uM[NA], uP[NA], fl[F];
        // own side: d flux / d q-_g
#pragma unroll
        for (int q = 0; q < NA; ++q) { uM[q] = 0.0; uP[q] = 0.0; }
        if constexpr (C != 0) { uM[0] = cm; uP[0] = cp; }
        uM[C + g] = 1.0;
        adj_flux_at<MODEL, DIM>(a.mp, bdry, kind, uM, uP, n, fl);
        double s = 0.0;
#pragma unroll
        for (int f = 0; f < F; ++f) s += we[f] * fl[f];
        // neighbour side: the neighbour's flux at its matched point, d / d q+_g
        if (nb >= 0) {
#pragma unroll
          for (int q = 0; q < NA; ++q) { uM[q] = 0.0; uP[q] = 0.0; }
          if constexpr (C != 0) { uM[0] = cp; uP[0] = cm; }
          uP[C + g] = 1.0;
          adj_flux_at<MODEL, DIM>(a.mp, false, 0, uM, uP, nnb, fl);
#pragma unroll
          for (int f = 0; f < F; ++f) s += wn[f] * fl[f];
        }
        w[g * NFPT] = s;
      }
      if constexpr (WC) {
        double uM[NA], uP[NA], fl[F], gc = 0.0;
        // own side: d flux / d c- (on a boundary c+ = c-, model_bc copies it)
        uM[0] = 1.0;
        uP[0] = 0.0;
#pragma unroll
        for (int f = 0; f < F; ++f) {
          uM[C + f] = sq[f * ENP + e * NP + lnode];
          uP[C + f] = qn[f];
        }
        adj_flux_at<MODEL, DIM>(a.mp, bdry, kind, uM, uP, n, fl);
#pragma unroll
        for (int f = 0; f < F; ++f) gc += we[f] * fl[f];
        if (nb >= 0) {
          // neighbour side: d flux_nb / d c+ (its c+ is this node's c)
          uM[0] = 0.0;
          uP[0] = 1.0;
#pragma unroll
          for (int f = 0; f < F; ++f) {
            uM[C + f] = qn[f];
            uP[C + f] = sq[f * ENP + e * NP + lnode];
          }
          adj_flux_at<MODEL, DIM>(a.mp, false, 0, uM, uP, nnb, fl);
#pragma unroll
          for (int f = 0; f < F; ++f) gc += wn[f] * fl[f];
        }
        w[F * NFPT] = gc;
      }
    }
    __syncthreads();
    gemm(a.afrag, ne * F);

    // ---- output ----
    for (int x = tid; x < ne * NP; x += THREADS) {
      const int e = x / NP, i = x - e * NP;
      const double* w = sw + e * CF * NFPT;
      const int p0 = snl[i], p1 = snl[i + 1];
#pragma unroll
      for (int g = 0; g < F; ++g) {
        double v = sum(e * F + g, i);
        for (int p = p0; p < p1; ++p) v += w[g * NFPT + snl[NP + 1 + p]];
        const int64_t gi = g * Knp + el0 * NP + x;
        if (a.fused) {
          a.lq[gi] += a.dt * v;
          a.lam[gi] = a.ra * sl[g * ENP + x];
        } else {
          a.q_bar[gi] = v;
        }
      }
      if constexpr (WC) {
        double v = sv[x];
        for (int p = p0; p < p1; ++p) v += w[F * NFPT + snl[NP + 1 + p]];
        const int64_t gi = el0 * NP + x;
        if (a.fused)
          a.c_bar[gi] += a.dt * v;
        else
          a.c_bar[gi] = v;
      }
    }
  }
}

// One adjoint call (all pointers of AdjArgs that the caller provides).
struct AdjCall {
  Op* op;
  AdjArgs a;
  cudaStream_t stream;
  bool configure, want_c;   // prepare the operator, without or with the c gradient
};

// The operator fragments of the adjoint, [LIFT^T | D^T | D], D where there is
// a c gradient, and the nodes' face points.
template <int MODEL, int DIM, int ORDER>
hb_status adj_fragments(Op* op, cudaStream_t s) {
  using S = AdjShape<MODEL, DIM, ORDER, false>;
  const Discr* d = op->d;
  const double* h = reinterpret_cast<const double*>(d->host_blob.data());
  const double* lift = h + (size_t)DIM * S::NP * S::NP;
  const size_t nl = (size_t)S::LW * S::LSTEPS * S::LMW * 64, na = (size_t)S::STEPS * S::MT * 64;
  const size_t ops = nl + (S::C ? 2 : 1) * na;
  std::vector<double> fr(ops + (S::NLIST + 7) / 8, 0.0);
  for (int p = 0; p < S::NFPT; ++p)
    for (int i = 0; i < S::NP; ++i) {
      const int w = p / (S::LMW * 8), row = p - w * S::LMW * 8;
      fr[(size_t)w * S::LSTEPS * S::LMW * 64 + dmma_afrag(row, i, S::LMW)] =
          lift[(size_t)p * S::NP + i];
    }
  // h holds D_r transposed, [r][j][i] = D_r[i][j]
  for (int r = 0; r < DIM; ++r)
    for (int i = 0; i < S::NP; ++i)
      for (int j = 0; j < S::NP; ++j) {
        const double v = h[((size_t)r * S::NP + j) * S::NP + i];
        fr[nl + dmma_afrag(j, r * S::NP + i, S::MT)] = v;
        if (S::C) fr[nl + na + dmma_afrag(i, r * S::NP + j, S::MT)] = v;
      }
  uint8_t* begin = reinterpret_cast<uint8_t*>(&fr[ops]);
  uint8_t* list = begin + S::NP + 1;
  int n = 0;
  for (int i = 0; i < S::NP; ++i) {
    begin[i] = (uint8_t)n;
    for (int p = 0; p < S::NFPT; ++p)
      if (d->fmask_host[p] == i) list[n++] = (uint8_t)p;
  }
  begin[S::NP] = (uint8_t)n;
  double* dev = nullptr;
  if (cudaMalloc(&dev, sizeof(double) * fr.size()) != cudaSuccess)
    return fail(HB_ERR_CUDA, "cannot allocate the adjoint's operator fragments");
  // waited for: another thread's stream may be the next to read it
  if (cudaMemcpyAsync(dev, fr.data(), sizeof(double) * fr.size(), cudaMemcpyHostToDevice, s) !=
          cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaFree(dev);
    return fail(HB_ERR_CUDA, "cannot upload the adjoint's operator fragments");
  }
  op->adjfrag = dev;
  return HB_OK;
}

template <typename KERN>
hb_status adj_launch(KERN kern, const AdjArgs& a, int threads, size_t smem, int slots,
                     cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<int64_t>(slots, a.nbatch));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  return HB_OK;
}

template <typename KERN>
hb_status adj_slots(KERN kern, int threads, size_t smem, int* slots) {
  if (*slots) return HB_OK;
  int dev, sms = 0, per_sm = 0;
  HB_CUDA(cudaGetDevice(&dev));
  HB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  HB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  HB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
  if (per_sm < 1) return fail(HB_ERR_UNSUPPORTED, "adjoint kernel does not fit on an SM");
  *slots = sms * per_sm;
  return HB_OK;
}

template <int MODEL, int DIM, int ORDER>
hb_status adj_one(const AdjCall& c) {
  using S = AdjShape<MODEL, DIM, ORDER, false>;
  constexpr bool CW = S::C != 0;
  using SC = AdjShape<MODEL, DIM, ORDER, CW>;
  static_assert(SC::total <= 227 * 1024 && S::total <= 227 * 1024 && S::ltotal <= 227 * 1024,
                "a batch exceeds the shared memory of a CTA");
  Op* op = c.op;
  const Discr* d = op->d;
  if (d->np != S::NP || d->nfp != S::NFP)
    return fail(HB_ERR_UNSUPPORTED, "element sizes do not match the order");
  if (c.configure) {
    hb_status st = adj_slots(adj_lift_kernel<MODEL, DIM, ORDER>, 128, S::ltotal,
                             &op->adj_slots[0]);
    if (st) return st;
    st = c.want_c ? adj_slots(adj_element_kernel<MODEL, DIM, ORDER, CW>, SC::THREADS, SC::total,
                              &op->adj_slots[2])
                  : adj_slots(adj_element_kernel<MODEL, DIM, ORDER, false>, S::THREADS, S::total,
                              &op->adj_slots[1]);
    if (st || op->adjfrag) return st;
    return adj_fragments<MODEL, DIM, ORDER>(op, c.stream);
  }
  const bool wc = c.a.c_bar != nullptr;
  AdjArgs a = c.a;
  a.K = d->K;
  a.nperm = d->nperm;
  a.lfrag = reinterpret_cast<const double2*>(op->adjfrag);
  a.afrag = a.lfrag + (size_t)S::LW * S::LSTEPS * S::LMW * 32;
  a.vfrag = a.afrag + (size_t)S::STEPS * S::MT * 32;
  a.nlist = reinterpret_cast<const uint8_t*>(a.vfrag + (CW ? (size_t)S::STEPS * S::MT * 32 : 0));
  a.geo = d->geo;
  a.conn = op->conn;
  a.fmask = d->fmask;
  a.shuffle = d->shuffle;
  a.mp = op->mp;
  a.err = op->err_flag;
  a.E = dmma_batch(d->K, S::LEB, S::F, op->adj_slots[0]);
  a.nbatch = (d->K + a.E - 1) / a.E;
  const hb_status st = adj_launch(adj_lift_kernel<MODEL, DIM, ORDER>, a, 128, S::ltotal,
                                  op->adj_slots[0], c.stream);
  if (st) return st;
  const int slots = op->adj_slots[wc ? 2 : 1];
  a.E = dmma_batch(d->K, wc ? SC::EB : S::EB, S::F, slots);
  a.nbatch = (d->K + a.E - 1) / a.E;
  if constexpr (CW) {
    if (wc)
      return adj_launch(adj_element_kernel<MODEL, DIM, ORDER, true>, a, SC::THREADS, SC::total,
                        slots, c.stream);
  }
  return adj_launch(adj_element_kernel<MODEL, DIM, ORDER, false>, a, S::THREADS, S::total, slots,
                    c.stream);
}

template <int MODEL, int DIM>
hb_status adj_orders(const AdjCall& c) {
  switch (c.op->d->order) {
    case 1: return adj_one<MODEL, DIM, 1>(c);
    case 2: return adj_one<MODEL, DIM, 2>(c);
    case 3: return adj_one<MODEL, DIM, 3>(c);
    case 4: return adj_one<MODEL, DIM, 4>(c);
    case 5: return adj_one<MODEL, DIM, 5>(c);
    case 6: return adj_one<MODEL, DIM, 6>(c);
    case 7: return adj_one<MODEL, DIM, 7>(c);
    default: return fail(HB_ERR_UNSUPPORTED, "FP64 tensor-core adjoint: orders 1 to 7");
  }
}

}  // namespace hb
