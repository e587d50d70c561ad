// FP64 fused DG right-hand side and LSRK stage on the FP64 tensor cores
// (mma.sync m8n8k4, FP64 operands and accumulators).
//
// On an affine element the operator is one contraction per (element, field)
// column: the chain rule and the model's volume map act pointwise, so
//
//   rhs = [ D_1 | .. | D_d | LIFT ] . [ z_1; ..; z_d; flux ]
//   z_r = vol( d r / d x  (outer)  q )     (model_volume is linear in grad q)
//
// with K = d Np + Nf Nfp rows and Np outputs.  This is the same number of
// products as differentiating first, but one accumulator per output instead
// of d per field, and one GEMM instead of two loops with a pass between.
//
// Persistent CTAs; per batch of up to EB elements (EB * F columns):
//   1. the state, geometry and face table arrive by cp.async one batch ahead;
//   2. every thread forms the z of its nodes and the fluxes of its face
//      points (the neighbour values of the first are requested before the z
//      phase, of the next before a flux is computed) into Z[column][k], whose
//      rows are consecutive k: conflict-free stores, 16-byte fragment loads;
//   3. warp (ng, kg) multiplies RN tiles of 8 columns by all MT tiles of 8
//      nodes over its share kg of the k range.  The operator fragments sit in
//      global memory in fragment order and are read through L1 (one copy per
//      SM serves all CTAs; a copy in each CTA's shared memory would cost a
//      resident CTA); a step's fragments are loaded while the previous step
//      multiplies;
//   4. the partial sums go to shared memory (over Z) and a pass in linear
//      order adds them, applies the source and the material divisor and
//      writes the RHS or the stage update.
// Splitting k over warps keeps the MT x RN register tile (its operand loads
// take 2/MT + 2/RN shared-memory wavefronts per MMA, against 4 cycles of the
// SM's FP64 pipe) and halves the chain of dependent MMAs on small meshes.
//
// Bound: the FP64 pipe, which the MMAs share with the fluxes' FP64 arithmetic
// (4 cycles per MMA and SM: 111 us of a C2 stage with the tile padding), and
// beside it the latency of the point phases at 16 warps per SM.  Measured per
// stage against the CUDA-core kernel: 3D Maxwell N = 4, K = 48000 454 -> 240
// us, N = 5, K = 13182 333 -> 123 us, variable material N = 2, K = 12960 33 ->
// 20 us; 3D wave N = 7, K = 10368 474 -> 239 us; 2D TM N = 5, K = 19594 33 ->
// 18 us; 2D wave N = 3, K = 684 8.3 -> 4.2 us.  Reference
// loops: jit/diff.py:137-175, jit/flux.py:311-353 and 429-472,
// jit/lift.py:110-141, jit/__init__.py:501-519,
// timestep/runge_kutta.py:123-128.
#pragma once

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "face.cuh"
#include "models.cuh"
#include "dmma.cuh"

namespace hb {

__host__ __device__ constexpr int f64_ru8(int x) { return (x + 7) / 8 * 8; }

// SB: bytes of a state value (8: FP64, 4: FP32 state and residual; the
// arithmetic is FP64 either way)
template <int MODEL, int DIM, int ORDER, int SB = 8>
struct F64Shape {
  static constexpr int F = Traits<MODEL, DIM>::F;
  static constexpr int C = Traits<MODEL, DIM>::COEFF;
  static constexpr int NP = DIM == 2 ? (ORDER + 1) * (ORDER + 2) / 2
                                     : (ORDER + 1) * (ORDER + 2) * (ORDER + 3) / 6;
  static constexpr int NFP = DIM == 2 ? ORDER + 1 : (ORDER + 1) * (ORDER + 2) / 2;
  static constexpr int NF = DIM + 1;
  static constexpr int NFPT = NF * NFP;
  static constexpr int G = DIM * DIM + NF * (DIM + 1);
  // k rows: volume [0, KV), padded to a whole step where the variable-c wave
  // scales the volume part by c at the node (KVP), then the face points
  static constexpr int KV = DIM * NP;
  static constexpr int KVP = C ? f64_ru8(KV) : KV;
  static constexpr int KP = f64_ru8(KVP + NFPT);
  static constexpr int PADS = KP - KV - NFPT;    // rows held at zero
  static constexpr int STEPS = KP / 8;           // two MMAs deep each
  // 16-byte fragment loads: columns 64 bytes apart modulo 128
  static constexpr int LDZ = KP % 16 == 8 ? KP : KP + 8;
  static constexpr int MT = (NP + 7) / 8;
  // few node tiles leave registers for more column tiles (and the batch then
  // has a node or a face point for every thread)
  static constexpr int RN = MT == 1 ? 8 : MT == 2 ? 4 : 2;
  // Two steps of the GEMM unrolled where the registers and the instruction
  // cache bear it, by measurement (stage times, one -> two): 3D Maxwell N = 5,
  // K = 13182 139 -> 123 us, N = 4, K = 48000 258 -> 240 us, 2D wave N = 3, K = 684
  // 4.6 -> 4.3 us; but 3D Maxwell N = 2, K = 48000 58.6 -> 61.4 us, 2D TM N = 6, K =
  // 33800 41.9 -> 44.7 us.
  static constexpr int UNROLL = (DIM == 3 ? MT >= 4 || F <= 3 : MT <= 3) ? 2 : 1;
  static constexpr int NGW = 2;
  // from 11 node tiles a CTA fills the SM: four k shares give it 8 warps
  static constexpr int KG = MT >= 11 ? 4 : 2;
  static constexpr int THREADS = 32 * NGW * KG;
  static constexpr int COLS = NGW * RN * 8;
  static constexpr int EB = COLS / F;
  // partial sums [KG][COLS][LDP]: the fragment stores of a half-warp (4
  // nodes x 4 column pairs) fall in distinct banks
  static constexpr int LDP = MT * 8 + 2;
  static constexpr int ENP = EB * NP;
  static constexpr int FR = (EB * NFPT + THREADS - 1) / THREADS;   // face points per thread
  // rounds of face points requested at once: all while they stay within 12
  // values a thread, else one round ahead (stage times: C2, 18 values, 273 us
  // all at once and 254 us one ahead; Maxwell N = 3, 12 values, 67 and 70 us)
  static constexpr int PF = FR * (F + C) <= 12 ? FR : 1;
  static constexpr int UR = (ENP + THREADS - 1) / THREADS;

  static constexpr size_t al(size_t x) { return (x + 15) & ~size_t(15); }
  static constexpr size_t zdoubles =
      COLS * LDZ > KG * COLS * LDP ? COLS * LDZ : KG * COLS * LDP;
  static constexpr size_t oZ = 0;
  static constexpr size_t oQ = al(oZ + 8 * zdoubles);          // [F][EB][NP]
  static constexpr size_t oC = al(oQ + SB * F * ENP);          // [2][EB][NP]
  static constexpr size_t oG = al(oC + 2 * 8 * C * ENP);       // [EB][G]
  static constexpr size_t oN = al(oG + 8 * EB * G);            // [EB][NF] int2
  static constexpr size_t oFm = al(oN + 8 * EB * NF);          // uint8 face nodes
  static constexpr size_t oSh = al(oFm + NFPT);                // uint8 neighbour nodes
  static constexpr size_t total = al(oSh + 6 * NFPT);
  // CTAs per SM: what shared memory holds, within the registers the tile needs
  // (variable material holds more: three CTAs there, 22 us against 25 at
  // K = 12960, N = 2)
  static constexpr int SMEM_CTAS = (int)((228 * 1024) / (total + 1024));
  static constexpr int min_ctas(bool vm) {
    const int regs = MT > 7 ? 1 : MT > 5 || vm ? 3 : 4;
    return SMEM_CTAS < 1 ? 1 : SMEM_CTAS < regs ? SMEM_CTAS : regs;
  }
};

template <typename IO>
struct F64Args {
  int64_t K, nbatch, e_begin, e_end;
  int E, nperm;
  FaceArgs<IO> face;         // neighbour, halo and boundary sources
  const double2* afrag;      // operator fragments [STEPS][MT][32]
  const double* geo;
  const int2* conn;
  const int* fmask;
  const int* shuffle;
  IO* q_out;
  IO* res;
  const double* source;
  double ra, rb, dt;
  double inv_eps, inv_mu;    // fixed material
  int mode;                  // 0: write rhs, 1: LSRK stage
  ModelParams mp;
};

// VM: Maxwell with variable material (coeff = [eps | mu])
template <int MODEL, int DIM, int ORDER, bool VM, typename IO>
__global__ void __launch_bounds__(F64Shape<MODEL, DIM, ORDER, sizeof(IO)>::THREADS,
                                  (F64Shape<MODEL, DIM, ORDER, sizeof(IO)>::min_ctas(VM)))
    rhs_fp64_kernel(const F64Args<IO> a) {
  using S = F64Shape<MODEL, DIM, ORDER, sizeof(IO)>;
  constexpr int F = S::F, C = S::C, NP = S::NP, NFP = S::NFP, NF = S::NF, NFPT = S::NFPT;
  constexpr int G = S::G, LDZ = S::LDZ, ENP = S::ENP, THREADS = S::THREADS;
  constexpr int MT = S::MT, RN = S::RN, KG = S::KG;
  extern __shared__ __align__(16) unsigned char smem[];
  double* sZ = reinterpret_cast<double*>(smem + S::oZ);
  uint8_t* sfm = smem + S::oFm;
  uint8_t* sse = smem + S::oSh;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kg = warp % KG, ng = warp / KG;
  const int64_t Knp = a.K * NP;

  for (int x = tid; x < NFPT; x += THREADS) sfm[x] = (uint8_t)a.fmask[x];
  // node of a neighbour seen through (perm, its face): fmask[f][shuffle[perm][k]]
  for (int x = tid; x < a.nperm * NFPT; x += THREADS) {
    const int perm = x / NFPT, r = x - perm * NFPT;
    const int f = r / NFP, k = r - f * NFP;
    sse[x] = (uint8_t)a.fmask[f * NFP + a.shuffle[perm * NFP + k]];
  }
  // the next launch may begin its set-up; this one waits for the previous
  // launch before it reads anything that one may have written
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  auto fetch = [&](int64_t batch, int buf) {
    const int64_t el0 = a.e_begin + batch * a.E;
    const int ne = (int)(a.e_end - el0 < a.E ? a.e_end - el0 : a.E);
    IO* dq = reinterpret_cast<IO*>(smem + S::oQ);
    for (int x = tid; x < ne * NP; x += THREADS) {
#pragma unroll
      for (int f = 0; f < F; ++f)
        cp_async_word(dq + f * ENP + x, a.face.q + f * Knp + el0 * NP + x);
      if constexpr (C != 0)
        cp_async8(reinterpret_cast<double*>(smem + S::oC) + buf * ENP + x,
                  a.face.coeff + el0 * NP + x);
    }
    double* dg = reinterpret_cast<double*>(smem + S::oG);
    for (int x = tid; x < ne * G; x += THREADS) cp_async8(dg + x, a.geo + el0 * G + x);
    int2* dn = reinterpret_cast<int2*>(smem + S::oN);
    for (int x = tid; x < ne * NF; x += THREADS) cp_async8(dn + x, a.conn + el0 * NF + x);
    cp_async_commit();
  };

  const IO* sq = reinterpret_cast<const IO*>(smem + S::oQ);
  const double* sgeo = reinterpret_cast<const double*>(smem + S::oG);
  const int2* sconn = reinterpret_cast<const int2*>(smem + S::oN);
  if (blockIdx.x < a.nbatch) fetch(blockIdx.x, 0);
  int buf = 0;   // of the coefficient, which the GEMM reads too
  for (int64_t batch = blockIdx.x; batch < a.nbatch; batch += gridDim.x, buf ^= 1) {
    const int64_t el0 = a.e_begin + batch * a.E;
    const int ne = (int)(a.e_end - el0 < a.E ? a.e_end - el0 : a.E);
    const double* sc = reinterpret_cast<const double*>(smem + S::oC) + buf * ENP;
    cp_async_wait_all();
    __syncthreads();   // the batch has arrived; the previous one is done with Z

    if (a.mode != 0) {
      constexpr int LINE = 128 / sizeof(IO), LINES = (ENP + LINE - 1) / LINE + 1;
      for (int x = tid; x < F * LINES; x += THREADS) {
        const int f = x / LINES, o = (x - f * LINES) * LINE;
        const IO* r = a.res + f * Knp + el0 * NP + (o < ne * NP ? o : ne * NP - 1);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(r));
      }
    }

    // ---- Z: face points and nodes ----
    // the exterior values of a thread's face points are requested ahead of
    // use: of all of them, or of the first, before the z phase
    const int nfi = ne * NFPT;
    auto load_ext = [&](int it, FaceExt<MODEL, DIM, double>& x) {
      if (it < nfi)
        face_load<MODEL, DIM, VM>(a.face, sconn[it / NFP], it % NFP, Knp, NP, NFP, NF, a.nperm,
                                  sse, x);
    };
    FaceExt<MODEL, DIM, double> ext[S::PF];
#pragma unroll
    for (int r = 0; r < S::PF; ++r) load_ext(tid + r * THREADS, ext[r]);
    for (int x = tid; x < ne * NP; x += THREADS) {
      const int e = x / NP, j = x - e * NP;
      double q[F];
#pragma unroll
      for (int f = 0; f < F; ++f) q[f] = (double)sq[f * ENP + x];
      const double* ge = sgeo + e * G;
      double* z = sZ + e * F * LDZ + j;
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        double g[DIM][F], vol[F];
#pragma unroll
        for (int d = 0; d < DIM; ++d)
#pragma unroll
          for (int f = 0; f < F; ++f) g[d][f] = ge[r * DIM + d] * q[f];
        model_volume<MODEL, DIM, double>(a.mp, g, 1.0, vol);
#pragma unroll
        for (int f = 0; f < F; ++f) z[f * LDZ + r * NP] = vol[f];
      }
    }
    if constexpr (S::PADS != 0) {
      for (int x = tid; x < ne * F * S::PADS; x += THREADS) {
        const int col = x / S::PADS, r = x - col * S::PADS;
        sZ[col * LDZ + (r < S::KVP - S::KV ? S::KV + r : NFPT + S::KV + r)] = 0.0;
      }
    }
    auto flux_at = [&](int it, FaceExt<MODEL, DIM, double>& x) {
      const int e = it / NFPT, p = it - e * NFPT, fc = p / NFP;
      const int lnode = sfm[p];
      double uM[F + C], n[DIM], fl[F];
      if constexpr (C != 0) uM[0] = sc[e * NP + lnode];
#pragma unroll
      for (int f = 0; f < F; ++f) uM[C + f] = (double)sq[f * ENP + e * NP + lnode];
      const double* gf = sgeo + e * G + DIM * DIM + fc * (DIM + 1);
#pragma unroll
      for (int d = 0; d < DIM; ++d) n[d] = gf[d];
      const bool have = face_flux<MODEL, DIM, VM>(
          a.face, a.mp, sconn[e * NF + fc], p - fc * NFP, NFP, (el0 + e) * NP + lnode, Knp, uM, n,
          x, fl);
      const double fscale = gf[DIM];
      double* z = sZ + e * F * LDZ + S::KVP + p;
#pragma unroll
      for (int f = 0; f < F; ++f) z[f * LDZ] = have ? fscale * fl[f] : 0.0;
    };
    if constexpr (S::PF == S::FR) {
#pragma unroll
      for (int r = 0; r < S::FR; ++r)
        if (tid + r * THREADS < nfi) flux_at(tid + r * THREADS, ext[r]);
    } else {
      // one copy of the flux code: unrolled, it outgrows the instruction cache
#pragma unroll 1
      for (int it = tid; it < nfi; it += THREADS) {
        FaceExt<MODEL, DIM, double> nxt;
        load_ext(it + THREADS, nxt);
        flux_at(it, ext[0]);
        ext[0] = nxt;
      }
    }
    __syncthreads();   // Z is complete; the state, geometry and face table are read
    if (batch + gridDim.x < a.nbatch) fetch(batch + gridDim.x, buf ^ 1);

    // ---- GEMM over this warp's share of k ----
    const bool work = ng * RN * 8 < ne * F;
    double acc[MT][RN][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int c = 0; c < RN; ++c) acc[m][c][0] = acc[m][c][1] = 0.0;
    if (work) {
      const int s0 = kg * S::STEPS / KG, s1 = (kg + 1) * S::STEPS / KG;
      const double2* ap = a.afrag + (size_t)s0 * MT * 32 + lane;
      const double* zp = sZ + (ng * RN * 8 + (lane >> 2)) * LDZ + 2 * (lane & 3) + 8 * s0;
      // volume part of the variable-c wave: times c at the output node
      auto scale_c = [&]() {
        if constexpr (C != 0) {
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int c = 0; c < RN; ++c)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int node = m * 8 + (lane >> 2);
                const int e = ((ng * RN + c) * 8 + 2 * (lane & 3) + h) / F;
                if (node < NP && e < ne) acc[m][c][h] *= sc[e * NP + node];
              }
        }
      };
      if constexpr (C != 0) {
        constexpr int SV = S::KVP / 8;
        const int nv = s1 < SV ? s1 - s0 : s0 < SV ? SV - s0 : 0;   // volume steps
        dmma_steps<MT, RN, LDZ, S::UNROLL>(acc, ap, zp, nv);
        if (nv > 0) scale_c();
        dmma_steps<MT, RN, LDZ, S::UNROLL>(acc, ap + (size_t)nv * MT * 32, zp + 8 * nv, s1 - s0 - nv);
      } else {
        dmma_steps<MT, RN, LDZ, S::UNROLL>(acc, ap, zp, s1 - s0);
      }
    }
    __syncthreads();   // all warps are done reading Z
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
    // the state and residual at this thread's outputs, requested before the
    // barrier (from L2: the state's shared copy is being refilled, the
    // residual was prefetched)
    IO rv[S::UR][F], qv[S::UR][F];
    const int64_t base = el0 * NP + tid;
    if (a.mode != 0) {
#pragma unroll
      for (int u = 0; u < S::UR; ++u)
        if (tid + u * THREADS < ne * NP) {
#pragma unroll
          for (int f = 0; f < F; ++f) {
            rv[u][f] = a.res[f * Knp + base + u * THREADS];
            qv[u][f] = a.face.q[f * Knp + base + u * THREADS];
          }
        }
    }
    __syncthreads();

    // ---- output in linear order ----
#pragma unroll
    for (int u = 0; u < S::UR; ++u) {
      const int n = tid + u * THREADS;
      if (n >= ne * NP) break;
      const int e = n / NP, i = n - e * NP;
      const double* P = sZ + e * F * S::LDP + i;
      const int64_t node = base + u * THREADS;
      double inv_eps = a.inv_eps, inv_mu = a.inv_mu;
      if constexpr (VM) {
        // one division for the fields of a kind
        inv_eps = 1.0 / a.face.coeff[node];
        inv_mu = 1.0 / a.face.coeff[Knp + node];
      }
#pragma unroll
      for (int f = 0; f < F; ++f) {
        double r = P[f * S::LDP];
#pragma unroll
        for (int g = 1; g < KG; ++g) r += P[g * S::COLS * S::LDP + f * S::LDP];
        const int64_t si = a.source ? model_src_index<MODEL>(f, node, Knp) : -1;
        const double src = si >= 0 ? a.source[si] : 0.0;
        if constexpr (IsMaxwell<MODEL>::value) {
          r *= f < maxwell_ne<MODEL>() ? inv_eps : inv_mu;
          if (f < maxwell_ne<MODEL>()) r += src;
        } else {
          r = model_finish<MODEL, DIM, double>(a.mp, f, r, 0.0, src);
        }
        const int64_t gi = f * Knp + node;
        if (a.mode == 0) {
          a.q_out[gi] = (IO)r;
        } else {
          const double nr = a.ra * (double)rv[u][f] + a.dt * r;
          a.res[gi] = (IO)nr;
          a.q_out[gi] = (IO)((double)qv[u][f] + a.rb * nr);
        }
      }
    }
  }
}

// One call of the FP64 path: configure an operator, or launch.
struct F64Call {
  Op* op;
  int mode;
  double ra, rb, dt;
  const void* q_in;
  void* q_out;
  void* res;
  const double* coeff;
  const double* bdry;
  const double* source;
  int64_t e0, e1;
  cudaStream_t stream;
  bool configure;
};

template <int MODEL, int DIM, int ORDER, bool VM, typename IO>
hb_status f64_one(const F64Call& c) {
  using S = F64Shape<MODEL, DIM, ORDER, sizeof(IO)>;
  Op* op = c.op;
  Discr* d = op->d;
  auto kern = rhs_fp64_kernel<MODEL, DIM, ORDER, VM, IO>;
  if (c.configure) {
    if (d->np != S::NP || d->nfp != S::NFP)
      return fail(HB_ERR_UNSUPPORTED, "element sizes do not match the order");
    int dev, sms = 0, max_optin = 0, per_sm = 0;
    HB_CUDA(cudaGetDevice(&dev));
    HB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    HB_CUDA(cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (S::total > (size_t)max_optin)
      return fail(HB_ERR_UNSUPPORTED, "FP64 kernel: batch exceeds shared memory");
    HB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)S::total));
    HB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, S::THREADS, S::total));
    if (per_sm < 1) return fail(HB_ERR_UNSUPPORTED, "FP64 kernel does not fit on an SM");
    op->f64_slots[VM] = sms * per_sm;
    if constexpr (VM) return HB_OK;   // the rest is the fixed-material kernel's
    op->elems_per_block = dmma_batch(d->K, S::EB, S::F, op->f64_slots[0]);
    op->blocks_per_sm = per_sm;
    op->threads = S::THREADS;
    op->smem = S::total;
    op->ops_in_smem = 0;
    op->grid = (int)std::min<int64_t>((d->K + op->elems_per_block - 1) / op->elems_per_block,
                                      op->f64_slots[0]);
    // operator fragments: lane (g, t) of step s and node tile m holds rows
    // m*8 + g, columns 8s + 2t and 8s + 2t + 1
    const double* h = reinterpret_cast<const double*>(d->host_blob.data());
    const double* lift = h + (size_t)DIM * S::NP * S::NP;
    std::vector<double> fr((size_t)S::STEPS * S::MT * 64, 0.0);
    for (int k = 0; k < S::KP; ++k) {
      const double* row = k < S::KV ? h + (size_t)k * S::NP
                          : k >= S::KVP && k < S::KVP + S::NFPT
                              ? lift + (size_t)(k - S::KVP) * S::NP : nullptr;
      if (!row) continue;
      for (int i = 0; i < S::NP; ++i)
        fr[dmma_afrag(i, k, S::MT)] = row[i];
    }
    if (cudaMalloc(&op->afrag, sizeof(double) * fr.size()) != cudaSuccess ||
        cudaMemcpy(op->afrag, fr.data(), sizeof(double) * fr.size(), cudaMemcpyHostToDevice) !=
            cudaSuccess)
      return fail(HB_ERR_CUDA, "cannot upload the FP64 operator fragments");
    return HB_OK;
  }
  F64Args<IO> a;
  a.K = d->K;
  a.e_begin = c.e0;
  a.e_end = c.e1;
  const int slots = op->f64_slots[VM];
  a.E = dmma_batch(c.e1 - c.e0, S::EB, S::F, slots);
  a.nbatch = (c.e1 - c.e0 + a.E - 1) / a.E;
  a.nperm = d->nperm;
  a.face.K = d->K;
  a.face.q = static_cast<const IO*>(c.q_in);
  a.face.coeff = c.coeff;
  a.face.bdry = c.bdry;
  a.face.n_given = op->n_given;
  a.face.halo = static_cast<const IO*>(op->halo);
  a.face.halo_c = op->halo_c;
  a.face.n_halo = op->n_halo;
  a.face.err = op->err_flag;
  a.afrag = reinterpret_cast<const double2*>(op->afrag);
  a.geo = d->geo;
  a.conn = op->conn;
  a.fmask = d->fmask;
  a.shuffle = d->shuffle;
  a.q_out = static_cast<IO*>(c.q_out);
  a.res = static_cast<IO*>(c.res);
  a.source = c.source;
  a.ra = c.ra;
  a.rb = c.rb;
  a.dt = c.dt;
  a.mode = c.mode;
  a.mp = op->mp;
  a.inv_eps = 1.0 / op->mp.eps;
  a.inv_mu = 1.0 / op->mp.mu;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<int64_t>(slots, a.nbatch));
  cfg.blockDim = dim3(S::THREADS);
  cfg.dynamicSmemBytes = S::total;
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
  return HB_OK;
}

// FP32 states that run here, in FP64 arithmetic, instead of on the split FP16
// planes (or, where no such instance is built, on the CUDA cores): the smaller
// elements, whose planes are mostly padding and whose batches are too short for
// the split kernel's pipeline.  LSRK4 step, split or CUDA cores -> here: 3D
// Maxwell N = 3, K = 9438 174 -> 141 us, K = 48000 709 -> 608 us, K = 1296 58 -> 39 us; 3D wave N = 3,
// K = 48000 417 -> 395 us; 2D wave N = 3, K = 45000 225 -> 97 us, N = 6, K = 20000
// 140 -> 137 us; against 3D Maxwell N = 4, K = 48000 716 -> 1152 us and 3D wave
// N = 4 489 -> 722 us, N = 5, K = 16464 252 -> 568 us.
// Beyond 16384 elements 2D advection and wave of order 6 and 3D wave of order 1
// and 2 stay where they were: the two sides are within 5 % of each other there
// (2D wave, order 6: K = 7200 81 -> 72 us, K = 20000 140 -> 137, K = 33800 201 -> 210; 3D
// wave, orders 1 and 2: K = 10368 52 -> 32 us, K = 34992 63 -> 67 and 143 -> 146 us).
constexpr bool f64_fp32_state(int dim, int order) { return dim == 2 || order <= 3; }
inline bool f64_fp32_mesh(int model, int dim, int order, int64_t k) {
  const bool wave = model == HB_MODEL_WAVE || model == HB_MODEL_VARWAVE;
  const bool even = dim == 2 ? order == 6 && (wave || model == HB_MODEL_ADVECTION)
                             : order <= 2 && wave;
  return !even || k <= 16384;
}

// Advection of low order on larger meshes stays on the CUDA cores: one field
// makes tiles of many small elements, whose point phases outweigh the product
// (stage times, CUDA cores -> here): 2D order 2, K = 24200 7.0 -> 7.7 us (K = 16200 6.5
// -> 6.6); 3D order 1, K = 24576 7.6 -> 8.0, K = 34992 8.5 -> 9.9 (FP32 states K = 13182 7.1 ->
// 8.0); 3D order 2, K = 1296 6.8 -> 7.1, K = 10368 8.7 -> 10.4, K = 48000 23 -> 29.  FP32
// states keep their FP64 arithmetic there; of 3D order 3 they go to the split
// planes (K = 16464 16.3 -> 16.8, K = 48000 35 -> 46).
inline bool f64_mesh(int model, int dim, int order, bool fp32, int64_t k) {
  if (model != HB_MODEL_ADVECTION) return true;
  if (dim == 2) return order != 2 || k <= 16384;
  return order == 1 ? k <= (fp32 ? 12288 : 16384) : order == 2 ? k <= 1024
                    : order != 3 || !fp32 || k <= 16384;
}

// Maxwell: the variable-material kernel where the call gives the material
template <int MODEL, int DIM, int ORDER, typename IO>
hb_status f64_material(const F64Call& c) {
  // (FP32 3D Maxwell of order 3 refuses a material: api.cu, check_inputs)
  if constexpr (IsMaxwell<MODEL>::value && !(DIM == 3 && ORDER >= 3 && sizeof(IO) == 4)) {
    if (c.configure || c.coeff != nullptr) {
      const hb_status st = f64_one<MODEL, DIM, ORDER, true, IO>(c);
      if (st || !c.configure) return st;
    }
  }
  return f64_one<MODEL, DIM, ORDER, false, IO>(c);
}

template <int MODEL, int DIM, int ORDER>
hb_status f64_order(const F64Call& c) {
  const bool fp32 = c.op->precision == HB_PREC_FP32;
  if (c.configure && !f64_mesh(MODEL, DIM, ORDER, fp32, c.op->d->K))
    return fail(HB_ERR_UNSUPPORTED, "FP64 tensor-core kernel: slower on this mesh");
  if (fp32) {
    // FP32 states: the elements and meshes that are faster here
    if constexpr (f64_fp32_state(DIM, ORDER)) {
      if (!c.configure || f64_fp32_mesh(MODEL, DIM, ORDER, c.op->d->K))
        return f64_material<MODEL, DIM, ORDER, float>(c);
    }
    return fail(HB_ERR_UNSUPPORTED, "FP64 tensor-core kernel: not for this FP32 state");
  }
  return f64_material<MODEL, DIM, ORDER, double>(c);
}

template <int MODEL, int DIM>
hb_status f64_orders(const F64Call& c) {
  switch (c.op->d->order) {
    case 1: return f64_order<MODEL, DIM, 1>(c);
    case 2: return f64_order<MODEL, DIM, 2>(c);
    case 3: return f64_order<MODEL, DIM, 3>(c);
    case 4: return f64_order<MODEL, DIM, 4>(c);
    case 5: return f64_order<MODEL, DIM, 5>(c);
    case 6: return f64_order<MODEL, DIM, 6>(c);
    case 7: return f64_order<MODEL, DIM, 7>(c);
    default: return fail(HB_ERR_UNSUPPORTED, "FP64 tensor-core kernel: orders 1 to 7");
  }
}

}  // namespace hb
