// Over-integrated right-hand side of the variable-coefficient advection
// operator (rhs_quad.cu's, same integrals) on the FP64 tensor cores.
//
// A warp owns 8 elements, the rows of its mma.sync m8n8k4 tiles; nodes and
// quadrature points are the columns.  A tile's accumulators sit in the same
// lanes, for the same element, as the left operand of the next product wants
// them (lane (g, t): element g, entries 2 t and 2 t + 1 of 8, with the k of a
// pair of MMAs permuted to match), so the whole chain
//
//   nodes -> volume points -> integrand -> projection
//   face nodes (both sides) -> face points -> flux -> lift
//
// stays in registers: no shared memory and no barrier, and a warp stalled on
// the neighbour gathers leaves the pipe to the others.  The matrices are read
// in fragment order through L1, which they share on an SM.
//
// Bound: FP64 pipe (N = 5, 64 volume points: 294 MMAs per 8 elements, 40 us at
// K = 80000) and L1 wavefronts of the scattered 8-byte gathers.  A stage at K =
// 80000, N = 5: 222 -> 69 us, N = 3 65 -> 37, N = 7 1185 -> 247 (rhs_quad.cu -> here); the
// sizes and meshes that stay there are in quad_on_cores.  The element sizes are
// run-time values except the number of 8-node tiles KS.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "dmma.cuh"

namespace hb {

namespace {

template <typename IO>
struct QuadF64Args {
  int64_t K, n_given;
  int np, nfp, nf, nperm, G, mode, flux_type;
  int nqt, nft;                 // tiles of 8 volume points, face points
  const double2* If;            // [nqt][KS][32]
  const double2* Pf;            // [dim][nqt][KS][32]
  const double2* Ff;            // [nf][nft][KF][32]
  const double2* Lf;            // [nf][nft][KS][32], negated
  const double* geo;
  const int2* conn;
  const int* fmask;
  const int* shuffle;
  const IO* q_in;
  IO* q_out;
  IO* res;
  const double* vel;            // [dim][K*np]
  const double* bdry;
  const double* elmax;          // element maxima of |v|^2 (LF flux)
  double ra, rb, dt;
  int* err;
};

// face-node tiles of the orders with KS node tiles
constexpr int quad_kf(int dim, int ks) { return dim == 2 || ks <= 2 ? 1 : ks <= 5 ? 2 : 3; }
constexpr int QUAD_THREADS = 64;

template <int DIM, int KS, typename IO>
__global__ void __launch_bounds__(QUAD_THREADS) quad_fp64_kernel(const QuadF64Args<IO> a) {
  constexpr int NV = 1 + DIM, KF = quad_kf(DIM, KS);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t group = blockIdx.x * (int64_t)(QUAD_THREADS / 32) + (threadIdx.x >> 5);
  if (group * 8 >= a.K) return;   // the whole warp
  // rows beyond the last element repeat it and store nothing
  const bool live = group * 8 + g < a.K;
  const int64_t el = live ? group * 8 + g : a.K - 1;
  const int64_t Knp = a.K * a.np;
  const int np = a.np, nfp = a.nfp;
  const IO* qe = a.q_in + el * np;
  const double* ve = a.vel + el * np;

  double w[NV][KS][2];
#pragma unroll
  for (int s = 0; s < KS; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 8 * s + 2 * t + h;
      const bool in = j < np;
      w[0][s][h] = in ? (double)__ldg(qe + j) : 0.0;
#pragma unroll
      for (int c = 0; c < DIM; ++c) w[1 + c][s][h] = in ? __ldg(ve + c * Knp + j) : 0.0;
    }
  const double* ge = a.geo + el * a.G;
  double acc[KS][2];
#pragma unroll
  for (int m = 0; m < KS; ++m) acc[m][0] = acc[m][1] = 0.0;

  // ---- volume points, 8 at a time ----
  {
    double rx[DIM][DIM];
#pragma unroll
    for (int r = 0; r < DIM; ++r)
#pragma unroll
      for (int x = 0; x < DIM; ++x) rx[r][x] = __ldg(ge + r * DIM + x);
    for (int qt = 0; qt < a.nqt; ++qt) {
      double c[NV][2];
#pragma unroll
      for (int v = 0; v < NV; ++v) c[v][0] = c[v][1] = 0.0;
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        const double2 b = __ldg(a.If + (qt * KS + s) * 32 + lane);
#pragma unroll
        for (int v = 0; v < NV; ++v) dmma(c[v], w[v][s][0], b.x);
#pragma unroll
        for (int v = 0; v < NV; ++v) dmma(c[v], w[v][s][1], b.y);
      }
#pragma unroll
      for (int r = 0; r < DIM; ++r) {
        double gr[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double s = 0.0;
#pragma unroll
          for (int x = 0; x < DIM; ++x) s += rx[r][x] * c[1 + x][h];
          gr[h] = c[0][h] * s;
        }
#pragma unroll
        for (int m = 0; m < KS; ++m) {
          const double2 b = __ldg(a.Pf + ((r * a.nqt + qt) * KS + m) * 32 + lane);
          dmma(acc[m], gr[0], b.x);
          dmma(acc[m], gr[1], b.y);
        }
      }
    }
  }

  // ---- faces ----
  for (int f = 0; f < a.nf; ++f) {
    const int2 cn = __ldg(a.conn + el * a.nf + f);
    const bool bdry = cn.x < 0;
    bool ok = true;
    const int nface = cn.y & 3, perm = cn.y >> 2;
    if (!bdry && (cn.x >= a.K || nface >= a.nf || perm < 0 || perm >= a.nperm)) {
      atomicCAS(a.err, 0, cn.x >= a.K ? DEV_BAD_NEIGHBOUR : DEV_BAD_CODE);
      ok = false;
    }
    if (bdry && cn.y != HB_BC_GIVEN && cn.y != HB_BC_DIRICHLET && cn.y != HB_BC_NONE)
      atomicCAS(a.err, 0, DEV_BAD_CODE);
    double wm[NV][KF][2], wp[NV][KF][2];
#pragma unroll
    for (int s = 0; s < KF; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = 8 * s + 2 * t + h;
#pragma unroll
        for (int v = 0; v < NV; ++v) wm[v][s][h] = wp[v][s][h] = 0.0;
        if (k < nfp) {
          const int own = __ldg(a.fmask + f * nfp + k);
          wm[0][s][h] = (double)__ldg(qe + own);
#pragma unroll
          for (int c = 0; c < DIM; ++c) wm[1 + c][s][h] = __ldg(ve + c * Knp + own);
          if (bdry) {
            // boundary: the given inflow values or zero, v from inside
#pragma unroll
            for (int c = 0; c < DIM; ++c) wp[1 + c][s][h] = wm[1 + c][s][h];
            if (cn.y == HB_BC_GIVEN) {
              const int64_t bi = (int64_t)(-1 - cn.x) * nfp + k;
              if (a.bdry == nullptr || bi >= a.n_given)
                atomicCAS(a.err, 0, a.bdry == nullptr ? DEV_MISSING_INPUT : DEV_BAD_BDRY_INDEX);
              else
                wp[0][s][h] = __ldg(a.bdry + bi);
            }
          } else if (ok) {
            const int64_t gi = (int64_t)cn.x * np +
                               __ldg(a.fmask + nface * nfp + __ldg(a.shuffle + perm * nfp + k));
            wp[0][s][h] = (double)__ldg(a.q_in + gi);
#pragma unroll
            for (int c = 0; c < DIM; ++c) wp[1 + c][s][h] = __ldg(a.vel + c * Knp + gi);
          }
        }
      }
    double n[DIM];
#pragma unroll
    for (int x = 0; x < DIM; ++x) n[x] = __ldg(ge + DIM * DIM + f * (DIM + 1) + x);
    const double fscale = __ldg(ge + DIM * DIM + f * (DIM + 1) + DIM);
    double cmax = 0.0;
    if (a.flux_type == 2) {
      const double cm = __ldg(a.elmax + el);
      const double cp = !bdry && ok ? __ldg(a.elmax + cn.x) : cm;
      cmax = cm > cp ? cm : cp;
    }
    const bool none = bdry && cn.y == HB_BC_NONE;
    __syncwarp();
    for (int pt = 0; pt < a.nft; ++pt) {
      double cm[NV][2], cp[NV][2];
#pragma unroll
      for (int v = 0; v < NV; ++v) cm[v][0] = cm[v][1] = cp[v][0] = cp[v][1] = 0.0;
#pragma unroll
      for (int s = 0; s < KF; ++s) {
        const double2 b = __ldg(a.Ff + ((f * a.nft + pt) * KF + s) * 32 + lane);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          dmma(cm[v], wm[v][s][0], b.x);
          dmma(cp[v], wp[v][s][0], b.x);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          dmma(cm[v], wm[v][s][1], b.y);
          dmma(cp[v], wp[v][s][1], b.y);
        }
      }
      double fl[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double nvm = 0.0, nvp = 0.0, navg = 0.0;
#pragma unroll
        for (int x = 0; x < DIM; ++x) {
          nvm += n[x] * cm[1 + x][h];
          nvp += n[x] * cp[1 + x][h];
          navg += n[x] * (0.5 * (cm[1 + x][h] + cp[1 + x][h]));
        }
        double v;
        if (a.flux_type == 0)
          v = (cm[0][h] * nvm + cp[0][h] * nvp) * 0.5;
        else if (a.flux_type == 2)
          v = 0.5 * (nvm * cm[0][h] + nvp * cp[0][h]) - 0.5 * (cp[0][h] - cm[0][h]) * cmax;
        else
          v = navg > 0.0 ? nvm * cm[0][h] : nvp * cp[0][h];
        fl[h] = none ? 0.0 : fscale * v;
      }
#pragma unroll
      for (int m = 0; m < KS; ++m) {
        const double2 b = __ldg(a.Lf + ((f * a.nft + pt) * KS + m) * 32 + lane);
        dmma(acc[m], fl[0], b.x);
        dmma(acc[m], fl[1], b.y);
      }
    }
  }

  // ---- output: lane (g, t) holds nodes 8 m + 2 t and + 1 of element g ----
  if (!live) return;
#pragma unroll
  for (int m = 0; m < KS; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = 8 * m + 2 * t + h;
      if (i >= np) continue;
      const int64_t node = el * np + i;
      if (a.mode == 0) {
        a.q_out[node] = (IO)acc[m][h];
      } else {
        const double rv = a.ra * (double)a.res[node] + a.dt * acc[m][h];
        a.res[node] = (IO)rv;
        a.q_out[node] = (IO)(w[0][m][h] + a.rb * rv);
      }
    }
}

struct QuadCall {
  Op* op;
  int mode;
  double ra, rb, dt;
  const void* q_in;
  void* q_out;
  void* res;
  const double* vel;
  const double* bdry;
  cudaStream_t stream;
};

template <int DIM, int KS, typename IO>
hb_status quad_run(const QuadCall& c) {
  Op* op = c.op;
  const Discr* d = op->d;
  QuadF64Args<IO> a;
  a.K = d->K;
  a.n_given = op->n_given;
  a.np = d->np;
  a.nfp = d->nfp;
  a.nf = d->nfaces;
  a.nperm = d->nperm;
  a.G = d->G;
  a.nqt = (op->nq + 7) / 8;
  a.nft = (op->nqf + 7) / 8;
  a.If = reinterpret_cast<const double2*>(op->quadfrag);
  a.Pf = a.If + (size_t)a.nqt * KS * 32;
  a.Ff = a.Pf + (size_t)DIM * a.nqt * KS * 32;
  a.Lf = a.Ff + (size_t)a.nf * a.nft * quad_kf(DIM, KS) * 32;
  a.geo = d->geo;
  a.conn = op->conn;
  a.fmask = d->fmask;
  a.shuffle = d->shuffle;
  a.q_in = static_cast<const IO*>(c.q_in);
  a.q_out = static_cast<IO*>(c.q_out);
  a.res = static_cast<IO*>(c.res);
  a.vel = c.vel;
  a.bdry = c.bdry;
  a.elmax = op->elmax;
  a.ra = c.ra;
  a.rb = c.rb;
  a.dt = c.dt;
  a.mode = c.mode;
  a.flux_type = op->mp.flux_type;
  a.err = op->err_flag;
  quad_fp64_kernel<DIM, KS, IO><<<(unsigned)op->grid, QUAD_THREADS, 0, c.stream>>>(a);
  HB_CUDA(cudaGetLastError());
  return HB_OK;
}

template <int DIM, int KS>
hb_status quad_io(const QuadCall& c) {
  return c.op->precision == HB_PREC_FP32 ? quad_run<DIM, KS, float>(c)
                                         : quad_run<DIM, KS, double>(c);
}

// node tiles built: orders 1 to 7 in 2D, 1 to 5 in 3D
bool quad_built(int dim, int ks) {
  return dim == 2 ? ks <= 5 : ks <= 3 || ks == 5 || ks == 7;
}

}  // namespace

// Uploads the four matrices in fragment order; HB_ERR_UNSUPPORTED for element
// sizes that are not built (rhs_quad.cu's kernel serves those).
hb_status prepare_quad_f64(Op* op, const hb_quad_desc* qd) {
  const Discr* d = op->d;
  const int np = d->np, nfp = d->nfp, nf = d->nfaces, dim = d->dim, nq = qd->nq, nqf = qd->nqf;
  const int ks = (np + 7) / 8, kf = quad_kf(dim, ks);
  if (!quad_built(dim, ks) || nfp > 8 * kf)
    return fail(HB_ERR_UNSUPPORTED, "FP64 tensor-core quadrature kernel: element too large");
  const int nqt = (nq + 7) / 8, nft = (nqf + 7) / 8;
  const size_t nI = (size_t)nqt * ks * 64, nP = (size_t)dim * nI;
  const size_t nF = (size_t)nf * nft * kf * 64, nL = (size_t)nf * nft * ks * 64;
  std::vector<double> h(nI + nP + nF + nL, 0.0);
  // column n, k of a tile: lane (n, k / 2), entry k % 2
  auto at = [](size_t tile, int n, int k) { return tile * 64 + (n * 4 + k / 2) * 2 + (k & 1); };
  double* I = h.data();
  double* P = I + nI;
  double* F = P + nP;
  double* L = F + nF;
  // the points that pad a tile repeat the last one, against zeros in the
  // projection and the lift: as 0 * w their values would not be zero where w is
  // not finite, also where the flux of the points does not see that w
  // (selecting zeros in the kernel instead: 69 -> 72 us a stage at N = 5, K = 80000)
  for (int q = 0; q < 8 * nqt; ++q)
    for (int j = 0; j < np; ++j)
      I[at((size_t)(q / 8) * ks + j / 8, q % 8, j % 8)] =
          qd->vol_interp[(size_t)std::min(q, nq - 1) * np + j];
  for (int q = 0; q < nq; ++q)
    for (int j = 0; j < np; ++j)
      for (int r = 0; r < dim; ++r)
        P[at(((size_t)r * nqt + q / 8) * ks + j / 8, j % 8, q % 8)] =
            qd->vol_project[((size_t)r * np + j) * nq + q];
  for (int f = 0; f < nf; ++f)
    for (int p = 0; p < 8 * nft; ++p) {
      for (int k = 0; k < nfp; ++k)
        F[at(((size_t)f * nft + p / 8) * kf + k / 8, p % 8, k % 8)] =
            qd->face_interp[((size_t)f * nqf + std::min(p, nqf - 1)) * nfp + k];
      if (p >= nqf) continue;
      for (int i = 0; i < np; ++i)
        L[at(((size_t)f * nft + p / 8) * ks + i / 8, i % 8, p % 8)] =
            -qd->face_lift[((size_t)i * nf + f) * nqf + p];
    }
  for (double x : h)
    if (!std::isfinite(x)) return fail(HB_ERR_INVALID_ARGUMENT, "non-finite quadrature matrix");
  if (cudaMalloc(&op->quadfrag, sizeof(double) * h.size()) != cudaSuccess ||
      cudaMemcpy(op->quadfrag, h.data(), sizeof(double) * h.size(), cudaMemcpyHostToDevice) !=
          cudaSuccess)
    return fail(HB_ERR_CUDA, "cannot upload the quadrature matrices");
  const int per_cta = 8 * (QUAD_THREADS / 32);
  op->elems_per_block = per_cta;
  op->threads = QUAD_THREADS;
  op->blocks_per_sm = 0;
  op->smem = 0;
  op->ops_in_smem = 0;
  op->grid = (int)((d->K + per_cta - 1) / per_cta);
  return HB_OK;
}

hb_status launch_quad_f64(Op* op, int mode, double ra, double rb, double dt, const void* q_in,
                          void* q_out, void* res, const double* vel, const double* bdry,
                          cudaStream_t s) {
  const QuadCall c = {op, mode, ra, rb, dt, q_in, q_out, res, vel, bdry, s};
  const int ks = (op->d->np + 7) / 8;
  if (op->d->dim == 2) {
    switch (ks) {
      case 1: return quad_io<2, 1>(c);
      case 2: return quad_io<2, 2>(c);
      case 3: return quad_io<2, 3>(c);
      case 4: return quad_io<2, 4>(c);
      default: return quad_io<2, 5>(c);
    }
  }
  switch (ks) {
    case 1: return quad_io<3, 1>(c);
    case 2: return quad_io<3, 2>(c);
    case 3: return quad_io<3, 3>(c);
    case 5: return quad_io<3, 5>(c);
    default: return quad_io<3, 7>(c);
  }
}

}  // namespace hb
