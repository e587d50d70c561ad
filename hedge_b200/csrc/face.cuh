// One face point of an element: the exterior values (neighbour element, halo
// buffer or boundary condition) and the numerical flux, in two steps so that
// the neighbour's values can be requested ahead of the arithmetic.
#pragma once

#include "models.cuh"

namespace hb {

template <typename S>
struct FaceArgs {
  int64_t K, n_given, n_halo;
  const S* q;               // [F][K*Np] state
  const double* coeff;      // c field, or [eps | mu] (variable material)
  const double* bdry;       // given boundary data
  const S* halo;            // [n_halo * nfp][F] ext values of halo faces
  const double* halo_c;     // [n_halo * nfp] ext c (var-c wave)
  int* err;
};

template <int MODEL, int DIM, typename T>
struct FaceExt {
  T u[Args<MODEL, DIM>::N];   // exterior flux arguments (not on a boundary)
  T eps, mu;                  // exterior material (variable material)
  bool ok;                    // the exterior is there (or a boundary's to form)
};

// Requests the exterior values of face node k; `nbr_node` maps (perm,
// neighbour's face, k) to the neighbour's volume node.
template <int MODEL, int DIM, bool VM, typename S>
__device__ __forceinline__ void face_load(const FaceArgs<S>& a, const int2 cn, int k,
                                          int64_t Knp, int np, int nfp, int nf, int nperm,
                                          const uint8_t* nbr_node,
                                          FaceExt<MODEL, DIM, double>& x) {
  constexpr int F = Traits<MODEL, DIM>::F, C = Traits<MODEL, DIM>::COEFF;
  x.ok = true;
  if (cn.x < 0) return;
  if (cn.x >= a.K) {
    // neighbour on another partition: ext values from the halo buffer (which
    // carries no material values)
    const int64_t h = (int64_t)cn.x - a.K;
    if (VM || h >= a.n_halo || a.halo == nullptr) {
      atomicCAS(a.err, 0, VM ? DEV_MISSING_INPUT : DEV_BAD_NEIGHBOUR);
      x.ok = false;
      return;
    }
    const int64_t hi = h * nfp + k;
    if constexpr (C != 0) x.u[0] = a.halo_c[hi];
#pragma unroll
    for (int f = 0; f < F; ++f) x.u[C + f] = (double)a.halo[hi * F + f];
    return;
  }
  const int nface = cn.y & 3, perm = cn.y >> 2;
  if (nface >= nf || perm < 0 || perm >= nperm) {
    atomicCAS(a.err, 0, DEV_BAD_CODE);
    x.ok = false;
    return;
  }
  const int64_t gi = (int64_t)cn.x * np + nbr_node[(perm * nf + nface) * nfp + k];
  if constexpr (C != 0) x.u[0] = a.coeff[gi];
#pragma unroll
  for (int f = 0; f < F; ++f) x.u[C + f] = (double)a.q[f * Knp + gi];
  if constexpr (VM) {
    x.eps = a.coeff[gi];
    x.mu = a.coeff[Knp + gi];
  }
}

// Flux of the interior values uM and the loaded exterior; own: this side's
// volume node.  False: the face carries no flux.
template <int MODEL, int DIM, bool VM, typename S>
__device__ __forceinline__ bool face_flux(const FaceArgs<S>& a, const ModelParams& mp,
                                          const int2 cn, int k, int nfp, int64_t own,
                                          int64_t Knp,
                                          const double (&uM)[Args<MODEL, DIM>::N],
                                          const double (&n)[DIM],
                                          FaceExt<MODEL, DIM, double>& x,
                                          double (&fl)[Traits<MODEL, DIM>::F]) {
  constexpr int F = Traits<MODEL, DIM>::F;
  const bool bdry = cn.x < 0;
  bool have = x.ok;
  // interior and exterior impedances; the interior one on boundary faces
  double Zi = 1.0, Ze = 1.0;
  if constexpr (VM) {
    Zi = sqrt(a.coeff[Knp + own] / a.coeff[own]);
    Ze = bdry || !have ? Zi : sqrt(x.mu / x.eps);
  }
  if (bdry) {
    double given = 0.0;
    const int64_t bi = (int64_t)(-1 - cn.x) * nfp + k;
    if (cn.y == HB_BC_GIVEN) {
      if (a.bdry == nullptr || bi >= a.n_given) {
        atomicCAS(a.err, 0, a.bdry == nullptr ? DEV_MISSING_INPUT : DEV_BAD_BDRY_INDEX);
        have = false;
      } else {
        given = a.bdry[bi];
      }
    }
    if (have) {
      if constexpr (VM) {
        ModelParams mpl = mp;
        mpl.Z = Zi;
        mpl.Y = 1.0 / Zi;
        have = model_bc<MODEL, DIM, double>(mpl, cn.y, uM, n, given, x.u);
      } else {
        have = model_bc<MODEL, DIM, double>(mp, cn.y, uM, n, given, x.u);
      }
    }
    if constexpr (IsMaxwell<MODEL>::value) {
      // incident data d (em.py:289-307): exterior state -d, field f's
      // values at bdry[f * n_given + node]; no data: zero exterior
      if (have && cn.y == HB_BC_INCIDENT && a.bdry != nullptr) {
        if (bi >= a.n_given) {
          atomicCAS(a.err, 0, DEV_BAD_BDRY_INDEX);
          have = false;
        } else {
#pragma unroll
          for (int f = 0; f < F; ++f) x.u[f] = -a.bdry[f * a.n_given + bi];
        }
      }
    }
  }
  if (!have) return false;
  if constexpr (VM)
    maxwell_flux_var<MODEL, DIM, double>(mp, bdry, uM, x.u, n, Zi, Ze, fl);
  else
    model_flux<MODEL, DIM, double>(mp, bdry, uM, x.u, n, fl);
  return true;
}

}  // namespace hb
