// The FP64 tensor-core adjoint's instances, one group of models per object
// file (HB_ADJ_PART), and their dispatch (part 0).
#include "adjoint_fp64.cuh"

namespace hb {

#if HB_ADJ_PART == 0
hb_status adj_advection(const AdjCall& c) {
  return c.op->d->dim == 2 ? adj_orders<HB_MODEL_ADVECTION, 2>(c)
                           : adj_orders<HB_MODEL_ADVECTION, 3>(c);
}
hb_status adj_wave(const AdjCall& c);
hb_status adj_varwave(const AdjCall& c);
hb_status adj_maxwell(const AdjCall& c);
hb_status adj_maxwell2(const AdjCall& c);

static hb_status adj_dispatch(const AdjCall& c) {
  switch (c.op->model) {
    case HB_MODEL_ADVECTION: return adj_advection(c);
    case HB_MODEL_WAVE: return adj_wave(c);
    case HB_MODEL_VARWAVE: return adj_varwave(c);
    case HB_MODEL_MAXWELL: return adj_maxwell(c);
    case HB_MODEL_MAXWELL_TM: case HB_MODEL_MAXWELL_TE: return adj_maxwell2(c);
    default: return fail(HB_ERR_UNSUPPORTED, "FP64 tensor-core adjoint: model not built");
  }
}

bool adjoint_f64_ready(Op* op, bool want_c, cudaStream_t s) {
  const int variant = want_c ? 1 : 0;
  if (op->adj.has(variant)) return true;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (op->d->order > 7 || cudaStreamIsCapturing(s, &cap) != cudaSuccess ||
      cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return false;
  }
  // (allocating here must not upset a capture on another thread)
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  const bool ok = op->adj.ready(
      variant,
      [&]() {
        AdjCall c = {};
        c.op = op;
        c.stream = s;
        c.configure = true;
        c.want_c = want_c;
        return adj_dispatch(c);
      },
      // the CUDA-core adjoint's launches ask for the last error
      []() { cudaGetLastError(); });
  cudaThreadExchangeStreamCaptureMode(&mode);
  return ok;
}

hb_status launch_adjoint_f64(Op* op, const double* q, const double* lam, double* q_bar,
                             double* c_bar, const double* coeff, double* work, cudaStream_t s) {
  AdjCall c = {};
  c.op = op;
  c.stream = s;
  c.a.q = q;
  c.a.lam_in = lam;
  c.a.q_bar = q_bar;
  c.a.c_bar = c_bar;
  c.a.coeff = coeff;
  c.a.work = work;
  return adj_dispatch(c);
}

hb_status launch_adjoint_stage(Op* op, double ra, double rb, double dt, const double* q,
                               double* lam, double* lq, double* c_bar, const double* coeff,
                               double* work, cudaStream_t s) {
  AdjCall c = {};
  c.op = op;
  c.stream = s;
  c.a.q = q;
  c.a.c_bar = c_bar;
  c.a.coeff = coeff;
  c.a.work = work;
  c.a.fused = 1;
  c.a.lam = lam;
  c.a.lq = lq;
  c.a.ra = ra;
  c.a.rb = rb;
  c.a.dt = dt;
  return adj_dispatch(c);
}
#elif HB_ADJ_PART == 1
hb_status adj_wave(const AdjCall& c) {
  return c.op->d->dim == 2 ? adj_orders<HB_MODEL_WAVE, 2>(c) : adj_orders<HB_MODEL_WAVE, 3>(c);
}
#elif HB_ADJ_PART == 2
hb_status adj_varwave(const AdjCall& c) {
  return c.op->d->dim == 2 ? adj_orders<HB_MODEL_VARWAVE, 2>(c)
                           : adj_orders<HB_MODEL_VARWAVE, 3>(c);
}
#else
hb_status adj_maxwell(const AdjCall& c) {
  return c.op->d->dim == 3 ? adj_orders<HB_MODEL_MAXWELL, 3>(c)
                           : fail(HB_ERR_UNSUPPORTED, "Maxwell adjoint: 3D only");
}
hb_status adj_maxwell2(const AdjCall& c) {
  return c.op->model == HB_MODEL_MAXWELL_TM ? adj_orders<HB_MODEL_MAXWELL_TM, 2>(c)
                                            : adj_orders<HB_MODEL_MAXWELL_TE, 2>(c);
}
#endif

}  // namespace hb
