// The FP64 tensor-core kernel's instances, one group of models per object
// file (HB_FP64_PART), and their dispatch (part 0).
#include "rhs_fp64.cuh"

namespace hb {

#if HB_FP64_PART == 0
hb_status f64_advection(const F64Call& c) {
  return c.op->d->dim == 2 ? f64_orders<HB_MODEL_ADVECTION, 2>(c)
                           : f64_orders<HB_MODEL_ADVECTION, 3>(c);
}
hb_status f64_wave2(const F64Call& c);
hb_status f64_wave3(const F64Call& c);
hb_status f64_varwave(const F64Call& c);
hb_status f64_maxwell(const F64Call& c);
hb_status f64_tm(const F64Call& c);
hb_status f64_te(const F64Call& c);

static hb_status f64_dispatch(const F64Call& c) {
  const int dim = c.op->d->dim;
  switch (c.op->model) {
    case HB_MODEL_ADVECTION: return f64_advection(c);
    case HB_MODEL_WAVE: return dim == 2 ? f64_wave2(c) : f64_wave3(c);
    case HB_MODEL_VARWAVE: return f64_varwave(c);
    case HB_MODEL_MAXWELL: return f64_maxwell(c);
    case HB_MODEL_MAXWELL_TM: return f64_tm(c);
    case HB_MODEL_MAXWELL_TE: return f64_te(c);
    default: return fail(HB_ERR_UNSUPPORTED, "FP64 tensor-core kernel: model not built");
  }
}

hb_status prepare_f64(Op* op) {
  F64Call c = {op, 0, 0, 0, 0, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
               0, op->d->K, nullptr, true};
  return f64_dispatch(c);
}

hb_status launch_f64(Op* op, int mode, double ra, double rb, double dt, const void* q_in,
                     void* q_out, void* res, const double* coeff, const double* bdry,
                     const double* source, int64_t e0, int64_t e1, cudaStream_t s) {
  F64Call c = {op, mode, ra, rb, dt, q_in, q_out, res, coeff, bdry, source, e0, e1, s, false};
  return f64_dispatch(c);
}
#elif HB_FP64_PART == 1
hb_status f64_wave2(const F64Call& c) { return f64_orders<HB_MODEL_WAVE, 2>(c); }
hb_status f64_wave3(const F64Call& c) { return f64_orders<HB_MODEL_WAVE, 3>(c); }
#elif HB_FP64_PART == 2
hb_status f64_varwave(const F64Call& c) {
  return c.op->d->dim == 2 ? f64_orders<HB_MODEL_VARWAVE, 2>(c)
                           : f64_orders<HB_MODEL_VARWAVE, 3>(c);
}
#elif HB_FP64_PART == 3
hb_status f64_maxwell(const F64Call& c) { return f64_orders<HB_MODEL_MAXWELL, 3>(c); }
#else
hb_status f64_tm(const F64Call& c) { return f64_orders<HB_MODEL_MAXWELL_TM, 2>(c); }
hb_status f64_te(const F64Call& c) { return f64_orders<HB_MODEL_MAXWELL_TE, 2>(c); }
#endif

}  // namespace hb
