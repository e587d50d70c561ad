"""hb_lsrk_step: the five stages of a step in one call equal five
hb_lsrk_stage calls bit for bit (same launches in the same order), with one
source per stage too; the stepper's two paths agree where the model's data
are constant in time; bad stage lists are refused on the host."""
import ctypes as C

import numpy as np
import pytest

import hedge_b200 as hb
from hedge_b200 import _native
from hedge_b200.timestep import RK4A, RK4B, RK4C, _A, _B

pytestmark = pytest.mark.gpu


def _problem(precision="fp64"):
    m = hb.make_box_tet_mesh(n=(2, 2, 2), jitter=0.03, seed=4)
    d = hb.Discretization(m, order=4, precision=precision)
    c = 1.0 + 0.2 * np.sin(d.nodes[:, 0])
    comp = hb.VariableVelocityStrongWaveOperator(c, 3).bind(d).compiled
    rng = np.random.default_rng(1)
    return d, comp, d.to_device(rng.uniform(-1, 1, (4, len(d))))


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp16x3"])
@pytest.mark.parametrize("with_source", [False, True])
def test_step_equals_stages(cuda_device, precision, with_source):
    import torch
    d, comp, q = _problem(precision)
    src = torch.rand((5, len(d)), dtype=torch.float64, device=d.device) if with_source else None
    bufs = [q] + [torch.empty_like(q) for _ in range(5)]
    ref = [q] + [torch.empty_like(q) for _ in range(5)]
    r1, r2 = torch.full_like(q, 0.5), torch.full_like(q, 0.5)
    comp.lsrk_step(_A, _B, 0.01, bufs, r1, source=src,
                   source_stride=len(d) if with_source else 0)
    for s in range(5):
        comp.lsrk_stage(RK4A[s], RK4B[s], 0.01, ref[s], ref[s + 1], r2,
                        source=src[s] if with_source else None)
    comp.check()
    for a, b in zip(bufs + [r1], ref + [r2]):
        assert torch.equal(a, b)


def test_stepper_with_constant_and_changing_data(cuda_device):
    import torch
    m = hb.make_regular_rect_mesh((-1, -1), (1, 1), (6, 6), jitter=0.02, seed=1,
                                  boundary_tagger=lambda *a: ["inflow"])
    d = hb.Discretization(m, order=3)
    f = lambda x: np.sin(3 * x[:, 0])                                    # noqa: E731
    y = d.to_device(np.cos(d.nodes.sum(1))).reshape(1, -1)
    out = []
    for data in (hb.TimeConstantGivenFunction(f),
                 hb.TimeDependentGivenFunction(lambda x, t: f(x))):
        op = hb.StrongAdvectionOperator(np.array([1.0, 0.5]), inflow_u=data, flux_type="upwind")
        rhs = op.bind(d)
        assert rhs.constant_context() == (type(data) is hb.TimeConstantGivenFunction)
        out.append(hb.LSRK4TimeStepper()(y, 0.0, 0.01, rhs))
    assert torch.equal(*out)
    # data that do change reach every stage at its own time
    op = hb.StrongAdvectionOperator(
        np.array([1.0, 0.5]), flux_type="upwind",
        inflow_u=hb.TimeDependentGivenFunction(lambda x, t: np.full(len(x), t)))
    rhs = op.bind(d)
    got = hb.LSRK4TimeStepper()(y, 0.0, 0.01, rhs)
    cur, res = y, torch.zeros_like(y)
    for a, b, c in zip(RK4A, RK4B, RK4C):
        nxt = torch.empty_like(cur)
        rhs.compiled.lsrk_stage(a, b, 0.01, cur, nxt, res,
                                bc_in=np.full(rhs.compiled.n_given, c * 0.01))
        cur = nxt
    assert torch.equal(got, cur)


def test_bad_stage_lists_are_refused(cuda_device):
    import torch
    d, comp, q = _problem()
    res, out = torch.zeros_like(q), torch.empty_like(q)
    lib, h, c = comp._lib, comp._handle, comp._coeff.data_ptr()

    def call(n, ptrs, r=res.data_ptr()):
        return lib.hb_lsrk_step(h, n, _A, _B, 0.01, (C.c_void_p * len(ptrs))(*ptrs), r, c, None,
                                None, 0, None)
    a, b = q.data_ptr(), out.data_ptr()
    bad = _native.HB_ERR_INVALID_ARGUMENT
    assert call(0, [a, b]) == bad and call(1, [a, a]) == bad and call(2, [a, b, b]) == bad
    assert call(1, [a, None]) == bad and call(1, [a, b], None) == bad
    assert lib.hb_lsrk_step(None, 1, _A, _B, 0.01, (C.c_void_p * 2)(a, b), res.data_ptr(), c,
                            None, None, 0, None) == bad
