"""LSRK4TimeStepper and the data that a model evaluates: data that may change
within a step reach each stage at that stage's own time, whoever evaluates
them (a model's own ``context``, a subclass's, a subclass of BoundRHS); only a
built-in ``context`` reading TimeConstantGivenFunctions is evaluated once a
step.  On the CPU with a stand-in for the compiled operator that records its
calls; on the GPU each step equals five lsrk_stage calls bit for bit."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import hedge_b200 as hb
from hedge_b200.discretization import BoundRHS
from hedge_b200.models import MODEL_ADVECTION, MODEL_MAXWELL, MODEL_VARADV, MODEL_WAVE
from hedge_b200.timestep import RK4A, RK4B, RK4C

CONST, CHANGING = hb.TimeConstantGivenFunction, hb.TimeDependentGivenFunction


class _Recorder:
    """What the stepper uses of a compiled operator; keeps each stage's data
    and coefficients."""

    def __init__(self, model, n_given=4):
        self.ot, self.n_given, self.stages = SimpleNamespace(model=model), n_given, []
        self.discr = SimpleNamespace(
            interpolate_boundary_function=lambda f, tag: f(np.zeros((4, 2))))

    def as_state(self, w):
        return w

    def lsrk_stage(self, a, b, dt, q_in, q_out, res, bc_in=None, coeff=None):
        self.stages.append((a, b, bc_in))

    def lsrk_step(self, a, b, dt, bufs, res, bc_in=None, coeff=None):
        self.stages += [(x, y, bc_in) for x, y in zip(a, b)]


class _OwnAdvection(hb.StrongAdvectionOperator):
    def context(self, discr, t, fields=None):
        return {"bc_in": np.full(4, t)}


class _OwnMaxwell(hb.MaxwellOperator):
    def context(self, discr, t, fields=None):
        return {"bc_in": np.full((6, 4), t)}


class _OwnRHS(BoundRHS):
    def context(self, t):
        return {"bc_in": np.full(4, t)}


def _advection(data, cls=hb.StrongAdvectionOperator):
    return cls(np.array([1.0, 0.5]), inflow_u=data)


def _with_attribute(model):
    model.context = lambda discr, t, fields=None: {"bc_in": np.full(4, t)}
    return model


def _wave(data):
    op = hb.StrongWaveOperator(1.0, 2)
    op.dirichlet_bc_f = data
    return op


ONE, TIME = (lambda x: np.ones(len(x))), (lambda x, t: np.full(len(x), t))
CHANGES = {
    "subclass": (MODEL_ADVECTION, BoundRHS, lambda: _advection(CONST(ONE), _OwnAdvection)),
    "maxwell": (MODEL_MAXWELL, BoundRHS, lambda: _OwnMaxwell(1.0, 1.0, 1)),
    "bound": (MODEL_ADVECTION, _OwnRHS, lambda: _advection(CONST(ONE))),
    "attribute": (MODEL_ADVECTION, BoundRHS, lambda: _with_attribute(_advection(CONST(ONE)))),
    "any object": (MODEL_WAVE, BoundRHS, lambda: _with_attribute(SimpleNamespace())),
    "given": (MODEL_ADVECTION, BoundRHS, lambda: _advection(CHANGING(TIME))),
    "wave": (MODEL_WAVE, BoundRHS, lambda: _wave(CHANGING(TIME))),
    "velocity": (MODEL_VARADV, BoundRHS, lambda: _with_attribute(
        hb.VariableCoefficientAdvectionOperator(2, CONST(ONE), bc_u_f=CONST(ONE)))),
}


@pytest.mark.parametrize("which", CHANGES)
def test_each_stage_has_its_own_time(which):
    model, bound, make = CHANGES[which]
    comp = _Recorder(model)
    rhs = bound(comp, make())
    assert not rhs.constant_context()
    hb.LSRK4TimeStepper()(torch.zeros(1, 4), 0.25, 0.5, rhs)
    assert [s[2].ravel()[0] for s in comp.stages] == [0.25 + c * 0.5 for c in RK4C]


@pytest.mark.parametrize("model,make", [(MODEL_ADVECTION, lambda: _advection(CONST(ONE))),
                                        (MODEL_WAVE, lambda: _wave(CONST(ONE))),
                                        (MODEL_WAVE, lambda: SimpleNamespace())])
def test_known_constant_data(model, make):
    comp = _Recorder(model, n_given=4 if hasattr(make(), "context") else 0)
    rhs = BoundRHS(comp, make())
    assert rhs.constant_context()
    hb.LSRK4TimeStepper()(torch.zeros(1, 4), 0.25, 0.5, rhs)
    assert [s[:2] for s in comp.stages] == list(zip(RK4A, RK4B))


@pytest.mark.parametrize("data", [CONST(ONE), CHANGING(TIME)])
@pytest.mark.parametrize("n", [4, 5])
def test_the_steppers_own_coefficients(data, n):
    comp = _Recorder(MODEL_ADVECTION)
    stepper = hb.LSRK4TimeStepper()
    stepper.coeffs = np.linspace(0.1, 0.9, 3 * n).reshape(n, 3)
    stepper(torch.zeros(1, 4), 0.25, 0.5, BoundRHS(comp, _advection(data)))
    assert [s[:2] for s in comp.stages] == [(a, b) for a, b, _ in stepper.coeffs]


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["advection", "maxwell", "any object"])
def test_step_equals_stages(cuda_device, which):
    from hedge_b200 import optemplate as ot
    if which == "maxwell":
        d = hb.Discretization(hb.make_box_tet_mesh(n=(2, 2, 2), jitter=0.03, seed=4), order=3)

        class Incident(hb.MaxwellOperator):
            def context(self, discr, t, fields=None):
                n = len(discr.get_boundary(hb.TAG_ALL).nodes)
                return {"bc_in": np.full((6, n), np.cos(t))}
        op = Incident(1.0, 1.0, flux_type=1, pec_tag=hb.TAG_NONE, incident_tag=hb.TAG_ALL,
                      incident_bc=lambda o, e, h: ot.make_sym_vector("inc", 6))
        rhs = op.bind(d)
    else:
        m = hb.make_regular_rect_mesh((-1, -1), (1, 1), (6, 6), jitter=0.02, seed=1,
                                      boundary_tagger=lambda *a: ["inflow"])
        d = hb.Discretization(m, order=3)
        n = len(d.get_boundary("inflow").nodes)

        class Inflow(hb.StrongAdvectionOperator):
            def context(self, discr, t, fields=None):
                return {"bc_in": np.full(n, np.cos(t))}
        op = Inflow(np.array([1.0, 0.5]), flux_type="upwind")
        rhs = op.bind(d)
        if which == "any object":
            rhs = rhs.compiled.bind_model(
                SimpleNamespace(context=lambda discr, t: {"bc_in": np.full(n, np.cos(t))}))
    comp = rhs.compiled
    rng = np.random.default_rng(1)
    y = d.to_device(rng.uniform(-1, 1, (comp.F, len(d))))
    t, dt = 0.3, 0.01
    got = hb.LSRK4TimeStepper()(y, t, dt, rhs)
    cur, res = y, torch.zeros_like(y)
    for a, b, c in zip(RK4A, RK4B, RK4C):
        nxt = torch.empty_like(cur)
        comp.lsrk_stage(a, b, dt, cur, nxt, res, **rhs.context(t + c * dt))
        cur = nxt
    comp.check()
    assert torch.equal(got, cur)
