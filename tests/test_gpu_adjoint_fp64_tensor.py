"""The FP64 tensor-core adjoint (adjoint_fp64.cu) at every order, order 8 (the
CUDA-core adjoint) among them, and on meshes where a batch, a column tile or
the persistent loop ends.  R is linear in q and, for the variable-velocity
wave, in c, so for random q and lam

    q_bar . q = lam . R(q; c)   and   c_bar . c = lam . R(q; c)

with R from the CPU oracle, to 1e-12 of |lam| |R| (FP64 sums); any wrong entry
of q_bar or c_bar breaks it.  One stage of the reversed LSRK recurrences
equals the same stage composed from the adjoint to 1e-13."""
import numpy as np
import pytest

import hedge_b200 as hb
from test_gpu_fp64_tensor import _mesh, _operator
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _check(model, dim, order, n, m):
    from oracle import OracleRHS
    d = hb.Discretization(_mesh(dim, n, m), order=order)
    op = _operator(model, dim, d)
    comp = d.compile(op.op_template())
    rng = np.random.default_rng(order)
    w, lam, lq = (rng.uniform(-1, 1, (comp.F, len(d))) for _ in range(3))
    bc = np.zeros(len(d.get_boundary("wall").nodes)) if model == "advection" else None
    ref = OracleRHS(d, op.descriptor())(w, bc_in=bc)
    want_c = model == "varwave"
    q, l = d.to_device(w), d.to_device(lam)
    q_bar, c_bar = comp.adjoint(l, q=q, want_c=want_c)
    plain, _ = comp.adjoint(l)
    comp.check()
    dot, scale = float((lam * ref).sum()), np.linalg.norm(lam) * np.linalg.norm(ref)
    assert abs(float((q_bar.cpu().numpy() * w).sum()) - dot) <= 1e-12 * scale
    assert rel_l2(plain.cpu().numpy(), q_bar.cpu().numpy()) <= 1e-13
    c0 = np.zeros(len(d))
    if want_c:
        assert abs(float((c_bar.cpu().numpy() * op.c).sum()) - dot) <= 1e-12 * scale
        c0 = rng.uniform(-1, 1, len(d))
    # one stage, in place: lam + b lq is the cotangent
    a, b, dt = -0.7, 0.4, 0.03
    l1, q1, c1 = d.to_device(lam).clone(), d.to_device(lq).clone(), d.to_device(c0).clone()
    comp.adjoint_stage(a, b, dt, l1, q1, q=q, c_bar=c1 if want_c else None)
    comp.check()
    l2 = lam + b * lq
    qb, cb = comp.adjoint(d.to_device(l2), q=q, want_c=want_c)
    assert rel_l2(l1.cpu().numpy(), a * l2) <= 1e-13
    assert rel_l2(q1.cpu().numpy(), lq + dt * qb.cpu().numpy()) <= 1e-13
    if want_c:
        assert rel_l2(c1.cpu().numpy(), c0 + dt * cb.cpu().numpy()) <= 1e-13


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("model,dim", [("advection", 2), ("advection", 3), ("wave", 2),
                                       ("wave", 3), ("varwave", 2), ("varwave", 3),
                                       ("maxwell", 3), ("tm", 2), ("te", 2)])
def test_every_order(cuda_device, model, dim, order):
    n, m = (3, 5) if dim == 2 else (1, 2 if order > 5 else 5)
    _check(model, dim, order, n, m)


@pytest.mark.parametrize("model,dim,n,m", [("advection", 2, 1, 1), ("maxwell", 3, 1, 1),
                                           ("varwave", 2, 150, 149), ("wave", 3, 16, 13)])
def test_mesh_sizes(cuda_device, model, dim, n, m):
    _check(model, dim, 2, n, m)
