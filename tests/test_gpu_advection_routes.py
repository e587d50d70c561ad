"""Advection of low order on both sides of the mesh sizes from which it stays
on the CUDA cores (rhs_fp64.cuh, f64_mesh), FP64 and FP32 states: right-hand
side and stage against the oracle, element ranges against the whole.  FP64:
1e-12 relative L2; FP32 states up to order 2 are computed in FP64 and rounded
once per value (6e-8), order 3 on larger meshes on split FP16 planes (1e-6, their
bound)."""
import numpy as np
import pytest

import hedge_b200 as hb
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dim,order,n,m", [
    (2, 2, 90, 90), (2, 2, 91, 91), (3, 1, 12, 13), (3, 1, 13, 13), (3, 1, 14, 14), (3, 1, 15, 14),
    (3, 2, 5, 6), (3, 2, 6, 6), (3, 3, 13, 16), (3, 3, 14, 14)])
def test_both_sides(cuda_device, dim, order, n, m, precision):
    import torch
    from hedge_b200 import _native
    from oracle import OracleRHS
    tag = lambda *a: ["inflow"]                                          # noqa: E731
    mesh = hb.make_regular_rect_mesh((-1, -1), (1, 1), (n + 1, m + 1), jitter=0.1 / n, seed=3,
                                     boundary_tagger=tag) if dim == 2 else \
        hb.make_box_tet_mesh(n=(n, n, m), jitter=0.1 / n, seed=3, boundary_tagger=tag)
    d = hb.Discretization(mesh, order=order, precision=precision)
    op = hb.StrongAdvectionOperator(np.array([1.0, 0.5, -0.3][:dim]), flux_type="upwind")
    comp = d.compile(op.op_template())
    rng = np.random.default_rng(order)
    u = rng.uniform(-1, 1, (1, len(d)))
    if precision == "fp32":
        u = u.astype(np.float32).astype(np.float64)
    bc = rng.uniform(-1, 1, comp.n_given)
    ref = OracleRHS(d, op.descriptor())(u, bc_in=bc)
    eps = 1e-12 if precision == "fp64" else 1e-6 if order == 3 else 1e-12 + 6e-8
    got = comp(w=u, bc_in=bc).double().cpu().numpy()
    comp.check()
    assert rel_l2(got.reshape(1, -1), ref) <= eps
    a, b, dt = -0.6, 0.4, 1e-3
    q = comp.as_state(u)
    r0 = torch.full_like(q, 0.25)
    res, out = r0.clone(), torch.empty_like(q)
    comp.lsrk_stage(a, b, dt, q, out, res, bc_in=bc)
    want = a * 0.25 + dt * ref
    assert rel_l2(res.double().cpu().numpy(), want) <= 2 * eps
    assert rel_l2(out.double().cpu().numpy(), u + b * want) <= 2 * eps
    # the same stage in two element ranges, bit for bit
    bcd = d.to_device(bc, torch.float64)
    res2, out2, k = r0.clone(), torch.empty_like(q), d.K // 3 + 1
    for e0, e1 in ((0, k), (k, d.K)):
        _native.check(comp._lib.hb_lsrk_stage_elements(
            comp._handle, e0, e1, a, b, dt, q.data_ptr(), out2.data_ptr(), res2.data_ptr(), None,
            bcd.data_ptr(), None, comp._stream()))
    comp.check()
    assert torch.equal(out, out2) and torch.equal(res, res2)
