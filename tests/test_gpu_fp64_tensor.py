"""The FP64 tensor-core right-hand side (rhs_fp64.cu) against the CPU oracle
at every order it is built for, at order 8 (which the CUDA-core kernel
serves), and where a batch, a column tile or the persistent loop ends: meshes
of 2 to 30 elements with all boundary kinds, and one with more batches than
resident CTAs.  The bound is the FP64 bound of a right-hand side, 1e-12
relative L2 (both sides sum at most a few hundred terms per value)."""
import numpy as np
import pytest

import hedge_b200 as hb
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _tagger(fvi, el, fn, points):
    c = points[list(fvi)].mean(axis=0)
    return ["open" if c[0] > 1 - 1e-9 else "mid" if c[0] < -1 + 1e-9 else "wall"]


def _mesh(dim, n, m):
    if dim == 2:
        return hb.make_regular_rect_mesh((-1, -1), (1, 1), (n + 1, m + 1), jitter=0.1 / n, seed=3,
                                         boundary_tagger=_tagger)
    return hb.make_box_tet_mesh(n=(n, n, m), jitter=0.1 / n, seed=3, boundary_tagger=_tagger)


def _operator(model, dim, d):
    x = d.nodes
    if model == "advection":
        return hb.StrongAdvectionOperator(np.array([1.0, 0.5, -0.3][:dim]), inflow_tag="wall",
                                          outflow_tag="open", flux_type="lf")
    if model == "wave":
        return hb.StrongWaveOperator(-0.8, dim, dirichlet_tag="wall", neumann_tag="mid",
                                     radiation_tag="open")
    if model == "varwave":
        return hb.VariableVelocityStrongWaveOperator(1.0 + 0.3 * np.sin(2 * x[:, 0]), dim,
                                                     dirichlet_tag="wall", neumann_tag="mid",
                                                     radiation_tag="open")
    cls = {"tm": hb.TMMaxwellOperator, "te": hb.TEMaxwellOperator}.get(model, hb.MaxwellOperator)
    eps, mu = (1.5 + 0.4 * np.sin(x[:, 0]), 1.2 + 0.3 * np.cos(x[:, 1])) \
        if model == "material" else (1.3, 0.7)
    return cls(eps, mu, flux_type=0.6, pec_tag="wall", pmc_tag="mid", absorb_tag="open")


def _check(model, dim, order, n, m):
    import torch
    from oracle import OracleRHS
    d = hb.Discretization(_mesh(dim, n, m), order=order)
    op = _operator(model, dim, d)
    comp = d.compile(op.op_template())
    F = comp.F
    rng = np.random.default_rng(order)
    x = d.nodes
    w = np.stack([np.sin((f + 1.3) * x[:, 0] + f) * np.cos(x[:, -1]) for f in range(F)]) \
        + 0.1 * rng.uniform(-1, 1, (F, len(d)))
    bc = np.sin(3 * d.get_boundary("wall").nodes[:, 0]) if model == "advection" else None
    ref = OracleRHS(d, op.descriptor())(w, bc_in=bc)
    q = d.to_device(w)
    out = torch.full_like(q, np.nan)
    comp.rhs_into(q, out, bc_in=bc)
    res0 = 0.01 * rng.uniform(-1, 1, w.shape)
    res, q1 = d.to_device(res0).clone(), torch.full_like(q, np.nan)
    comp.lsrk_stage(-0.4, 0.3, 0.01, q, q1, res, bc_in=bc)
    comp.check()
    assert rel_l2(out.cpu().numpy(), ref) <= 1e-12
    rref = -0.4 * res0 + 0.01 * ref
    assert rel_l2(res.cpu().numpy(), rref) <= 1e-12
    assert rel_l2(q1.cpu().numpy(), w + 0.3 * rref) <= 1e-12


MODELS = [("advection", 2), ("advection", 3), ("wave", 2), ("wave", 3), ("varwave", 2),
          ("varwave", 3), ("maxwell", 3), ("material", 3), ("tm", 2), ("te", 2)]


@pytest.mark.parametrize("order", range(1, 9))
@pytest.mark.parametrize("model,dim", MODELS)
def test_every_order(cuda_device, model, dim, order):
    n, m = (3, 5) if dim == 2 else (1, 2 if order > 5 else 5)
    _check(model, dim, order, n, m)


@pytest.mark.parametrize("model,dim,n,m", [("advection", 2, 1, 1), ("maxwell", 3, 1, 1),
                                           ("tm", 2, 150, 149), ("maxwell", 3, 13, 11),
                                           ("varwave", 3, 16, 13)])
def test_mesh_sizes(cuda_device, model, dim, n, m):
    _check(model, dim, 2, n, m)


@pytest.mark.parametrize("order", range(1, 8))
@pytest.mark.parametrize("model,dim", [m for m in MODELS if m[0] != "material"])
def test_fp32_state(cuda_device, model, dim, order):
    """FP32 states, on this kernel or (3D from order 4) on the split planes:
    1e-5 relative L2, the FP32 path's bound, on FP32-rounded inputs."""
    _check_fp32(model, dim, order, *((3, 5) if dim == 2 else (1, 2 if order > 5 else 5)))


@pytest.mark.parametrize("n,m", [(90, 91), (91, 91)])
def test_fp32_state_on_both_sides_of_the_mesh_rule(cuda_device, n, m):
    """2D wave of order 6 with 16380 and 16562 elements: this kernel, the split
    planes."""
    _check_fp32("wave", 2, 6, n, m)


def _check_fp32(model, dim, order, n, m):
    from oracle import OracleRHS
    d = hb.Discretization(_mesh(dim, n, m), order=order, precision="fp32")
    op = _operator(model, dim, d)
    comp = d.compile(op.op_template())
    x = d.nodes
    w = np.stack([np.sin((f + 1.3) * x[:, 0] + f) * np.cos(x[:, -1]) for f in range(comp.F)])
    w = w.astype(np.float32).astype(np.float64)
    bc = np.sin(3 * d.get_boundary("wall").nodes[:, 0]) if model == "advection" else None
    ref = OracleRHS(d, op.descriptor())(w, bc_in=bc)
    q = d.to_device(w)
    out = q.new_empty(q.shape)
    comp.rhs_into(q, out, bc_in=bc)
    comp.check()
    assert rel_l2(out.double().cpu().numpy(), ref) <= 1e-5


@pytest.mark.parametrize("order", [2, 3])
def test_fp32_material_and_incident_data(cuda_device, order):
    """HB_PREC_FP32 Maxwell through the C ABI: variable material and incident
    data are taken at order 2 and refused from order 3 on, where the precision
    is the split kernels'."""
    import ctypes as C

    from hedge_b200 import _native
    from hedge_b200.discretization import op_descriptor
    from oracle import OracleRHS
    d = hb.Discretization(_mesh(3, 1, 5), order=order, precision="fp32")
    op = _operator("material", 3, d)
    comp = d.compile(op.op_template())
    desc = op_descriptor(comp.ot, _native.PREC_FP32, comp.conn, comp.n_given)
    h = C.c_void_p()
    _native.check(comp._lib.hb_op_create(d._native_handle(), C.byref(desc), C.byref(h)))
    rng = np.random.default_rng(5)
    w = rng.uniform(-1, 1, (6, len(d))).astype(np.float32).astype(np.float64)
    q = d.to_device(w)
    out = q.new_empty(q.shape)
    st = comp._lib.hb_rhs(h, q.data_ptr(), out.data_ptr(), comp._coeff.data_ptr(), None, None,
                          comp._stream())
    if order == 3:
        assert st == _native.HB_ERR_UNSUPPORTED
        assert comp._lib.hb_rhs(h, q.data_ptr(), out.data_ptr(), None, q.data_ptr(), None,
                                comp._stream()) == _native.HB_ERR_UNSUPPORTED
    else:
        _native.check(st)
        ref = OracleRHS(d, op.descriptor())(w)
        assert rel_l2(out.double().cpu().numpy(), ref) <= 1e-5
    _native.check(comp._lib.hb_op_destroy(h))
