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
