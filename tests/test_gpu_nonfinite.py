"""A value that is not finite reaches only what depends on it.  The result is
formed with two finite values in one element first: what does not change
between them does not depend on that element, and stays bit for bit as it is
with infinities and NaN there (neither the padding of a tile
nor a product with a 0/1 matrix may spread them)."""
import numpy as np
import pytest

import hedge_b200 as hb

pytestmark = pytest.mark.gpu


def _mesh(dim):
    if dim == 2:
        return hb.make_regular_rect_mesh((-1, -1), (1, 1), (6, 6), jitter=0.03, seed=1)
    return hb.make_box_tet_mesh(n=(3, 3, 3), jitter=0.03, seed=1)


def _inner(d):
    """An element away from the boundary."""
    centres = d.nodes.reshape(d.K, d.Np, -1).mean(axis=1)
    return int(np.abs(centres).sum(axis=1).argmin())


def _unaffected(run, x, d):
    """Runs with finite values in one element, then with others; returns the
    mask of the outputs (that element's left out) that agree, by field and
    element, and checks them with infinities and NaN there."""
    import torch
    e = _inner(d)
    cols = slice(e * d.Np, (e + 1) * d.Np)
    base = run(x)
    other = x.clone()
    other[..., cols] = -1.7 * x[..., cols] + 0.3
    same = base == run(other)
    same = same.reshape(-1, d.K, d.Np).all(dim=2, keepdim=True).expand(-1, -1, d.Np)
    same = same.reshape(base.shape).clone()
    same[..., cols] = False
    assert bool(torch.isfinite(base).all())
    for bad in (float("inf"), float("-inf"), float("nan")):
        other[..., cols] = bad
        got = run(other)
        assert not bool(torch.isfinite(got[..., cols]).all())
        assert torch.equal(got[same], base[same])
    return same


@pytest.mark.parametrize("dim,order,degree", [(2, 2, 6), (2, 4, 9), (2, 5, 15), (3, 2, 5),
                                              (3, 3, 8)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_quadrature_upwind(cuda_device, dim, order, degree, precision):
    """Over-integrated advection: upwind neighbours do not see the element."""
    d = hb.Discretization(_mesh(dim), order=order, precision=precision,
                          quad_min_degrees={"quad": degree})
    v = np.array([1.0, 0.6, 0.35])[:dim]
    op = hb.VariableCoefficientAdvectionOperator(
        dim, hb.TimeConstantGivenFunction(lambda x: np.outer(v, np.ones(len(x)))),
        bc_u_f=hb.TimeConstantGivenFunction(lambda x: np.ones(len(x))), flux_type="upwind")
    rhs = op.bind(d)
    u = d.to_device(np.random.default_rng(order).uniform(0.5, 1.5, len(d))).reshape(1, -1)
    u = u.to(rhs.compiled.state_dtype)
    same = _unaffected(lambda x: rhs(0.0, x).reshape(1, -1), u, d)
    # at least one neighbour, and no node of the elements further away, is upwind
    e = _inner(d)
    neighbours = [k for k in set(rhs.compiled.conn.reshape(d.K, -1, 2)[e, :, 0])]
    kept = [bool(same.reshape(d.K, d.Np)[k].all()) for k in neighbours]
    assert any(kept) and not all(kept)
    rhs.compiled.check()


@pytest.mark.parametrize("order", [1, 3, 5, 7, 8])
@pytest.mark.parametrize("model,dim", [("advection", 2), ("varwave", 2), ("wave", 3),
                                       ("varwave", 3), ("maxwell", 3), ("tm", 2)])
def test_adjoint(cuda_device, model, dim, order):
    """The cotangent in an element, and the state for the c gradient, reach the
    neighbours' nodes on the shared faces and no others (orders 1 to 7 and the
    CUDA-core kernel beyond)."""
    import torch
    from test_gpu_fp64_tensor import _mesh as tagged, _operator
    mesh = tagged(dim, 5, 5) if dim == 2 else tagged(dim, 2, 2)
    d = hb.Discretization(mesh, order=order)
    op = _operator(model, dim, d)
    comp = d.compile(op.op_template())
    e = _inner(d)
    mine = torch.zeros(len(d), dtype=torch.bool, device=d.device)
    mine[e * d.Np:(e + 1) * d.Np] = True
    inner, outer = comp.gather_map()
    reached = mine.clone()
    inside = outer >= 0
    reached[inner[inside][mine[outer[inside]]]] = True
    assert int(reached.sum()) > d.Np
    rng = np.random.default_rng(order)
    q, lam = (d.to_device(rng.uniform(-1, 1, (comp.F, len(d)))) for _ in range(2))
    want_c = model == "varwave"
    q_bar, c_bar = comp.adjoint(lam, q=q, want_c=want_c)
    for bad in (float("inf"), float("nan")):
        x = torch.where(mine, bad, lam)
        got, _ = comp.adjoint(x, q=q)
        assert torch.equal(got[:, ~reached], q_bar[:, ~reached])
        assert not bool(torch.isfinite(got[:, mine]).all())
        if want_c:
            for l, s in ((x, q), (lam, torch.where(mine, bad, q))):
                _, got = comp.adjoint(l, q=s, want_c=True)
                assert torch.equal(got[~reached], c_bar[~reached])
                assert not bool(torch.isfinite(got[mine]).all())
    comp.check()
