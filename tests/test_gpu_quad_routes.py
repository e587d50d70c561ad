"""The over-integrated advection on both sides of the rule that chooses its
kernel (rhs_quad.cu: 256 threads a CTA; quad_fp64.cu: 64), right-hand side and
stage, FP64 and FP32 states, against the template executor on one copy of a
small mesh; the larger meshes are copies of it, not connected to one another.
FP64: 1e-12 relative L2, the bound of a right-hand side; FP32 states are
computed in FP64 and rounded once per value (6e-8)."""
import numpy as np
import pytest

import hedge_b200 as hb
from conftest import rel_l2
from test_quadrature import state, velocity

pytestmark = pytest.mark.gpu


def _copies(mesh, n):
    points, elements = mesh.points, mesh.elements
    return hb.Mesh(np.tile(points, (n, 1)), np.concatenate(
        [elements + k * len(points) for k in range(n)]))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("dim,order,degree,K,threads", [
    (2, 1, 3, 20466, 64), (2, 1, 3, 20484, 256),
    (2, 6, 13, 18, 256), (2, 6, 13, 1332, 256), (2, 6, 13, 3204, 64),
    (2, 7, 15, 18, 256), (2, 7, 15, 2070, 256), (2, 7, 15, 4140, 64),
    (3, 2, 5, 6, 256), (3, 2, 5, 12, 64),
    (3, 3, 9, 6, 256), (3, 3, 9, 1776, 256), (3, 3, 9, 1782, 64),
    (3, 4, 9, 1032, 256), (3, 4, 9, 1044, 64), (3, 4, 12, 24, 64),
    (3, 5, 11, 12, 256), (3, 5, 11, 3072, 64), (3, 5, 15, 6, 64), (3, 6, 13, 6, 256)])
def test_both_sides(cuda_device, dim, order, degree, K, threads, precision):
    import torch
    from optemplate_exec import TemplateExecutor
    mesh = hb.make_regular_rect_mesh((-1, -1), (1, 1), (4, 4), jitter=0.05, seed=2) if dim == 2 \
        else hb.make_box_tet_mesh(n=(1, 1, 1), jitter=0.05, seed=2)
    n = K // len(mesh.elements)
    assert n * len(mesh.elements) == K
    op = hb.VariableCoefficientAdvectionOperator(dim, None, bc_u_f=1, flux_type="upwind")
    tpl = op.op_template()
    small = hb.Discretization(mesh, order=order, quad_min_degrees={"quad": degree})
    u, v = state(small, 3), velocity(small)
    if precision == "fp32":
        u = u.astype(np.float32).astype(np.float64)
    bc = lambda d: np.sin(3 * d.get_boundary(hb.TAG_ALL).nodes[:, 0])     # noqa: E731
    ref = np.tile(TemplateExecutor(small)(tpl, u=u, v=v, bc_u=bc(small))[0], n)
    d = hb.Discretization(_copies(mesh, n), order=order, precision=precision,
                          quad_min_degrees={"quad": degree})
    comp = d.compile(tpl)
    assert comp.launch_info()["threads"] == threads
    u, v = np.tile(u, n), np.tile(v, (1, n))
    got = comp(u=u, v=v, bc_u=bc(d)).double().cpu().numpy()
    comp.check()
    eps = 1e-12 if precision == "fp64" else 1e-12 + 6e-8
    assert rel_l2(got, ref) <= eps
    # a stage: res = a res + dt rhs, q = u + b res
    a, b, dt = -0.6, 0.4, 1e-2
    q = comp.as_state(u)
    res, out = torch.full_like(q, 0.25), torch.empty_like(q)
    comp.lsrk_stage(a, b, dt, q, out, res, bc_in=bc(d),
                    coeff=d.to_device(v, torch.float64).reshape(-1).contiguous())
    comp.check()
    want = a * 0.25 + dt * ref
    assert rel_l2(res.double().cpu().numpy()[0], want) <= 2 * eps
    assert rel_l2(out.double().cpu().numpy()[0], u + b * want) <= 2 * eps
