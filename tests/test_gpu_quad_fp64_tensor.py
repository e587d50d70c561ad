"""The quadrature kernel on the FP64 tensor cores (quad_fp64.cu) at every
number of node tiles it is built for, beyond them (order 8 in 2D: the
CUDA-core kernel), and on meshes that end within a warp's 8 elements, against
the template executor.  FP64: 1e-12 relative L2, the bound of a right-hand
side (the rules of high degree have weights of both signs; the executor sums
the same terms)."""
import numpy as np
import pytest

import hedge_b200 as hb
from conftest import rel_l2
from test_quadrature import state, velocity

pytestmark = pytest.mark.gpu


def _check(dim, order, n, m, degree, flux):
    from optemplate_exec import TemplateExecutor
    mesh = hb.make_regular_rect_mesh((-1, -1), (1, 1), (n + 1, m + 1), jitter=0.1 / n, seed=2) \
        if dim == 2 else hb.make_box_tet_mesh(n=(n, n, m), jitter=0.1 / n, seed=2)
    d = hb.Discretization(mesh, order=order, quad_min_degrees={"quad": degree})
    op = hb.VariableCoefficientAdvectionOperator(dim, None, bc_u_f=1, flux_type=flux)
    tpl = op.op_template()
    env = {"u": state(d, 3), "v": velocity(d),
           "bc_u": np.sin(3 * d.get_boundary(hb.TAG_ALL).nodes[:, 0])}
    ref = TemplateExecutor(d)(tpl, **env)[0]
    comp = d.compile(tpl)
    got = comp(**env).cpu().numpy()
    comp.check()
    assert rel_l2(got, ref) <= 1e-12


@pytest.mark.parametrize("dim,order", [(2, o) for o in range(1, 9)] + [(3, o) for o in (1, 2, 3, 4)])
def test_every_order(cuda_device, dim, order):
    _check(dim, order, 3 if dim == 2 else 1, 5 if dim == 2 else 2, 2 * order + 1, "upwind")


@pytest.mark.parametrize("n,m", [(1, 1), (2, 2), (3, 3), (40, 37)])
@pytest.mark.parametrize("flux", ["central", "lf"])
def test_mesh_sizes(cuda_device, n, m, flux):
    _check(2, 2, n, m, 6, flux)
