"""The batched ensemble kernel at the orders its element sizes are compile-time
constants for and at order 8 (run-time sizes), in 2D and 3D: one step
of every member against the CPU oracle.  The bound is the ensemble's, 1e-5
relative L2 of the step's increment (FP32 right-hand side)."""
import numpy as np
import pytest

import hedge_b200 as hb
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
def test_every_order(cuda_device, dim):
    from oracle import OracleRHS
    from hedge_b200.ensemble import Ensemble, Member
    from hedge_b200.timestep import RK4A, RK4B
    members = []
    # (3D operators of order 7 on exceed the batch's shared memory: refused)
    for order in range(1, 9 if dim == 2 else 7):
        if dim == 2:
            mesh = hb.make_regular_rect_mesh((-1, -1), (1, 1), (4 + order, 5), jitter=0.05, seed=order,
                                             periodicity=(True, True))
            models = [hb.StrongAdvectionOperator(np.array([0.8, -0.4]), flux_type="upwind"),
                      hb.StrongWaveOperator(0.9, 2)]
        else:
            mesh = hb.make_box_tet_mesh(n=(1, 1, 2), jitter=0.05, seed=order)
            models = [hb.StrongWaveOperator(0.9, 3)]
        d = hb.Discretization(mesh, order=order)
        x = d.nodes
        for m in models:
            F = 1 if isinstance(m, hb.StrongAdvectionOperator) else dim + 1
            q = np.stack([np.sin((f + 1) * x[:, 0] + f) * np.cos(x[:, -1]) for f in range(F)])
            members.append(Member(d, m, q))
    ens = Ensemble(members)
    ens.step(1)
    ens.check()
    for k, m in enumerate(members):
        q = m.q0.astype(np.float32).astype(np.float64)
        orc = OracleRHS(m.discr, m.model.op_template())
        res, y = np.zeros_like(q), q.copy()
        for a, b in zip(RK4A, RK4B):
            res = a * res + m.dt * orc(y)
            y = y + b * res
        got = ens.state(k).double().cpu().numpy()
        # the state is stored in FP32: its rounding enters the increment
        round_off = 2.0 ** -24 * np.linalg.norm(q) * 5 ** 0.5
        assert np.linalg.norm((got - q) - (y - q)) <= 1e-5 * np.linalg.norm(y - q) + round_off, \
            (k, m.discr.order, rel_l2(got - q, y - q))
