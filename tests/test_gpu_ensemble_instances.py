"""The ensemble kernel's two builds, for batches mostly of orders 1 to 7 and
mostly beyond: members of every order step bit for bit alike in both (the same
arithmetic with compile-time and run-time sizes)."""
import numpy as np
import pytest

import hedge_b200 as hb

pytestmark = pytest.mark.gpu


def test_builds_agree(cuda_device):
    import torch
    from hedge_b200.ensemble import Ensemble, Member

    def members(orders, n=6):
        out = []
        for order in orders:
            mesh = hb.make_regular_rect_mesh((-1, -1), (1, 1), (4 + order, n), jitter=0.05 / n,
                                             seed=order, periodicity=(True, True))
            d = hb.Discretization(mesh, order=order)
            x = d.nodes
            for m in (hb.StrongAdvectionOperator(np.array([0.8, -0.4]), flux_type="upwind"),
                      hb.StrongWaveOperator(0.9, 2)):
                F = 1 if isinstance(m, hb.StrongAdvectionOperator) else 3
                out.append(Member(d, m, np.stack([np.sin((f + 1) * x[:, 0] + f) * np.cos(x[:, 1])
                                                  for f in range(F)])))
        return out
    states = []
    for extra in ([], members([8]), members([9], 80)):
        ens = Ensemble(members(range(1, 8)) + extra)
        ens.step(2)
        ens.check()
        states.append([ens.state(k) for k in range(14)])
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert bool(torch.isfinite(a).all()) and torch.equal(a, b)
