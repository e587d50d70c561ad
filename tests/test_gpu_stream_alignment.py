"""The streamed-operator split kernel on vectors at every 8-byte alignment (its
state loads are 32 and its update accesses 16 bytes wide where the addresses
allow): bit for bit what it gives on aligned ones.  And its 12- and 16-warp
builds on partitions: parts of more than one batch, with halo faces and a
ragged last batch, against the oracle."""
import numpy as np
import pytest

import hedge_b200 as hb
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _model(kind):
    return hb.MaxwellOperator(1.0, 1.0, flux_type=1) if kind == "maxwell" else \
        hb.StrongWaveOperator(1.0, 3, flux_type="upwind")


def _at(x, doubles):
    """A copy of x that many doubles behind a 256-byte boundary."""
    import torch
    buf = torch.empty(x.numel() + 32 + doubles, dtype=x.dtype, device=x.device)
    start = (-buf.data_ptr() // 8) % 32 + doubles
    out = buf[start:start + x.numel()].view(x.shape)
    assert out.data_ptr() % 256 == 8 * doubles
    return out.copy_(x)


@pytest.mark.parametrize("precision", ["fp16x3", "bf16x3"])
@pytest.mark.parametrize("kind,order", [("maxwell", 5), ("wave", 5), ("wave", 6), ("wave", 7),
                                        ("maxwell", 6)])
def test_alignments(cuda_device, kind, order, precision):
    import torch
    d = hb.Discretization(hb.make_box_tet_mesh(n=(2, 2, 3), jitter=0.03, seed=2), order=order,
                          precision=precision)
    comp = _model(kind).bind(d).compiled
    rng = np.random.default_rng(1)
    q = d.to_device(rng.uniform(-1, 1, (comp.F, len(d))))
    r = d.to_device(rng.uniform(-1, 1, (comp.F, len(d))))

    def stage(iq, io, ir):
        x, out, res = _at(q, iq), _at(torch.zeros_like(q), io), _at(r, ir)
        comp.lsrk_stage(-0.6, 0.4, 1e-3, x, out, res)
        rhs = _at(torch.zeros_like(q), io)
        comp.rhs_into(x, rhs)
        comp.check()
        return out, res, rhs
    want = stage(0, 0, 0)
    assert all(bool(torch.isfinite(x).all()) for x in want)
    for offsets in ((1, 0, 0), (2, 0, 0), (3, 2, 1), (0, 1, 0), (0, 0, 1), (2, 2, 2), (1, 1, 1)):
        for a, b in zip(want, stage(*offsets)):
            assert torch.equal(a, b), offsets


@pytest.mark.parametrize("precision", ["fp16x3", "bf16x3"])
@pytest.mark.parametrize("kind,order", [("maxwell", 5), ("wave", 6), ("wave", 7)])
def test_partitioned_wide_builds(cuda_device, kind, order, precision):
    import ctypes as C
    from oracle import OracleRHS
    from hedge_b200.partition import LocalExchange, PartitionPlan, PartitionedOperator
    from test_gpu_parity import _fields
    d = hb.Discretization(hb.make_box_tet_mesh(n=(3, 3, 3), jitter=0.03, seed=5), order=order)
    model = _model(kind)
    F = 6 if kind == "maxwell" else 4
    plan = PartitionPlan(d, model.op_template(), 3)
    parts = [PartitionedOperator(d, model, plan, r, precision=precision) for r in range(3)]
    ex = LocalExchange(plan, parts)
    q = _fields(d, F, 12)
    ref = OracleRHS(d, model.op_template())(q).reshape(F, -1)
    ql = [p.scatter(q) for p in parts]
    for p, x in zip(parts, ql):
        p.pack(x)
    ex.exchange_all()
    for p, x in zip(parts, ql):
        info = (C.c_int64 * 6)()
        p.lib.hb_op_launch_info(p._h, info, 6)
        assert p.part.n_halo_faces > 0 and info[1] == (384 if order == 6 else 512)
        for by_ranges in (False, True):
            got = p.rhs(x, exchanged=True, by_ranges=by_ranges)
            p.check()
            assert rel_l2(got.double().cpu().numpy(), ref[:, p.local_nodes()]) <= \
                (1e-6 if precision == "fp16x3" else 1e-5)
