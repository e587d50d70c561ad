"""ReceiverTraces with receivers of the user's own: what ``transpose`` returns
(a buffer that it keeps, a strided, expanded or FP32 tensor) is read, never
updated in place, and FP32 states give gradients too.  On the CPU with a
stand-in for the compiled operator that checks what the kernels would be
given; on the GPU against the built-in receivers."""
import numpy as np
import pytest
import torch

import hedge_b200 as hb
from hedge_b200 import adjoint

F, N = 2, 6


class _Linear:
    """dq/dt = -q: as_state, stages and their adjoint on CPU tensors."""
    var_material = False

    def __init__(self, dtype):
        self.dtype = dtype

    def as_state(self, q):
        return q.to(self.dtype).reshape(F, N).contiguous()

    def lsrk_step(self, a, b, dt, bufs, res, coeff=None):
        for s in range(len(a)):
            assert bufs[s].dtype == self.dtype and bufs[s].is_contiguous()
            res.mul_(a[s]).sub_(bufs[s], alpha=dt)
            bufs[s + 1].copy_(bufs[s]).add_(res, alpha=b[s])

    def adjoint_step(self, a, b, dt, lam, lq, states, coeff=None, c_bar=None):
        for x in (lam, lq):
            assert x.dtype == torch.float64 and x.is_contiguous() and x.shape == (F, N)
        for s in reversed(range(len(states))):
            lam.add_(lq, alpha=b[s])
            lq.sub_(lam, alpha=dt)
            lam.mul_(a[s])


class _Plain:
    """Every value of the state's first field is a trace."""

    def __call__(self, q):
        return q[0].clone()

    def transpose(self, g, like):
        out = torch.zeros(like.shape, dtype=torch.float64, device=like.device)
        out[0] = g
        return out


class _Kept(_Plain):
    def __init__(self):
        self.kept = []

    def transpose(self, g, like):
        x = super().transpose(g, like)
        self.kept.append((x, x.clone()))
        return x


class _Strided(_Plain):
    def transpose(self, g, like):
        out = super().transpose(g, like)
        return out.T.contiguous().T


class _Single(_Plain):
    def transpose(self, g, like):
        return super().transpose(g, like).float()


def _gradient(comp, receivers, q0, dt=0.125, steps=4):
    q0 = q0.clone().requires_grad_(True)
    traces = adjoint.ReceiverTraces.apply(q0, None, comp, receivers, dt, steps, None, 2)
    (traces.double() ** 2).sum().backward()
    return q0.grad.double()


@pytest.mark.parametrize("kind", [_Kept, _Strided, _Single])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_transpose_is_only_read(kind, dtype):
    q0 = torch.linspace(-1, 1, F * N, dtype=torch.float64).reshape(F, N)
    want = _gradient(_Linear(torch.float64), _Plain(), q0)
    rec = kind()
    got = _gradient(_Linear(dtype), rec, q0)
    # traces and cotangents of one or the other are rounded to FP32
    assert torch.allclose(got, want, rtol=0,
                          atol=1e-14 if dtype == torch.float64 and kind is not _Single else 1e-5)
    if kind is _Kept:
        assert all(torch.equal(a, b) for a, b in rec.kept)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_own_receivers(cuda_device, precision):
    m = hb.make_regular_rect_mesh((-1, -1), (1, 1), (6, 6), jitter=0.03, seed=1)
    grads = []
    for prec, kind in (("fp64", None), (precision, "kept"), (precision, "strided")):
        d = hb.Discretization(m, order=3, precision=prec)
        comp = hb.StrongWaveOperator(1.0, 2).bind(d).compiled
        rec = base = adjoint.Receivers(d, [(0.1, 0.2), (-0.4, 0.3)])
        if kind:
            buffers = []

            def transpose(g, like, base=base, kind=kind, buffers=buffers):
                x = base.transpose(g, like.double())
                x = x.T.contiguous().T if kind == "strided" else x
                buffers.append((x, x.clone()))
                return x
            rec = type("Own", (), {"__call__": lambda self, q: base(q),
                                   "transpose": staticmethod(transpose)})()
        q0 = d.to_device(np.random.default_rng(5).uniform(-1, 1, (3, len(d))))
        q0 = q0.double().requires_grad_(True)
        tr = adjoint.ReceiverTraces.apply(q0, None, comp, rec, 0.01, 5, None, 2)
        adjoint.trace_loss(tr.double()).backward()
        comp.check()
        grads.append(q0.grad)
        if kind:
            assert all(torch.equal(a, b) for a, b in buffers)
    for g in grads[1:]:
        err = float((g - grads[0]).norm() / grads[0].norm())
        # FP32: 25 stages of rounding at 6e-8, the trace differences carried over
        assert err <= (1e-13 if precision == "fp64" else 1e-5), err
