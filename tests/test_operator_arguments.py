"""CompiledOperator hands raw pointers to the native library: what does not fit
is refused before the call.  On the CPU, with a stand-in for the library."""
import ctypes as C
from types import SimpleNamespace

import pytest
import torch

from hedge_b200.discretization import CompiledOperator
from hedge_b200.models import MODEL_VARWAVE

N, F = 12, 3


class _Discr(SimpleNamespace):
    def __len__(self):
        return N


class _Library:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *args: self.calls.append((name, args)) or 0


def _operator(**kw):
    op = CompiledOperator.__new__(CompiledOperator)
    op.__dict__.update(discr=_Discr(device=torch.device("cpu"), dimensions=2), F=F, n_given=0,
                       ot=SimpleNamespace(model=MODEL_VARWAVE), var_material=False, _n_e=0,
                       _coeff=torch.ones(N, dtype=torch.float64), _source=None, _handle=None,
                       _lib=_Library(), _stream=lambda: 0,
                       _adj_work=torch.empty(4, dtype=torch.float64))
    op.__dict__.update(kw)
    return op


def _vec(*shape, dtype=torch.float64):
    return torch.ones(shape, dtype=dtype)


def _doubles(n):
    return (C.c_double * n)(*range(n))


def test_step_takes_a_complete_stage_list():
    op = _operator()
    op.lsrk_step(_doubles(2), _doubles(2), 0.1, [_vec(F, N) for _ in range(3)], _vec(F, N),
                 source=_vec(2, N), source_stride=N)
    assert [c[0] for c in op._lib.calls] == ["hb_lsrk_step"]


@pytest.mark.parametrize("a,b,buffers,kw", [
    (2, 2, 2, {}), (2, 1, 3, {}), (1, 2, 3, {}),
    (2, 2, 3, dict(source=_vec(N + 1), source_stride=N)),
    (2, 2, 3, dict(source=_vec(2, N, dtype=torch.float32), source_stride=N)),
    (2, 2, 3, dict(source=_vec(N, 2).T, source_stride=N)),
    (2, 2, 3, dict(source=_vec(2, N), source_stride=-N)),
])
def test_step_refuses(a, b, buffers, kw):
    op = _operator()
    with pytest.raises(ValueError):
        op.lsrk_step(_doubles(a), _doubles(b), 0.1, [_vec(F, N) for _ in range(buffers)],
                     _vec(F, N), **kw)
    assert not op._lib.calls


def test_step_refuses_other_coefficient_types():
    op = _operator()
    with pytest.raises(ValueError):
        op.lsrk_step((C.c_float * 2)(), _doubles(2), 0.1, [_vec(F, N) for _ in range(3)],
                     _vec(F, N))
    assert not op._lib.calls


def test_step_refuses_stage_sources_with_variable_material():
    # the material divides a source before the kernel sees it
    op = _operator(var_material=True, _n_e=3, _coeff=_vec(2 * N))
    with pytest.raises(ValueError):
        op.lsrk_step(_doubles(2), _doubles(2), 0.1, [_vec(F, N) for _ in range(3)], _vec(F, N),
                     source=_vec(2, 3 * N), source_stride=3 * N)
    assert not op._lib.calls


def test_adjoint_stage_takes_device_vectors():
    op = _operator()
    q = _vec(F, N, dtype=torch.float32)          # converted, as adjoint() does
    op.adjoint_stage(0.1, 0.2, 0.3, _vec(F, N), _vec(F * N), q=q, c_bar=_vec(N))
    (name, args), = op._lib.calls
    assert name == "hb_adjoint_stage" and args[4] not in (None, q.data_ptr())


def test_adjoint_step_takes_the_stages_last_first():
    op = _operator()
    op.adjoint_step((0.1, 0.2), (0.3, 0.4), 0.5, _vec(F, N), _vec(F, N), (_vec(F, N), None))
    assert [(c[1][1], c[1][2]) for c in op._lib.calls] == [(0.2, 0.4), (0.1, 0.3)]
    assert op._lib.calls[0][1][4] is None and op._lib.calls[1][1][4] is not None


@pytest.mark.parametrize("bad", [_vec(F, N, dtype=torch.float32), _vec(F, N - 1), _vec(N, F).T,
                                 _vec(F, 2 * N)[:, ::2], torch.ones(1, 1).double().expand(F, N)])
@pytest.mark.parametrize("which", ["lam", "lq"])
def test_adjoint_stage_refuses_vectors(which, bad):
    op = _operator()
    x = dict(lam=_vec(F, N), lq=_vec(F, N), q=_vec(F, N))
    x[which] = bad
    with pytest.raises(ValueError):
        op.adjoint_stage(0.1, 0.2, 0.3, **x)
    assert not op._lib.calls


@pytest.mark.parametrize("which", ["c_bar", "coeff"])
@pytest.mark.parametrize("bad", [_vec(N, dtype=torch.float32), _vec(N - 1), _vec(2 * N)[::2]])
def test_adjoint_stage_refuses_coefficients(which, bad):
    op = _operator()
    with pytest.raises(ValueError):
        op.adjoint_stage(0.1, 0.2, 0.3, _vec(F, N), _vec(F, N), q=_vec(F, N), **{which: bad})
    assert not op._lib.calls


def test_adjoint_stage_refuses_a_short_state():
    op = _operator()
    with pytest.raises(RuntimeError):
        op.adjoint_stage(0.1, 0.2, 0.3, _vec(F, N), _vec(F, N), q=_vec(F, N - 1))
    assert not op._lib.calls
