"""An operator may be destroyed after its discretization (as the garbage
collector does with a cycle): nothing of the discretization is read then, and
no error is left for the next launch."""
import ctypes as C
import gc

import numpy as np
import pytest

import hedge_b200 as hb

pytestmark = pytest.mark.gpu


def test_operator_outlives_its_discretization(cuda_device):
    lib = None
    for k in range(20):
        d = hb.Discretization(hb.make_regular_rect_mesh((-1, -1), (1, 1), (4, 4 + k % 3)), order=2)
        comp = hb.StrongWaveOperator(1.0, 2).bind(d).compiled
        lib = comp._lib
        op, comp._handle = comp._handle, None
        discr = d._native_handle()
        assert lib.hb_discr_destroy(discr) == 0
        d._handle = None
        del comp, d
        gc.collect()
        # memory that the discretization had goes to others
        junk = [np.full(n, 0x5A, dtype=np.uint8) for n in (64, 128, 256, 384, 512, 1024) * 20]
        assert lib.hb_op_destroy(op) == 0 and len(junk) == 120
    d = hb.Discretization(hb.make_regular_rect_mesh((-1, -1), (1, 1), (4, 4)), order=2)
    rhs = hb.StrongWaveOperator(1.0, 2).bind(d)
    out = rhs(0.0, np.ones((3, len(d))))
    rhs.compiled.check()
    assert bool((out == out).all()) and isinstance(op, C.c_void_p)
