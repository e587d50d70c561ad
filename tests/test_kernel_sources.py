"""What the kernel sources have to keep to and no run shows: with programmatic
dependent launch a kernel starts before the launch that writes its input has
ended, so a load of such data may not be moved before griddepcontrol.wait, nor
go through the read-only path where a buffer may be read, written and read
again by launches that overlap."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hedge_b200",
                    "csrc")


def _source(name):
    return re.sub(r"//.*", "", open(os.path.join(CSRC, name)).read())


def test_inline_loads_are_ordered():
    for name in os.listdir(CSRC):
        for m in re.finditer(r"\basm\s*(volatile)?\s*\(\s*\"([^\"]*)", _source(name)):
            if re.match(r"(ld|st|cp|red|atom|prefetch|griddepcontrol|mbarrier|tcgen05)\b", m.group(2)):
                assert m.group(1), (name, m.group(2))


def test_mutable_data_is_not_loaded_as_constant():
    # these kernels release the next launch before they wait for the previous
    # one, so three overlap.  The operator's own tables are constant; the state,
    # coefficient, source, boundary and halo values, the residual and the
    # adjoint's scratch are not
    constant = r"a\.(geo|conn|fmask|shuffle|afrag|vfrag|lfrag|nlist)\b|ap\b"
    for name in ("rhs_fp64.cuh", "face.cuh", "adjoint_fp64.cuh", "dmma.cuh"):
        for m in re.finditer(r"__ldg\(([^;]*)", _source(name)):
            assert re.match(constant, m.group(1)), (name, m.group(1))
        assert "ld.global.nc" not in _source(name), name
