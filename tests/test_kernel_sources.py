"""What the kernel sources have to keep to and no run shows: with programmatic
dependent launch a kernel starts before the launch that writes its input has
ended, so a load of such data may not be moved before griddepcontrol.wait."""
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
