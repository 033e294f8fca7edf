"""What the kernels' sources must keep to, where a run would not show a breach (or only by chance)."""
import os
import re

import pytest

from serve_b200.kernels.build import CSRC

SOURCES = {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def _body_before(text, at):
    """What stands between the opening brace of the function that holds position ``at`` and that position."""
    start = max(m.end() for m in re.finditer(r"^__device__ __forceinline__ [^;]*?\{", text[:at], re.M | re.S))
    assert text.find("\n}", start) > at, "an instruction outside a function of its own"
    return text[start:at]


@pytest.mark.parametrize("name", [f for f, s in SOURCES.items() if "tcgen05.ld" in s])
def test_a_warp_meets_before_its_tensor_memory_instructions(name):
    """tcgen05.ld, .st, the wait for stores and barriers are ``.aligned``: all lanes execute them together. Branches that rows beyond the last
    and lanes that wait alone take stand before them, so the functions that issue them begin with the warp's meeting."""
    text = SOURCES[name]
    found = list(re.finditer(r'"(\{\\n .reg .pred p, q;\\n setp[^;]*;\\n )?(tcgen05\.(ld|st|wait::st)\.sync\.aligned|bar\.(sync|red))', text))
    assert found
    for m in found:
        assert "__syncwarp();" in _body_before(text, m.start()), text[m.start():m.end()]


@pytest.mark.parametrize("name", [f for f, s in SOURCES.items() if "tcgen05.ld" in s])
def test_lanes_that_load_from_tensor_memory_give_up_together(name):
    """A lane that left such a loop by itself would not come to the next meeting: only single-lane loops may leave on one lane's wait."""
    text = SOURCES[name]
    for m in re.finditer(r"if \(!(tc::)?mbar_wait\([^\n]*(break|failed)", text):
        block = text[:m.start()]
        single = max(block.rfind("if (lane == 0) {"), block.rfind("if (lane == 0 && "))
        assert single > block.rfind("} else {\n"), text[m.start():m.end()]
