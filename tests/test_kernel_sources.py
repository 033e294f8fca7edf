"""What the kernels' sources must keep to, where a run would not show a breach (or only by chance)."""
import os
import re

import pytest

from serve_b200.kernels.build import CSRC

SOURCES = {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def _function(text, at):
    """(name, what stands between its opening brace and ``at``) of the function that holds position ``at``."""
    start = max(re.finditer(r"^__device__ __forceinline__ \w+ (\w+)\([^;]*?\{", text[:at], re.M | re.S), key=lambda m: m.end())
    assert text.find("\n}", start.end()) > at or text.find("}\n", start.end()) > at, "an instruction outside a function of its own"
    return start.group(1), text[start.end():at]


TENSOR_MEMORY = [f for f, s in SOURCES.items() if "tcgen05." in s]


@pytest.mark.parametrize("name", TENSOR_MEMORY)
def test_a_warp_meets_before_its_tensor_memory_instructions(name):
    """tcgen05.ld, .st, the wait for stores and barriers are ``.aligned``: all lanes execute them together. Branches that rows beyond the last
    and lanes that wait alone take stand before them, so the functions that issue them begin with the warp's meeting. Those named _met do
    not: before their calls no lane has gone its own way since the warp met last."""
    text = SOURCES[name]
    found = list(re.finditer(r'"(\{\\n .reg .pred p, q;\\n setp[^;]*;\\n )?(tcgen05\.(ld|st|wait::st)\.sync\.aligned|bar\.(sync|red))', text))
    assert found or name not in ("tcgen05_ops.cuh", "attention_tc.cu")
    for m in found:
        function, before = _function(text, m.start())
        assert "__syncwarp();" in before or function.endswith("_met"), function
    for m in re.finditer(r"(?<!void )\b\w+_met\(", text):
        line = text[text.rfind("\n", 0, m.start()) + 1:m.start()]
        if "__forceinline__" in line or "__syncwarp();\n" in text[m.start() - 60:m.start()]:
            continue                                        # (one that hands on to another, or a meeting and such a call)
        met = max(text.rfind(s, 0, m.start()) for s in ("__syncwarp();", "pair_any(", "tc::load32(", "tc_store32("))
        between = text[met + 1:m.start()]
        assert met > 0 and not re.search(r"mbar_|if \(lane|row_ok|\breturn\b", between), between


@pytest.mark.parametrize("name", TENSOR_MEMORY)
def test_lanes_that_load_from_tensor_memory_give_up_together(name):
    """A lane that left such a loop by itself would not come to the next meeting: only single-lane loops may leave on one lane's wait."""
    text = SOURCES[name]
    for m in re.finditer(r"if \(!(tc::)?mbar_wait\([^\n]*(break|failed)", text):
        block = text[:m.start()]
        single = max(block.rfind("if (lane == 0) {"), block.rfind("if (lane == 0 && "))
        assert single > block.rfind("} else {\n"), text[m.start():m.end()]


# file -> what is read with __ldg: weights, which no kernel of a step writes
WEIGHTS = {"projection_ops.cu": ["reinterpret_cast<const uint32_t*>(wr"], "decode_stack.cu": ["reinterpret_cast<const float4*>(weight)", "reinterpret_cast<const uint2*>(weight)"],
           "talking_attention.cu": ["a)", "a +", "ta +", "tb +"]}
EARLY_EXPERTS = ["moe_route_kernel", "moe_route_bias_kernel", "moe_sort_kernel", "moe_combine_rows_kernel", "moe_gather_kernel"]


def test_only_weights_are_read_as_unchanging():
    """A kernel that begins before its predecessors have ended must not tell the compiler that nobody writes what they leave it."""
    for name, text in SOURCES.items():
        for m in re.finditer(r"__ldg\(([^\n]*)", text):
            assert any(m.group(1).startswith(w) for w in WEIGHTS.get(name, [])), (name, m.group(0))
    for kernel in EARLY_EXPERTS:
        text = SOURCES["experts_tcgen05.cu" if kernel == "moe_gather_kernel" else "routed_experts.cu"]
        signature = re.search(r"__global__ void [^;{]*?\b" + kernel + r"\([^{]*\{", text).group(0)
        assert "__restrict__" not in signature and "pdl_wait();" in text[text.index(signature):][:1200], kernel
