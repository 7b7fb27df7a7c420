"""Kernels that are launched before the kernel ahead of them has ended (q4b_launch): each waits for it, and nothing that a
kernel ahead may have written is read with a load that the compiler may move over the wait: __ldg, the non-volatile
cache-hint intrinsics, or a `const __restrict__` pointer.  Weights and tables may be."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "suzuku-engine-q4_b200", "csrc")
CONSTANT = {"w", "W", "w4", "g4", "norm_w", "bg", "bu", "bd", "grid3", "grid2", "codes"}
# device functions that such kernels run
HELPERS = ("stream_items", "stack_body", "softmax_topk_regs", "small_group", "quant_planes", "layer_pick")


def _functions():
    """(name of the kernel or the names of the device functions, text) of everything up to a closing brace in the first
    column."""
    for path in sorted(glob.glob(os.path.join(CSRC, "q4b_*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for part in re.split(r"(?<=\n)}\n", text):
            kernel = re.findall(r"__global__(?:\s+static)?\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)", part)
            yield kernel[-1:], re.findall(r"\b(\w+)\s*\(", part) if "__device__" in part else [], part


def test_every_dependent_kernel_waits_and_reads_plainly():
    parts = list(_functions())
    launched = set()
    for _, _, text in parts:
        for args in re.findall(r"\bq4b_launch\(((?:[^(),]|\([^()]*\))+)", text):
            launched |= set(re.findall(r"\b(\w+_k)\b", args))
        launched |= set(re.findall(r"const auto k = (\w+_k)\b", text))
    launched |= {"moe_decode_stack_k", "moe_decode_session_k"}
    assert len(launched) > 25, sorted(launched)
    seen = set()
    for kernel, functions, text in parts:
        dependent = bool(kernel) and kernel[0] in launched
        if not dependent and (kernel or not set(HELPERS) & set(functions)):
            continue
        if dependent:
            seen.add(kernel[0])
            assert re.search(r"\b(q4b_pdl_wait|stream_items|stack_body)\b", text), kernel[0] + " does not wait"
            head = text[text.rindex("__global__"):]
            for arg in re.findall(r"const \w+ \*\s*__restrict__ (\w+)", head[:head.index("{")]):
                assert arg in CONSTANT, "%s: %s may be written by the kernel ahead" % (kernel[0], arg)
        for expr in re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?([\w.]+)", text):
            assert expr.split(".")[-1] in CONSTANT, "%s: __ldg of %s" % (kernel or functions[:3], expr)
        assert not re.search(r"\b__ld(cg|cs|ca|lu|cv)\(", text), kernel or functions[:3]
    assert seen == launched, launched - seen
