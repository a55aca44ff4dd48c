"""Kernels that request a cache row before their dependency is met rely on an order: the steps that wrote the row have ended.  It is
given by the first kernel of a step, whose successors start only behind its own wait, and is checked in the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vui_b200", "csrc")


def _source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def test_a_step_starts_behind_all_that_came_before():
    src = _source("decode_kernels.cuh")
    body = src[src.index("{", src.index("k_embed_codes(")):]
    assert body.index("pdl_wait()") < body.index("pdl_trigger()") < body.index("__global__")


def test_early_requests_only_in_steps():
    """The step's first launch is that kernel; a prefill, whose rows may follow one another in a slot, asks for nothing early."""
    src = _source("vuib200.cu")
    step = src[src.index('extern "C" int32_t vuib_backbone_step('):]
    launches = re.findall(r"launch\((\w+)|(run_layers)\(", step[: step.index("\n}")])
    assert launches[0][0] == "k_embed_codes" and launches[1][1] == "run_layers"
    last = [m.strip() for m in re.findall(r"AttnArgs aa\{.*?,\s*([^,{}]+)\};", src, flags=re.S)]
    tables = {"!prefill": 1, "0": len(last) - 2, "1": 1}   # 1: the test hook
    assert {v: last.count(v) for v in set(last)} == tables
