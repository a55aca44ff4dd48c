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


def test_early_requests_are_coherent():
    """The preceding kernel may be writing what a stale place leads to, and the second look must see it: no read-only loads."""
    for name, kernel in (("decode_kernels.cuh", "k_attn_wide("), ("fused_blocks.cuh", "k_attn_block("), ("fused_rows.cuh", "k_attn_rows(")):
        src = _source(name)
        body = src[src.index("{", src.index(kernel)):]
        body = body[: body.index("\n}")]
        assert "ld_l2" in body[: body.index("pdl_wait()")] and not re.search(r"ldg_stream|\.nc\b|__ldg\([^)]*(?:kb|vb|k_cache|v_cache)", body)
    src = _source("decode_kernels.cuh")
    for load in ("uint4 ld_l2(", "void ld_l2_if("):
        body = src[src.index(load):]
        assert "ld.global.cg.v4" in body[: body.index("\n}")]
