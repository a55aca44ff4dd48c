"""A CTA may touch a peer's shared memory only once every CTA of its cluster is known to run.  A kernel that does it too early can fault,
so the order is checked in the sources: in the body of every kernel the first store to a peer comes behind a cluster barrier."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vui_b200", "csrc")
# what stores to a peer: the instructions, and the device functions that issue them
REMOTE = re.compile(r"st\.shared::cluster|st\.async|\bpush_f32\w*\(|\bdt_push_\w+[<(]|\bdt_residual_exchange[<(]|\.send\(")
WAIT = re.compile(r"barrier\.cluster\.wait|\bcluster_wait\(\)")
ARRIVE = re.compile(r"barrier\.cluster\.arrive|\bcluster_arrive(_relaxed)?\(\)")


def kernels():
    """(file, name, body) of every kernel, comments left out."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
        for m in re.finditer(r"__global__", src):
            name = re.search(r"\b(k_\w+)\s*\(", src[m.start():])
            at = src.index("{", src.index(")", m.start() + name.end()))
            depth, end = 0, at
            for end in range(at, len(src)):
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                if depth == 0:
                    break
            yield os.path.basename(path), name.group(1), src[at:end]


CLUSTERED = [k for k in kernels() if REMOTE.search(k[2])]


def test_the_cluster_kernels_are_found():
    assert {k[1] for k in CLUSTERED} == {"k_ervq", "k_sg", "k_gemm_tc", "k_depth_tc", "k_attn_block", "k_mlp_block", "k_attn_rows", "k_mlp_rows"}


@pytest.mark.parametrize("file,name,body", CLUSTERED, ids=[k[1] for k in CLUSTERED])
def test_no_store_to_a_peer_before_the_cluster_has_met(file, name, body):
    first, met = REMOTE.search(body), WAIT.search(body)
    assert met and met.start() < first.start(), f"{file}: {name} stores to a peer before it has waited for the cluster"
    assert ARRIVE.search(body).start() < met.start()


def test_a_wait_is_not_given_up_while_peers_are_sending():
    """The host lets no cluster kernel wait for less than 2^18 polls, and no bound overflow when a kernel multiplies it."""
    src = open(os.path.join(CSRC, "vuib200.cu")).read()
    for args in ("aa", "ma", "a"):
        for m in re.finditer(rf"\b{args}\.spin_limit = ([^;]+);", src):
            assert m.group(1) == "cluster_limit(e)"
    assert re.search(r"cluster_limit\(const VuibEngine\* e\) \{ return e->spin_limit > 1u << 18 \? e->spin_limit : 1u << 18; \}", src)
    assert "e->spin_limit = polls < 1u << 26 ? polls : 1u << 26;" in src
    factors = [int(f) for name in sorted(glob.glob(os.path.join(CSRC, "*.cuh"))) for f in re.findall(r"\b(\d+)u? \* a\.spin_limit", open(name).read())]
    assert factors and max(factors) * 2 ** 26 < 2 ** 32


def test_the_quantisers_winners_have_two_buffers():
    """Between a thread's reads of a codebook's winners and the next codebook's writes stands no barrier of the CTA: the wait in between is
    for the peers' answers to this CTA, and the reading thread may be answering another.  So the codebooks take turns."""
    body = next(k[2] for k in CLUSTERED if k[1] == "k_ervq")
    assert re.search(r"\bwon\[2\]\[RV_WARPS\]\[F\];", body)
    uses = re.findall(r"\bwon\[(\w+)\]", body)
    assert uses.pop(0) == "2" and len(uses) >= 2 and set(uses) == {"buf"} and "const int buf = cb & 1;" in body
