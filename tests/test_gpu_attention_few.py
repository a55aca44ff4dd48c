"""Decode attention at the edges of its tiles (16 keys a warp, 128 a pass, 512 a CTA, splits of 256 beyond; splits of 128 with more
rows or in longer caches), against softmax attention in 64 bits, and with infinite values."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 15, 16, 17, 127, 128, 129, 255, 256, 257, 383, 384, 511, 512, 513, 640, 767, 768, 769, 1000, 1023, 1024]


@pytest.fixture(scope="module", params=[1024, 1088])
def eng(nano_model, request):
    from vui_b200 import Engine

    return Engine(model=nano_model, max_rows=64, max_seq=request.param)


def _reference(eng, layer, q, slots, pos):
    kc, vc = eng.flash_kv_caches[layer].k_cache.double(), eng.flash_kv_caches[layer].v_cache.double()
    out = []
    for r in range(q.shape[0]):
        n = int(pos[r]) + 1
        k, v = (c[int(slots[r]), :n].repeat_interleave(2, 1) for c in (kc, vc))
        p = (torch.einsum("hd,nhd->hn", q[r].double().view(16, 64), k) / 8).softmax(-1)
        out.append(torch.einsum("hn,nhd->hd", p, v).reshape(-1))
    return torch.stack(out)


@pytest.mark.parametrize("rows", [1, 18, 45])
def test_attention_at_tile_edges(eng, rows):
    g = torch.Generator(device="cuda").manual_seed(rows)
    layer = 1
    eng.flash_kv_caches[layer].k_cache.normal_(generator=g)
    eng.flash_kv_caches[layer].v_cache.normal_(generator=g)
    for first in ([0, 7, 13] if rows == 1 else [0]):
        pos = torch.tensor([LENGTHS[(first + i) % len(LENGTHS)] - 1 for i in range(rows)], dtype=torch.int32)
        slots = torch.tensor([(5 * i) % 64 for i in range(rows)], dtype=torch.int32)
        q = torch.randn(rows, 1024, device="cuda", generator=g).to(torch.bfloat16)
        out = eng._attention(layer, q, slots, pos)
        assert torch.equal(out, eng._attention(layer, q, slots, pos))
        ref = _reference(eng, layer, q, slots, pos)
        # one rounding to bf16 (half a unit in the last of 8 digits: 2^-8 of the value), and fp32 sums of at most 1024 terms of up to 5 (1024 ulps of 2^-24, far from all in one direction)
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()
        eng.check_device()


@pytest.mark.parametrize("rows", [3, 45])
def test_infinite_values_stay_infinite(eng, rows):
    layer, n = 2, 300
    kc, vc = eng.flash_kv_caches[layer].k_cache, eng.flash_kv_caches[layer].v_cache
    kc.fill_(0.5)
    vc.fill_(1.0)
    vc[:, 17, :, 3] = float("inf")
    vc[:, n:] = float("nan")   # behind the context: never looked at
    q = torch.ones(rows, 1024, device="cuda", dtype=torch.bfloat16)
    out = eng._attention(layer, q, torch.zeros(rows, dtype=torch.int32), torch.full((rows,), n - 1, dtype=torch.int32)).view(rows, 16, 64)
    assert (out[:, :, 3] == float("inf")).all()
    out[:, :, 3] = 1.0
    assert (out == 1.0).all()


@pytest.mark.parametrize("rows", [1, 5, 18])
@pytest.mark.parametrize("moved", ["not", "position", "slot", "wildly"])
def test_keys_requested_before_the_place_is_final(eng, rows, moved):
    """As a step asks for them: where the table changes behind the early look (or does not), the result is that of the final place."""
    import ctypes as C

    g = torch.Generator(device="cuda").manual_seed(rows)
    layer = 3
    eng.flash_kv_caches[layer].k_cache.normal_(generator=g)
    eng.flash_kv_caches[layer].v_cache.normal_(generator=g)
    q = torch.randn(rows, 1024, device="cuda", generator=g).to(torch.bfloat16)
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    for first in range(0, len(LENGTHS), rows):
        pos = torch.tensor([LENGTHS[(first + i) % len(LENGTHS)] - 1 for i in range(rows)], dtype=torch.int32, device="cuda")
        slots = torch.tensor([(5 * i) % 64 for i in range(rows)], dtype=torch.int32, device="cuda")
        old_pos = {"position": (pos - 1).clamp(min=0), "wildly": (pos * 7919) % 3000 - 900}.get(moved, pos).to(torch.int32)
        old_slots = {"slot": (slots + 1) % 64, "wildly": slots - 40}.get(moved, slots).to(torch.int32)
        out = torch.empty_like(q)
        eng._ck(eng._lib.vuib_debug_attention_moved(eng._handle, layer, rows, P(q), P(old_slots), P(old_pos), P(slots), P(pos), P(out), eng._stream))
        assert torch.equal(out, eng._attention(layer, q, slots, pos))
    eng.check_device()
