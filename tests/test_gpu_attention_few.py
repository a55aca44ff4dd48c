"""Decode attention at the edges of its tiles (4 keys a step of a warp, splits of 128; for few rows in caches of up to 1024 positions four
splits a CTA, else one), against softmax attention in 64 bits and against itself with other rows, and with infinite values."""
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
@pytest.mark.parametrize("moved", ["not", "on", "back", "slot", "wildly"])
def test_keys_requested_before_the_place_is_final(eng, rows, moved):
    """As a step asks for them: where the table changes behind the early look (or does not), the result is that of the final place, with
    the row's own key as the preceding kernel wrote it, also where the early look has seen what was there before (back)."""
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
        old_pos = {"on": (pos - 1).clamp(min=0), "back": (pos + 40).clamp(max=1023), "wildly": (pos * 7919) % 3000 - 900}.get(moved, pos).to(torch.int32)
        old_slots = {"slot": (slots + 1) % 64, "wildly": slots - 40}.get(moved, slots).to(torch.int32)
        out = torch.empty_like(q)
        own = torch.randn(2, rows, 512, device="cuda", generator=g).to(torch.bfloat16)
        own[0] = q.view(rows, 8, 2, 64)[:, :, 0].reshape(rows, 512)   # a key that weighs: the head's own query
        eng._ck(eng._lib.vuib_debug_attention_moved(eng._handle, layer, rows, P(q), P(old_slots), P(old_pos), P(slots), P(pos), P(own[0]), P(own[1]),
                                                    P(out), eng._stream))
        assert torch.equal(out, eng._attention(layer, q, slots, pos))
        ref = _reference(eng, layer, q, slots, pos)
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()   # as above
    eng.check_device()


def test_a_rows_bits_are_its_own(nano_model):
    """Whatever kernel the number of rows or the size of the cache leads to: a row alone, among few, among many, in a longer cache."""
    from vui_b200 import Engine

    layer, outs = 0, []
    for max_seq in (1024, 1088):
        eng = Engine(model=nano_model, max_rows=64, max_seq=max_seq)
        g = torch.Generator(device="cuda").manual_seed(7)
        for c in (eng.flash_kv_caches[layer].k_cache, eng.flash_kv_caches[layer].v_cache):
            c[:, :1024] = torch.randn(65, 1024, 8, 64, device="cuda", generator=g)
        q = torch.randn(46, 1024, device="cuda", generator=g).to(torch.bfloat16)
        pos = torch.tensor([LENGTHS[i % len(LENGTHS)] - 1 for i in range(46)], dtype=torch.int32)
        slots = torch.arange(46, dtype=torch.int32) % 23
        outs.append(eng._attention(layer, q, slots, pos))
        for first, n in [(i, 1) for i in range(23)] + [(0, 5), (18, 5), (0, 18), (5, 18), (0, 19), (20, 24)]:
            part = slice(first, first + n)
            assert torch.equal(eng._attention(layer, q[part], slots[part], pos[part]), outs[0][part]), (max_seq, first, n)
    assert torch.equal(*outs)


def test_a_streams_step_does_not_depend_on_the_others(nano_model):
    """The backbone's step from five rows on, bit for bit: few and many rows, caches on either side of the rule."""
    from vui_b200 import Engine

    seen = {}
    for max_seq in (1024, 1088):
        eng = Engine(model=nano_model, max_rows=33, max_seq=max_seq)
        g = torch.Generator(device="cuda").manual_seed(8)
        eng._kv[:, :, :, :1024] = torch.randn(eng._kv[:, :, :, :1024].shape, device="cuda", generator=g, dtype=torch.bfloat16) * 0.5
        codes = torch.randint(0, 2048, (33, 16), generator=torch.Generator().manual_seed(8)).cuda()
        lens = torch.tensor([(37 * i + 3) % 700 for i in range(33)], dtype=torch.int32, device="cuda")
        eng._g_slot_idx[:] = torch.arange(33, dtype=torch.int32, device="cuda")
        eng._g_seq_inc.fill_(1)
        for B in (33, 19, 18, 5):
            eng.seq_lens[:33] = lens
            eng._g_codes_in.copy_(codes)
            eng._apply_cfg(None, greedy=True)
            eng._frame_call(B)
            got = (eng._g_hidden_out[:B].clone(), torch.stack([eng._kv[:, :, b, int(lens[b])] for b in range(B)]))
            for a, b in zip(got, seen.setdefault("first", got)):
                assert torch.equal(a, b[:B]), (max_seq, B)
        eng.check_device()
