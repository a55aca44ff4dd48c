"""Decode steps of one and of several streams at the edges of the kernels' row ranges (one row, fused rows up to 4, tensor-core tiles of
16 / 32 / 64, clusters of 8 depth streams up to 120) and of their key ranges (64 keys a CTA and 512 a cluster requested in advance,
splits of 128) against the register-tile GEMV kernels, on the same caches and input codes."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


def _sure(nano_sd):
    """The seeded weights with every code following from the one before (as in a trained model): no near ties between codes."""
    sd, g = dict(nano_sd), torch.Generator().manual_seed(1)
    code, audio = (sd[n].float() / sd[n].float().std() for n in ("rq_transformer.code_emb.embedding.weight", "audio_emb.embedding.weight"))
    head = torch.empty_like(sd["rq_transformer.head_W"])
    for i in range(15):
        head[i, torch.randperm(2048, generator=g)] = code[i * 2048:(i + 1) * 2048].to(head.dtype) * 0.1
    sd["rq_transformer.head_W"] = head
    sd["codec_head.weight"] = (audio[torch.randperm(2048, generator=g)] * 0.1).to(head.dtype)
    sd["rq_transformer.code_emb.embedding.weight"], sd["audio_emb.embedding.weight"] = code.to(head.dtype), audio.to(head.dtype)
    return sd


@pytest.fixture(scope="module")
def sure_model(nano_sd):
    from vui_b200 import VuiB200, VuiShape

    return VuiB200(VuiShape(), _sure(nano_sd), device="cuda")


@pytest.fixture(scope="module")
def deep_model(nano_sd):
    """Five depth layers: more than the one-launch depth loop takes, so that each layer runs as kernels of its own."""
    from vui_b200 import VuiB200, VuiShape

    sd = _sure(nano_sd)
    for name in list(sd):
        if name.startswith("rq_transformer.blocks.0."):
            sd[name.replace("blocks.0.", "blocks.4.")] = sd[name].flip(0).contiguous()
    return VuiB200(VuiShape(n_layers=2, rq_n_layers=5), {k: v for k, v in sd.items()}, device="cuda")


LENGTHS = [0, 1, 63, 64, 511, 513, 600, 97]


@pytest.mark.parametrize("B", [1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 65, 120, 121, 241])
def test_decode_step_matches_gemv_kernels(sure_model, B):
    _check_step(sure_model, B, [LENGTHS[i % 8] for i in range(B)], 640)


@pytest.mark.parametrize("B,first", [(1, n) for n in range(1, 8)] + [(2, 4), (2, 6), (3, 4), (4, 2), (4, 4)])
def test_few_streams_at_every_length(sure_model, B, first):
    _check_step(sure_model, B, [LENGTHS[(first + i) % 8] for i in range(B)], 640)


@pytest.mark.parametrize("B", [1, 2, 3, 4, 6, 17])
def test_long_contexts(sure_model, B):
    _check_step(sure_model, B, [[2047, 1024, 513, 1537, 2000, 640][i % 6] for i in range(B)], 2048)


@pytest.mark.parametrize("B", [5, 16, 33])
def test_depth_layers_as_kernels_of_their_own(deep_model, B):
    _check_step(deep_model, B, [LENGTHS[i % 8] for i in range(B)], 640)


@pytest.mark.parametrize("width", [1024, 1536])
def test_wider_depth_transformers(width):
    """Widths that the library takes besides the 512 of the one-launch depth loop (VuiShape itself derives no ffn for them)."""
    from vui_b200 import VuiB200, VuiShape
    from vui_b200.model import state_dict_shapes

    class Wide(VuiShape):
        rq_ffn = property(lambda self: 1536)

    shape, g = Wide(n_layers=2, vocab_size=64, rq_d_model=width, rq_n_heads=width // 64), torch.Generator().manual_seed(width)
    sd = {n: torch.ones(s) if n.endswith("norm.weight") else torch.randn(s, generator=g) * 0.02 for n, s in state_dict_shapes(shape).items()}
    model = VuiB200(shape, _sure({n: t.to(torch.bfloat16) for n, t in sd.items()}), device="cuda")
    _check_step(model, 6, LENGTHS[:6], 640)


def _check_step(model, B, lengths, max_seq):
    from vui_b200 import Engine

    eng = Engine(model=model, max_rows=B, max_seq=max_seq)
    lens = torch.tensor(lengths, dtype=torch.int32)
    kv = torch.randn(eng._kv[0].shape, device="cuda", dtype=torch.bfloat16, generator=torch.Generator(device="cuda").manual_seed(B)) * 0.5
    codes_in = torch.randint(0, 2048, (B, 16), generator=torch.Generator().manual_seed(B)).cuda()
    eng._apply_cfg(None, greedy=True)
    res = {}
    for off in ("1", ""):
        os.environ["VUIB_NO_TC"] = os.environ["VUIB_NO_FUSED"] = off
        try:
            for layer in eng._kv:
                layer.copy_(kv)
            eng.seq_lens[:B] = lens.cuda()
            eng._g_slot_idx[:B] = torch.arange(B, dtype=torch.int32).cuda()
            eng._g_seq_inc[:B] = 1
            eng._g_codes_in[:B] = codes_in
            rq = torch.zeros(B, 15, 2048, device="cuda", dtype=torch.bfloat16)
            eng._set_taps(None, rq)
            eng._frame_call(B)
            torch.cuda.synchronize()
            eng.check_device()
            new = torch.stack([eng._kv[-1, :, b, int(lens[b])] for b in range(B)])
            res[off] = [t[:B].float().cpu() for t in (eng._g_hidden_out, eng._g_cb0_out, new)] + [rq.float().cpu(), eng._g_codes_in[:B].cpu()]
            assert eng.seq_lens[:B].cpu().tolist() == (lens + 1).tolist()
        finally:
            os.environ["VUIB_NO_TC"] = os.environ["VUIB_NO_FUSED"] = ""
            eng._set_taps(None, None)
    for a, b in zip(res[""][:3], res["1"][:3]):   # hidden, first-codebook logits, the last layer's new K/V: every row
        rel = (a - b).flatten(1).norm(dim=1) / b.flatten(1).norm(dim=1)
        assert rel.max() < 2e-2, rel
    (rq, codes), (rq_ref, codes_ref) = res[""][3:], res["1"][3:]
    assert (codes[:, 0] == codes_ref[:, 0]).float().mean() > 0.8
    seen = 0
    for b in range(B):   # depth logits for as long as the codes drawn so far are the same (near ties may fall either way)
        for i in range(15):
            if not torch.equal(codes[b, :i + 1], codes_ref[b, :i + 1]):
                break
            assert (rq[b, i] - rq_ref[b, i]).norm() / rq_ref[b, i].norm() < 3e-2, (b, i)
            seen += 1
    assert seen > 10 * B
