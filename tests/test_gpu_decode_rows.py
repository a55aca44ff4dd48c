"""Decode steps of several streams at the edges of the kernels' row ranges (fused rows up to 4, tensor-core tiles of 16 / 32 / 64,
clusters of 8 depth streams up to 120) against the register-tile GEMV kernels, on the same caches and input codes."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sure_model(nano_sd):
    """The seeded weights with every code following from the one before (as in a trained model): no near ties between codes."""
    from vui_b200 import VuiB200, VuiShape

    sd, g = dict(nano_sd), torch.Generator().manual_seed(1)
    code, audio = (sd[n].float() / sd[n].float().std() for n in ("rq_transformer.code_emb.embedding.weight", "audio_emb.embedding.weight"))
    head = torch.empty_like(sd["rq_transformer.head_W"])
    for i in range(15):
        head[i, torch.randperm(2048, generator=g)] = code[i * 2048:(i + 1) * 2048].to(head.dtype) * 0.1
    sd["rq_transformer.head_W"] = head
    sd["codec_head.weight"] = (audio[torch.randperm(2048, generator=g)] * 0.1).to(head.dtype)
    sd["rq_transformer.code_emb.embedding.weight"], sd["audio_emb.embedding.weight"] = code.to(head.dtype), audio.to(head.dtype)
    return VuiB200(VuiShape(), sd, device="cuda")


@pytest.mark.parametrize("B", [2, 3, 4, 5, 8, 9, 16, 17, 33, 65, 120, 121, 241])
def test_decode_step_matches_gemv_kernels(sure_model, B):
    from vui_b200 import Engine

    eng = Engine(model=sure_model, max_rows=B, max_seq=640)
    lens = torch.tensor([[0, 1, 63, 64, 511, 513, 600, 97][i % 8] for i in range(B)], dtype=torch.int32)
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
