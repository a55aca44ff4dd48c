"""A second speaker given by an embedding alone: Row.prefill(segments, spk_emb=a, spk_emb_2=b) and RenderRequest."""
import zlib
from types import SimpleNamespace

import pytest
import torch

from vui_b200.engine import Engine, GenConfig, RenderRequest, Segment


def test_prompt_sets_both_speaker_tokens():
    """Without a device: the prompt of a row keeps the second speaker's token whether or not that speaker has segments."""
    eng = SimpleNamespace(device="cpu", _embed_speaker=lambda e: e, _speaker_segments_emb=lambda segs, tok, final: [(tok, len(segs))])
    a, b = torch.zeros(1), torch.ones(1)
    row = SimpleNamespace(_codec_ctx=None)
    parts = Engine._prompt_parts(eng, row, [Segment("Hello there.")], a, None, b)
    assert row._spk_token is a and row._spk_token_2 is b and parts == [(a, 1)]
    parts = Engine._prompt_parts(eng, row, [Segment("Hello there.")], a, [Segment("One."), Segment("Two.")], b)
    assert row._spk_token_2 is b and parts == [(a, 1), (b, 2)]
    Engine._prompt_parts(eng, row, [Segment("Hello there.")], a)
    assert row._spk_token_2 is None and row._active_speaker == 0


class StubTok:
    special_to_id = {"[SC]": 151900}

    def encode(self, text):
        return torch.tensor([zlib.crc32(w.encode()) % 151000 for w in text.split()] or [1], dtype=torch.long)


@pytest.mark.gpu
def test_sc_switches_the_speaker(nano_sd, monkeypatch):
    """Every chunk of a text is spoken with the token of the speaker whose turn it is: rows that stream and render, and requests."""
    from vui_b200 import VuiB200, VuiShape

    sd = dict(nano_sd)
    sd["spk_proj.weight"] = torch.empty(1024, 1024).normal_(0, 0.01, generator=torch.Generator().manual_seed(9)).bfloat16()
    model = VuiB200(VuiShape(), sd, device="cuda", tokenizer=StubTok())
    eng = Engine(model=model, max_rows=1, max_seq=256)
    a, b = (torch.randn(1024, generator=torch.Generator().manual_seed(s)) for s in (1, 2))
    used = []
    token_of = Engine._active_spk_token
    monkeypatch.setattr(Engine, "_active_spk_token", lambda self, row: used.append(token_of(self, row)) or used[-1])
    segs = [Segment("A short prompt.", torch.randint(0, 2048, (4, 16), generator=torch.Generator().manual_seed(3)))]
    cfg = GenConfig(temperature=0.8, top_k=50, max_turn_secs=0.3, eos_threshold=1.0)
    text = "One two three. [SC] Four five six. [SC] Seven eight nine."
    want = [eng._embed_speaker(e) for e in (a, b, a)]

    def check():
        assert len(used) == 3 and all(torch.equal(u, w) for u, w in zip(used, want))
        used.clear()

    row = eng.new_row()
    assert row.prefill(segs, spk_emb=a, spk_emb_2=b) == 1 + 3 + 1 + 4   # [spk] text [SC] codes, nothing of the second speaker
    list(eng._stream_codes(row, text, cfg))
    check()
    row.close()
    eng.render_continuous_codes([RenderRequest(segments=segs, spk_emb=a, spk_emb_2=b, text=text)], cfg)
    check()
    eng.check_device()
