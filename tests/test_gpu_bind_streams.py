"""Objects built on a stream of the caller's while that stream is busy: what binding lays out in the workspace is made of the weights
as that stream leaves them, and stays."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _on_a_busy_stream(make):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(400_000_000)   # about 0.2 s
        obj = make()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    return obj


def test_engine(nano_model):
    from vui_b200 import Engine

    def codes(eng):   # six streams: the depth loop in one launch, from the weights laid out at binding
        rows = [eng.new_row() for _ in range(6)]
        h = torch.stack([eng.prefill_ids(r, torch.arange(5 + i)) for i, r in enumerate(rows)])
        return eng.generate_frames(rows, h, 2, greedy=True)

    make = lambda: Engine(model=nano_model, max_rows=6, max_seq=64)  # noqa: E731
    want = codes(make())   # first: loading a kernel waits for the device
    assert torch.equal(codes(_on_a_busy_stream(make)), want)


def test_decoder():
    from vui_b200.codec import QwenCodecDecoder, random_codec_state

    sd = {k: v.cuda() for k, v in random_codec_state(0).items()}
    codes = torch.randint(0, 2048, (1, 16, 4), generator=torch.Generator().manual_seed(1)).cuda()
    make = lambda: QwenCodecDecoder({k: v * 1.0 for k, v in sd.items()})  # noqa: E731
    want = make()(codes)
    assert torch.equal(_on_a_busy_stream(make)(codes), want)


def test_encoder():
    from oracle.codec_enc_oracle import test_audio
    from vui_b200.codec_encoder import QwenCodecEncoder, random_encoder_state

    sd = {k: v.cuda() for k, v in random_encoder_state(0).items()}
    audio = test_audio(4 * 1920, seed=1).cuda()
    make = lambda: QwenCodecEncoder({k: v * 1.0 for k, v in sd.items()})  # noqa: E731
    want = make()(audio)
    assert torch.equal(_on_a_busy_stream(make)(audio), want)
