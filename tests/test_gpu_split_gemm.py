"""The split GEMMs under the codec (split_gemm.cuh) at row counts around their tiles, clusters and splits: whole inputs decoded and
encoded in one pass against the CPU oracles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def codec():
    from oracle.codec_oracle import CodecOracle
    from vui_b200.codec import QwenCodecDecoder, random_codec_state

    sd = random_codec_state(0)
    return QwenCodecDecoder(sd, device="cuda"), CodecOracle(sd)


@pytest.mark.parametrize("frames,n_q", [(2, 16), (7, 1), (16, 16), (33, 8)])
def test_decode_in_one_pass(codec, frames, n_q):
    dec, oracle = codec
    codes = torch.randint(0, 2048, (1, n_q, frames), generator=torch.Generator().manual_seed(frames))
    got = dec(codes.cuda()).cpu()
    dec.check_device()
    assert dec.position() == frames
    ref = oracle.decode_offline(codes)
    assert got.shape == ref.shape and (got - ref).abs().max().item() <= 5e-5 * ref.abs().max().item()


@pytest.mark.parametrize("frames", [2, 9, 250])
def test_a_frame_after_a_whole_input_is_a_first_frame(codec, frames):
    """The library's own calls, without the resets of the Python class between them: 250 is all the positions that there are."""
    dec, _ = codec
    codes = torch.randint(0, 2048, (1, 16, frames), generator=torch.Generator().manual_seed(frames)).cuda()
    nxt = torch.randint(0, 2048, (3, 16), generator=torch.Generator().manual_seed(1)).cuda()

    def stream():
        out = torch.zeros(3, 1920, device="cuda")
        for i in range(3):
            dec._check(dec._lib.vuib_codec_decode_frame(dec._h, nxt[i].data_ptr(), 16, out[i].data_ptr(), dec._stream()))
            assert dec.position() == i + 1
        return out

    dec.reset_streaming()
    fresh = stream()
    dec(codes)
    assert dec.position() == frames
    assert torch.equal(stream(), fresh)
    dec.check_device()
    dec.reset_streaming()
    assert dec.position() == 0


@pytest.mark.parametrize("frames", [1, 2, 17, 32])
def test_encode_in_one_pass(frames):
    from oracle.codec_enc_oracle import EncoderOracle, test_audio
    from vui_b200.codec_encoder import QwenCodecEncoder, random_encoder_state

    enc, oracle = QwenCodecEncoder(random_encoder_state(0)), EncoderOracle(random_encoder_state(0))
    audio = test_audio(frames * 1920, seed=frames)
    got, ref = enc(audio.cuda())[0].cpu(), oracle.encode(audio)[0]
    # a code may differ where two are equally near; what follows from it in its frame then differs too
    assert got.shape == ref.shape and (got != ref).float().mean().item() <= 0.02


def test_encoder_takes_weights_at_any_float():
    """A state dict on the device whose tensors are views one float into their buffers, as slices of one flat parameter buffer are."""
    from oracle.codec_enc_oracle import test_audio
    from vui_b200.codec_encoder import QwenCodecEncoder, random_encoder_state

    sd = random_encoder_state(0)
    odd = {}
    for name, t in sd.items():
        flat = torch.empty(t.numel() + 1, device="cuda")
        odd[name] = flat[1:].view(t.shape).copy_(t)
        assert odd[name].data_ptr() % 16 == 4
    audio = test_audio(17 * 1920, seed=17).cuda()
    assert torch.equal(QwenCodecEncoder(odd)(audio), QwenCodecEncoder(sd)(audio))


def test_encoder_reports_a_wait_that_ran_out():
    """The flag that the kernels set, set by hand in the workspace: reported once, and the encoder goes on."""
    from vui_b200 import _lib
    from vui_b200.codec_encoder import QwenCodecEncoder

    enc = QwenCodecEncoder.random_init(0)
    enc.check_device()
    enc._ws[:4].view(torch.int32).fill_(4)
    with pytest.raises(_lib.VuibError, match="wait") as err:
        enc.check_device()
    assert err.value.code == -7
    enc(torch.zeros(1, 1, 1920, device="cuda"))
    enc.check_device()


def test_a_streaming_decoder_takes_whole_inputs_frame_by_frame(codec):
    from vui_b200.codec import QwenCodecDecoder, random_codec_state

    whole, _ = codec
    dec = QwenCodecDecoder(random_codec_state(0), whole_inputs=False)
    assert dec._ws.numel() < 40e6 < whole._ws.numel()
    codes = torch.randint(0, 2048, (1, 16, 5), generator=torch.Generator().manual_seed(5)).cuda()
    for _ in range(2):   # each call starts from zero padding
        got = dec(codes)
        assert dec.position() == 5 and (got - whole(codes)).abs().max().item() <= 5e-5 * got.abs().max().item()
    with dec.streaming(1):
        assert torch.equal(torch.cat([dec(codes[:, :, t:t + 1]) for t in range(5)], dim=-1), got)
    dec.check_device()
