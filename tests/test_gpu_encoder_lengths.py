"""The quantiser and the codec's attention where their split changes: frames of a cluster (8, or 9 where that saves a wave), one and several
clusters, 64 keys a CTA.  The codes against the nearest ones in 64 bits for the encoder's own latents, followed codebook by codebook as long
as the distance to the runner-up leaves no doubt; a prefix's frames against those of the whole."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def encoder():
    from vui_b200.codec_encoder import QwenCodecEncoder, random_encoder_state

    sd = random_encoder_state(0)
    return QwenCodecEncoder(sd), sd


def _sound(n):
    return (torch.randn(1, 1, n * 1920, generator=torch.Generator().manual_seed(3)) * 0.1).cuda()


@pytest.fixture(scope="module")
def long_encoder(encoder):
    """Of 20 s, the longest buffer."""
    from vui_b200.codec_encoder import QwenCodecEncoder

    return QwenCodecEncoder(encoder[1], max_secs=20.0), encoder[1]


@pytest.mark.parametrize("frames", [1, 7, 8, 9, 31, 32, 33, 64, 65, 120, 121, 125])
def test_codes_are_the_nearest(encoder, frames):
    _check_nearest(*encoder, frames)


@pytest.mark.parametrize("frames", [120, 121, 135, 136, 240, 241, 250])
def test_codes_of_long_inputs_are_the_nearest(long_encoder, frames):
    _check_nearest(*long_encoder, frames)


def _check_nearest(enc, sd, frames):
    codes = enc(_sound(frames))[0].cpu()
    lat = enc.read_latent(frames).double()
    followed = 0
    for part, first, n in (("semantic", 0, 1), ("acoustic", 1, 15)):
        r = (sd[f"quantizer.{part}.input_proj.weight"][:, :, 0].double() @ lat).T
        sure = torch.ones(frames, dtype=torch.bool)
        for i in range(n):
            e = sd[f"quantizer.{part}.codebooks.{i}.embed"].double()
            d = (e * e).sum(1)[None] - 2 * r @ e.T
            best = d.topk(2, largest=False)
            # sums of 256 products in 32 bits, residuals of up to 15 subtractions: 1e-5 of the largest distance is some hundred roundings
            sure &= best.values[:, 1] - best.values[:, 0] > 1e-5 * d.abs().amax(1)
            assert torch.equal(codes[first + i][sure], best.indices[sure, 0])
            followed += int(sure.sum())
            r = r - e[codes[first + i]]
    assert followed > 0.9 * 16 * frames
    enc.check_device()


@pytest.mark.parametrize("frames", [16, 32, 33, 64, 65, 80, 121])
def test_a_prefix_has_the_frames_of_the_whole(encoder, frames):
    enc, _ = encoder
    x = _sound(125)
    enc(x)
    whole = enc.read_latent(125)[:, :frames]
    enc(x[:, :, :frames * 1920])
    part = enc.read_latent(frames)
    # 32-bit sums in another order through some forty layers
    assert (part - whole).abs().max() <= 5e-5 * whole.abs().max()
