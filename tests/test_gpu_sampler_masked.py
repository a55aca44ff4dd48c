"""Draws from logits of which most are masked out with -inf (constrained decoding), by both rules of the sampler."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng(nano_model):
    from vui_b200 import Engine

    return Engine(model=nano_model, max_rows=8, max_seq=64)


@pytest.mark.parametrize("cb0", [False, True])
@pytest.mark.parametrize("top_k", [0, 2, 50, 2047])
def test_masked_codes_are_never_drawn(eng, cb0, top_k):
    """Four codes are left, so a top-k of 50 or 2047 keeps masked ones, whose probability is exactly 0; the draws follow the softmax
    over what the rule keeps."""
    allowed = torch.tensor([3, 700, 1500, 2040])
    lg = torch.full((2048,), float("-inf"))
    lg[allowed] = torch.tensor([1.0, 0.5, 0.25, -0.5])
    T, n = 0.7, 2000
    eng._ws_reset_counters()
    eng._set_sampling(T, top_k, top_k, 1.0, 0, 0)
    draws = eng._sample_rows(lg[None].expand(8, -1).contiguous(), n // 8, cb0=cb0).flatten()
    p = torch.softmax(lg[allowed] / T, 0)
    if top_k == 2:
        p = torch.tensor([p[0], p[1], 0, 0]) / (p[0] + p[1])
    counts = torch.stack([(draws == a).sum() for a in allowed]).float()
    assert counts.sum() == n
    assert (counts - n * p).abs().max() < 5 * (n * 0.25) ** 0.5   # five standard deviations of a count
    eng.check_device()
