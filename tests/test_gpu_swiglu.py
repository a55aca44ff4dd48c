"""SiLU(w1 h) * (w3 h) of every path that a decode step can take, over all finite bf16 gate values, against 64 bits: a
one-layer model whose rows are one-hot and whose matrices pass single values through unchanged."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu

D, UNITS, ROWS = 1024, 1022, 64   # output column 0 stays free, the rows' own columns are left out of the comparison


@pytest.fixture(scope="module")
def gates():
    """Every finite bf16, each once or more, as the (UNITS, ROWS) values that w1 . h takes."""
    bits = torch.arange(65536, dtype=torch.int32)
    bits = bits[(bits & 0x7F80) != 0x7F80].to(torch.int16)
    bits = torch.cat([bits, bits[: UNITS * ROWS - bits.numel()]])
    return bits.view(torch.bfloat16).reshape(UNITS, ROWS)


@pytest.fixture(scope="module")
def engine(nano_sd, gates):
    from vui_b200 import Engine, VuiB200, VuiShape

    shape = VuiShape(n_layers=1, vocab_size=8, norm_eps=0.0)
    sd = {k: v for k, v in nano_sd.items() if not k.startswith("decoder.blocks.") or k.startswith("decoder.blocks.0.")}
    sd["token_emb.weight"] = sd["token_emb.weight"][:8]
    zero = lambda k: torch.zeros_like(sd[k])  # noqa: E731
    p = "decoder.blocks.0."
    sd[p + "mlp_norm.weight"] = torch.ones_like(sd[p + "mlp_norm.weight"])
    # code r of the first codebook embeds as the unit vector of column r; RMSNorm turns its 1 into sqrt(1024) = 32
    emb = zero("audio_emb.embedding.weight")
    emb[torch.arange(ROWS), torch.arange(ROWS)] = 1.0
    out_proj, w1, w3, w2 = (zero(p + n) for n in ("attn.out_proj.weight", "mlp.w1.weight", "mlp.w3.weight", "mlp.w2.weight"))
    w1[:UNITS, :ROWS] = gates / 32
    w3[:UNITS, :ROWS] = 1.0 / 32
    w2[torch.arange(UNITS) + 1, torch.arange(UNITS)] = 1.0
    sd.update({"audio_emb.embedding.weight": emb, p + "attn.out_proj.weight": out_proj, p + "mlp.w1.weight": w1, p + "mlp.w3.weight": w3,
               p + "mlp.w2.weight": w2})
    return Engine(model=VuiB200(shape, sd, device="cuda"), max_rows=ROWS, max_seq=64)


@pytest.mark.parametrize("rows,per_phase", [(64, False), (64, True), (4, False), (1, False)])
def test_swiglu_over_all_gate_values(engine, gates, rows, per_phase):
    eng = engine
    codes = torch.full((ROWS, 16), 2047, device="cuda")   # the other codebooks' rows embed as zeros
    got = torch.zeros(ROWS, UNITS, dtype=torch.bfloat16)
    os.environ["VUIB_NO_TC"] = os.environ["VUIB_NO_FUSED"] = "1" if per_phase else ""
    try:
        for r0 in range(0, ROWS, rows):
            taps = torch.zeros(1, ROWS, D, device="cuda", dtype=torch.bfloat16)
            eng._set_taps(taps, None)
            codes[:rows, 0] = torch.arange(r0, r0 + rows)
            eng.seq_lens.zero_()
            P = lambda t: t.data_ptr()  # noqa: E731
            eng._ck(eng._lib.vuib_backbone_step(eng._handle, rows, P(eng._g_slot_idx), None, P(codes), P(eng._g_hidden_out),
                                                P(eng._g_cb0_out), P(eng._g_eos_out), eng._stream))
            eng.check_device()
            got[r0:r0 + rows] = taps[0, :rows, 1:UNITS + 1].cpu()
    finally:
        os.environ["VUIB_NO_TC"] = os.environ["VUIB_NO_FUSED"] = ""
        eng._set_taps(None, None)
    a = ((gates / 32).double() * 32).t()   # what w1 holds of a gate: the smallest ones are rounded by the division
    want = (a / (1 + torch.exp(-a))).to(torch.bfloat16)
    keep = torch.ones(ROWS, UNITS, dtype=torch.bool)
    for r in range(1, ROWS):
        keep[r, r - 1] = False   # the row's own 1 in the residual is added there
    g, w = got.float()[keep], want.float()[keep]
    # A few ulp of fp32 before the rounding to bf16 may turn a near tie, which is one step of a bf16.  Below x = -88.7 exp(-x) is
    # infinite in fp32 and the plain quotient 0 instead of -2.6e-37 and less.
    least = torch.tensor(2.0 ** -120)
    assert ((g - w).abs() <= torch.maximum(w.abs() * 2.0 ** -7, least)).all()
    wrong = int((g != w)[w.abs() >= least].sum())
    print(f"\n[swiglu] rows {rows}, per-phase kernels {per_phase}: {wrong} of {w.numel()} not the nearest bf16")
    assert wrong < 20
