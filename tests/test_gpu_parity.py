"""Parity of the CUDA path (through the C ABI, via vui_b200.Engine) against the
oracle on the same seeded weights and inputs.  Needs a B200."""
import os

import pytest
import torch

from oracle.vui_oracle import FrameTrace, Oracle, OracleConfig

pytestmark = pytest.mark.gpu

BF16_ULP_AT_1 = 2.0 ** -7  # spacing of bf16 values in [1, 2)
REL_TOL = 2e-2             # max-abs error / max-abs value against the fp32 result of the same algorithm
REL_TOL_BF16 = 4e-2        # against another bf16 evaluation (both sit ~1.5-2e-2 from fp32 after 24 blocks; max over many frames)
COS_TOL = 0.999


def _rel(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return ((a - b).abs().max() / b.abs().max()).item()


def _cos(a, b):
    return torch.nn.functional.cosine_similarity(a.float().cpu().flatten(), b.float().cpu().flatten(), dim=0).item()


@pytest.fixture(scope="module")
def eng1(nano_model):
    from vui_b200 import Engine

    return Engine(model=nano_model, max_rows=1, max_seq=1024)


@pytest.fixture(scope="module")
def eng8(nano_model):
    from vui_b200 import Engine

    return Engine(model=nano_model, max_rows=8, max_seq=640)


@pytest.fixture(scope="module")
def oracle_gpu(nano_sd):
    """The oracle on the GPU (torch ops -> cuBLAS bf16, fp32 accumulation kept in full):
    the reference's arithmetic stack."""
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    return Oracle(OracleConfig(), nano_sd, n_slots=1, max_seq=1024, dtype=torch.bfloat16, device="cuda")


@pytest.fixture(scope="module")
def oracle_fp32(nano_sd):
    """The same algorithm without the bf16 roundings (fp32, TF32 off): the value both bf16
    evaluations approximate."""
    torch.backends.cuda.matmul.allow_tf32 = False
    return Oracle(OracleConfig(), nano_sd, n_slots=1, max_seq=1024, dtype=torch.float32, device="cuda")


def _ids(n, seed):
    return torch.randint(0, 151936, (n,), generator=torch.Generator().manual_seed(seed))


def test_library_loaded_and_no_fallback(eng1):
    import vui_b200._lib as L

    assert os.path.exists(L.LIB_PATH)
    assert eng1.launch_count() >= 0


def test_gather_sum_bit_exact(eng1, golden_dir):
    """Codebook gather-sum (backbone input) against the reference's AudioEmbedding output."""
    fx = torch.load(os.path.join(golden_dir, "ops_bf16.pt"))
    emb_k = eng1._embed_codes_kernel(fx["emb_codes"].cuda())
    assert torch.equal(emb_k.cpu(), fx["emb_out"])
    # fp32 view: the sums agree bit for bit after widening, too
    assert torch.equal(emb_k.float().cpu(), fx["emb_out"].float())


@pytest.mark.parametrize("tensor_cores", [False, True])
def test_rmsnorm_and_rope_bit_exact(eng1, golden_dir, tensor_cores):
    """The RMSNorm staging and the RoPE epilogue of both kernel families against the reference
    modules' bf16 outputs (RMSNorm.forward model.py:292-297; apply_rotary_emb rope.py:50), bit for
    bit: an identity matrix as the Linear passes the staged row through unchanged."""
    fx = torch.load(os.path.join(golden_dir, "ops_bf16.pt"))
    eye = torch.eye(1024, dtype=torch.bfloat16)
    y = eng1._debug_norm_linear(fx["norm_x"], fx["norm_w"], eye, tensor_cores).cpu()
    assert torch.equal(y, fx["norm_y"])
    q = fx["rope_q"].reshape(5, 1024)
    out = eng1._debug_linear_rope(q, eye, fx["rope_pos"], tensor_cores).cpu()
    assert torch.equal(out.view(5, 16, 64), fx["rope_out"])
    # and with the real Wqkv of layer 0 behind the norm: the reference's Linear output within bf16 rounding
    w = eng1.model.sd["decoder.blocks.0.attn.Wqkv.weight"]
    ones = torch.ones(1024, dtype=torch.bfloat16)
    got = eng1._debug_norm_linear(fx["mlp_x"], ones, w, tensor_cores).float().cpu()
    h = fx["mlp_x"].float()
    want = torch.nn.functional.linear((h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-5)).bfloat16().float(), w.float().cpu())
    assert (got - want).abs().max().item() <= 2.0 ** -8 * want.abs().max().item() + 1e-6
    eng1.check_device()


def test_prefill_and_frame0_vs_oracle(eng1, oracle_gpu, oracle_fp32):
    """64-token prefill -> final hidden, cb0 logits, depth logits of frame 0."""
    eng, o = eng1, oracle_gpu
    ids = _ids(64, 0)
    eng.reset()
    o.seq_lens = [0]
    oracle_fp32.seq_lens = [0]
    row = eng.new_row()
    h = eng.prefill_ids(row, ids)
    ho = o.prefill_text(0, ids)[-1]
    h32 = oracle_fp32.prefill_text(0, ids)[-1]
    print(f"\n[prefill hidden] engine vs fp32 {_rel(h, h32):.4f}; bf16 oracle vs fp32 {_rel(ho, h32):.4f}; "
          f"engine vs bf16 oracle {_rel(h, ho):.4f}")
    assert _rel(h, h32) < REL_TOL and _cos(h, h32) > COS_TOL
    assert _rel(h, h32) < 1.25 * _rel(ho, h32) + 2e-3
    assert _rel(h, ho) < REL_TOL_BF16 and _cos(h, ho) > COS_TOL
    rq_tap = torch.zeros(1, 15, 2048, device="cuda", dtype=torch.bfloat16)
    eng._set_taps(None, rq_tap)
    eng._apply_cfg(None, greedy=True)
    codes = eng._first_frames([row], h[None])
    hid, cb0, eos = eng._last_first
    cb0_o = torch.nn.functional.linear(ho[None], o.w["codec_head.weight"])
    assert _rel(cb0, cb0_o) < REL_TOL
    # teacher-force the oracle with the engine's codes: logits of all 15 heads
    c_o, lg_o = o.rq_generate(h[None], codes[:, 0], top_k=1, return_logits=True, forced=codes)
    torch.cuda.synchronize()
    assert _rel(rq_tap, lg_o) < REL_TOL and _cos(rq_tap, lg_o) > COS_TOL
    for q in (codes[0] != c_o[0]).nonzero().flatten().tolist():
        top2 = lg_o[0, q - 1].float().topk(2).values
        assert (top2[0] - top2[1]).item() <= 2 * BF16_ULP_AT_1, (q, top2)
    eng._set_taps(None, None)
    row.close()


def test_per_layer_hidden_vs_oracle(eng1, oracle_gpu, oracle_fp32):
    """One decode step after a prefill: residual stream after every block, against the fp32
    evaluation (tolerance 2e-2) and the bf16 oracle."""
    eng, o, o32 = eng1, oracle_gpu, oracle_fp32
    ids = _ids(48, 3)
    eng.reset()
    o.seq_lens = [0]
    o32.seq_lens = [0]
    row = eng.new_row()
    eng.prefill_ids(row, ids)
    o.prefill_text(0, ids)
    o32.prefill_text(0, ids)
    codes = torch.randint(0, 2048, (1, 16), generator=torch.Generator().manual_seed(5))
    taps = torch.zeros(24, 1, 1024, device="cuda", dtype=torch.bfloat16)
    eng._set_taps(taps, None)
    eng._g_codes_in[0] = codes[0].cuda()
    hidden, cb0, eos = eng._decode_step()
    torch.cuda.synchronize()
    o.taps, o32.taps = {}, {}
    ho, cb0_o, eos_o = o.backbone_step([0], codes)
    h32, cb0_32, _ = o32.backbone_step([0], codes)
    worst = (0.0, 0.0, 0.0)
    for li in range(24):
        ref, ref32 = o.taps[f"layer{li}"][0], o32.taps[f"layer{li}"][0]
        e32, o32e, eo = _rel(taps[li, 0], ref32), _rel(ref, ref32), _rel(taps[li, 0], ref)
        worst = max(worst, (e32, o32e, eo))
        assert e32 < REL_TOL and _cos(taps[li, 0], ref32) > COS_TOL, (li, e32)
        assert eo < REL_TOL_BF16 and _cos(taps[li, 0], ref) > COS_TOL, (li, eo)
    print(f"\n[per-layer] worst layer: engine vs fp32 {worst[0]:.4f}, bf16 oracle vs fp32 {worst[1]:.4f}, "
          f"engine vs bf16 oracle {worst[2]:.4f}")
    o.taps, o32.taps = None, None
    assert _rel(hidden[0], h32[0]) < REL_TOL and _cos(hidden[0], h32[0]) > COS_TOL
    assert _rel(hidden[0], ho[0]) < REL_TOL_BF16 and _cos(hidden[0], ho[0]) > COS_TOL
    assert _rel(cb0[0], cb0_32[0]) < REL_TOL
    assert _rel(cb0[0], cb0_o[0]) < REL_TOL_BF16
    assert abs(eos.float().item() - eos_o.float().item()) < 2e-2
    assert row.offset == 49
    eng._set_taps(None, None)
    row.close()


def _ref_attention(q, k_cache, v_cache, slot, pos):
    """fp32 softmax attention of one row: q (16, 64), caches (slots, S, 8, 64)."""
    k = k_cache[slot, : pos + 1].float().repeat_interleave(2, dim=1)  # (T, 16, 64)
    v = v_cache[slot, : pos + 1].float().repeat_interleave(2, dim=1)
    s = torch.einsum("hd,thd->ht", q.float(), k) * 0.125
    return torch.einsum("ht,thd->hd", torch.softmax(s, dim=-1), v)


def test_attention_kernel_ragged(eng8):
    """The attention kernel alone on random K/V: one key, a partial split, exact split boundaries,
    several splits, two rows on one slot; against fp32 softmax attention."""
    eng = eng8
    g = torch.Generator().manual_seed(7)
    layer = 5
    kv = eng.model.decoder.flash_kv_caches[layer]
    saved = (kv.k_cache.clone(), kv.v_cache.clone())
    kv.k_cache.copy_(torch.randn(kv.k_cache.shape, generator=g).to(torch.bfloat16))
    kv.v_cache.copy_(torch.randn(kv.v_cache.shape, generator=g).to(torch.bfloat16))
    slots = torch.tensor([0, 1, 2, 3, 4, 4, 7, 8])
    pos = torch.tensor([0, 5, 127, 128, 300, 301, 639, 255])
    q = torch.randn(8, 1024, generator=g).to(torch.bfloat16)
    out = eng._attention(layer, q, slots, pos).float().cpu()
    out2 = eng._attention(layer, q, slots, pos).float().cpu()
    assert torch.equal(out, out2)  # split merge order is fixed: bitwise repeatable
    kc, vc = kv.k_cache.cpu(), kv.v_cache.cpu()
    for r in range(8):
        ref = _ref_attention(q[r].view(16, 64), kc, vc, int(slots[r]), int(pos[r])).reshape(-1)
        err = (out[r] - ref).abs().max().item()
        assert err <= 2.0 ** -8 * max(1.0, ref.abs().max().item()) + 1e-3, (r, err)
    kv.k_cache.copy_(saved[0])
    kv.v_cache.copy_(saved[1])


def _greedy_engine(eng, ids, n_frames):
    eng.reset()
    row = eng.new_row()
    h = eng.prefill_ids(row, ids)
    codes = eng.generate_frames([row], h[None], n_frames, greedy=True)
    torch.cuda.synchronize()
    row.close()
    return codes[0].cpu()


def test_greedy_tokens_vs_oracle(eng1, oracle_gpu, nano_sd):
    """Greedy codec ids for 32 frames against the oracle on the GPU (cuBLAS bf16 GEMMs).
    Ids must be identical up to the first argmax whose top-2 logits are within 2 bf16 ulps in
    the oracle; a divergence anywhere else fails.  The count of identical frames is printed.
    (With random-init weights the bf16 logits of a 2048-way head tie exactly at the top in
    about one argmax in fifteen, so two bf16 evaluations that differ by one ulp anywhere
    upstream part ways within a frame or two; the teacher-forced test below is the strict one.)"""
    ids = _ids(256, 0)
    mine = _greedy_engine(eng1, ids, 32)
    o = oracle_gpu
    o.seq_lens = [0]
    tr = FrameTrace()
    ref = o.generate_greedy(0, ids, 32, record=tr).cpu()
    same = (mine == ref).all(dim=1)
    n_same = int(same.cumprod(0).sum())
    print(f"\n[greedy parity] frames identical to the GPU oracle before first divergence: {n_same}/32")
    if n_same < 32:
        f = n_same
        q = int((mine[f] != ref[f]).nonzero()[0])
        lg = tr.cb0[f] if q == 0 else tr.rq_logits[f][q - 1]
        top2 = lg.topk(2).values
        margin = (top2[0] - top2[1]).item()
        print(f"[greedy parity] first divergence frame {f} codebook {q}: oracle top-2 margin {margin:.5f}")
        assert margin <= 2 * BF16_ULP_AT_1 * max(1.0, abs(top2[0].item())), "diverged at a clear argmax"


def test_teacher_forced_32_frames(eng1, oracle_gpu):
    """Feed the oracle's own greedy frames to the engine one by one: every frame's 16 argmaxes
    must equal the oracle's except where the oracle's top-2 margin is within 2 bf16 ulps."""
    eng, o = eng1, oracle_gpu
    ids = _ids(256, 1)
    o.seq_lens = [0]
    tr = FrameTrace()
    ref = o.generate_greedy(0, ids, 32, record=tr).cpu()
    eng.reset()
    row = eng.new_row()
    h = eng.prefill_ids(row, ids)
    eng._apply_cfg(None, greedy=True)
    eng._g_slot_idx[0] = row.idx
    eng._g_seq_inc[0] = 1
    mism, wide, total = 0, 0, 0
    rq_tap = torch.zeros(1, 15, 2048, device="cuda", dtype=torch.bfloat16)
    eng._set_taps(None, rq_tap)
    c0 = eng._first_frames([row], h[None])[0].cpu()
    frames, mine_logits = [c0], [[eng._last_first[1][0].float().cpu()] + list(rq_tap[0].float().cpu())]
    for f in range(1, 32):
        eng._g_codes_in[0] = ref[f - 1].cuda()
        eng._frame_step(1)
        frames.append(eng._g_codes_in[0].cpu())
        mine_logits.append([eng._g_cb0_out[0].float().cpu()] + list(rq_tap[0].float().cpu()))
        assert _rel(eng._g_hidden_out[0], tr.hidden[f]) < REL_TOL_BF16
        assert _rel(eng._g_cb0_out[0], tr.cb0[f]) < REL_TOL_BF16
    eng._set_taps(None, None)
    # the depth loop is autoregressive inside a frame: compare up to its first internal divergence.  An argmax
    # may differ only where the oracle's top-2 margin is within two bf16 steps, or within twice the largest
    # difference between the two logit vectors themselves (each of the two candidates moves by at most that)
    for f in range(32):
        for q in range(16):
            total += 1
            if frames[f][q] != ref[f][q]:
                lg = tr.cb0[f] if q == 0 else tr.rq_logits[f][q - 1]
                top2 = lg.topk(2).values
                margin = (top2[0] - top2[1]).item()
                two_steps = 2 * BF16_ULP_AT_1 * max(1.0, abs(top2[0].item()))
                delta = (mine_logits[f][q] - lg).abs().max().item()
                assert delta <= REL_TOL_BF16 * lg.abs().max().item(), (f, q, delta)
                assert margin <= max(two_steps, 2 * delta), (f, q, margin, delta)
                wide += margin > two_steps
                mism += 1
                break
    print(f"\n[teacher-forced] frames whose first differing argmax is a near-tie: {mism}/32 "
          f"({wide} of them wider than two bf16 steps but within twice the logit difference; every other argmax identical)")
    assert wide <= 2
    row.close()


def test_batch_invariance_and_ragged(eng8, eng1):
    """Four streams with ragged prompt lengths decoded together give, bit for bit, what each
    gives alone (every row is computed in the same order whatever the batch; up to 4 rows run
    in the fused layers' form for several rows, more go to the tensor-core GEMMs, which sum in another order)."""
    lens = [64, 17, 130, 255]
    idss = [_ids(n, 10 + i) for i, n in enumerate(lens)]
    # a lone row normally takes kernels of its own, which sum out_proj / w2 in another order: VUIB_NO_FUSED switches
    # them off, so that one row and four rows run the same kernels
    os.environ["VUIB_NO_FUSED"] = "1"
    eng1._graphs = {}
    try:
        solo = [_greedy_engine(eng1, ids, 6) for ids in idss]
    finally:
        os.environ["VUIB_NO_FUSED"] = ""
        eng1._graphs = {}
    eng = eng8
    eng.reset()
    rows = [eng.new_row() for _ in lens]
    hs = eng._prefill_many([(r, eng.model.token_emb(ids[None])) for r, ids in zip(rows, idss)])
    h = torch.stack([x[-1] for x in hs])
    codes = eng.generate_frames(rows, h, 6, greedy=True).cpu()
    for i in range(len(lens)):
        assert torch.equal(codes[i], solo[i]), i
    assert [r.offset for r in rows] == [n + 5 for n in lens]
    eng.check_device()
    for r in rows:
        r.close()


def test_fused_layers_match_per_phase_kernels(eng1, oracle_fp32):
    """A lone row runs each layer as two cluster kernels (attention block, MLP block; partial sums of
    out_proj and w2 exchanged as fp32 rows); without them and without the tensor cores it takes five kernels
    per layer.  Same rounding points, another fp32 summation order: after a prefill + decode steps the residual stream after every
    block, the final hidden, the cb0 and depth logits and the K/V rows written agree closely, both are
    equally close to the fp32 oracle, and the greedy codes agree except at near-ties."""
    eng = eng1
    ids = _ids(200, 77)
    res = {}
    for off in ("1", ""):
        eng._graphs = {}
        eng.reset()
        row = eng.new_row()
        h = eng.prefill_ids(row, ids)   # the same kernels on both sides
        os.environ["VUIB_NO_FUSED"] = os.environ["VUIB_NO_TC"] = off   # VUIB_NO_FUSED alone: the fused layers' form for several rows
        taps = torch.zeros(24, 1, 1024, device="cuda", dtype=torch.bfloat16)
        rq_tap = torch.zeros(1, 15, 2048, device="cuda", dtype=torch.bfloat16)
        eng._set_taps(taps, rq_tap)
        eng._apply_cfg(None, greedy=True)
        eng._g_slot_idx[0] = row.idx
        eng._g_seq_inc[0] = 1
        codes_in = torch.randint(0, 2048, (16,), generator=torch.Generator().manual_seed(8)).cuda()
        frames = []
        for f in range(3):  # teacher-forced on fixed input codes: both runs see the same history
            eng._g_codes_in[0] = (codes_in + f) % 2048
            eng._frame_call(1)
            frames.append(eng._g_codes_in[0].clone())
        torch.cuda.synchronize()
        eng.check_device()
        res[off] = dict(taps=taps.clone(), rq=rq_tap.clone(), hidden=eng._g_hidden_out.clone(), cb0=eng._g_cb0_out.clone(),
                        eos=eng._g_eos_out.clone(), codes=torch.stack(frames).cpu(),
                        k=torch.stack([eng._kv[li, 0, row.idx, 200:203].clone() for li in (0, 11, 23)]),
                        v=torch.stack([eng._kv[li, 1, row.idx, 200:203].clone() for li in (0, 11, 23)]), off=row.offset)
        eng._set_taps(None, None)
        row.close()
        os.environ["VUIB_NO_FUSED"] = os.environ["VUIB_NO_TC"] = ""
    eng._graphs = {}
    a, b = res[""], res["1"]  # fused, per-phase
    assert a["off"] == b["off"] == 203 and a["k"].float().abs().max() > 0
    worst = max(_rel(a["taps"][li], b["taps"][li]) for li in range(24))
    print(f"\n[fused vs per-phase] worst per-layer hidden {worst:.5f}, final hidden {_rel(a['hidden'], b['hidden']):.5f}, "
          f"cb0 {_rel(a['cb0'], b['cb0']):.5f}, depth logits {_rel(a['rq'], b['rq']):.5f}, K {_rel(a['k'], b['k']):.5f}")
    # two bf16 evaluations that round at different summation orders: the bound the oracle tests use
    assert worst < REL_TOL_BF16 and all(_cos(a["taps"][li], b["taps"][li]) > COS_TOL for li in range(24))
    assert _rel(a["hidden"], b["hidden"]) < REL_TOL_BF16 and _cos(a["hidden"], b["hidden"]) > COS_TOL
    assert _rel(a["cb0"], b["cb0"]) < REL_TOL_BF16 and _rel(a["k"], b["k"]) < REL_TOL_BF16 and _rel(a["v"], b["v"]) < REL_TOL_BF16
    assert abs(a["eos"].float().item() - b["eos"].float().item()) < 3e-2
    assert _cos(a["rq"], b["rq"]) > COS_TOL
    # and the fused path is as close to the fp32 evaluation as the per-phase path is
    o32 = oracle_fp32
    o32.seq_lens = [0]
    o32.prefill_text(0, ids)
    codes_in = torch.randint(0, 2048, (16,), generator=torch.Generator().manual_seed(8))
    for f in range(3):
        h32, cb32, _ = o32.backbone_step([0], ((codes_in + f) % 2048)[None])
    ea, eb = _rel(a["hidden"], h32[0]), _rel(b["hidden"], h32[0])
    print(f"[fused vs per-phase] final hidden vs fp32: fused {ea:.4f}, per-phase {eb:.4f}")
    assert ea < REL_TOL + 5e-3 and ea < 1.25 * eb + 2e-3


def test_tensor_core_path_matches_gemv_path(nano_model, oracle_fp32):
    """A prefill, and decode steps of five rows and more, run on the tcgen05 GEMM (TMA-fed, accumulators in tensor
    memory); with VUIB_NO_TC on the register-tile GEMV.  Same rounding points, different fp32 summation order: a 40-token
    prefill must agree between the two and with the fp32 oracle within the bf16 tolerance, and a
    16-stream decode step must agree with the same streams decoded one by one (in the fused layers)."""
    from vui_b200 import Engine

    eng = Engine(model=nano_model, max_rows=16, max_seq=256)
    ids = _ids(40, 77)
    outs = {}
    for off in ("", "1"):
        os.environ["VUIB_NO_TC"] = off
        eng.reset()
        row = eng.new_row()
        outs[off] = eng._prefill_emb(row, eng.model.token_emb(ids[None]))[0].clone()
        eng.check_device()
        row.close()
    os.environ["VUIB_NO_TC"] = ""
    tc, gemv = outs[""], outs["1"]
    oracle_fp32.seq_lens = [0]
    ref = oracle_fp32.prefill_text(0, ids)
    print(f"\n[tc vs gemv] prefill hidden: tc vs fp32 {_rel(tc, ref):.4f}, gemv vs fp32 {_rel(gemv, ref):.4f}, "
          f"tc vs gemv {_rel(tc, gemv):.4f}")
    # The maximum over 40x1024 elements after 24 blocks sits at 2-2.5e-2 from fp32 for ANY bf16
    # evaluation (the GEMV path included), so the bound here is relative: the tensor-core result
    # must be as close to fp32 as the GEMV result is, and both within the two-bf16-paths bound.
    assert _cos(tc, ref) > COS_TOL and _cos(tc, gemv) > COS_TOL
    assert _rel(tc, ref) < REL_TOL_BF16 and _rel(tc, ref) < 1.25 * _rel(gemv, ref) + 2e-3
    assert _rel(tc, gemv) < REL_TOL_BF16
    # 16 streams in one step (tensor cores) vs each alone (fused layers)
    lens = [20 + 3 * i for i in range(16)]
    eng.reset()
    rows = [eng.new_row() for _ in lens]
    hs = eng._prefill_many([(r, eng.model.token_emb(_ids(n, 200 + i)[None])) for i, (r, n) in enumerate(zip(rows, lens))])
    codes_in = torch.randint(0, 2048, (16, 16), generator=torch.Generator().manual_seed(9))
    eng._g_codes_in.copy_(codes_in.cuda())
    hidden_b, cb0_b, eos_b = (t.clone() for t in eng._decode_step())
    torch.cuda.synchronize()
    eng.check_device()
    assert [r.offset for r in rows] == [n + 1 for n in lens]
    eng1 = Engine(model=nano_model, max_rows=1, max_seq=256)
    for i in (0, 7, 15):
        eng1.reset()
        r1 = eng1.new_row()
        eng1.prefill_ids(r1, _ids(lens[i], 200 + i))
        eng1._g_codes_in[0] = codes_in[i].cuda()
        h1, c1, e1 = eng1._decode_step()
        assert _rel(hidden_b[i], h1[0]) < REL_TOL_BF16 and _cos(hidden_b[i], h1[0]) > COS_TOL, i
        assert _rel(cb0_b[i], c1[0]) < REL_TOL_BF16, i
        r1.close()
    # a whole sampled frame for 16 streams runs and yields valid codes
    from vui_b200 import GenConfig
    h = torch.stack([x[-1] for x in hs])
    codes = eng.generate_frames(rows, h, 3, GenConfig(temperature=0.8, top_k=50, rep_penalty=1.0)).cpu()
    eng.check_device()
    assert codes.shape == (16, 3, 16) and codes.min() >= 0 and codes.max() < 2048


def test_prefill_chunking_equals_single_call(eng8):
    """A 300-token prompt in one call and in pieces of 50 give the same hidden (test_gpu_prefill_cut.py: cut by the engine)."""
    eng = eng8
    ids = _ids(300, 21)
    eng.reset()
    r1, r2 = eng.new_row(), eng.new_row()
    h1 = eng.prefill_ids(r1, ids)
    for t in range(0, 300, 50):
        h2 = eng.prefill_ids(r2, ids[t:t + 50])
    assert torch.equal(h1, h2)
    assert r1.offset == r2.offset == 300
    r1.close(), r2.close()


def test_determinism_and_seeded_sampling(eng8):
    from vui_b200 import GenConfig

    eng = eng8
    cfg = GenConfig(temperature=0.8, top_k=50, rep_penalty=1.0)
    outs = []
    for _ in range(2):
        eng.reset()
        eng._ws_reset_counters()
        rows = [eng.new_row() for _ in range(3)]
        hs = eng._prefill_many([(r, eng.model.token_emb(_ids(40 + 7 * i, 30 + i)[None])) for i, r in enumerate(rows)])
        h = torch.stack([x[-1] for x in hs])
        outs.append(eng.generate_frames(rows, h, 8, cfg).cpu())
        for r in rows:
            r.close()
    assert torch.equal(outs[0], outs[1])
    assert outs[0].min() >= 0 and outs[0].max() < 2048
    assert not torch.equal(outs[0][0], outs[0][1])


def _chi2(counts, probs, n):
    exp = probs * n
    return ((counts - exp) ** 2 / exp).sum().item()


def test_sampler_distribution_cb0(eng8, golden_dir):
    """cb0 draws at T=0.8, top-k 50 (Engine._sample_cb0, engine.py:855-863: softmax, top-k over the
    probabilities, renormalise) against the distribution the reference computed for the same logits:
    chi-square on the 50 kept entries, nothing outside the support."""
    fx = torch.load(os.path.join(golden_dir, "ops_bf16.pt"))
    eng = eng8
    for row in (0, 1):
        lg = fx["cb0_logits"][row].cuda()
        probs = fx["cb0_probs_t0.8_k50"][row]
        n = 4000
        eng._ws_reset_counters()
        eng._set_sampling(0.8, 50, 3, 1.0, 0, 0)  # the depth rule's k (3) must not leak into cb0
        draws = eng._sample_rows(lg[None].expand(8, -1).contiguous(), n // 8, cb0=True)
        counts = torch.bincount(draws.flatten(), minlength=2048).float()
        support = probs > 0
        assert int(support.sum()) == 50
        # bf16 logits tie: torch.topk keeps exactly 50 entries and breaks a tie at the 50th value arbitrarily,
        # the kernel keeps every entry that ties with it (documented difference).  The kept set must be the
        # reference's 50 plus nothing but such ties, and the distribution over it the renormalised softmax.
        sc = lg.float().cpu() / 0.8
        kth = sc.topk(50).values[-1]
        kept = sc >= kth
        assert bool((kept | ~support).all()) and int(kept.sum()) - 50 <= 4
        assert bool((sc[kept & ~support] == kth).all())
        assert counts[~kept].sum() == 0
        want = torch.softmax(sc.masked_fill(~kept, float("-inf")), dim=-1)
        # on the reference's own support the two distributions agree up to the renormalisation constant
        ratio = want[support] / probs[support]
        assert (ratio / ratio[0] - 1).abs().max() < 1e-3
        chi2 = _chi2(counts[kept], want[kept], n)
        assert chi2 < 100.0, chi2  # ~49 dof: mean 49, p(chi2 > 100) ~ 2e-5


def test_sampler_distribution_depth_rule(eng8, golden_dir):
    """Depth codebooks (model.py:955-962): logits / T, keep entries >= the k-th value, softmax, draw."""
    fx = torch.load(os.path.join(golden_dir, "ops_bf16.pt"))
    eng = eng8
    lg = fx["cb0_logits"][0]
    sc = lg.float() / 0.8
    kth = sc.topk(50).values[-1]
    probs = torch.softmax(sc.masked_fill(sc < kth, float("-inf")), dim=-1)
    n = 4000
    eng._ws_reset_counters()
    eng._set_sampling(0.8, 3, 50, 1.0, 0, 0)
    draws = eng._sample_rows(lg[None].expand(8, -1).contiguous().cuda(), n // 8)
    counts = torch.bincount(draws.flatten(), minlength=2048).float()
    support = probs > 0
    assert counts[~support].sum() == 0
    assert _chi2(counts[support], probs[support], n) < 60.0 + 1.5 * int(support.sum())


def test_first_frame_cb0_ignores_top_k(eng8, golden_dir):
    """cb0 of a chunk's first frame is drawn from the WHOLE distribution even when top-k is set
    (engine.py:936-937, 1416-1424): draws land outside the top-50 at the rate softmax(l/T) gives, and
    32 equal-count bins of the codebook (sorted by probability) pass a chi-square test."""
    fx = torch.load(os.path.join(golden_dir, "ops_bf16.pt"))
    eng = eng8
    lg = fx["cb0_logits"][0]
    probs = torch.softmax(lg.float() / 0.8, dim=-1)
    order = probs.argsort(descending=True)
    n = 4000
    eng._ws_reset_counters()
    eng._set_sampling(0.8, 50, 1, 1.0, 0, 2)  # two codebooks: the depth loop after the draw stays short
    draws = eng._sample_first_frame(lg[None].expand(8, -1).contiguous(), n // 8)
    eng._set_sampling(1.0, 1, 1, 1.0, 0, 0)
    counts = torch.bincount(draws.flatten(), minlength=2048).float()
    p_out = probs[order[50:]].sum().item()
    frac_out = counts[order[50:]].sum().item() / n
    assert p_out > 0.5  # these logits are flat: most of the mass lies outside the top 50
    assert abs(frac_out - p_out) < 5 * (p_out * (1 - p_out) / n) ** 0.5, (frac_out, p_out)
    binned_c = counts[order].reshape(32, 64).sum(1)
    binned_p = probs[order].reshape(32, 64).sum(1)
    assert _chi2(binned_c, binned_p, n) < 80.0  # 31 dof
    # greedy (top_k_cb0 == 1) stays greedy on the first frame
    eng._set_sampling(1.0, 1, 1, 1.0, 0, 2)
    g = eng._sample_first_frame(lg[None].expand(8, -1).contiguous(), 1)
    assert g.flatten().tolist() == [int(torch.argmax(lg.float()))] * 8
    eng._set_sampling(1.0, 1, 1, 1.0, 0, 0)


def test_greedy_first_index_on_ties(eng8):
    eng = eng8
    lg = torch.zeros(8, 2048, device="cuda", dtype=torch.bfloat16)
    lg[:, 100] = 1.5
    lg[:, 7] = 1.5
    lg[:, 2047] = 1.5
    eng._set_sampling(1.0, 1, 1, 1.0, 0, 0)
    assert eng._sample_rows(lg, 1).flatten().tolist() == [7] * 8


def test_rep_penalty_window(eng8):
    """With a huge penalty the sampler never repeats a code inside the window and may after it."""
    eng = eng8
    lg = torch.full((8, 2048), -4.0, device="cuda", dtype=torch.bfloat16)
    lg[:, :4] = 4.0  # four strong candidates
    eng._rep_reset()
    eng._set_sampling(1.0, 1, 1, 1000.0, 3, 0)
    seq = eng._sample_rows(lg, 12, cb0=True)[:, 0].tolist()
    for i in range(3, 12):
        assert seq[i] not in seq[i - 3:i], seq
    assert set(seq) == {0, 1, 2, 3}
    eng._rep_reset()


def test_device_flag_reports_bad_code(eng8):
    from vui_b200._lib import VuibError

    eng = eng8
    eng.reset()
    row = eng.new_row()
    eng.prefill_ids(row, _ids(8, 1))
    eng._g_codes_in.zero_()
    eng._g_codes_in[0, 3] = 5000  # outside [0, 2048)
    eng._decode_step()
    with pytest.raises(VuibError):
        eng.check_device()
    eng.check_device()  # flag cleared
    row.close()


def test_host_side_errors(nano_model):
    from vui_b200 import Engine

    with pytest.raises(ValueError):
        Engine(model=nano_model, max_rows=1, max_seq=10 ** 6)
    eng = Engine(model=nano_model, max_rows=1, max_seq=128)
    r = eng.new_row()
    with pytest.raises(RuntimeError):
        eng.new_row()
    with pytest.raises(RuntimeError):
        eng.prefill_ids(r, _ids(200, 0))  # overflows max_seq
    r.close()
    eng2 = Engine(model=nano_model, max_rows=2, max_seq=128)
    with pytest.raises(RuntimeError):
        next(eng2.new_row().stream("hello"))


def test_older_single_stream_api_decode_step(nano_model, oracle_fp32):
    """`setup_decode_graph()` / `decode_step(codes, pos)` of the reference's older single-stream API
    (model.py:1228-1300): four frames of codes fed at positions 0..3 give, bit for bit, what the
    engine's own backbone step gives (that step is held to the oracle by the tests above; here the
    fp32 oracle bounds it loosely, a single bf16 evaluation sits up to ~2.3e-2 from it), and stepping
    back to a position overwrites it."""
    from vui_b200 import Engine

    m = nano_model
    m.setup_decode_graph(max_seq=256)
    eng = Engine(model=m, max_rows=1, max_seq=256)
    eng.new_row()
    g = torch.Generator().manual_seed(5)
    frames = torch.randint(0, 2048, (4, 16), generator=g)
    oracle_fp32.seq_lens = [0]
    for pos in range(4):
        hid, cb0, eos = m.decode_step(frames[pos].cuda(), pos)
        assert hid.shape == (1, 1024) and cb0.shape == (1, 2048) and eos.shape == (1, 1)
        eng._g_codes_in[0].copy_(frames[pos])
        eh, ec, ee = eng._decode_step()
        torch.cuda.synchronize()
        assert torch.equal(hid, eh[:1]) and torch.equal(cb0, ec[:1]) and torch.equal(eos.reshape(-1), ee[:1].reshape(-1)), pos
        rh, rc, re_ = oracle_fp32.backbone_step([0], frames[pos][None])
        assert _rel(hid, rh) < 3e-2 and _cos(hid, rh) > COS_TOL, pos
        assert _rel(cb0, rc) < 3e-2 and _cos(cb0, rc) > COS_TOL, pos
        assert abs(float(eos) - float(re_)) < 3e-2 * max(1.0, float(rc.abs().max())), pos
    first = m.decode_step(frames[3].cuda(), 3)[0].clone()
    again = m.decode_step(frames[3].cuda(), 3)[0]
    assert torch.equal(first, again)  # same position, same history: bit-identical
    with pytest.raises(RuntimeError):
        type(m).decode_step(type(m).__new__(type(m)), frames[0], 0)


def test_bad_slot_and_position_are_clamped_and_flagged(eng8):
    """Out-of-range slots / positions handed to the C ABI never index outside the cache: the kernels
    clamp them and record the device flag (prefill rows, the attention entry point, the sampler)."""
    import ctypes as C

    from vui_b200._lib import VuibError

    eng = eng8
    eng.reset()
    eng.check_device()
    guard_k = eng._kv.clone()
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    emb = torch.randn(3, 1024, generator=torch.Generator().manual_seed(1)).to("cuda", torch.bfloat16)
    out = torch.empty_like(emb)
    for slots, poss in (([0, 99, 1], [0, 0, 0]), ([0, -5, 1], [0, 0, 0]), ([0, 1, 2], [0, 10 ** 6, 0]), ([0, 1, 2], [0, -1, 0])):
        slot = torch.tensor(slots, dtype=torch.int32, device="cuda")
        pos = torch.tensor(poss, dtype=torch.int32, device="cuda")
        eng._ck(eng._lib.vuib_prefill(eng._handle, 3, P(slot), P(pos), P(emb), P(out), eng._stream))
        with pytest.raises(VuibError) as ei:
            eng.check_device()
        assert ei.value.code == -7
        eng.check_device()  # cleared
        assert torch.isfinite(out.float()).all()
    # only slots 0..2, 8 (clamped high slot) and positions 0 / max_seq-1 of them may have been written
    touched = (eng._kv != guard_k).any(dim=-1).any(dim=-1)  # (L, 2, slots, max_seq)
    allowed = torch.zeros_like(touched)
    allowed[:, :, :, 0] = True
    allowed[:, :, :, eng.max_seq - 1] = True
    assert not (touched & ~allowed).any()
    # attention entry: bad position and slot
    q = torch.randn(2, 1024, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16)
    o = eng._attention(0, q, torch.tensor([0, 50]), torch.tensor([10 ** 6, 3]))
    torch.cuda.synchronize()
    assert torch.isfinite(o.float()).all()
    with pytest.raises(VuibError):
        eng.check_device()
    # sampler: slot outside the per-slot state
    lg = torch.zeros(2, 2048, device="cuda", dtype=torch.bfloat16)
    codes = torch.zeros(2, device="cuda", dtype=torch.long)
    bad = torch.tensor([0, 1000], dtype=torch.int32, device="cuda")
    eng._ck(eng._lib.vuib_sample_rows(eng._handle, 2, P(bad), P(lg), 0, P(codes), eng._stream))
    with pytest.raises(VuibError):
        eng.check_device()
    eng._ws_reset_counters()
    eng.check_device()


def test_bounded_wait_runs_out_and_reports(nano_model):
    """A wait inside a kernel that cannot complete (the tensor-core GEMM's mailbox told to expect one value
    more than is sent to it by a test hook) gives up after the configured number of polls, records the device flag and
    the kernel returns; after vuib_reset_state the same call is bit-identical to a clean run."""
    from vui_b200 import Engine
    from vui_b200._lib import VuibError

    eng = Engine(model=nano_model, max_rows=1, max_seq=64, max_prefill_rows=16)
    ids = _ids(8, 4)  # 8 rows: the tensor-core path, K split over several CTAs per tile
    row = eng.new_row()
    clean = eng.prefill_ids(row, ids).clone()
    eng.check_device()
    eng._rewind_row(row, 0)
    eng._ck(eng._lib.vuib_set_wait_limit(eng._handle, 20000))
    eng._ck(eng._lib.vuib_debug_withhold_arrival(eng._handle, eng._stream))
    eng.prefill_ids(row, ids)
    torch.cuda.synchronize()  # the kernels returned: nothing hangs
    with pytest.raises(VuibError) as ei:
        eng.check_device()
    assert ei.value.code == -7 and "wait" in str(ei.value)
    eng._ck(eng._lib.vuib_set_wait_limit(eng._handle, 1 << 22))
    eng._ws_reset_counters()
    eng._rewind_row(row, 0)
    again = eng.prefill_ids(row, ids)
    eng.check_device()
    assert torch.equal(again, clean)


def test_a_withheld_arrival_does_not_outlive_a_reset(nano_model):
    """The hook armed, but no GEMM of it run before vuib_reset_state: the calls after that are clean."""
    from vui_b200 import Engine

    eng = Engine(model=nano_model, max_rows=1, max_seq=64, max_prefill_rows=16)
    row = eng.new_row()
    clean = eng.prefill_ids(row, _ids(8, 4)).clone()
    eng._ck(eng._lib.vuib_set_wait_limit(eng._handle, 20000))
    eng._ck(eng._lib.vuib_debug_withhold_arrival(eng._handle, eng._stream))
    eng._ws_reset_counters()
    eng._rewind_row(row, 0)
    again = eng.prefill_ids(row, _ids(8, 4))
    eng.check_device()
    assert torch.equal(again, clean)


@pytest.mark.parametrize("polls", [16, 2 ** 32 - 1])
def test_wait_limit_at_its_ends(nano_model, polls):
    """One to four streams run in kernels whose CTAs send to one another: the shortest limit does not make them give up, and the
    longest does not overflow into a short one, in them or in the GEMMs of more streams."""
    from vui_b200 import Engine

    for n in (1, 3) if polls == 16 else (1, 3, 6):
        eng = Engine(model=nano_model, max_rows=n, max_seq=64)
        rows = [eng.new_row() for _ in range(n)]
        out = []
        for limit in (1 << 22, polls):
            if limit != 16:   # GEMMs, in a prefill or of five streams and more, do take so short a limit
                eng._ck(eng._lib.vuib_set_wait_limit(eng._handle, limit))
            for r in rows:
                eng._rewind_row(r, 0)
            h = torch.stack([eng.prefill_ids(r, _ids(5 + i, i)) for i, r in enumerate(rows)])
            eng._ck(eng._lib.vuib_set_wait_limit(eng._handle, limit))
            eng._graphs = {}
            out.append(eng.generate_frames(rows, h, 3, greedy=True))
            eng.check_device()
        assert torch.equal(out[0], out[1])
