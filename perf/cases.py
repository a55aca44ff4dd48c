"""What users of this package have it do, as cases that can be timed: text and voice prompts taken in, frames of codes generated
for one to 256 streams, text spoken as audio for one listener and for a queue of requests, codes decoded to audio and audio encoded
to codes.  Model shapes are the package's own (VuiShape, QwenCodecDecoder, QwenCodecEncoder); weights are seeded random ones.

Random matrices alone give flat distributions over the 2048 codes, whose near-ties fall the other way with every change of a
rounding; a trained model is sure of its code nearly always.  So the embeddings here are as large as what the layers add, and each
output head is aligned with the embedding that it follows (a seeded permutation of it): every code is likely given the one before.
"""

import math
import random
import zlib

import torch

from vui_b200 import Engine, GenConfig, RenderRequest, Segment, VuiB200, VuiShape
from vui_b200.codec import QwenCodecDecoder, codec_param_shapes
from vui_b200.codec_encoder import QwenCodecEncoder, StreamingCodecEncoder, encoder_param_shapes
from vui_b200.model import state_dict_shapes

SHAPE = VuiShape()
SAMPLES = 1920  # of one codec frame (80 ms at 24 kHz)


def listed():
    return [
        # one listener, codes only: latency of every single frame counts
        {"name": "frames-1", "kind": "frames", "streams": 1, "prompt_min": 256, "prompt_max": 256, "frames": 25, "greedy": True, "codebooks": 0},
        # a handful of listeners on one card
        {"name": "frames-3", "kind": "frames", "streams": 3, "prompt_min": 40, "prompt_max": 200, "frames": 25, "greedy": False, "codebooks": 0},
        # sixteen cloned voices
        {"name": "frames-16", "kind": "frames", "streams": 16, "prompt_min": 253, "prompt_max": 253, "frames": 20, "greedy": True, "codebooks": 0},
        # a busy server: 64 conversations of different lengths
        {"name": "frames-64", "kind": "frames", "streams": 64, "prompt_min": 64, "prompt_max": 512, "frames": 20, "greedy": False, "codebooks": 0},
        # the most that a card is given
        {"name": "frames-256", "kind": "frames", "streams": 256, "prompt_min": 64, "prompt_max": 512, "frames": 12, "greedy": False, "codebooks": 0},
        # one sentence of text ids read in: the smallest call
        {"name": "ids-37", "kind": "ids", "tokens": 37},
        # sixteen voice prompts (transcript and 10 s of codes each) read in, row after row
        {"name": "prompts-16", "kind": "prompts", "rows": 16, "words": 128, "frames": 125},
        # one turn of a conversation: a sentence in, audio out frame by frame
        {"name": "talk-6", "kind": "talk", "words": 6, "prompt_words": 20, "prompt_frames": 75, "codebooks": 0},
        # a queue of requests over fewer rows, each to its whole audio
        {"name": "render-6", "kind": "render", "rows": 4, "requests": 6, "words": 7, "prompt_words": 12, "prompt_frames": 36},
        # the codes of 10 s to audio in one call
        {"name": "decode-125", "kind": "decode", "frames": 125, "codebooks": 16},
        # a 10 s recording to codes in one call
        {"name": "encode-125", "kind": "encode", "frames": 125},
        # a user speaking for about 5 s: chunks of audio as they come in, codes as soon as they are known
        {"name": "listen-5", "kind": "listen", "chunks": 5, "chunk_samples": 24000},
    ]


def _log_int(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(("frames", "frames", "frames", "ids", "prompts", "talk", "render", "decode", "encode", "listen"))
    if kind == "frames":
        streams = _log_int(rng, 1, 256)
        low = _log_int(rng, 16, 256)
        return {"kind": kind, "streams": streams, "prompt_min": low, "prompt_max": rng.randint(low, min(512, 2 * low)),
                "frames": rng.randint(6, max(8, min(32, 3072 // streams))), "greedy": rng.random() < 0.3, "codebooks": rng.choice((0, 0, 0, 8, 12))}
    if kind == "ids":
        return {"kind": kind, "tokens": _log_int(rng, 4, 2000)}
    if kind == "prompts":
        return {"kind": kind, "rows": _log_int(rng, 1, 16), "words": _log_int(rng, 6, 128), "frames": _log_int(rng, 12, 125)}
    if kind == "talk":
        words = rng.randint(8, 40)
        return {"kind": kind, "words": rng.randint(2, 12), "prompt_words": words, "prompt_frames": round(words * rng.uniform(2.5, 4.5)), "codebooks": rng.choice((0, 0, 8))}
    if kind == "render":
        rows, words = rng.randint(1, 5), rng.randint(8, 20)
        return {"kind": kind, "rows": rows, "requests": rng.randint(rows, 6), "words": rng.randint(3, 7), "prompt_words": words,
                "prompt_frames": round(words * rng.uniform(2.0, 3.0))}
    if kind == "decode":
        return {"kind": kind, "frames": _log_int(rng, 2, 240), "codebooks": rng.choice((16, 16, 8))}
    if kind == "encode":
        return {"kind": kind, "frames": _log_int(rng, 2, 125)}
    return {"kind": kind, "chunks": rng.randint(1, 6), "chunk_samples": rng.randint(24000, 38400)}


# ------------------------------------------------------------------------------------------------ what a user's program has in hand
class Words:
    """A tokenizer with what Engine reads of one: an id for each word."""

    special_to_id = {"[SC]": 151900}

    def encode(self, text):
        return torch.tensor([zlib.crc32(w.encode()) % 151000 for w in text.split()] or [1], dtype=torch.long)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _model(seed):
    g, s = _generator(seed), SHAPE
    sd = {}
    for name, shape in state_dict_shapes(s).items():
        if name.endswith("norm.weight"):
            sd[name] = torch.ones(shape, device="cuda", dtype=torch.bfloat16)
        else:
            sd[name] = torch.randn(shape, device="cuda", dtype=torch.bfloat16, generator=g).mul_(0.02)
    cs, permutation = s.codebook_size, lambda: torch.randperm(s.codebook_size, device="cuda", generator=g)
    audio, code, text = (sd[n] for n in ("audio_emb.embedding.weight", "rq_transformer.code_emb.embedding.weight", "token_emb.weight"))
    for table in (audio, code):
        table.mul_(50.0)
    sd["codec_head.weight"] = torch.empty_like(audio[:cs])
    sd["codec_head.weight"][permutation()] = audio[:cs] * 0.1
    for i in range(s.n_quantizers - 1):
        sd["rq_transformer.head_W"][i, permutation()] = code[i * cs : (i + 1) * cs] * 0.1
    # a word leads to a first code as surely as a code to the next
    text.mul_(25.0).add_(audio[torch.arange(s.vocab_size, device="cuda") % cs])
    sd["eos_head.bias"] = torch.full((1,), -8.0, device="cuda")  # a turn's length is set by its text
    return VuiB200(s, sd, device="cuda", tokenizer=Words())


def _random_state(shapes, seed, gain_of):
    """Matrices ~ N(0, 1 / fan_in), scales around their usual values, so that every path of the codec is live."""
    g, out = _generator(seed), {}
    for name, shape in shapes.items():
        leaf = name.rsplit(".", 1)[-1]
        t = torch.randn(shape, device="cuda", generator=g)
        if leaf in ("alpha", "beta"):
            t = t * 0.3
        elif leaf in ("attn_scale", "mlp_scale", "gamma"):
            t = 0.5 + 0.1 * t
        elif leaf == "bias":
            t = t * 0.05
        elif len(shape) == 1:
            t = 1.0 + 0.1 * t
        elif leaf != "embed":
            t = t * gain_of(name) / math.sqrt(_fan_in(name, shape))
        out[name] = t
    return out


def _fan_in(name, shape):
    if ".block.1.conv.weight" in name and name.startswith("decoder"):
        return 2 * shape[0]  # transposed, two taps overlap
    if name.startswith("upsample") and name.endswith("0.conv.weight"):
        return shape[0]
    return math.prod(shape[1:])


def _decoder(seed):
    gain = lambda n: 0.25 if "conv2.conv.weight" in n or n == "decoder.6.conv.weight" else 1.0  # noqa: E731  audio inside the clamp
    dec = QwenCodecDecoder(_random_state(codec_param_shapes(), seed, gain))
    dec.setup_streaming_graph()
    return dec


def _encoder(seed):
    gain = lambda n: 4.0 if n.endswith("input_proj.weight") else 1.0  # noqa: E731  latents on the codebooks' scale
    return QwenCodecEncoder(_random_state(encoder_param_shapes(), seed, gain))


def _codes(seed, *shape):
    return torch.randint(0, SHAPE.codebook_size, shape, generator=torch.Generator().manual_seed(seed))


def _text(rng, words):
    """Words in sentences of seven."""
    out = []
    for i in range(words):
        w = "".join(rng.choice("bdfgklmnprstvz") + rng.choice("aeiou") for _ in range(rng.randint(1, 3)))
        out.append(w + ("." if i % 7 == 6 or i == words - 1 else ""))
    return " ".join(out)


def _sound(seed, samples):
    """Voiced sound with a syllable's rise and fall, and some noise."""
    g = _generator(seed)
    t = torch.arange(samples, device="cuda", dtype=torch.float32) / 24000.0
    f = 90.0 + 120.0 * float(torch.rand((), device="cuda", generator=g))
    a = torch.rand(12, device="cuda", generator=g)
    x = sum(a[k] / (k + 1) * torch.sin(2 * math.pi * f * (k + 1) * t) for k in range(12))
    return 0.2 * x * (0.6 + 0.4 * torch.sin(2 * math.pi * 3.0 * t)) + 0.01 * torch.randn(samples, device="cuda", generator=g)


def _cfg(case):
    return GenConfig(temperature=0.8, top_k=50, rep_penalty=1.0, n_codebooks=case["codebooks"] % SHAPE.n_quantizers)


def _room(positions):
    return 64 * -(-positions // 64)


def _prompt_lengths(case, rng):
    return [rng.randint(case["prompt_min"], case["prompt_max"]) for _ in range(case["streams"])]


@torch.inference_mode()
def prepare(case, seed):
    kind, rng = case["kind"], random.Random(seed)
    s = {"case": dict(case)}
    if kind == "frames":
        lengths = _prompt_lengths(case, rng)
        eng = Engine(model=_model(seed), max_rows=case["streams"], max_seq=_room(case["prompt_max"] + case["frames"] + 8), max_prefill_rows=1024, seed=seed)
        rows = [eng.new_row() for _ in lengths]
        ids = [_ids(seed + 1 + i, n) for i, n in enumerate(lengths)]
        hidden = eng._prefill_many([(r, eng.model.token_emb(i[None])) for r, i in zip(rows, ids)])
        for r, n in zip(rows, lengths):
            r._prompt_offset = n
        s.update(eng=eng, rows=rows, hidden=torch.stack([h[-1] for h in hidden]))
    elif kind == "ids":
        eng = Engine(model=_model(seed), max_rows=1, max_seq=_room(case["tokens"] + 8), seed=seed)
        s.update(eng=eng, rows=[eng.new_row()], ids=_ids(seed + 1, case["tokens"]))
    elif kind == "prompts":
        eng = Engine(model=_model(seed), max_rows=case["rows"], max_seq=_room(case["words"] + case["frames"] + 9), max_prefill_rows=1024, seed=seed)
        prompts = []
        for i in range(case["rows"]):  # up to an eighth shorter, each another length
            words, frames = (n - rng.randint(0, n // 8) for n in (case["words"], case["frames"]))
            prompts.append([Segment(_text(rng, words), _codes(seed + i, frames, SHAPE.n_quantizers))])
        s.update(eng=eng, rows=[eng.new_row() for _ in prompts], prompts=prompts)
    elif kind == "talk":
        eng = Engine(model=_model(seed), codec=_decoder(seed), max_rows=1, max_seq=1024, seed=seed)
        row = eng.new_row()
        row.prefill([Segment(_text(rng, case["prompt_words"]), _codes(seed, case["prompt_frames"], SHAPE.n_quantizers))])
        s.update(eng=eng, rows=[row], text=_text(rng, case["words"]))
    elif kind == "render":
        eng = Engine(model=_model(seed), codec=_decoder(seed), max_rows=case["rows"], max_seq=512, seed=seed)
        requests = [RenderRequest(segments=[Segment(_text(rng, case["prompt_words"]), _codes(seed + i, case["prompt_frames"], SHAPE.n_quantizers))],
                                  text=_text(rng, case["words"])) for i in range(case["requests"])]
        s.update(eng=eng, requests=requests)
    elif kind == "decode":
        s.update(dec=_decoder(seed), codes=_codes(seed, 1, case["codebooks"], case["frames"]).cuda())
    elif kind == "encode":
        s.update(enc=_encoder(seed), audio=_sound(seed, case["frames"] * SAMPLES)[None, None])
    else:
        listener = StreamingCodecEncoder(_encoder(seed))
        listener.setup_graph()
        s.update(listener=listener, sound=_sound(seed, case["chunks"] * case["chunk_samples"]).cpu())
    return s


def _ids(seed, n):
    return torch.randint(0, SHAPE.vocab_size, (n,), generator=torch.Generator().manual_seed(seed))


# ------------------------------------------------------------------------------------------------ one pass
@torch.inference_mode()
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frames":
        for row in s["rows"]:
            row.rewind()
        codes = s["eng"].generate_frames(s["rows"], s["hidden"], case["frames"], _cfg(case), greedy=case["greedy"])
        return {"codes": codes, **_cache(s["eng"], case["streams"], case["prompt_min"] + case["frames"] - 1)}
    if kind == "ids":
        s["rows"][0].reset()
        return {"hidden": s["eng"].prefill_ids(s["rows"][0], s["ids"]), **_cache(s["eng"], 1, case["tokens"])}
    if kind == "prompts":
        ends = []
        for row, segments in zip(s["rows"], s["prompts"]):
            row.reset()
            ends.append(row.prefill(segments))
        return {"ends": ends[0], **_cache(s["eng"], case["rows"], case["words"] - case["words"] // 8 + case["frames"] - case["frames"] // 8)}
    if kind == "talk":
        s["rows"][0].rewind()
        return torch.cat(list(s["rows"][0].stream(s["text"], GenConfig(n_codebooks=case["codebooks"]))), dim=-1)
    if kind == "render":
        return s["eng"].render_continuous(s["requests"], GenConfig())
    if kind == "decode":
        return s["dec"].decode(s["codes"])
    if kind == "encode":
        return s["enc"].encode(s["audio"])
    n, got = case["chunk_samples"], []
    s["listener"].reset()
    for i in range(case["chunks"]):
        got.append(s["listener"].feed(s["sound"][i * n : (i + 1) * n]))
    got.append(s["listener"].flush())
    return torch.cat([c for c in got if c is not None])


def _cache(eng, rows, positions):
    """The updated K/V of the last layer, which depends on all that was computed before it, where every row has some."""
    last = eng.flash_kv_caches[-1]
    return {"k": last.k_cache[:rows, :positions], "v": last.v_cache[:rows, :positions], "lengths": eng.seq_lens[:rows]}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
_LAYER = 2048 * 1024 + 1024 * 1024 + 3 * 3072 * 1024            # parameters of a backbone layer
_BACKBONE = SHAPE.n_layers * _LAYER
_HEAD = SHAPE.codebook_size * SHAPE.d_model
_DEPTH = SHAPE.rq_n_layers * (4 * 512 * 512 + 3 * 512 * SHAPE.rq_ffn)
_DEPTH_HEAD = SHAPE.codebook_size * SHAPE.rq_d_model
_KV = SHAPE.n_layers * 2 * SHAPE.n_kv_heads * SHAPE.head_dim * 2  # bytes of one position
_SCORES = SHAPE.n_layers * SHAPE.n_heads * SHAPE.head_dim * 4     # operations of one query on one key


def _generate(streams, mean_prompt, frames, codebooks):
    q = codebooks or SHAPE.n_quantizers
    weights = 2 * (_BACKBONE + _HEAD + _DEPTH + (q - 1) * _DEPTH_HEAD)
    keys = mean_prompt + frames / 2
    return {"bytes": frames * (weights + streams * (_KV * (keys + 1) + q * 3072)),
            "flops": frames * streams * (2 * (_BACKBONE + _HEAD + q * _DEPTH + (q - 1) * _DEPTH_HEAD) + _SCORES * keys)}


def _prefill(positions, mean_keys, calls=1):
    return {"bytes": calls * 2 * _BACKBONE + positions * (_KV + 2 * SHAPE.d_model),
            "flops": positions * (2 * _BACKBONE + _SCORES * mean_keys)}


def _codec_work(shapes, columns):
    """(bytes of the weights once, operations of one frame), columns(name): how many columns of a frame a matrix meets."""
    size = {n: math.prod(shape) for n, shape in shapes.items() if not n.endswith("embed")}
    return 4 * sum(v for n, v in size.items() if columns(n)), 2 * sum(v * columns(n) for n, v in size.items())


def _decoder_columns(name):
    if name.startswith("quantizer"):
        return 0 if "input_proj" in name else 1
    if name.startswith("upsample"):
        return (1, 2)[int(name[9])] * (1 if ".0.conv" in name else 2)
    if name.startswith("decoder"):
        i = int(name[8])
        out = (4, 32, 160, 640, 1920, 1920, 1920)[i]
        return (0, 4, 32, 160, 640)[i] if 1 <= i <= 4 and ".block.1." in name else out
    return 1


def _encoder_columns(name):
    if name.startswith("conv_encoder"):
        i = int(name.split(".")[2])
        return {0: 1920, 1: 1920, 3: 480, 4: 480, 6: 96, 7: 96, 9: 16, 10: 16, 12: 2, 14: 2}[i]
    return 2 if name.startswith("transformer") else 0 if "output_proj" in name else 1


def _decode(frames, calls):
    weights, ops = _codec_work(codec_param_shapes(), _decoder_columns)
    return {"bytes": calls * weights + frames * (4 * SAMPLES + 128), "flops": frames * ops}


def _encode(frames, calls):
    weights, ops = _codec_work(encoder_param_shapes(), _encoder_columns)
    books = 16 * 2048 * 256
    return {"bytes": calls * (weights + 4 * books) + frames * (4 * SAMPLES + 128), "flops": frames * (ops + 2 * books)}


def _sum(*parts):
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def _turn_frames(words, prompt_words, prompt_frames):
    return GenConfig().max_turn_frames(words, prompt_words / (prompt_frames / 12.5))


def work(case):
    kind = case["kind"]
    if kind == "frames":
        return _generate(case["streams"], (case["prompt_min"] + case["prompt_max"]) / 2, case["frames"], case["codebooks"])
    if kind == "ids":
        return _prefill(case["tokens"], case["tokens"] / 2)
    if kind == "prompts":
        each = case["words"] + case["frames"] + 1
        return _prefill(15 / 16 * each * case["rows"], each / 2, case["rows"])
    if kind == "talk":
        frames = _turn_frames(case["words"], case["prompt_words"], case["prompt_frames"])
        prompt = case["prompt_words"] + case["prompt_frames"]
        return _sum(_prefill(case["words"], prompt), _generate(1, prompt, frames, case["codebooks"]), _decode(frames, frames))
    if kind == "render":
        frames = _turn_frames(case["words"], case["prompt_words"], case["prompt_frames"])
        prompt, rows, n = case["prompt_words"] + case["prompt_frames"], case["rows"], case["requests"]
        return _sum(_prefill(n * (prompt + case["words"]), prompt / 2, n), *[_generate(b, prompt, frames, 0) for b in [rows] * (n // rows) + [n % rows] * (n % rows > 0)],
                    _decode(n * frames, n))
    if kind == "decode":
        return _decode(case["frames"], 1)
    if kind == "encode":
        return _encode(case["frames"], 1)
    return _encode(case["chunks"] * case["chunk_samples"] / SAMPLES, case["chunks"])


def tolerance(case):
    kind = case["kind"]
    if kind in ("encode", "listen"):
        return {"differ": 0.01}  # two codes equally near: the other one, and what follows from it in that frame
    if kind in ("decode", "talk", "render"):
        return {"rel": 5e-5, "max": 5e-3}  # 32-bit sums through some hundred layers
    return {"rel": 2e-2, "differ": 0.005}  # bf16 through 24 layers; a draw at the edge between two codes
