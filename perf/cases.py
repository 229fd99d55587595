"""What a program built on asrq_b200 has the library do, as cases that can be timed and compared.

Four kinds, by the entry point a program calls:

* ``linear``   one packed ``LinearQ`` layer on 16-bit activations (``forward`` / ``forward_fused``): a user of the drop-in
  layer inside a model of their own.  One token up to a batch of encoder windows, 2- and 4-bit weights, both activation
  types, with the step that follows the layer in a block (GELU, residual) or without.
* ``linear_qq`` one W4A4 ``LinearQQ`` layer (online Hadamard, per-token int4 activations), one token up to a batch of windows.
* ``whisper``  ``WhisperEngine.generate``: log-mel windows in, greedy token ids out, at the Whisper-large-v3 shape.
* ``speech``   ``SpeechLM.generate``: FastConformer-shaped W4A4 encoder, Qwen3-1.7B-shaped W4A16 decoder.

Weights are seeded and random (there are no checkpoints here).  The two whole models get an output head that is a
permutation of their token embedding and an embedding large enough to lead the residual stream, so that every step's
choice is decided by a clear margin, as a trained model's is, and equal arithmetic gives equal ids.
"""
import math
import random
from types import SimpleNamespace

import torch

import asrq_b200
from asrq_b200 import conformer, packing, qwen3, whisper

DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}

# (in_features, out_features, group_size, bias) of the models' quantized layers; fused q/k/v, k/v and gate/up included
WHISPER_LAYERS = [(1280, 1280, 128, True), (1280, 2560, 128, True), (1280, 3840, 128, True), (1280, 5120, 128, True),
                  (5120, 1280, 128, True)]
QWEN_LAYERS = [(2048, 2048, 128, False), (2048, 4096, 64, False), (2048, 6144, 64, False), (2048, 12288, 128, False),
               (6144, 2048, 64, False)]
CONFORMER_LAYERS = [(1024, 1024), (1024, 4096), (4096, 1024)]

WHISPER = dict(d_model=1280, heads=20, ffn=5120, layers=32, vocab=51866, mel=128, src=1500)   # large-v3 shape
SPEECH = dict(d_model=1024, ffn=4096, enc_layers=32, mel=80, hidden=2048, inter=6144, dec_layers=28, q_heads=16, kv_heads=8,
              head_dim=128, vocab=151936, prompt=8)


def listed():
    def linear(name, k, n, m, bits=4, group=128, bias=True, dtype="f16", then="none"):
        return {"name": name, "kind": "linear", "k": k, "n": n, "m": m, "bits": bits, "group": group, "bias": bias, "dtype": dtype,
                "then": then}

    return [
        # one new token through a gate or up projection of the Qwen3 decoder: launch and call latency
        linear("linear w4 1 token", 2048, 6144, 1, group=64, bias=False),
        # sixteen sequences decoding, 2-bit down projection, bf16
        linear("linear w2 16 tokens", 6144, 2048, 16, bits=2, group=64, bias=False, dtype="bf16"),
        # a decoder batch of 32 through fc1 with its GELU
        linear("linear w4 32 tokens gelu", 1280, 5120, 32, then="gelu"),
        # the prompt of one utterance (250 frames, 8 text tokens and a start token) through a fused q/k/v, bf16
        linear("linear w4 259 tokens", 2048, 4096, 259, group=64, bias=False, dtype="bf16"),
        # one 30-second window through an encoder's fc1
        linear("linear w4 1500 tokens", 1280, 5120, 1500),
        # 32 windows through fc2 with the residual
        linear("linear w4 48000 tokens res", 5120, 1280, 48000, then="residual"),
        # one 20-second utterance through the first feed-forward layer of a FastConformer block
        {"name": "w4a4 250 tokens", "kind": "linear_qq", "k": 1024, "n": 4096, "m": 250, "bias": True, "dtype": "f16"},
        # sixteen 30-second utterances through the second
        {"name": "w4a4 6000 tokens", "kind": "linear_qq", "k": 4096, "n": 1024, "m": 6000, "bias": True, "dtype": "f16"},
        # one utterance, as an interactive user sends it
        {"name": "whisper 1 window", "kind": "whisper", "batch": 1, "steps": 64},
        # a full batch of windows, as bulk transcription runs
        {"name": "whisper 32 windows", "kind": "whisper", "batch": 32, "steps": 128},
        {"name": "speech 1 utterance", "kind": "speech", "batch": 1, "frames": 2000, "steps": 64},
        {"name": "speech 64 utterances", "kind": "speech", "batch": 64, "frames": 2000, "steps": 200},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random):
    p = rng.random()
    if p < 0.45:
        k, n, group, bias = rng.choice(WHISPER_LAYERS + QWEN_LAYERS)
        m = _log(rng, 1, 48000)
        return {"kind": "linear", "k": k, "n": n, "m": m, "bits": rng.choice((4, 4, 2)), "group": group, "bias": bias,
                "dtype": rng.choice(("f16", "f16", "bf16")), "then": rng.choice(("none", "none", "gelu", "residual"))}
    if p < 0.7:
        k, n = rng.choice(CONFORMER_LAYERS)
        return {"kind": "linear_qq", "k": k, "n": n, "m": _log(rng, 1, 16000), "bias": True, "dtype": rng.choice(("f16", "f16", "bf16"))}
    if p < 0.85:
        return {"kind": "whisper", "batch": _log(rng, 1, 32), "steps": rng.randint(16, 128)}
    return {"kind": "speech", "batch": _log(rng, 1, 64), "frames": rng.randint(400, 2000), "steps": rng.randint(16, 200)}


# ---- what a program has in hand before the call --------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weight(gen, n, k):
    """N(0, 0.02) with one value in a thousand ten times larger."""
    w = torch.randn(n, k, generator=gen, device="cuda") * 0.02
    return torch.where(torch.rand(n, k, generator=gen, device="cuda") < 1e-3, w * 10, w)


def _prepare_linear(c, seed):
    gen, dt = _gen(seed), DTYPES[c["dtype"]]
    m, n, k = c["m"], c["n"], c["k"]
    layer = asrq_b200.LinearQ(k, n, c["bits"], c["group"], bias=c["bias"]).cuda()
    weight, scales, zeros = packing.rtn_pack_cuda(_weight(gen, n, k).half(), c["bits"], c["group"])
    layer.load_quantized_params(scales, zeros, weight)
    if c["bias"]:
        layer.bias = (torch.randn(n, generator=gen, device="cuda") * 0.02).half()
    x = torch.randn(m, k, generator=gen, device="cuda").to(dt)
    residual = torch.randn(m, n, generator=gen, device="cuda").to(dt) if c["then"] == "residual" else None
    return {"kind": "linear", "layer": layer, "x": x, "residual": residual, "then": c["then"]}


def _prepare_linear_qq(c, seed):
    gen, dt = _gen(seed), DTYPES[c["dtype"]]
    m, n, k = c["m"], c["n"], c["k"]
    layer = asrq_b200.LinearQQ(k, n, 4, 4, 128, bias=c["bias"]).cuda()
    weight, scales = packing.pack_w4a4_cuda(_weight(gen, n, k), 128, True)
    layer.load_quantized_params(scales, torch.zeros_like(scales), weight)
    if c["bias"]:
        layer.bias = (torch.randn(n, generator=gen, device="cuda") * 0.02).half()
    # activations with heavy tails (Student t, 4 degrees of freedom) and eight outlier channels
    x = torch.randn(m, k, generator=gen, device="cuda")
    chi2 = sum(torch.randn(m, k, generator=gen, device="cuda").square_() for _ in range(4))
    x = x / (chi2 / 4).sqrt_()
    x[:, torch.randperm(k, generator=gen, device="cuda")[:8]] *= 20
    return {"kind": "linear_qq", "layer": layer, "x": x.to(dt)}


_models = {}   # the two whole models: a program loads its model once and keeps it


def _decided(engine, gen):
    """Embedding of unit size, output head = the embedding's rows in another order: each token's successor is clear."""
    e = engine.embed
    engine.head = e[torch.randperm(e.shape[0], generator=gen, device=e.device)].contiguous()
    engine.embed = e * 50


def _whisper():
    if "whisper" not in _models:
        w = WHISPER
        cfg = SimpleNamespace(vocab_size=w["vocab"], num_mel_bins=w["mel"], encoder_layers=w["layers"], decoder_layers=w["layers"],
                              encoder_attention_heads=w["heads"], decoder_attention_heads=w["heads"], d_model=w["d_model"],
                              encoder_ffn_dim=w["ffn"], decoder_ffn_dim=w["ffn"], max_source_positions=w["src"],
                              max_target_positions=448, decoder_start_token_id=50258)
        eng = whisper.WhisperEngine.random_init(cfg, "cuda", seed=0, bits=4, group_size=128)
        _decided(eng, _gen(1))
        _models["whisper"] = eng
    return _models["whisper"]


def _speech():
    if "speech" not in _models:
        s = SPEECH
        enc = conformer.FastConformerStandIn("cuda", n_layers=s["enc_layers"], d_model=s["d_model"], ffn=s["ffn"], mel=s["mel"], seed=0)
        cfg = SimpleNamespace(vocab_size=s["vocab"], hidden_size=s["hidden"], intermediate_size=s["inter"], num_hidden_layers=s["dec_layers"],
                              num_attention_heads=s["q_heads"], num_key_value_heads=s["kv_heads"], head_dim=s["head_dim"],
                              rms_norm_eps=1e-6, tie_word_embeddings=True, rope_theta=1000000.0)
        dec = qwen3.Qwen3Engine.random_init(cfg, "cuda", seed=1, bits=4, group_size=128)
        _decided(dec, _gen(2))
        _models["speech"] = conformer.SpeechLM(enc, dec, prompt_tokens=s["prompt"], seed=0)
    return _models["speech"]


def prepare(case, seed):
    if case["kind"] == "linear":
        return _prepare_linear(case, seed)
    if case["kind"] == "linear_qq":
        return _prepare_linear_qq(case, seed)
    if case["kind"] == "whisper":
        model, shape = _whisper(), (case["batch"], WHISPER["mel"], 2 * WHISPER["src"])
    else:
        model, shape = _speech(), (case["batch"], SPEECH["mel"], case["frames"])
    x = torch.randn(*shape, generator=_gen(seed), device="cuda").half()   # log-mel features, normalised
    return {"kind": case["kind"], "model": model, "x": x, "steps": case["steps"]}


# ---- one pass ------------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "linear":
        if state["then"] == "none":
            return state["layer"](state["x"])
        return state["layer"].forward_fused(state["x"], residual=state["residual"], gelu=state["then"] == "gelu")
    if kind == "linear_qq":
        return state["layer"](state["x"])
    model = state["model"]
    ids = model.generate(state["x"], steps=state["steps"])
    # the ids, and the last step's logits, which depend on everything that was cached before
    return {"ids": ids, "logits": model.logits if kind == "whisper" else model.dec.last_logits}


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _linear_work(m, n, k, bits, group, bias=False, residual=False):
    return {"bytes": 2 * m * k + n * k * bits // 8 + 4 * n * (k // group) + (2 * n if bias else 0) + 2 * m * n * (2 if residual else 1),
            "flops": 2 * m * n * k}


def work(case):
    if case["kind"] == "linear":
        return _linear_work(case["m"], case["n"], case["k"], case["bits"], case["group"], case["bias"], case["then"] == "residual")
    if case["kind"] == "linear_qq":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * m * k + n * k // 2 + 2 * n * (k // 128) + 2 * n + 2 * m * n, "flops": 2 * m * n * k + m * k * int(math.log2(k))}
    b, steps = case["batch"], case["steps"]
    # Weights and caches are read once per token: the next token needs this one's, and they exceed what the chip holds.
    q4 = 0.5 + 4 / 128   # bytes of a packed weight with its share of the group's scale and zero
    if case["kind"] == "whisper":
        d, f, nl, src, v = WHISPER["d_model"], WHISPER["ffn"], WHISPER["layers"], WHISPER["src"], WHISPER["vocab"]
        enc_w, dec_w, xkv_w = nl * (4 * d * d + 2 * d * f), nl * (6 * d * d + 2 * d * f), nl * 2 * d * d
        conv = 3 * d * WHISPER["mel"] * 2 + 3 * d * d
        flops = 2 * b * src * (enc_w + xkv_w + conv) + 4 * b * src * src * d * nl
        flops += steps * (2 * b * (dec_w + v * d) + 4 * b * d * nl * (src + steps / 2))
        nbytes = 2 * b * WHISPER["mel"] * 2 * src + (enc_w + xkv_w) * q4 + 4 * b * src * d * nl
        nbytes += steps * (dec_w * q4 + 2 * v * d + 4 * b * d * nl * (src + steps / 2))
        return {"bytes": nbytes, "flops": flops}
    s = SPEECH
    d, f, h, i, v = s["d_model"], s["ffn"], s["hidden"], s["inter"], s["vocab"]
    t = -(-case["frames"] // 8)
    p = t + s["prompt"]
    kv = s["kv_heads"] * s["head_dim"]
    enc_w, dec_w = s["enc_layers"] * (4 * d * f + 4 * d * d), s["dec_layers"] * (h * (h + 2 * kv) + h * h + 3 * h * i)
    enc_pw = s["enc_layers"] * 3 * d * d                      # pointwise convolutions, 16-bit
    flops = 2 * b * t * (enc_w + enc_pw) + 4 * b * t * t * d * s["enc_layers"] + 2 * b * p * dec_w + 2 * b * p * p * h * s["dec_layers"]
    flops += steps * (2 * b * (dec_w + v * h) + 4 * b * h * s["dec_layers"] * (p + steps / 2))
    nbytes = 2 * b * s["mel"] * case["frames"] + enc_w * (0.5 + 2 / 128) + 2 * enc_pw + 4 * b * p * kv * s["dec_layers"]
    nbytes += steps * (dec_w * q4 + 2 * v * h + 4 * b * kv * s["dec_layers"] * (p + steps / 2))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] in ("linear", "linear_qq"):
        # one rounding of the result; in bf16 the weights may be rounded to it too
        return {"rel": 1e-3, "max": 1e-2} if case["dtype"] == "f16" else {"rel": 1e-2, "max": 5e-2}
    if case["kind"] == "whisper":
        return {"rel": 1e-2, "max": 1e-1, "differ": 0.01}      # fp16 through 64 layers
    # 4-bit activations: where a value sits on the edge between two codes, a last-place difference moves it by a code
    return {"rel": 2e-2, "max": 2e-1, "differ": 0.01}
