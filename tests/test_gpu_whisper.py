"""Whisper*Q on the GPU against the reference's own classes (fixture: the reference model's fp32 CPU
outputs on a toy configuration), and the CUDA-graph engine against the model classes."""
import pytest
import torch

import asrq_b200
from asrq_b200 import whisper as W
from tests.gpu_util import DEV
from tests.whisper_util import load_fixture

transformers = pytest.importorskip("transformers")
pytestmark = pytest.mark.gpu


def _model():
    cfg, sd, x, ids, logits, enc = load_fixture()
    m = W.WhisperForConditionalGenerationQ(transformers.WhisperConfig(**cfg))
    m.load_state_dict(sd)
    m = m.half().to(DEV).eval()
    return cfg, m, x, ids, logits, enc


def _close(a, ref, tol, what):
    err = float((a.float().cpu() - ref).abs().max())
    scale = float(ref.abs().max())
    assert err <= tol * scale, f"{what}: max error {err:.3e} against scale {scale:.3e}"
    return err / scale


def test_model_classes_match_reference_outputs():
    """fp16 on the GPU (LinearQ through the CUDA kernels) against the reference classes in fp32 on the CPU:
    encoder states and teacher-forced logits within 1e-2 of the largest magnitude, greedy ids equal
    wherever the reference's top-2 margin is not within the error."""
    cfg, m, x, ids, logits, enc = _model()
    with torch.no_grad():
        e = m.model.encoder(x.half().to(DEV)).last_hidden_state
        _close(e, enc, 1e-2, "encoder states")
        start = torch.full((ids.shape[0], 1), cfg["decoder_start_token_id"], dtype=torch.long)
        out = m(input_features=x.half().to(DEV), decoder_input_ids=torch.cat([start, ids[:, :-1]], 1).to(DEV)).logits
    rel = _close(out, logits, 1e-2, "teacher-forced logits")
    top2 = logits.topk(2, dim=-1).values
    margin = top2[..., 0] - top2[..., 1]
    clear = margin > 4 * rel * float(logits.abs().max())
    assert int(clear.sum()) >= clear.numel() // 2
    assert torch.equal(out.argmax(-1).cpu()[clear], ids[clear])
    asrq_b200.check_status()


def test_engine_matches_model_classes_and_reference():
    cfg, m, x, ids, logits, enc = _model()
    eng = W.WhisperEngine.from_model(m)
    e = eng.encode(x)
    _close(e, enc, 1e-2, "engine encoder states")
    steps = ids.shape[1]
    got, lg = eng.decode(e, steps, forced_ids=ids.t().contiguous(), keep_logits=True, use_graph=False)
    rel = _close(lg.transpose(0, 1), logits, 1e-2, "engine logits, teacher-forced")
    top2 = logits.topk(2, dim=-1).values
    clear = (top2[..., 0] - top2[..., 1]) > 4 * rel * float(logits.abs().max())
    assert torch.equal(got.cpu()[clear], ids[clear])
    # free-running greedy decoding: the captured graph and the eager step give the same tokens
    a = eng.generate(x, steps=steps, use_graph=False).clone()
    b = eng.generate(x, steps=steps, use_graph=True).clone()
    c = eng.generate(x, steps=steps, use_graph=True).clone()     # a second replay of the same graph
    assert torch.equal(a, b) and torch.equal(b, c)
    # and against the reference's greedy ids up to the first position where its margin was not clear
    for r in range(ids.shape[0]):
        n_clear = int((~clear[r]).nonzero()[0]) if bool((~clear[r]).any()) else steps
        assert torch.equal(a[r, :n_clear].cpu(), ids[r, :n_clear])
    asrq_b200.check_status()


def test_engine_random_init_large_width_runs_and_is_deterministic():
    """Whisper-large-v3 widths at reduced depth: the shapes the whole-model benchmark runs (d_model 1280,
    20 heads, FFN 5120, 1500 source positions), batch 4, through the graph."""
    cfg = transformers.WhisperConfig(vocab_size=51866, num_mel_bins=128, encoder_layers=2, decoder_layers=2,
                                     encoder_attention_heads=20, decoder_attention_heads=20, d_model=1280,
                                     encoder_ffn_dim=5120, decoder_ffn_dim=5120, max_source_positions=1500,
                                     max_target_positions=448, decoder_start_token_id=50258)
    eng = W.WhisperEngine.random_init(cfg, DEV, seed=0)
    gen = torch.Generator().manual_seed(0)
    x = torch.randn(4, 128, 3000, generator=gen).half()
    a = eng.generate(x, steps=8).clone()
    b = eng.generate(x, steps=8).clone()
    assert a.shape == (4, 8) and torch.equal(a, b)
    assert int(a.min()) >= 0 and int(a.max()) < 51866
    e = eng.encode(x)
    assert bool(torch.isfinite(e).all())
    # utterances are independent: a shard of the batch gives the same tokens (data-parallel split)
    c = eng.generate(x[:2], steps=8)
    assert torch.equal(c, a[:2])
    asrq_b200.check_status()


def test_engine_captures_again_for_replaced_operands():
    """The captured step is replayed only while the weights are the ones that it was captured with."""
    cfg, m, x, ids, logits, enc = _model()
    eng = W.WhisperEngine.from_model(m)
    eng.generate(x, steps=4)
    first, held = eng._graph, (eng.head, eng.dec_layers[0]["fc1"].weight)
    eng.generate(x, steps=4)
    assert eng._graph is first
    for change in (lambda: setattr(eng, "head", eng.head.flip(0).contiguous()),
                   lambda: eng.dec_layers[0]["fc1"].load_quantized_params(eng.dec_layers[0]["fc1"].scales, eng.dec_layers[0]["fc1"].zeros,
                                                                          eng.dec_layers[0]["fc1"].weight.flip(0).contiguous())):
        change()
        want = eng.generate(x, steps=4, use_graph=False).clone(), eng.logits.clone()
        got = eng.generate(x, steps=4).clone(), eng.logits.clone()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert len(held) == 2
    asrq_b200.check_status()
