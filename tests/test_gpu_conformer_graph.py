"""The encoder's joined layers and captured shapes give the blocks' own bits, and step aside for replaced parameters."""
import threading

import pytest
import torch

from asrq_b200 import conformer as C

pytestmark = pytest.mark.gpu


def _feats(b, frames, seed=5):
    return torch.randn(b, 80, frames, generator=torch.Generator().manual_seed(seed)).half().cuda()


@pytest.mark.parametrize("b,frames", [(1, 400), (2, 600), (3, 1001)])
def test_encode_is_the_blocks_bit_for_bit(b, frames):
    enc = C.FastConformerStandIn("cuda", n_layers=3, d_model=256, ffn=1024, heads=4, mel=80, sub_channels=64, seed=4)
    plain = lambda f: enc.encode(f, hook=lambda *_: None)  # noqa: E731
    for seed in (5, 6, 7):  # eager, captured, replayed
        assert torch.equal(enc.encode(_feats(b, frames, seed)), plain(_feats(b, frames, seed)))
    assert len(enc._graphs) == 1
    q = enc.layers[1]["q"]
    q.scales.mul_(2)                               # in place: the rows of the joined buffer too
    assert enc._joined_ok() and torch.equal(enc.encode(_feats(b, frames)), plain(_feats(b, frames)))
    q.load_quantized_params(q.scales * 2, q.zeros, q.weight.clone())
    assert not enc._joined_ok() and torch.equal(enc.encode(_feats(b, frames)), plain(_feats(b, frames)))


def test_a_captured_shape_keeps_its_derived_operands(monkeypatch):
    """Operands derived anew (another 8-bit form in between) are other memory: the captured encode is not replayed over what
    the first ones left, and an unchanged encoder captures once."""
    enc = C.FastConformerStandIn("cuda", n_layers=2, d_model=256, ffn=512, heads=4, mel=80, sub_channels=64, seed=4)
    f = _feats(1, 800)
    want = [enc.encode(f) for _ in range(4)][0]
    graph = next(iter(enc._graphs.values()))["graph"]
    enc.encode(f)
    assert next(iter(enc._graphs.values()))["graph"] is graph
    with monkeypatch.context() as m:
        m.setattr(C.LinearQQ, "operand", "int8")
        assert torch.equal(enc.encode(_feats(1, 960)), enc.encode(_feats(1, 960), hook=lambda *_: None))
    torch.cuda.synchronize()
    junk = [torch.full((256 * n,), 77, dtype=torch.uint8, device="cuda") for n in (256, 512, 768) for _ in range(32)]
    assert torch.equal(enc.encode(f), want) and len(junk) == 96


def test_captured_shapes_are_bounded_and_shared_by_streams():
    enc = C.FastConformerStandIn("cuda", n_layers=2, d_model=256, ffn=512, heads=4, mel=80, sub_channels=64, seed=4)
    for frames in range(400, 400 + 16 * (enc.graph_shapes + 2), 16):
        for _ in range(2):
            enc.encode(_feats(1, frames))
    assert len(enc._graphs) == enc.graph_shapes
    f = [_feats(2, 800, s) for s in range(4)]
    want = [enc.encode(x, hook=lambda *_: None) for x in f]
    enc.encode(f[0])
    bad = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(10):
                y = enc.encode(f[i])
                torch.cuda.current_stream().synchronize()
                if not torch.equal(y, want[i]):
                    bad.append(i)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
