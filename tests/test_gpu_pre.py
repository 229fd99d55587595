"""A layer with the step ahead of it in the same kernel (asrq_linearq_a16_pre): the norm of one or two rows, silu(gate) * up of one."""
import weakref

import pytest
import torch

import asrq_b200
from asrq_b200 import _lib, linear, packing, qwen3, whisper
from asrq_b200.linear import PRE_LAYERNORM, PRE_RMSNORM, PRE_SILU_MUL, linear_after
from gpu_util import DEV
from tests.qwen3_util import toy_models

pytestmark = pytest.mark.gpu


def _layer(k, n, bits, group, bias=True):
    gen = torch.Generator(device=DEV).manual_seed(k + n + bits)
    layer = asrq_b200.LinearQ(k, n, bits, group, bias=bias).to(DEV)
    w, s, z = packing.rtn_pack_cuda((torch.randn(n, k, generator=gen, device=DEV) * 0.02).half(), bits, group)
    layer.load_quantized_params(s, z, w)
    if bias:
        layer.bias = (torch.randn(n, generator=gen, device=DEV) * 0.02).half()
    return layer, gen


SHAPES = [(1280, 1280, 128, 4), (1280, 3840, 128, 4), (1280, 5120, 128, 4), (2048, 4096, 64, 4), (2048, 12288, 128, 4), (512, 48, 32, 4),
          (1280, 1280, 256, 2), (2048, 2048, 64, 2), (1280, 5120, 128, 2)]


@pytest.mark.parametrize("k,n,group,bits", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows", [1, 2])
@pytest.mark.parametrize("pre", [PRE_LAYERNORM, PRE_RMSNORM])
def test_norm_ahead(k, n, group, bits, dtype, rows, pre):
    layer, gen = _layer(k, n, bits, group)
    x = torch.randn(rows, k, generator=gen, device=DEV) + 0.5
    x[:, 3] = 300.0                                   # a channel that carries most of the row, as residual streams have
    x = x.to(dtype)
    g = (1 + 0.1 * torch.randn(k, generator=gen, device=DEV)).to(dtype)
    b = (0.1 * torch.randn(k, generator=gen, device=DEV)).to(dtype)
    r = torch.randn(rows, n, generator=gen, device=DEV).to(dtype)
    h = asrq_b200.add_layernorm(x, None, g, b, 1e-5)[1] if pre == PRE_LAYERNORM else asrq_b200.add_rmsnorm(x, None, g, 1e-6)[1]
    for kw in ({}, {"gelu": True}, {"residual": r}):
        y = linear_after(layer, pre, x, g, b if pre == PRE_LAYERNORM else None, 1e-5 if pre == PRE_LAYERNORM else 1e-6, **kw)
        assert y is not None
        assert torch.equal(y, layer.forward_fused(h, **kw)), kw  # the same statistics, the same split of K: the same bits


@pytest.mark.parametrize("k,n,group,bits", [(6144, 2048, 64, 4), (6144, 2048, 128, 4), (2048, 2048, 128, 2), (512, 48, 32, 4)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_silu_ahead_has_the_bits_of_two_calls(k, n, group, bits, dtype):
    layer, gen = _layer(k, n, bits, group, bias=False)
    gu = (4 * torch.randn(1, 2 * k, generator=gen, device=DEV)).to(dtype)
    gu[0, :8] = torch.tensor([-87.6, -88.4, 80.0, -20.0, 0.0, -0.0, 11.0, -1e-4], device=DEV)
    r = torch.randn(1, n, generator=gen, device=DEV).to(dtype)
    y = linear_after(layer, PRE_SILU_MUL, gu, residual=r)
    x = asrq_b200.silu_mul(gu)
    assert torch.equal(y, layer.forward_fused(x, residual=r))


def test_what_is_not_covered_is_left_to_the_caller():
    layer, gen = _layer(1280, 1280, 4, 128)
    x = torch.randn(3, 1280, generator=gen, device=DEV).half()
    g = torch.ones(1280, device=DEV, dtype=torch.float16)
    assert linear_after(layer, PRE_LAYERNORM, x, g, g, 1e-5) is None                                 # three rows
    assert linear_after(layer, PRE_LAYERNORM, x[:2].t().contiguous().t(), g, g, 1e-5) is None        # strided rows
    assert linear_after(layer, PRE_SILU_MUL, torch.randn(2, 2560, device=DEV).half()) is None        # two rows of gate and up
    assert linear_after(layer, PRE_LAYERNORM, x[:1].float(), g, g, 1e-5) is None
    with pytest.raises(_lib.AsrqError):
        _lib.call("asrq_linearq_a16_pre", 4, PRE_RMSNORM, x.data_ptr(), g.data_ptr(), None, 1e-5, layer.weight.data_ptr(), layer.scales.data_ptr(),
                  layer.zeros.data_ptr(), None, None, x.data_ptr(), 3, 1280, 1280, 128, _lib.F16, 0, torch.cuda.current_stream().cuda_stream)


class _Doubling(asrq_b200.LinearQ):
    def forward(self, input):
        return 2 * super().forward(input)


def test_a_layer_that_does_more_than_its_product_is_called():
    layer, gen = _layer(1280, 1280, 4, 128)
    x = torch.randn(1, 1280, generator=gen, device=DEV).half()
    norm = whisper._Norm(torch.ones(1280, device=DEV).half(), torch.zeros(1280, device=DEV).half())
    want = layer(norm(x))
    assert torch.equal(whisper._norm_then(norm, layer, x), want)
    seen = []
    hook = layer.register_forward_hook(lambda m, i, o: seen.append(o))
    assert linear_after(layer, PRE_LAYERNORM, x, norm.w, norm.b, norm.eps) is None
    assert torch.equal(whisper._norm_then(norm, layer, x), want) and len(seen) == 1
    hook.remove()
    layer.__class__ = _Doubling
    assert torch.equal(whisper._norm_then(norm, layer, x), 2 * want)
    assert torch.equal(whisper._norm_then(torch.nn.Identity(), torch.nn.Flatten(), x), x)   # neither the engine's own


@pytest.mark.parametrize("name", ["qkv", "o", "gu", "down"])
def test_qwen_step_of_one_sequence_runs_the_hooks_of_its_layers(name):
    _, _, model = toy_models()
    eng = qwen3.Qwen3Engine.from_model(model.half().to(DEV))
    emb = torch.randn(1, 5, eng.embed.shape[1], generator=torch.Generator().manual_seed(0)).half().to(DEV)
    want = eng.generate(emb, 3, use_graph=False).clone()
    calls = []
    eng.layers[0][name].register_forward_hook(lambda m, i, o: calls.append(o.shape))
    assert torch.equal(eng.generate(emb, 3, use_graph=False), want)
    assert len(calls) == 3                                                                  # the prompt and two steps


def test_the_query_is_asked_on_the_tensors_device(monkeypatch):
    """asrq_linearq_a16_pre_covers answers for the current device, as asrq_linearq_a16_pre runs on it."""
    layer, gen = _layer(1280, 1280, 4, 128)
    x, g = torch.randn(1, 1280, generator=gen, device=DEV).half(), torch.ones(1280, device=DEV, dtype=torch.float16)
    inside, asked = [], []

    class OnDevice(linear._on_device):
        def __enter__(self):
            inside.append(self.idx)
            return super().__enter__()

        def __exit__(self, *exc):
            inside.pop()
            return super().__exit__(*exc)

    class Lib:
        def __getattr__(self, name):
            fn = getattr(lib, name)
            return (lambda *a: asked.append(list(inside)) or fn(*a)) if name == "asrq_linearq_a16_pre_covers" else fn
    lib = _lib.load()
    monkeypatch.setattr(linear, "_on_device", OnDevice)
    monkeypatch.setattr(_lib, "load", Lib)
    assert linear_after(layer, PRE_LAYERNORM, x, g, g, 1e-5) is not None
    assert asked == [[x.device.index]]


@pytest.mark.parametrize("way", ["linear_after", "forward_fused"])
def test_operands_are_held_while_the_library_is_called(way, monkeypatch):
    """Another thread may replace a layer's buffers during the call: those whose addresses were passed stay."""
    layer, gen = _layer(1280, 1280, 4, 128)
    x, g = torch.randn(1, 1280, generator=gen, device=DEV).half(), torch.ones(1280, device=DEV, dtype=torch.float16)
    names, gone, call = ("weight", "scales", "zeros", "bias"), [], _lib.call

    def replacing(name, *args):
        for n in names:
            old = weakref.ref(getattr(layer, n))
            setattr(layer, n, getattr(layer, n).clone())
            if old() is None:
                gone.append(n)
        return call(name, *args)
    layer(x)                                          # the stream's workspace exists
    monkeypatch.setattr(linear, "_native", None)
    monkeypatch.setattr(_lib, "call", replacing)
    if way == "linear_after":
        assert linear_after(layer, PRE_LAYERNORM, x, g, g, 1e-5) is not None
    else:
        layer.forward_fused(x, gelu=True)
    assert not gone
