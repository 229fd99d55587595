"""The module calls' native host path against the Python one: same bits, the same errors, and it sees replaced and
modified buffers."""
import pytest
import torch

import asrq_b200
from asrq_b200 import linear, packing
from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


def _layers(k, n, bias, seed=0):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    w = torch.randn(n, k, generator=gen, device=DEV) * 0.02
    q = asrq_b200.LinearQ(k, n, 4, 128, bias=bias).to(DEV)
    weight, scales, zeros = packing.rtn_pack_cuda(w.half(), 4, 128)
    q.load_quantized_params(scales, zeros, weight)
    qq = asrq_b200.LinearQQ(k, n, 4, 4, 128, bias=bias).to(DEV)
    weight, scales = packing.pack_w4a4_cuda(w, 128, True)
    qq.load_quantized_params(scales, torch.zeros_like(scales), weight)
    if bias:
        q.bias = torch.randn(n, generator=gen, device=DEV).half()
        qq.bias = q.bias
    torch.cuda.synchronize()
    return q, qq


def _python(monkeypatch, call):
    with monkeypatch.context() as m:
        m.setattr(linear, "_native", None)
        return call()


@pytest.mark.parametrize("m", [1, 5, 16, 33, 63, 64, 300])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bias", [True, False])
def test_native_call_gives_the_python_path_bits(m, dtype, bias, monkeypatch):
    q, qq = _layers(512, 256, bias)
    x = torch.randn(m, 512, device=DEV).to(dtype)
    r = torch.randn(m, 256, device=DEV).to(dtype)
    for call in (lambda: q(x), lambda: q.forward_fused(x, residual=r), lambda: q.forward_fused(x, gelu=True), lambda: qq(x)):
        _python(monkeypatch, call)                      # workspace and prepared weight exist
        before = linear._native.calls()
        y = call()
        assert linear._native.calls() > before          # and it was the native path that ran
        assert torch.equal(y, _python(monkeypatch, call))
    assert q(x.view(1, m, 512)).shape == (1, m, 256)
    asrq_b200.check_status()


def test_replaced_and_modified_buffers_are_seen():
    q, qq = _layers(512, 256, True)
    q2, qq2 = _layers(512, 256, True, seed=1)
    x = torch.randn(80, 512, device=DEV).half()
    q(x), qq(x)
    q.load_quantized_params(q2.scales, q2.zeros, q2.weight)
    q.bias = q2.bias
    assert torch.equal(q(x), q2(x))
    qq.weight.copy_(qq2.weight)                         # in place: the derived 8-bit operand is stale
    qq.scales, qq.bias = qq2.scales, qq2.bias
    torch.cuda.synchronize()
    assert torch.equal(qq(x), qq2(x))


def test_unusual_calls_go_the_python_way():
    q, qq = _layers(512, 256, True)
    x = torch.randn(512, 6, device=DEV).half().t()      # not contiguous
    assert torch.equal(q(x), q(x.contiguous())) and torch.equal(qq(x), qq(x.contiguous()))
    assert q(x[:0]).shape == (0, 256) and qq(x[:0]).shape == (0, 256)
    with pytest.raises(TypeError):
        q(x.float())
    with pytest.raises(ValueError):
        q(x[:, :256])
    with pytest.raises(RuntimeError, match="no CPU path"):
        qq(x.cpu())
    with pytest.raises(ValueError):
        q.forward_fused(x.contiguous(), residual=x.contiguous())
    q.group_size = 96                                   # the library's own refusal
    with pytest.raises(asrq_b200._lib.AsrqError):
        q(x.contiguous())
