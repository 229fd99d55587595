"""Kernels that start while the one before them still runs (programmatic dependent launch) read what that one writes, and not what
was there before: every kind of kernel behind a layer whose output is new in every call, in memory that is used again and again,
against the same calls one after the other."""
import pytest
import torch

import asrq_b200
from asrq_b200 import linear, packing
from gpu_util import DEV, lib_option

pytestmark = pytest.mark.gpu
CALLS = 64


def _layer(k, n, group, bits=4):
    gen = torch.Generator(device=DEV).manual_seed(k + n)
    layer = asrq_b200.LinearQ(k, n, bits, group, bias=False).to(DEV)
    weight, scales, zeros = packing.rtn_pack_cuda((torch.randn(n, k, generator=gen, device=DEV) * 0.02).half(), bits, group)
    layer.load_quantized_params(scales, zeros, weight)
    return layer


def _consumers(dtype):
    """name -> (rows, width of the layer's output, what follows it)."""
    gen = torch.Generator(device=DEV).manual_seed(5)

    def rand(*shape):
        return torch.randn(*shape, generator=gen, device=DEV).to(dtype)
    out = {}
    for rows, dim in ((4, 1280), (400, 1280), (4, 1008), (400, 1008)):  # a block, a warp of vectors and a warp of values per row
        gamma, beta = rand(dim), rand(dim)
        out[f"layer norm {rows}x{dim}"] = rows, dim, lambda h, gamma=gamma, beta=beta: linear.add_layernorm(h, h, gamma, beta)[1]
    for rows, dim in ((4, 2048), (400, 2048), (400, 1008)):
        gamma = rand(dim)
        out[f"rms norm {rows}x{dim}"] = rows, dim, lambda h, gamma=gamma: linear.add_rmsnorm(h, h, gamma)[1]
    out["silu"] = 4, 4096, linear.silu_mul
    cos, sin, qw, kw = rand(8, 128), rand(8, 128), rand(128), rand(128)

    def rope(h):
        k, v = torch.zeros(2, 4, 2, 8, 128, dtype=dtype, device=DEV)
        return torch.cat([linear.qk_norm_rope(h, qw, kw, cos, sin, k, v, 3, 4, 1, 4, 2, 1e-6).reshape(-1), k.reshape(-1), v.reshape(-1)])
    out["norm and rotary embedding"] = 4, 8 * 128, rope
    head = rand(5001, 1280)
    out["head"] = 4, 1280, lambda h: linear.dense_head(h, head)
    scratch = torch.zeros(8, dtype=torch.int64, device=DEV)

    def argmax(h):
        tokens = torch.empty(4, dtype=torch.int64, device=DEV)
        linear.argmax_rows(h, tokens, scratch)
        return tokens
    out["argmax"] = 4, 5120, argmax
    out["argmax of an odd width"] = 4, 5120, lambda h: argmax(h.reshape(-1)[:4 * 5119].reshape(4, 5119))
    after = {"split K": _layer(1024, 512, 256), "decode": _layer(1024, 512, 128)}
    for name, layer in after.items():
        out[name] = 4, 1024, layer
    out["decode of 12 rows"] = 12, 1024, after["decode"]   # (from three rows on, a small layer starts the next launch behind its own wait)
    residual = rand(4, 512)
    out["residual pass"] = 4, 1024, lambda h: after["split K"].forward_fused(h, residual=residual, gelu=True)
    return out


NAMES = ["layer norm 4x1280", "layer norm 400x1280", "layer norm 4x1008", "layer norm 400x1008", "rms norm 4x2048", "rms norm 400x2048",
         "rms norm 400x1008", "silu", "norm and rotary embedding", "head", "argmax", "argmax of an odd width", "split K", "decode",
         "decode of 12 rows", "residual pass"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_reads_what_the_kernel_before_wrote(name, dtype):
    rows, width, then = _consumers(dtype)[name]
    layer = _layer(4096, width, 128)
    xs = torch.randn(CALLS, rows, 4096, device=DEV).to(dtype)
    torch.cuda.synchronize()
    with lib_option("no_pdl", 1):
        want = [then(layer(x)) for x in xs]
    torch.cuda.synchronize()
    for _ in range(4):
        got = [then(layer(x)) for x in xs]                 # (the layer's output: one block of the allocator's, over and over)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        then(layer(xs[0]))                                 # the stream's workspace exists
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = [then(layer(x)) for x in xs]
    for _ in range(4):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    asrq_b200.check_status()
