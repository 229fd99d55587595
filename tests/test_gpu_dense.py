"""Large W{2,4}A16 calls that dequantise the weights once (csrc/gemm_a16_dense.cu): the same bits as the kernels that unpack inside
the GEMM, at the edges of its tiles and of its shares of a round."""
import threading

import pytest
import torch

import asrq_b200
from asrq_b200 import _lib, packing
from gpu_util import CANARY, DEV, check_canary, lib_option, padded

pytestmark = pytest.mark.gpu


def _layer(k, n, bits, group, bias):
    gen = torch.Generator(device=DEV).manual_seed(k + n + bits)
    layer = asrq_b200.LinearQ(k, n, bits, group, bias=bias).to(DEV)
    w, s, z = packing.rtn_pack_cuda((torch.randn(n, k, generator=gen, device=DEV) * 0.02).half(), bits, group)
    layer.load_quantized_params(s, z, w)
    if bias:
        layer.bias = (torch.randn(n, generator=gen, device=DEV) * 0.02).half()
    return layer, gen


# one K block; a single narrow tile; tiles of 256 with half a one left; more than one round with a ragged rest; 128 features beyond 256s
@pytest.mark.parametrize("k,n,group", [(64, 128, 64), (128, 256, 64), (640, 1408, 128), (1280, 5120, 128), (2048, 2048, 64)])
@pytest.mark.parametrize("m", [17, 31, 128, 257, 1500, 6001])
@pytest.mark.parametrize("bits,dtype", [(4, torch.float16), (2, torch.bfloat16), (4, torch.bfloat16), (2, torch.float16)])
def test_same_bits_as_unpacking_inside(m, k, n, group, bits, dtype):
    layer, gen = _layer(k, n, bits, group, bias=m != 31)
    asrq_b200.linear._workspace(torch.device(DEV), _lib.workspace_bytes(_lib.WS_LINEARQ, 1 << 14, n, k))
    x = torch.randn(m, k, generator=gen, device=DEV).to(dtype)
    r = torch.randn(m, n, generator=gen, device=DEV).to(dtype)
    times = -(-512 // m)  # few tokens go to other kernels: the reference takes the rows several times over
    for kw in ({}, {"gelu": True}, {"residual": r}, {"gelu": True, "residual": r}):
        with lib_option("tc_pair", 0), lib_option("mid_kernel", 1), lib_option("tc_split", 1):
            rep = {q: v.repeat(times, 1) if q == "residual" else v for q, v in kw.items()}
            want = layer.forward_fused(x.repeat(times, 1), **rep)[:m]
        with lib_option("tc_pair", 2):
            assert _scratch_bytes(m, n, k, group) == 2 * n * k
            got = layer.forward_fused(x, **kw)
        assert torch.equal(got, want), kw
    asrq_b200.check_status()


def _scratch_bytes(m, n, k, group, act=_lib.ACT_NONE, residual=False):
    return _lib.load().asrq_linearq_a16_scratch_bytes(m, n, k, group, act, residual)


@pytest.mark.parametrize("room", [None, 2 * 5120 * 1280 - 16, 2 * 5120 * 1280])
def test_a_call_without_scratch_unpacks_inside(room):
    """No scratch, or too little for the 16-bit weights: the kernels that unpack in the GEMM, with the same bits.  The scratch is
    written up to its end and not beyond."""
    layer, gen = _layer(1280, 5120, 4, 128, True)
    x = torch.randn(6000, 1280, generator=gen, device=DEV).half()
    want = layer(x)
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device=DEV)
    assert _scratch_bytes(6000, 5120, 1280, 128) == 2 * 5120 * 1280
    scratch = padded((room,), torch.uint8, fill=CANARY) if room else None
    got = torch.empty_like(want)
    operands = (x.data_ptr(), layer.weight.data_ptr(), layer.scales.data_ptr(), layer.zeros.data_ptr(), layer.bias.data_ptr())
    _lib.call("asrq_linearq_a16_scratch", 4, *operands, None, got.data_ptr(), 6000, 5120, 1280, 128, _lib.F16, _lib.ACT_NONE, ws.data_ptr(), ws.numel(),
              scratch.data_ptr() if room else None, room or 0, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(got, want)
    if room:
        check_canary(scratch, "scratch")
        assert bool((scratch == CANARY).all()) == (room < 2 * 5120 * 1280)
    got.zero_()
    _lib.call("asrq_linearq_a16", 4, *operands, got.data_ptr(), 6000, 5120, 1280, 128, _lib.F16, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert torch.equal(got, want)


def test_scratch_is_asked_for_where_it_is_used():
    """The query and the dispatch are one rule: nothing for calls that unpack inside."""
    assert _scratch_bytes(48000, 1280, 5120, 128, residual=True) == 2 * 1280 * 5120
    assert _scratch_bytes(1500, 5120, 1280, 128) == 0          # the pair kernel's
    assert _scratch_bytes(48000, 1280, 5120, 96) == 0          # not a group size of this form
    assert _scratch_bytes(48000, 1280, 5120, 32) == 0
    assert [_scratch_bytes(m, 1280, 5120, 128) for m in (0, 1, 16, 17, 33, 767)] == [0] * 6
    with lib_option("tc_pair", 0):
        assert _scratch_bytes(48000, 1280, 5120, 128) == 0
    with lib_option("tc_pair", 2):
        assert _scratch_bytes(17, 1280, 5120, 128) == 2 * 1280 * 5120 and _scratch_bytes(16, 1280, 5120, 128) == 0


@pytest.mark.parametrize("native", [True, False])
def test_no_memory_for_scratch_is_no_error(native, monkeypatch):
    layer, gen = _layer(2048, 12288, 4, 128, True)
    x = torch.randn(2000, 2048, generator=gen, device=DEV).half()
    want = layer(x)
    if not native:
        monkeypatch.setattr(asrq_b200.linear, "_native", None)
    need = _scratch_bytes(2000, 12288, 2048, 128)
    assert need == 2 * 12288 * 2048
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    block = torch.empty_like(want)                             # the output's memory stays at hand, nothing else is to be had
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(need, dtype=torch.uint8, device=DEV)
        del block
        got = layer(x)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want)


def test_graphs_of_one_capture_stream_replayed_on_two():
    """Two layers captured one after the other on one stream; the graphs then run at the same time.  Each has its own 16-bit weights."""
    layers = [_layer(1280, 5120, 4, 128, True), _layer(5120, 1280, 4, 128, True)]
    xs = [torch.randn(6000, lq.in_features, generator=gen, device=DEV).half() for lq, gen in layers]
    want = [lq(x) for (lq, _), x in zip(layers, xs)]
    capture, streams = torch.cuda.Stream(), [torch.cuda.Stream(), torch.cuda.Stream()]
    with torch.cuda.stream(capture):
        layers[0][0](xs[0])                                    # the stream's workspace exists
    torch.cuda.synchronize()
    graphs, outs = [torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()], []
    for g, (lq, _), x in zip(graphs, layers, xs):
        with torch.cuda.graph(g, stream=capture):
            outs.append(lq(x))
    for _ in range(20):
        for out in outs:
            out.zero_()
        torch.cuda.synchronize()
        for _ in range(5):
            for g, s in zip(graphs, streams):
                with torch.cuda.stream(s):
                    g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(out, ref) for out, ref in zip(outs, want))
    asrq_b200.check_status()


def test_threads_on_one_stream():
    """Two threads' calls on one stream, whose launches may alternate: neither call's weights are the other's."""
    layers = [_layer(1280, 5120, 4, 128, True), _layer(5120, 1280, 4, 128, True)]
    xs = [torch.randn(2000, lq.in_features, generator=gen, device=DEV).half() for lq, gen in layers]
    want = [lq(x) for (lq, _), x in zip(layers, xs)]
    assert all(_scratch_bytes(2000, lq.out_features, lq.in_features, 128) for lq, _ in layers)
    stream, start, wrong = torch.cuda.Stream(), threading.Barrier(2), []
    with torch.cuda.stream(stream):
        layers[0][0](xs[0])
    torch.cuda.synchronize()

    def work(lq, x, ref):
        with torch.cuda.stream(stream):
            start.wait(30)
            for _ in range(20):
                wrong.extend(1 for y in [lq(x) for _ in range(20)] if not torch.equal(y, ref))
    threads = [threading.Thread(target=work, args=(lq, x, ref)) for (lq, _), x, ref in zip(layers, xs, want)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not wrong
    asrq_b200.check_status()
