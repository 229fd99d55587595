"""The module calls' native host path against the Python one: same bits, the same errors, and it sees replaced and
modified buffers."""
import copy
import pickle
import threading
import time

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


def _in_threads(works):
    errors = []

    def guarded(work):
        try:
            work()
        except BaseException as e:  # noqa: BLE001 (reported by the test's own thread)
            errors.append(e)
    threads = [threading.Thread(target=guarded, args=(w,)) for w in works]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors


def test_threads_on_streams_of_their_own():
    q, qq = _layers(512, 256, True)
    xs = [torch.randn(m, 512, device=DEV).half() for m in (1, 16, 33, 80)]
    want = [(q(x), q.forward_fused(x, gelu=True), qq(x)) for x in xs]
    torch.cuda.synchronize()

    def work(x, w):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(200):
                for got, ref in zip((q(x), q.forward_fused(x, gelu=True), qq(x)), w):
                    assert torch.equal(got, ref)
    _in_threads([lambda x=x, w=w: work(x, w) for x, w in zip(xs, want)])
    asrq_b200.check_status()


@pytest.mark.parametrize("quantized_activations", [False, True])
def test_a_waiting_launch_leaves_the_interpreter_to_others(quantized_activations):
    """A thread fills the launch queue of a stream that a timed kernel holds up for about two seconds, and waits in a launch for
    room; this thread's Python goes on meanwhile."""
    layer = _layers(512, 256, True)[quantized_activations]
    x = torch.randn(80, 512, device=DEV).half()
    stream = torch.cuda.Stream()
    done, took = threading.Event(), []

    def work():
        with torch.cuda.stream(stream):
            layer(x)                                    # workspace and prepared weight exist
            stream.synchronize()
            torch.cuda._sleep(int(4e9))
            t0 = time.perf_counter()
            for _ in range(4000):                       # several times what the queue holds
                layer(x)
            took.append(time.perf_counter() - t0)
            done.set()
    worker = threading.Thread(target=work)
    worker.start()
    gap, last = 0.0, time.perf_counter()
    while not done.is_set() and worker.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    worker.join()
    torch.cuda.synchronize()
    assert took and took[0] > 1.0, took                 # the launches did have to wait
    assert gap < 0.5, gap
    asrq_b200.check_status()


def test_prepared_weight_is_the_weights_own():
    """The derived 8-bit operand goes with the memory of the packed weight, not with its address; a copied layer derives its own."""
    x = torch.randn(80, 512, device=DEV).half()
    a, b, c = (_layers(512, 256, True, seed=s)[1] for s in (0, 1, 2))
    want_a, want_c = a(x), c(x)
    for other in (copy.deepcopy(a), pickle.loads(pickle.dumps(a))):
        assert torch.equal(other(x), want_a)
    address = a.weight.data_ptr()
    a.load_quantized_params(b.scales, b.zeros, b.weight.clone())   # gives the first weight back, no call with this one
    held = []
    for _ in range(64):                                            # the third weight at the first one's address, if that is free
        held.append(c.weight.clone())
        if held[-1].data_ptr() == address:
            break
    a.load_quantized_params(c.scales, c.zeros, held[-1])
    a.bias = c.bias
    assert torch.equal(a(x), want_c)


def test_prepared_weight_derived_under_capture():
    """What a capture derives exists only once the graph has run: a call outside makes its own."""
    qq = _layers(512, 256, True)[1]
    x = torch.randn(80, 512, device=DEV).half()
    want = _layers(512, 256, True)[1](x)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = qq(x)
    assert torch.equal(qq(x), want)
    graph.replay()
    assert torch.equal(y, want)


def test_prepared_weight_on_another_stream():
    """A stream that did not derive the operand waits for the one that did."""
    x = torch.randn(80, 512, device=DEV).half()
    want = _layers(512, 256, True)[1](x)
    qq = _layers(512, 256, True)[1]
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(two):
        _layers(512, 256, True)[1](x)                              # this stream's workspace exists
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        torch.cuda._sleep(int(2e8))                                # about a tenth of a second
        qq(x)
    with torch.cuda.stream(two):
        first, second = qq(x), qq(x)                               # by the Python path, then by the native one
    torch.cuda.synchronize()
    assert torch.equal(first, want) and torch.equal(second, want)
    asrq_b200.check_status()


def test_prepared_weight_outlives_the_streams_that_use_it():
    """The layer gets another weight while a call on a second stream is still to run: that call's operand is not reused for
    the first stream's tensors meanwhile."""
    x = torch.randn(80, 512, device=DEV).half()
    qq, other = (_layers(512, 256, True, seed=s)[1] for s in (0, 1))
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(one):
        want = qq(x)                                               # derives
        other(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(two):
        qq(x)
        torch.cuda._sleep(int(2e8))                                # about a tenth of a second
        y = qq(x)
    held = qq.scales, qq.zeros, qq.weight                          # a program's own part of it
    with torch.cuda.stream(one):
        qq.load_quantized_params(other.scales, other.zeros, other.weight)
        qq(x)                                                      # gives the first operand back
        junk = [torch.full((512 * 256,), 255, dtype=torch.uint8, device=DEV) for _ in range(32)]
    torch.cuda.synchronize()
    assert torch.equal(y, want) and len(junk) == 32 and len(held) == 3


def test_a_workspace_that_was_outgrown_stays():
    """A captured graph holds the address of the workspace that its stream had: that memory is given to nobody else when a
    wider layer needs more, and what is kept is bounded by what is in use."""
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        key = (torch.cuda.current_device(), stream.cuda_stream)
        linear._workspaces.pop(key, None)
        small = linear._workspace(torch.device(DEV), 1 << 20)
        address, kept = small.data_ptr(), len(linear._outgrown)
        del small
        for n in (3 << 20, 9 << 20, 10 << 20, 30 << 20):
            linear._workspace(torch.device(DEV), n)
        others = [torch.empty(1 << 20, dtype=torch.uint8, device=DEV) for _ in range(64)]
        assert all(t.data_ptr() != address for t in others)
        assert sum(t.numel() for t in linear._outgrown[kept:]) <= linear._workspaces[key].numel()


def test_a_workspace_made_under_capture():
    """Two layers captured one after the other on a stream that has no workspace yet: the second graph runs without the first
    ever having run.  (Scales at an odd address take the kernel that counts in the workspace.)"""
    q = _layers(2048, 256, False)[0]
    q.scales = torch.cat((q.scales.new_zeros(1), q.scales.flatten()))[1:].view_as(q.scales)
    x = torch.randn(1, 2048, device=DEV).half()
    want = q(x)
    stream = torch.cuda.Stream()
    linear._workspaces.pop((torch.cuda.current_device(), stream.cuda_stream), None)
    first = torch.cuda.CUDAGraph()
    with torch.cuda.graph(first, stream=stream):
        torch.full((1 << 20,), 255, dtype=torch.uint8, device=DEV)     # what the graphs' memory holds then
    first.replay()
    torch.cuda.synchronize()
    graphs, ys = [torch.cuda.CUDAGraph() for _ in range(2)], []
    for graph in graphs:
        with torch.cuda.graph(graph, stream=stream, pool=first.pool()):
            ys.append(q(x))
    ws = linear._workspaces[(torch.cuda.current_device(), stream.cuda_stream)]
    assert not bool(ws[:256 + 4 * 4096].any())                     # status and counters
    for y, graph in zip(ys[::-1], graphs[::-1]):
        graph.replay()
        assert torch.equal(y, want)
    asrq_b200.check_status()


def test_workspaces_of_many_streams_and_threads():
    """Every stream of torch's pool under capture in its turn, none of them with a workspace yet; then threads that ask for one
    stream's workspace at once and get the same."""
    q = _layers(512, 256, True)[0]
    x = torch.randn(4, 512, device=DEV).half()
    want = q(x)
    for _ in range(40):
        stream = torch.cuda.Stream()
        linear._workspaces.pop((torch.cuda.current_device(), stream.cuda_stream), None)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            y = q(x)
        graph.replay()
        assert torch.equal(y, want)
    stream, got = torch.cuda.Stream(), []
    linear._workspaces.pop((torch.cuda.current_device(), stream.cuda_stream), None)

    def work():
        with torch.cuda.stream(stream):
            got.append(linear._workspace(torch.device(DEV), 1 << 20).data_ptr())
    _in_threads([work] * 8)
    assert len(got) == 8 and len(set(got)) == 1
