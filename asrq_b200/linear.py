"""Drop-in ``LinearQ`` / ``LinearQQ`` modules backed by the B200 kernels.

Same constructor, buffer names, shapes and dtypes, ``state_dict`` keys and
``forward(input)`` contract as the reference module (asrq/core/linear.py:8-86), so the
``Whisper*Q`` / ``Qwen3*Q`` / ``Conformer*Q`` classes can import it unchanged.  The
forward pass calls the C ABI (``include/asrq_b200.h``); there is no CPU or PyTorch
fallback -- a CPU tensor, or a missing library, raises.
"""
from __future__ import annotations

import os
import threading

import torch
import torch.nn as nn

from . import _lib

_DTYPES = {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}
_CHECK = os.environ.get("ASRQ_B200_CHECK_STATUS", "0") == "1"

# one scratch buffer per (device, stream): kernels on one stream run in order, so they can share it
_workspaces: dict = {}
_outgrown: list = []  # earlier, smaller ones: a captured graph may hold their address
_growing = threading.Lock()

_native = None


def _load_native() -> None:
    """The ordinary case of a module call in native code (csrc/host.cpp); built together with the library."""
    global _native
    from . import _native as module
    module.bind(_workspaces, _lib.check)
    _native = module


try:
    _load_native()
except ImportError:  # not built, or it does not load: packing works without it, the first call raises (see _lib.load)
    pass


def _workspace(device: torch.device, nbytes: int) -> torch.Tensor:
    key = (device.index, torch.cuda.current_stream(device).cuda_stream)
    ws = _workspaces.get(key)
    if ws is None or ws.numel() < nbytes:
        with _growing:  # one thread makes it; a second one that another thread had in use would not outlive its call
            ws = _workspaces.get(key)
            if ws is None or ws.numel() < nbytes:
                if ws is not None:
                    _outgrown.append(ws)
                    nbytes = max(nbytes, 2 * ws.numel())  # what is kept stays below what is in use
                from . import _native as native  # (not the switch between the two call paths above)
                ws = native.zeros_now(max(nbytes, 1 << 20), device.index)
                _workspaces[key] = ws
    return ws


def _weights_scratch(nbytes: int, device: torch.device):
    """Memory of a large call's own for its weights as 16-bit values (asrq_linearq_a16_scratch): unlike the workspace not shared by
    what runs on a stream.  None where the call needs none, and where there is none to be had: it then unpacks inside the GEMM."""
    if nbytes == 0:
        return None
    try:
        return torch.empty(nbytes, dtype=torch.uint8, device=device)
    except torch.OutOfMemoryError:
        return None


def check_status(device=None) -> None:
    """Synchronises the device and raises if a kernel on any of its streams reported a bounded wait that gave up."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    idx = device.index if device.index is not None else torch.cuda.current_device()
    torch.cuda.synchronize(idx)
    for (dev, stream), ws in list(_workspaces.items()):
        if dev == idx:
            with _on_device(torch.device("cuda", idx)):
                _lib.call("asrq_check_status", ws.data_ptr(), stream)


class _on_device:
    """Makes the tensor's device current around C-ABI calls (the library works on the current device:
    per-device facts, occupancy queries, launches).  Free when it already is."""

    def __init__(self, device: torch.device):
        self.idx = device.index if device.index is not None else torch.cuda.current_device()
        self.prev = None

    def __enter__(self):
        cur = torch.cuda.current_device()
        if cur != self.idx:
            self.prev = cur
            torch.cuda.set_device(self.idx)
        return self

    def __exit__(self, *exc):
        if self.prev is not None:
            torch.cuda.set_device(self.prev)
        return False


def _expect(ok: bool, what: str) -> None:
    """What a kernel takes as given about its operands (it gets addresses and sizes only)."""
    if not ok:
        raise ValueError(what)


def add_layernorm(x: torch.Tensor, delta, weight: torch.Tensor, bias: torch.Tensor, eps: float = 1e-5, write_sum: bool = True):
    """``(x + delta, layer_norm(x + delta) * weight + bias)`` in one kernel (``delta`` may be None: then the
    first result is ``x`` itself).  16-bit tensors on a CUDA device; the last dimension is normalised."""
    dt = _require_cuda_16bit(x, "add_layernorm")
    dim = x.shape[-1]
    x2 = x.reshape(-1, dim)
    x2 = x2 if x2.is_contiguous() else x2.contiguous()
    d2 = None
    if delta is not None:
        d2 = delta.reshape(-1, dim)
        d2 = d2 if d2.is_contiguous() else d2.contiguous()
    h = torch.empty_like(x2)
    xo = torch.empty_like(x2) if (delta is not None and write_sum) else None
    with _on_device(x.device):
        _lib.call("asrq_add_layernorm", x2.data_ptr(), None if d2 is None else d2.data_ptr(), weight.data_ptr(),
                  bias.data_ptr(), float(eps), None if xo is None else xo.data_ptr(), h.data_ptr(), x2.shape[0], dim, dt,
                  torch.cuda.current_stream(x.device).cuda_stream)
    return (x if xo is None else xo.reshape(x.shape)), h.reshape(x.shape)


def add_rmsnorm(x: torch.Tensor, delta, weight: torch.Tensor, eps: float = 1e-6, write_sum: bool = True):
    """``(x + delta, rms_norm(x + delta) * weight)`` in one kernel, with the rounding of the Qwen3 norm module (the
    normalised value is rounded to the tensor's type before the weight multiplies it).  ``delta`` may be None."""
    dt = _require_cuda_16bit(x, "add_rmsnorm")
    dim = x.shape[-1]
    x2 = x.reshape(-1, dim)
    x2 = x2 if x2.is_contiguous() else x2.contiguous()
    d2 = None
    if delta is not None:
        d2 = delta.reshape(-1, dim)
        d2 = d2 if d2.is_contiguous() else d2.contiguous()
    h = torch.empty_like(x2)
    xo = torch.empty_like(x2) if (delta is not None and write_sum) else None
    with _on_device(x.device):
        _lib.call("asrq_add_rmsnorm", x2.data_ptr(), None if d2 is None else d2.data_ptr(), weight.data_ptr(), float(eps),
                  None if xo is None else xo.data_ptr(), h.data_ptr(), x2.shape[0], dim, dt,
                  torch.cuda.current_stream(x.device).cuda_stream)
    return (x if xo is None else xo.reshape(x.shape)), h.reshape(x.shape)


def silu_mul(gate_up: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up`` for the output of a fused gate/up projection: ``gate_up`` is ``(..., 2 * I)`` with the
    gate features first; returns ``(..., I)``."""
    dt = _require_cuda_16bit(gate_up, "silu_mul")
    inter = gate_up.shape[-1] // 2
    g2 = gate_up.reshape(-1, 2 * inter)
    g2 = g2 if g2.is_contiguous() else g2.contiguous()
    out = torch.empty((g2.shape[0], inter), dtype=gate_up.dtype, device=gate_up.device)
    with _on_device(gate_up.device):
        _lib.call("asrq_silu_mul", g2.data_ptr(), out.data_ptr(), g2.shape[0], inter, dt,
                  torch.cuda.current_stream(gate_up.device).cuda_stream)
    return out.reshape(*gate_up.shape[:-1], inter)


def qk_norm_rope(qkv: torch.Tensor, q_weight: torch.Tensor, k_weight: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor,
                 k_cache: torch.Tensor, v_cache: torch.Tensor, pos, B: int, T: int, n_q: int, n_kv: int, eps: float) -> torch.Tensor:
    """Per-head RMS norm of queries and keys, rotary embedding, and the cache write for ``T`` new positions of ``B``
    sequences, in one kernel.  ``qkv``: (B*T, (n_q + 2 n_kv) * head_dim) from a fused projection; ``cos``/``sin``:
    (max_len, head_dim) tables; caches (B, n_kv, max_len, head_dim); ``pos``: first position, an int or a one-element int64
    CUDA tensor (read on the device).  Returns the queries (B, n_q, T, head_dim)."""
    dt = _require_cuda_16bit(qkv, "qk_norm_rope")
    hd = k_cache.shape[-1]
    q = torch.empty((B, n_q, T, hd), dtype=qkv.dtype, device=qkv.device)
    on_dev = isinstance(pos, torch.Tensor)
    with _on_device(qkv.device):
        _lib.call("asrq_qk_norm_rope", qkv.data_ptr(), q_weight.data_ptr(), k_weight.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                  pos.data_ptr() if on_dev else None, 0 if on_dev else int(pos), q.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(),
                  B, T, n_q, n_kv, hd, k_cache.shape[2], float(eps), dt, torch.cuda.current_stream(qkv.device).cuda_stream)
    return q


def decode_self_attention(qkv: torch.Tensor, kv_cache: torch.Tensor, pos: torch.Tensor, scale: float = 1.0, settled: bool = False) -> torch.Tensor:
    """Self-attention of one decoding step with the cache write: ``qkv`` (B, 3 * d) from a fused projection, ``kv_cache``
    (2, B, heads, max_len, head_dim), ``pos`` a one-element int64 CUDA tensor (the new token's position).  Returns (B, d).
    ``settled``: the position and the cache below it are older than the library's kernels just ahead on the stream (a decoder's
    are), so they may be fetched while these still run."""
    dt = _require_cuda_16bit(qkv, "decode_self_attention")
    _, B, H, max_len, hd = kv_cache.shape
    _expect(kv_cache.is_contiguous() and kv_cache.shape[0] == 2 and kv_cache.dtype == qkv.dtype and kv_cache.device == pos.device == qkv.device and
            pos.dtype == torch.int64, "decode_self_attention: kv_cache must be contiguous (2, B, heads, max_len, head_dim) of qkv's type, pos int64")
    q2 = qkv.reshape(B, 3 * H * hd)
    q2 = q2 if q2.is_contiguous() else q2.contiguous()
    out = torch.empty((B, H * hd), dtype=qkv.dtype, device=qkv.device)
    with _on_device(qkv.device):
        _lib.call("asrq_decode_self_attention_settled" if settled else "asrq_decode_self_attention", q2.data_ptr(), kv_cache.data_ptr(), pos.data_ptr(), out.data_ptr(), B, H, hd, max_len,
                  float(scale), dt, torch.cuda.current_stream(qkv.device).cuda_stream)
    return out


def argmax_rows(logits: torch.Tensor, tokens: torch.Tensor, scratch: torch.Tensor, ids: torch.Tensor = None, pos: torch.Tensor = None) -> None:
    """``tokens.copy_(logits.argmax(-1))`` for contiguous (B, N) 16-bit logits; with ``ids`` (steps, B) and ``pos`` (one int64 on the
    device) also ``ids[pos] = tokens``.  ``scratch``: 2 B int64, zero before the first call, which every call leaves at zero."""
    dt = _require_cuda_16bit(logits, "argmax_rows")
    B, n = logits.shape
    _expect(logits.is_contiguous() and all(t is None or (t.is_contiguous() and t.dtype == torch.int64 and t.device == logits.device)
                                           for t in (tokens, scratch, ids, pos)) and tokens.numel() >= B and scratch.numel() >= 2 * B and
            (ids is None or (pos is not None and ids.numel() % max(B, 1) == 0)),
            "argmax_rows: contiguous (B, N) logits, int64 tokens (B), scratch (2 B), ids (steps, B) with pos on the same device")
    with _on_device(logits.device):
        _lib.call("asrq_argmax_rows", logits.data_ptr(), tokens.data_ptr(), None if ids is None else ids.data_ptr(), None if pos is None else pos.data_ptr(),
                  scratch.data_ptr(), B, n, dt, torch.cuda.current_stream(logits.device).cuda_stream)


def _conv_step(fn: str, tensors, out: torch.Tensor, sizes) -> torch.Tensor:
    dt = _require_cuda_16bit(tensors[0], fn)
    _expect(all(t.dtype == out.dtype and t.device == out.device for t in tensors), f"{fn}: tensors of one type on one device")
    tensors = [t if t.is_contiguous() else t.contiguous() for t in tensors]
    with _on_device(out.device):
        _lib.call(fn, *(t.data_ptr() for t in tensors), out.data_ptr(), *sizes, dt, torch.cuda.current_stream(out.device).cuda_stream)
    return out


def bias_glu(x: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """``glu(x + bias)`` over the channels of a (B, 2C, T) convolution output, in one pass."""
    B, c2, T = x.shape
    _expect(c2 % 2 == 0 and bias.numel() == c2, f"bias_glu: an even number of channels and a bias of as many values (x {tuple(x.shape)}, bias {bias.numel()})")
    return _conv_step("asrq_bias_glu", (x, bias), x.new_empty(B, c2 // 2, T), (B, c2 // 2, T))


def bias_affine_silu(x: torch.Tensor, bias: torch.Tensor, scale: torch.Tensor, shift: torch.Tensor) -> torch.Tensor:
    """``silu((x + bias) * scale + shift)`` per channel of a (B, C, T) convolution output, in one pass."""
    _expect(bias.numel() == scale.numel() == shift.numel() == x.shape[1], "bias_affine_silu: bias, scale and shift of one value per channel")
    return _conv_step("asrq_bias_affine_silu", (x, bias, scale, shift), x.new_empty(x.shape), x.shape)


def half_step(x: torch.Tensor, y: torch.Tensor) -> torch.Tensor:
    """``x + 0.5 * y``, tensors of as many values, a multiple of 8, in one pass."""
    _expect(x.numel() == y.numel(), f"half_step: {tuple(x.shape)} and {tuple(y.shape)}")
    return _conv_step("asrq_half_step", (x, y), x.new_empty(x.shape), (x.numel(),))


def bias_add_transposed(x: torch.Tensor, conv: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """``x + (conv + bias).transpose(1, 2)``: x (B, T, C), conv (B, C, T), in one pass."""
    _expect(conv.shape == (x.shape[0], x.shape[2], x.shape[1]) and bias.numel() == x.shape[2],
            f"bias_add_transposed: x {tuple(x.shape)}, conv {tuple(conv.shape)}, bias {bias.numel()}")
    return _conv_step("asrq_bias_add_transposed", (x, conv, bias), x.new_empty(x.shape), x.shape)


def decode_cross_attention(q: torch.Tensor, kv: torch.Tensor, heads: int, scale: float = 1.0, settled: bool = False) -> torch.Tensor:
    """Cross-attention of one decoding step: ``q`` (B, d), ``kv`` (B, T, 2 d) with keys and values side by side (a fused
    projection's output).  Returns (B, d).  ``settled``: ``kv`` is older than the kernels just ahead on the stream (a step's cross
    keys are), so it may be fetched while these still run."""
    dt = _require_cuda_16bit(q, "decode_cross_attention")
    B, T, d2 = kv.shape
    d = d2 // 2
    _expect(kv.is_contiguous() and kv.dtype == q.dtype and kv.device == q.device and d2 == 2 * d and d % heads == 0 and q.numel() == B * d,
            f"decode_cross_attention: contiguous kv (B, T, 2 d) of q's type and q (B, d) (kv {tuple(kv.shape)}, q {tuple(q.shape)}, {heads} heads)")
    q2 = q.reshape(B, d)
    q2 = q2 if q2.is_contiguous() else q2.contiguous()
    out = torch.empty((B, d), dtype=q.dtype, device=q.device)
    with _on_device(q.device):
        _lib.call("asrq_decode_cross_attention", q2.data_ptr(), kv.data_ptr(), kv.data_ptr() + 2 * d, out.data_ptr(), B, heads, d // heads, T,
                  2 * d, float(scale), int(settled), dt, torch.cuda.current_stream(q.device).cuda_stream)
    return out


def decode_grouped_attention(qkv: torch.Tensor, q_weight: torch.Tensor, k_weight: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor,
                             k_cache: torch.Tensor, v_cache: torch.Tensor, pos: torch.Tensor, n_q: int, eps: float, scale: float) -> torch.Tensor:
    """:func:`qk_norm_rope` for one new position and the attention over the cache in one kernel: ``qkv`` (B, (n_q + 2 n_kv) * 128),
    caches (B, n_kv, max_len, 128), ``pos`` a one-element int64 CUDA tensor; two query heads per key head.  Returns (B, n_q * 128).
    The position and the cache below it are fetched ahead of the stream dependency: behind :func:`qk_norm_rope` into the same
    cache an ordinary kernel or copy has to come first."""
    dt = _require_cuda_16bit(qkv, "decode_grouped_attention")
    B, nkv, max_len, hd = k_cache.shape
    _expect(v_cache.shape == k_cache.shape and qkv.numel() == B * (n_q + 2 * nkv) * hd and min(cos.numel(), sin.numel()) >= max_len * hd and
            q_weight.numel() == k_weight.numel() == hd and pos.dtype == torch.int64 and pos.device == qkv.device and
            all(t.is_contiguous() and t.dtype == qkv.dtype and t.device == qkv.device for t in (qkv, q_weight, k_weight, cos, sin, k_cache, v_cache)),
            "decode_grouped_attention: contiguous tensors of one type; qkv (B, (n_q + 2 n_kv) head_dim), caches (B, n_kv, max_len, head_dim), "
            "tables (max_len, head_dim), pos int64")
    out = torch.empty((B, n_q * hd), dtype=qkv.dtype, device=qkv.device)
    with _on_device(qkv.device):
        _lib.call("asrq_decode_grouped_attention", qkv.data_ptr(), q_weight.data_ptr(), k_weight.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                  pos.data_ptr(), k_cache.data_ptr(), v_cache.data_ptr(), out.data_ptr(), B, n_q, nkv, hd, max_len, float(eps), float(scale), dt,
                  torch.cuda.current_stream(qkv.device).cuda_stream)
    return out


def dense_head(x: torch.Tensor, weight: torch.Tensor, out: torch.Tensor = None) -> torch.Tensor:
    """``x @ weight.T`` for the floating-point output head of a decoding step (``weight`` is (vocabulary, K) in the
    activations' 16-bit type): this library's kernel for up to 32 rows of ``x`` and K a multiple of 32 up to 3200,
    ``torch.matmul`` otherwise."""
    dt = _require_cuda_16bit(x, "dense_head")
    k = x.shape[-1]
    x2 = x.reshape(-1, k)
    m, n = x2.shape[0], weight.shape[0]
    if out is None:
        out = torch.empty((m, n), dtype=x.dtype, device=x.device)
    if (m > 32 or k % 32 or k > 3200 or weight.dtype != x.dtype or not weight.is_contiguous() or weight.shape[1] != k or out.numel() != m * n or
            out.dtype != x.dtype or not out.is_contiguous()):
        torch.matmul(x2, weight.t(), out=out)
        return out.reshape(*x.shape[:-1], n)
    x2 = x2 if x2.is_contiguous() else x2.contiguous()
    with _on_device(x.device):
        _lib.call("asrq_dense_head", x2.data_ptr(), weight.data_ptr(), out.data_ptr(), m, n, k, dt,
                  torch.cuda.current_stream(x.device).cuda_stream)
    return out.reshape(*x.shape[:-1], n)


def _as_2d(x: torch.Tensor, k: int) -> torch.Tensor:
    if x.shape[-1] != k:
        raise ValueError(f"last dimension of the input is {x.shape[-1]}, expected in_features={k}")
    x2 = x.reshape(-1, k)
    return x2 if x2.is_contiguous() else x2.contiguous()


def _require_cuda_16bit(x: torch.Tensor, who: str) -> int:
    if not x.is_cuda:
        raise RuntimeError(f"{who}: input is on {x.device}; asrq_b200 runs on CUDA (sm_100a) only and has no CPU path")
    try:
        return _DTYPES[x.dtype]
    except KeyError:
        raise TypeError(f"{who}: input dtype {x.dtype} is not supported (float16 or bfloat16)") from None


class LinearQ(nn.Module):
    """Linear layer with packed 2-/4-bit weights and per-group fp16 scales and zeros.

    Mirrors asrq/core/linear.py:8-66: ``weight`` uint8 (out, in*bits/8), ``scales`` and
    ``zeros`` fp16 (out, ceil(in/group_size)), ``bias`` fp16 (out) or None;
    ``W[n,k] = q[n,k]*scales[n,k//g] + zeros[n,k//g]``; ``forward`` returns
    ``input @ W.T (+ bias)`` in the input dtype with the input's leading dimensions.
    """

    def __init__(self, in_features, out_features, bits, group_size=128, bias=True):
        super().__init__()
        self.in_features = in_features
        self.out_features = out_features
        self.group_size = group_size
        self.bits = bits
        self.register_buffer("weight", torch.zeros((out_features, in_features // (8 // bits)), dtype=torch.uint8))
        if bias:
            self.register_buffer("bias", torch.zeros(out_features, dtype=torch.float16))
        else:
            self.bias = None
        ngroups = (in_features + group_size - 1) // group_size
        self.register_buffer("scales", torch.zeros((out_features, ngroups), dtype=torch.float16))
        self.register_buffer("zeros", torch.zeros((out_features, ngroups), dtype=torch.float16))

    def load_quantized_params(self, scales, zeros, quantized_weight):
        """Binds already-packed parameters, moving them to the module's device (linear.py:27-31)."""
        self.scales = scales.to(self.scales.device)
        self.zeros = zeros.to(self.zeros.device)
        self.weight = quantized_weight.to(self.weight.device)

    def dequantize_weight(self, device="cpu", dtype=torch.float32):
        """Full (out, in) weight in ``dtype`` with the reference's two-step rounding
        (linear.py:33-54).  A debugging aid; ``forward`` never calls it."""
        g, k = self.group_size, self.in_features
        scale = self.scales.repeat_interleave(g, dim=1).to(device).to(dtype)[:, :k]
        zero = self.zeros.repeat_interleave(g, dim=1).to(device).to(dtype)[:, :k]
        wq = self.weight.to(device)
        q = torch.zeros((self.out_features, k), device=device, dtype=dtype)
        if self.bits == 4:
            q[:, 0::2] = (wq & 0x0F).to(dtype)
            q[:, 1::2] = (wq >> 4).to(dtype)
        elif self.bits == 2:
            for e in range(4):
                q[:, e::4] = ((wq >> (2 * e)) & 0x03).to(dtype)
        else:
            raise NotImplementedError("bits must be 2 or 4")
        return q * scale + zero

    def _check_buffers(self, x: torch.Tensor):
        """(weight, scales, zeros, bias) as the kernels take them.  The caller passes and holds these tensors, read once: another
        thread may replace the layer's."""
        held = []
        for name in ("weight", "scales", "zeros"):
            t = getattr(self, name)
            if t.device != x.device:
                raise RuntimeError(f"LinearQ.{name} is on {t.device} but the input is on {x.device}")
            if not t.is_contiguous():
                t = t.contiguous()
                setattr(self, name, t)
            held.append(t)
        weight, scales, zeros = held
        bias = self.bias
        if scales.dtype != torch.float16 or zeros.dtype != torch.float16:
            raise TypeError("LinearQ.scales and LinearQ.zeros must be float16")
        if weight.dtype != torch.uint8:
            raise TypeError("LinearQ.weight must be uint8")
        if bias is not None and (bias.dtype != torch.float16 or bias.device != x.device):
            raise TypeError("LinearQ.bias must be float16 on the input's device")
        return weight, scales, zeros, bias

    def forward(self, input):
        if _native is not None and not _CHECK:
            y = _native.linearq_forward(self, input, None, False)
            if y is not None:
                return y
        return self.forward_fused(input)

    def forward_fused(self, input, residual=None, gelu=False):
        """``forward`` with the step that follows the layer in a transformer block done in the kernel's
        epilogue: ``gelu(layer(input))`` or ``residual + layer(input)`` (``residual``: the output's shape and
        dtype).  Same bits as the unfused module sequence."""
        if _native is not None and not _CHECK:
            y = _native.linearq_forward(self, input, residual, bool(gelu))
            if y is not None:
                return y
        # fp16 / bf16 only (the reference computes in whatever dtype the input has, asrq/core/linear.py:58-59;
        # an fp32 input raises here rather than silently running a slower path)
        dt = _require_cuda_16bit(input, "LinearQ.forward")
        if self.bits not in (2, 4):
            raise NotImplementedError("LinearQ.forward: bits must be 2 or 4")
        weight, scales, zeros, bias = self._check_buffers(input)
        n, k = self.out_features, self.in_features
        x2 = _as_2d(input, k)
        m = x2.shape[0]
        y = torch.empty((m, n), dtype=input.dtype, device=input.device)
        if m == 0:
            return y.reshape(*input.shape[:-1], n)
        ws = _workspace(input.device, _lib.workspace_bytes(_lib.WS_LINEARQ, m, n, k))
        stream = torch.cuda.current_stream(input.device).cuda_stream
        with _on_device(input.device):
            r2 = None
            if residual is not None:
                if residual.dtype != input.dtype or residual.numel() != m * n or residual.device != input.device:
                    raise ValueError("forward_fused: residual must have the output's shape, dtype and device")
                r2 = residual.reshape(m, n)
                r2 = r2 if r2.is_contiguous() else r2.contiguous()
            act = _lib.ACT_GELU if gelu else _lib.ACT_NONE
            w16 = _weights_scratch(_lib.load().asrq_linearq_a16_scratch_bytes(m, n, k, self.group_size, act, residual is not None), input.device)
            args = (self.bits, x2.data_ptr(), weight.data_ptr(), scales.data_ptr(), zeros.data_ptr(), None if bias is None else bias.data_ptr())
            if w16 is not None:
                _lib.call("asrq_linearq_a16_scratch", *args, None if r2 is None else r2.data_ptr(), y.data_ptr(), m, n, k, self.group_size, dt, act,
                          ws.data_ptr(), ws.numel(), w16.data_ptr(), w16.numel(), stream)
            elif r2 is None and not gelu:
                _lib.call("asrq_linearq_a16", *args, y.data_ptr(), m, n, k, self.group_size, dt, ws.data_ptr(), ws.numel(), stream)
            else:
                _lib.call("asrq_linearq_a16_fused", *args, None if r2 is None else r2.data_ptr(), y.data_ptr(), m, n, k, self.group_size, dt, act,
                          ws.data_ptr(), ws.numel(), stream)
        if _CHECK:
            check_status(input.device)
        return y.reshape(*input.shape[:-1], n)

    def extra_repr(self):
        return (f"in_features={self.in_features}, out_features={self.out_features}, bits={self.bits}, "
                f"group_size={self.group_size}, bias={self.bias is not None}")


PRE_LAYERNORM, PRE_RMSNORM, PRE_SILU_MUL = 1, 2, 3  # asrq_linearq_a16_pre


def calls_only_linearq(layer) -> bool:
    """Whether calling ``layer`` runs :meth:`LinearQ.forward` and nothing else: no subclass or stand-in, no hooks, no replaced method."""
    return (type(layer) is LinearQ and not layer._forward_hooks and not layer._forward_pre_hooks and "forward" not in layer.__dict__ and
            "forward_fused" not in layer.__dict__ and not nn.modules.module._global_forward_hooks and
            not nn.modules.module._global_forward_pre_hooks)


def linear_after(layer: LinearQ, pre: int, x: torch.Tensor, weight=None, bias=None, eps: float = 0.0, residual=None, gelu: bool = False):
    """``layer.forward_fused(h, residual, gelu)`` where ``h`` is the step ahead of the layer: the layer norm or RMS norm of the
    residual stream ``x``, or ``silu(gate) * up`` of a fused projection's output ``x``.  For one or two rows (one for the last)
    both are one kernel; otherwise None, and the caller does them one after the other; so also where a call of the layer does
    more than its product (:func:`calls_only_linearq`)."""
    if not calls_only_linearq(layer):
        return None
    k, n = layer.in_features, layer.out_features
    width = 2 * k if pre == PRE_SILU_MUL else k
    rows = x.numel() // width
    if rows > 2 or not x.is_cuda or x.shape[-1] != width or not x.is_contiguous() or x.dtype not in _DTYPES:
        return None
    with _on_device(x.device):
        if _lib.load().asrq_linearq_a16_pre_covers(layer.bits, pre, rows, n, k, layer.group_size, _DTYPES[x.dtype]) != 1:
            return None
    packed, scales, zeros, layer_bias = layer._check_buffers(x)
    if residual is not None and not (residual.numel() == rows * n and residual.is_contiguous() and residual.dtype == x.dtype and residual.device == x.device):
        return None
    if layer_bias is not None and not layer_bias.is_contiguous():
        return None
    for t in (weight, bias):
        if t is not None and not (t.numel() == k and t.is_contiguous() and t.dtype == x.dtype and t.device == x.device):
            return None
    if any(t is not None and t.data_ptr() % 16 for t in (x, packed, scales, zeros, weight, bias)):
        return None
    y = torch.empty((*x.shape[:-1], n), dtype=x.dtype, device=x.device)

    def ptr(t):
        return None if t is None else t.data_ptr()

    with _on_device(x.device):
        _lib.call("asrq_linearq_a16_pre", layer.bits, pre, x.data_ptr(), ptr(weight), ptr(bias), float(eps), packed.data_ptr(),
                  scales.data_ptr(), zeros.data_ptr(), ptr(layer_bias), ptr(residual), y.data_ptr(), rows, n, k, layer.group_size,
                  _DTYPES[x.dtype], _lib.ACT_GELU if gelu else _lib.ACT_NONE, torch.cuda.current_stream(x.device).cuda_stream)
    return y


class _Prepared(tuple):
    """(operand, an alias of the packed weight it was derived from, that weight's version, the operand's format, the streams that
    are ordered behind the derivation, its event).  The alias keeps the weight's memory, so that an equal address means the same
    memory; another stream waits for the event once.  A copy of a layer, or a pickled one, derives its own."""
    __slots__ = ()

    def of(self, weight: torch.Tensor, operand: str) -> bool:
        src = self[1]
        return (src.data_ptr(), src.device, self[2], self[3]) == (weight.data_ptr(), weight.device, weight._version, operand)

    def __reduce_ex__(self, protocol):
        return type(None), ()


class LinearQQ(LinearQ):
    """W4A4 linear: online Hadamard rotation + per-token int4 activations, grouped int4 weights.

    Constructor signature of the reference stub (asrq/core/linear.py:69-75), whose
    ``forward`` returns None.  ``weight`` holds two's-complement signed nibbles
    (asrq/matmulq/test.py:141-142), ``scales`` the per-(row, group) weight scales;
    ``zeros`` is unused and stays zero.  ``forward`` computes

        v = hadU(x) (if ``hadamard``);  s = absmax(v)/7 per token;  q = rint(v/s)
        y[m,n] = s[m] * sum_g (sum_{k in g} q[m,k]*qw[n,k]) * scales[n,g]  (+ bias[n])

    which equals ``x @ W.T`` up to quantisation error when ``weight`` was produced by
    :func:`asrq_b200.packing.pack_w4a4` with the same ``hadamard`` flag.
    """

    def __init__(self, in_features, out_features, wbits, abits, group_size=128, bias=True, hadamard=True):
        if wbits != 4 or abits != 4:
            raise NotImplementedError("LinearQQ supports wbits=4, abits=4")
        super().__init__(in_features, out_features, wbits, group_size, bias)
        self.register_buffer("act_scales", torch.ones(in_features))
        self.amax = 2 ** (abits - 1) - 1
        self.abits = abits
        self.hadamard = hadamard

    def _quantize(self, input):
        dt = _require_cuda_16bit(input, "LinearQQ")
        x2 = _as_2d(input, self.in_features)
        m, k = x2.shape
        qa = torch.empty((m, k // 2), dtype=torch.uint8, device=input.device)
        sa = torch.empty((m,), dtype=torch.float32, device=input.device)
        stream = torch.cuda.current_stream(input.device).cuda_stream
        _lib.call("asrq_hadamard_quant_int4", x2.data_ptr(), qa.data_ptr(), sa.data_ptr(), m, k,
                  1 if self.hadamard else 0, dt, stream)
        return qa, sa, dt, stream

    def quantize_activation(self, input):
        """(codes, scales): integer-valued float codes (M,K) and per-token scales (M,1), the
        return convention of the reference method (linear.py:77-82), computed by the CUDA prologue."""
        _require_cuda_16bit(input, "LinearQQ")
        with _on_device(input.device):
            qa, sa, _, _ = self._quantize(input)
        p = qa.to(torch.int32)
        lo, hi = p & 0xF, (p >> 4) & 0xF
        lo = torch.where(lo >= 8, lo - 16, lo)
        hi = torch.where(hi >= 8, hi - 16, hi)
        q = torch.stack((lo, hi), dim=-1).reshape(qa.shape[0], -1).to(torch.float32)
        return q, sa.reshape(-1, 1)

    # 8-bit operand family of the tensor-core path: "f8" (e4m3 bytes holding the code, tcgen05 kind::f8f6f4,
    # fp32 group sums) or "int8" (16x the code, kind::i8, int32 group sums).  Same bits out; f8 is faster.
    operand = os.environ.get("ASRQ_B200_W4A4_OPERAND", "f8")

    def _entry(self, stem: str) -> str:
        if self.operand not in ("f8", "int8"):
            raise ValueError(f"LinearQQ.operand must be 'f8' or 'int8', got {self.operand!r}")
        if stem == "prepare":
            return "asrq_w4a4_prepare_weight_f8" if self.operand == "f8" else "asrq_w4a4_prepare_weight"
        return f"asrq_{stem}_{self.operand}"

    def _prepared_weight(self) -> torch.Tensor:
        """8-bit operand form of ``weight`` (natural k order), derived on first use and whenever the
        packed buffer is replaced or modified; not part of ``state_dict``.  (A change that the tensor's version
        counter does not see, as through ``weight.data``, is not seen here either.)"""
        weight, operand = self.weight, self.operand
        stream = torch.cuda.current_stream(weight.device)
        capturing = torch.cuda.is_current_stream_capturing()
        p = getattr(self, "_w8", None)
        if type(p) is _Prepared and p.of(weight, operand):
            if stream.cuda_stream not in p[4] and not capturing:
                stream.wait_event(p[5])
                p[0].record_stream(stream)  # replaced, its memory waits for this stream's work too
                p[4].add(stream.cuda_stream)
            return p[0]
        w8 = torch.empty((self.out_features, self.in_features), dtype=torch.uint8, device=weight.device)
        _lib.call(self._entry("prepare"), weight.data_ptr(), w8.data_ptr(), self.out_features, self.in_features, stream.cuda_stream)
        if not capturing:  # what is being captured exists only once the graph has run: its own calls derive it again
            self._w8 = _Prepared((w8, weight.detach(), weight._version, operand, {stream.cuda_stream}, stream.record_event()))
        return w8

    def _tensor_core_ok(self, m: int) -> bool:
        n, k, g = self.out_features, self.in_features, self.group_size
        return m >= 64 and n % 128 == 0 and k % 128 == 0 and g % 128 == 0 and k % g == 0

    def forward(self, input, acc_dump=None, two_call=False):
        if acc_dump is None and not two_call and _native is not None and not _CHECK:
            y = _native.linearqq_forward(self, input)
            if y is not None:
                return y
        _require_cuda_16bit(input, "LinearQQ")
        with _on_device(input.device):
            return self._forward(input, acc_dump, two_call)

    def _forward(self, input, acc_dump=None, two_call=False):
        """``two_call=True`` forces the packed-activation sequence (asrq_hadamard_quant_int4 then
        asrq_w4a4_gemm); the default for large M is the prologue writing 8-bit operands directly.
        Both produce the same bits."""
        weight, scales, _, bias = self._check_buffers(input)
        if input.numel() == 0:
            _require_cuda_16bit(input, "LinearQQ")
            return input.new_empty(*input.shape[:-1], self.out_features)
        n, k = self.out_features, self.in_features
        bias_ptr = None if bias is None else bias.data_ptr()
        dump = None if acc_dump is None else acc_dump.data_ptr()
        if two_call or not self._tensor_core_ok(input.numel() // k):
            qa, sa, dt, stream = self._quantize(input)
            m = qa.shape[0]
            y = torch.empty((m, n), dtype=input.dtype, device=input.device)
            ws = _workspace(input.device, _lib.workspace_bytes(_lib.WS_W4A4_GEMM, m, n, k))
            _lib.call("asrq_w4a4_gemm", qa.data_ptr(), sa.data_ptr(), weight.data_ptr(), scales.data_ptr(),
                      bias_ptr, y.data_ptr(), dump, m, n, k, self.group_size, dt, ws.data_ptr(), ws.numel(), stream)
        else:
            dt = _require_cuda_16bit(input, "LinearQQ")
            x2 = _as_2d(input, k)
            m = x2.shape[0]
            w8 = self._prepared_weight()
            a8 = torch.empty((m, k), dtype=torch.uint8, device=input.device)
            sa = torch.empty((m,), dtype=torch.float32, device=input.device)
            y = torch.empty((m, n), dtype=input.dtype, device=input.device)
            ws = _workspace(input.device, _lib.STATUS_BYTES)
            stream = torch.cuda.current_stream(input.device).cuda_stream
            _lib.call(self._entry("hadamard_quant"), x2.data_ptr(), a8.data_ptr(), sa.data_ptr(), m, k,
                      1 if self.hadamard else 0, dt, stream)
            _lib.call(self._entry("w4a4_gemm"), a8.data_ptr(), sa.data_ptr(), w8.data_ptr(), scales.data_ptr(),
                      bias_ptr, y.data_ptr(), dump, m, n, k, self.group_size, dt, ws.data_ptr(), ws.numel(), stream)
        if _CHECK:
            check_status(input.device)
        return y.reshape(*input.shape[:-1], n)
