"""W4A16 / W2A16 parity on the GPU, through the C ABI, against the CPU oracle.

Bar: |y - y_fp32| <= 2e-3 * ||row||_inf of the fp32 CPU result (fp16 outputs); bf16 outputs
additionally get half a bf16 ulp of the reference value, because rounding the output to
bf16 alone can cost 3.9e-3 of the row maximum.
"""
import glob
import os

import numpy as np
import pytest
import torch

from oracle import linearq_oracle as O
from asrq_b200 import _lib
from tests.gpu_util import DEV, assert_close_rows, bf16_half_ulp, f16, lib_option, make_layer, run_a16_abi

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def _ref32(case, dtype=torch.float16):
    x = case["x"].to(dtype)
    return O.linearq_forward_fp32(x, case["weight"], case["scales"], case["zeros"], case["bias"], case["bits"],
                                  case["group_size"])


def _golden_cases():
    out = []
    for p in sorted(glob.glob(os.path.join(GOLDEN, "linearq_*.npz"))):
        d = np.load(p)
        bits, g, k, n = int(d["bits"]), int(d["group_size"]), int(d["in_features"]), int(d["out_features"])
        chunk = 128 if bits == 4 else 256
        if k % chunk or n % 16 or g % (128 // bits):
            continue
        out.append(os.path.basename(p))
    return out


@pytest.mark.parametrize("name", _golden_cases())
def test_golden_fixture_through_module(name):
    """The reference's own outputs (fixtures): our fp16 output vs the reference fp32 forward."""
    d = np.load(os.path.join(GOLDEN, name))
    case = dict(x=f16(d["x"]), weight=torch.from_numpy(d["weight"]), scales=f16(d["scales"]), zeros=f16(d["zeros"]),
                bias=f16(d["bias"]) if "bias" in d else None, bits=int(d["bits"]), group_size=int(d["group_size"]))
    lq = make_layer(case)
    y = lq(case["x"].to(DEV))
    assert y.dtype == torch.float16 and y.shape == (case["x"].shape[0], case["weight"].shape[0])
    assert_close_rows(y, torch.from_numpy(d["y_f32"]), what=name)


@pytest.mark.parametrize("bits", [4, 2])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 8, 9, 16])
@pytest.mark.parametrize("kn", [(2048, 6144), (6144, 2048), (2048, 4096)])
def test_decode_shapes_gemv(bits, m, kn):
    k, n = kn
    case = O.make_c3(seed=1000 + m, m=m, k=k, n=n, bits=bits, group_size=64)
    y = run_a16_abi(f"asrq_w{bits}a16_gemv", case)
    assert_close_rows(y, _ref32(case), what=f"gemv w{bits} m{m} {k}x{n}")


@pytest.mark.parametrize("bits,g,m,k,n,bias", [
    (4, 128, 5, 1280, 5120, True),    # Whisper fc1, K not a power of two
    (4, 128, 7, 5120, 1280, True),    # Whisper fc2: K > 2048 forces a K split
    (2, 128, 16, 1280, 1280, False),
    (4, 32, 3, 256, 48, True),        # N not a multiple of the block's 128 rows; smallest group
    (2, 64, 1, 256, 16, False),       # one warp strip
    (4, 128, 17, 1024, 256, True),    # M > 16: two row blocks
    (2, 64, 40, 512, 128, True),      # M > 32 through the skinny entry point
])
def test_gemv_edge_shapes(bits, g, m, k, n, bias):
    gen = torch.Generator().manual_seed(bits * 1000 + m)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, g, False)
    case = dict(x=torch.randn(m, k, generator=gen).half(), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half() if bias else None,
                bits=bits, group_size=g)
    y = run_a16_abi(f"asrq_w{bits}a16_gemv", case)
    assert_close_rows(y, _ref32(case), what=f"gemv edge w{bits} g{g} m{m} {k}x{n}")


@pytest.mark.parametrize("bits,g,m,k,n,bias,dtype", [
    (4, 128, 1, 16384, 256, False, torch.float16),    # K beyond 16 warps x 4 steps: 8 rounds per warp
    (4, 64, 5, 16384, 128, True, torch.float16),
    (4, 32, 16, 8192, 64, False, torch.float16),      # four groups per step: two steps per round
    (2, 64, 2, 32768, 64, True, torch.float16),
    (2, 256, 20, 16384, 128, False, torch.bfloat16),  # two launches (16 + 4 tokens)
    (4, 128, 3, 8192, 4096, False, torch.float16),    # 16 MiB of weights: more than one resident wave
])
def test_gemv_rounds(bits, g, m, k, n, bias, dtype):
    """Long K and large layers run on small blocks whose warps walk K in rounds."""
    gen = torch.Generator().manual_seed(bits * 13 + m)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, g, False)
    case = dict(x=torch.randn(m, k, generator=gen).to(dtype), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half() if bias else None,
                bits=bits, group_size=g)
    y = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=dtype)
    ref = _ref32(case, dtype)
    extra = bf16_half_ulp(ref) if dtype == torch.bfloat16 else None
    if extra is None:
        assert_close_rows(y, ref, what=f"gemv rounds w{bits} g{g} m{m} {k}x{n}")
    else:
        assert_close_rows(y, ref, rel=2e-3, extra=extra, what=f"gemv rounds bf16 w{bits} g{g} m{m} {k}x{n}")
    y2 = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=dtype)
    assert torch.equal(y, y2)


def test_gemv_deterministic_and_workspace_clean():
    """Split-K partial sums are added in slice order: repeated runs are bit-identical."""
    case = O.make_c3(seed=7, m=4, k=6144, n=2048, bits=4, group_size=64)
    lq = make_layer(case)
    x = case["x"].to(DEV)
    ys = [lq(x).clone() for _ in range(3)]
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[1], ys[2])


@pytest.mark.parametrize("bits", [4, 2])
def test_gemv_bf16(bits):
    case = O.make_c3(seed=11, m=4, k=2048, n=4096, bits=bits, group_size=64, dtype=torch.bfloat16)
    y = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=torch.bfloat16)
    ref = _ref32(case, torch.bfloat16)
    assert_close_rows(y, ref, extra=bf16_half_ulp(ref), what=f"gemv bf16 w{bits}")


def test_config1_w4a16_prefill():
    """Whisper-large-v3 encoder fc1 as one layer: K=1280 N=5120 M=1500, RTN g128 asymmetric, 0.1 % weight
    outliers x10, bias."""
    case = O.make_c1(seed=0)
    y = run_a16_abi("asrq_w4a16_gemm", case)
    assert_close_rows(y, _ref32(case), what="config 1")


@pytest.mark.parametrize("bits,g,m,k,n,bias", [
    (4, 128, 32, 256, 128, False),     # one tile, smallest M
    (4, 64, 33, 64, 128, True),        # one K block, ragged M
    (4, 128, 200, 1280, 1280, True),   # Whisper attention projection
    (2, 128, 256, 1280, 5120, True),
    (2, 64, 1500, 2048, 256, False),
    (4, 64, 777, 6144, 2048, False),   # long K: many ring wraps
    (4, 128, 6000, 1024, 4096, True),  # many tiles per block: accumulator double-buffering
])
def test_gemm_tc_shapes(bits, g, m, k, n, bias):
    gen = torch.Generator().manual_seed(bits * 7 + m)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, g, False)
    case = dict(x=torch.randn(m, k, generator=gen).half(), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half() if bias else None,
                bits=bits, group_size=g)
    y = run_a16_abi(f"asrq_w{bits}a16_gemm", case)
    assert_close_rows(y, _ref32(case), what=f"gemm w{bits} g{g} m{m} {k}x{n}")


@pytest.mark.parametrize("bits,g,m,k,n,bias,dtype", [
    (4, 128, 32, 2048, 6144, False, torch.float16),   # decode batch 32: 48 tiles, K in 3 parts
    (4, 128, 64, 5120, 1280, True, torch.float16),    # 20 tiles, K in 7 parts
    (2, 64, 40, 1280, 1280, True, torch.float16),     # ragged M, two token tiles
    (4, 64, 100, 6144, 2048, False, torch.bfloat16),
    (4, 128, 256, 1280, 1280, True, torch.float16),   # widest M that still splits
])
def test_gemm_tc_split_k(bits, g, m, k, n, bias, dtype):
    """Mid-size M: the K range of a tile is divided among blocks and the fp32 parts are added in a
    fixed order by the last block to arrive.  Same workspace for two calls: the tile counters must
    come back to zero, and the result must not depend on timing."""
    gen = torch.Generator().manual_seed(bits * 11 + m)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, g, False)
    case = dict(x=torch.randn(m, k, generator=gen).to(dtype), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half() if bias else None,
                bits=bits, group_size=g)
    from asrq_b200 import _lib
    x, wq = case["x"].to(DEV), case["weight"].to(DEV)
    sc, ze = case["scales"].to(DEV), case["zeros"].to(DEV)
    b = None if case["bias"] is None else case["bias"].to(DEV)
    ws = torch.zeros(_lib.workspace_bytes(_lib.WS_A16_GEMM, m, n, k), dtype=torch.uint8, device=DEV)
    assert ws.numel() > 16640
    ys = []
    for _ in range(2):
        y = torch.empty(m, n, dtype=dtype, device=DEV)
        _lib.call(f"asrq_w{bits}a16_gemm", x.data_ptr(), wq.data_ptr(), sc.data_ptr(), ze.data_ptr(),
                  None if b is None else b.data_ptr(), y.data_ptr(), m, n, k, g,
                  _lib.F16 if dtype == torch.float16 else _lib.BF16, ws.data_ptr(), ws.numel(),
                  torch.cuda.current_stream().cuda_stream)
        _lib.call("asrq_check_status", ws.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert int(ws[:16640].view(torch.int32).abs().sum()) == 0, "status block or tile counters not clean"
        ys.append(y)
    assert torch.equal(ys[0], ys[1])
    ref = _ref32(case, dtype)
    if dtype == torch.float16:
        assert_close_rows(ys[0], ref, what=f"split-K gemm w{bits} m{m} {k}x{n}")
    else:
        wd = O.dequantize_weight(case["weight"], case["scales"], case["zeros"], bits, g, k, torch.float32)
        xf = case["x"].float()
        w_round = 6.0 * 2.0 ** -9 / 3 ** 0.5 * torch.sqrt((xf * xf) @ (wd * wd).t())
        assert_close_rows(ys[0], ref, rel=2e-3, extra=bf16_half_ulp(ref) + w_round, what="split-K gemm bf16")


@pytest.mark.parametrize("bits", [4, 2])
def test_gemm_tc_bf16(bits):
    gen = torch.Generator().manual_seed(bits)
    m, k, n, g = 300, 1024, 512, 128
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, g, False)
    case = dict(x=torch.randn(m, k, generator=gen), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=None, bits=bits, group_size=g)
    y = run_a16_abi(f"asrq_w{bits}a16_gemm", case, dtype=torch.bfloat16)
    ref = _ref32(case, torch.bfloat16)
    # The bf16 MMA takes bf16 weights: each dequantised weight is rounded once to 8 significand bits
    # (relative error <= 2^-9, independent per weight).  Its effect on an output is a sum of K
    # independent terms with standard deviation <= 2^-9/sqrt(3) * sqrt(sum_k x_k^2 w_k^2); six sigma
    # of that is allowed on top of the fp16 bar and the output's own bf16 rounding.
    wd = O.dequantize_weight(case["weight"], case["scales"], case["zeros"], bits, g, k, torch.float32)
    xf = case["x"].to(torch.bfloat16).float()
    w_round = 6.0 * 2.0 ** -9 / 3 ** 0.5 * torch.sqrt((xf * xf) @ (wd * wd).t())
    assert_close_rows(y, ref, rel=2e-3, extra=bf16_half_ulp(ref) + w_round, what=f"gemm bf16 w{bits}")


def test_gemm_matches_gemv_and_linearity():
    """Size-independent properties: both kernels agree, and the layer is linear in x."""
    case = O.make_c3(seed=3, m=64, k=2048, n=1024, bits=4, group_size=64)
    y_tc = run_a16_abi("asrq_w4a16_gemm", case).float()
    y_gv = run_a16_abi("asrq_w4a16_gemv", case).float()
    scale = y_gv.abs().max(dim=-1, keepdim=True).values
    assert float(((y_tc - y_gv).abs() / scale).max()) < 2e-3
    lq = make_layer(case)
    x = case["x"].to(DEV)
    y2 = lq(2 * x).float()
    assert float(((y2 - 2 * lq(x).float()).abs() / scale.to(DEV)).max()) < 2e-3


def test_module_dispatch_and_leading_dims():
    case = O.make_c1(seed=1, m=96, k=1280, n=1280)
    lq = make_layer(case)
    x = case["x"].to(DEV).reshape(2, 3, 16, 1280)
    y = lq(x)
    assert y.shape == (2, 3, 16, 1280)
    assert_close_rows(y.reshape(96, 1280), _ref32(case), what="module 4-D input")
    y1 = lq(x[0, 0, :1])
    assert_close_rows(y1, _ref32(case)[:1], what="module M=1")
    empty = lq(x[:0])
    assert empty.shape == (0, 3, 16, 1280)
    with pytest.raises(TypeError):
        lq(x.float())


@pytest.mark.parametrize("m,k,n,bits", [(64, 256, 256, 4), (300, 1280, 1024, 4), (1500, 1280, 5120, 4), (200, 1024, 512, 2)])
def test_gemm_cta_pair_variant(m, k, n, bits):
    """The tcgen05 cta_group::2 kernel (two CTAs share one 256-row MMA; the default for M > 256), forced
    also for smaller M, against the fp32 CPU result."""
    gen = torch.Generator().manual_seed(m + n)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, 128, False)
    case = dict(x=torch.randn(m, k, generator=gen).half(), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half(), bits=bits, group_size=128)
    with lib_option("tc_pair", 1):
        y = run_a16_abi(f"asrq_w{bits}a16_gemm", case)
    assert_close_rows(y, _ref32(case, torch.float16), what=f"pair gemm w{bits} m{m}")


@pytest.mark.parametrize("m,k,n,bits", [(1500, 1280, 5120, 4), (6000, 1024, 4096, 4), (777, 6144, 2048, 2)])
def test_gemm_single_cta_kernel_large_m(m, k, n, bits):
    """The one-CTA-per-tile kernel on large M (where the CTA-pair kernel is the default), and both agree."""
    gen = torch.Generator().manual_seed(m + n + 5)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, 128, False)
    case = dict(x=torch.randn(m, k, generator=gen).half(), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half(), bits=bits, group_size=128)
    y_pair = run_a16_abi(f"asrq_w{bits}a16_gemm", case)
    with lib_option("tc_pair", 0):
        y_single = run_a16_abi(f"asrq_w{bits}a16_gemm", case)
    ref = _ref32(case, torch.float16)
    assert_close_rows(y_single, ref, what=f"single-CTA gemm w{bits} m{m}")
    assert_close_rows(y_pair, ref, what=f"pair gemm w{bits} m{m}")


def _sample_rows(m, tile=224, count=768, seed=0):
    """Rows to check on a large M: the first and last rows, the rows either side of token-tile
    boundaries, and a seeded random sample."""
    gen = torch.Generator().manual_seed(seed)
    rows = {0, 1, m - 2, m - 1}
    for t in (tile, 256, 192):
        for b in range(t, m, t * max(1, m // (t * 24))):
            rows.update((b - 1, b))
    rows.update(torch.randint(0, m, (count,), generator=gen).tolist())
    return torch.tensor(sorted(r for r in rows if 0 <= r < m))


@pytest.mark.parametrize("m,k,n,g", [
    (48000, 1280, 1280, 128),   # Whisper-large-v3 encoder, batch 32 x 1500 frames: attention projections
    (48000, 1280, 5120, 128),   # ... and fc1
    (16000, 1024, 4096, 128),   # FastConformer FFN, batch 64 x 250 frames
])
def test_encoder_sized_m(m, k, n, g):
    """The whole-model encoder token counts through the module (CTA-pair kernel, hundreds of tiles per
    block), checked on a row sample against the fp32 CPU result."""
    gen = torch.Generator().manual_seed(m + n)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, 4, g, False)
    bias = (torch.randn(n, generator=gen) * 0.02).half()
    x = torch.randn(m, k, generator=gen).half()
    case = dict(x=x, weight=O.pack_codes(codes, 4), scales=scales.half(), zeros=zeros.half(), bias=bias, bits=4,
                group_size=g)
    y = run_a16_abi("asrq_w4a16_gemm", case)
    rows = _sample_rows(m)
    sub = dict(case, x=x[rows])
    assert_close_rows(y[rows.to(DEV)], _ref32(sub), what=f"encoder M={m} {k}->{n}")
    # every row was written (the output buffer starts as canary bytes, 0xA5A5 = -0.0216 as fp16)
    assert bool((y.view(torch.int16) != torch.tensor(-0x5A5B, dtype=torch.int16, device=DEV)).any(dim=1).all())


@pytest.mark.parametrize("release", [0, 1])
def test_pair_kernel_bitwise_stress(release):
    """The CTA-pair kernel hands dequantised weights from the peer CTA's shared memory to an MMA issued
    by the other CTA.  Both forms of that hand-off (relaxed remote arrival, and release/acquire at
    cluster scope) must give the bits of the one-CTA kernel, launch after launch."""
    for (m, k, n) in ((1500, 1280, 5120), (4096, 2048, 1024)):
        gen = torch.Generator().manual_seed(m)
        w = torch.randn(n, k, generator=gen) * 0.02
        codes, scales, zeros, _ = O.rtn_codes(w, 4, 128, False)
        case = dict(x=torch.randn(m, k, generator=gen).half(), weight=O.pack_codes(codes, 4), scales=scales.half(),
                    zeros=zeros.half(), bias=None, bits=4, group_size=128)
        lq = make_layer(case)
        x = case["x"].to(DEV)
        with lib_option("tc_pair", 0):
            y_single = lq(x).clone()
        with lib_option("tc_pair", 1), lib_option("tc_pair_release", release):
            for _ in range(40):
                assert torch.equal(lq(x), y_single)
    import asrq_b200
    asrq_b200.check_status()


def test_pair_kernel_repeats_bit_for_bit_in_a_chain():
    """The sequence of a transformer block's prefill at Qwen3-1.7B widths and M = 2560 (norm -> gate/up -> silu*up ->
    down, the pair kernel launched behind other launches of the library), repeated: every repetition gives the bits
    of the first, and those of the one-CTA kernel.  (With the packed-weight slot released before the warp had
    provably finished reading it, one K block of a few weight rows was wrong about once in 300 such chains.)"""
    m, h, inter = 2560, 2048, 6144
    gen = torch.Generator().manual_seed(7)

    def layer(n, k):
        w = torch.randn(n, k, generator=gen) * 0.02
        codes, scales, zeros, _ = O.rtn_codes(w, 4, 128, False)
        return make_layer(dict(x=torch.zeros(1, k), weight=O.pack_codes(codes, 4), scales=scales.half(), zeros=zeros.half(),
                               bias=None, bits=4, group_size=128))

    import asrq_b200
    gu, down = layer(2 * inter, h), layer(h, inter)
    x = torch.randn(m, h, generator=gen).half().to(DEV)
    g = torch.ones(h, dtype=torch.float16, device=DEV)

    def chain():
        hn = asrq_b200.add_rmsnorm(x, None, g, 1e-6)[1]
        a = gu(hn)
        return a, down(asrq_b200.silu_mul(a))

    with lib_option("tc_pair", 0):
        a0, d0 = [t.clone() for t in chain()]
    for _ in range(150):
        a, d = chain()
        assert torch.equal(a, a0)
        assert torch.equal(d, d0)
    asrq_b200.check_status()


def test_bf16_prefill_error_is_reported():
    """bf16 activations on the prefill kernel: the MMA takes bf16 weights, so every dequantised weight is
    rounded to 8 significand bits first.  On Whisper fc1 (K=1280 N=5120 M=1500) the result stays within
    2e-3 of the row maximum plus half an output ulp for all but a small fraction of outputs; the
    measured excess is asserted here so that the documented figure cannot drift."""
    case = O.make_c1(seed=0)
    y = run_a16_abi("asrq_w4a16_gemm", case, dtype=torch.bfloat16)
    ref = _ref32(case, torch.bfloat16)
    err = (y.float().cpu() - ref).abs()
    tol = O.row_tolerance(ref) + bf16_half_ulp(ref)
    frac_out = float((err > tol).float().mean())
    worst = float((err / tol).max())
    print(f"bf16 prefill on fc1: {frac_out:.2e} of outputs beyond 2e-3*rowmax + half ulp, worst {worst:.2f}x")
    assert worst < 2.0 and frac_out < 1e-2


def test_injected_timeout_status_raises_and_clears():
    """A kernel whose bounded wait gives up writes (1, site) into the workspace status block.  That
    path is exercised from the host: the words are written by a copy, no device-side wait runs out."""
    import asrq_b200
    case = O.make_c3(seed=5, m=2, k=2048, n=256, bits=4, group_size=64)
    lq = make_layer(case)
    lq(case["x"].to(DEV))
    dev = torch.device(DEV)
    from asrq_b200 import linear as L
    ws = L._workspaces[(dev.index, torch.cuda.current_stream(dev).cuda_stream)]
    ws[:8].copy_(torch.tensor([1, 0, 0, 0, 14, 0, 0, 0], dtype=torch.uint8))
    with pytest.raises(_lib.AsrqError) as e:
        asrq_b200.check_status()
    assert e.value.code == -7 and "site 14" in str(e.value)
    assert int(ws[:256].view(torch.int32).abs().sum()) == 0      # cleared
    asrq_b200.check_status()                                       # and the next check is clean
    y = lq(case["x"].to(DEV))                                      # the workspace is usable again
    assert_close_rows(y, _ref32(case), what="after an injected status")


@pytest.mark.skipif(torch.cuda.is_available() and torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_module_on_non_current_device():
    """A layer on cuda:1 called while cuda:0 is the current device."""
    dev1 = torch.device("cuda", 1)
    case = O.make_c3(seed=6, m=3, k=2048, n=512, bits=4, group_size=64)
    lq = make_layer(case, device=dev1)
    assert torch.cuda.current_device() == 0
    y = lq(case["x"].to(dev1))
    assert y.device == dev1
    assert_close_rows(y, _ref32(case), what="layer on cuda:1, current device cuda:0")


@pytest.mark.parametrize("bits,g,m,k,n,bias,dtype", [
    (4, 64, 1, 2048, 6144, False, torch.float16),    # decode-sweep shapes, three tiles per block
    (4, 64, 16, 6144, 2048, False, torch.float16),   # one 48 KB tile per block, K split over all warps
    (2, 64, 8, 2048, 4096, False, torch.float16),
    (2, 64, 16, 6144, 2048, True, torch.float16),
    (4, 128, 32, 1280, 1280, True, torch.float16),   # whole-model decode batch: two token groups, one launch
    (4, 128, 32, 1280, 3840, True, torch.float16),   # fused q/k/v
    (4, 128, 32, 5120, 1280, True, torch.float16),
    (4, 128, 17, 1280, 5120, True, torch.bfloat16),  # ragged second token group
    (4, 128, 40, 1280, 1280, False, torch.float16),  # > 32 tokens: two launches
    (4, 32, 3, 256, 48, True, torch.float16),        # four groups per step, three tiles on three blocks
    (2, 256, 5, 512, 64, False, torch.float16),
    (4, 128, 4, 384, 4096, False, torch.float16),    # row bytes not a multiple of 128
])
def test_gemv_staged_kernel(bits, g, m, k, n, bias, dtype):
    """The staged decode kernel (weights prefetched into shared memory ahead of the stream dependency)
    against the fp32 CPU result, and against the strip-per-block kernel it replaces."""
    gen = torch.Generator().manual_seed(bits * 31 + m + n)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, g, False)
    case = dict(x=torch.randn(m, k, generator=gen).to(dtype), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half() if bias else None,
                bits=bits, group_size=g)
    with lib_option("gemv_kernel", 3):
        y = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=dtype)
        y2 = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=dtype)
    with lib_option("gemv_kernel", 1):
        y_old = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=dtype)
    ref = _ref32(case, dtype)
    extra = bf16_half_ulp(ref) if dtype == torch.bfloat16 else None
    assert_close_rows(y, ref, extra=extra, what=f"staged gemv w{bits} g{g} m{m} {k}x{n}")
    assert_close_rows(y_old, ref, extra=extra, what=f"strip gemv w{bits} g{g} m{m} {k}x{n}")
    assert torch.equal(y, y2)


@pytest.mark.parametrize("m", [1, 16, 32])
def test_decode_chain_orders_dependent_launches(m):
    """A chain of layers in which every launch consumes the previous launch's output, replayed as one CUDA
    graph: launches prefetch their weights before they wait for their predecessor, and must still see its
    output.  Same bits as the chain run without programmatic dependent launch."""
    gen = torch.Generator().manual_seed(m)
    d = 1280
    layers = []
    for i in range(6):
        w = torch.randn(d, d, generator=gen) * (1.0 / d ** 0.5)
        codes, scales, zeros, _ = O.rtn_codes(w, 4, 128, False)
        layers.append(make_layer(dict(x=torch.zeros(1, d), weight=O.pack_codes(codes, 4), scales=scales.half(),
                                      zeros=zeros.half(), bias=None, bits=4, group_size=128)))
    x = torch.randn(m, d, generator=gen).half().to(DEV)

    def chain():
        h = x
        for L in layers:
            h = L(h)
        return h
    with lib_option("no_pdl", 1):
        ref = chain().clone()
    torch.cuda.synchronize()
    eager = chain().clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = chain()
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(20):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(eager, ref) and torch.equal(out, ref)
    import asrq_b200
    asrq_b200.check_status()


@pytest.mark.parametrize("bits,g,m,k,n,bias,dtype", [
    (4, 128, 32, 1280, 1280, True, torch.float16),    # whole-model decode batch: 10 tiles x 8 K parts
    (4, 128, 32, 1280, 3840, True, torch.float16),    # fused q/k/v: 30 tiles x 4 parts
    (4, 128, 32, 1280, 5120, True, torch.float16),    # 40 tiles x 3 parts
    (4, 128, 32, 5120, 1280, True, torch.float16),    # long K: 12 parts of 6-7 K blocks
    (4, 128, 17, 1280, 1280, False, torch.bfloat16),  # ragged token tile
    (4, 128, 64, 1280, 5120, True, torch.float16),    # 64-token tile
    (4, 128, 50, 1024, 4096, False, torch.float16),
    (2, 64, 24, 512, 256, True, torch.float16),       # one K block per part
    (2, 128, 33, 2048, 1024, False, torch.bfloat16),
    (4, 64, 20, 64, 128, True, torch.float16),        # a single K block, a single tile, no split
])
def test_mid_m_tensor_core_kernel(bits, g, m, k, n, bias, dtype):
    """17..64 tokens on the chain-oriented tcgen05 kernel (weights fetched and unpacked ahead of the stream
    dependency, K parts meeting through the workspace) against the fp32 CPU result; two runs give the same
    bits and the tile counters come back to zero (checked by the call helper); against the kernels it replaces."""
    from asrq_b200 import _lib
    gen = torch.Generator().manual_seed(bits * 17 + m + n)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, g, False)
    case = dict(x=torch.randn(m, k, generator=gen).to(dtype), weight=O.pack_codes(codes, bits), scales=scales.half(),
                zeros=zeros.half(), bias=(torch.randn(n, generator=gen) * 0.02).half() if bias else None,
                bits=bits, group_size=g)
    ref = _ref32(case, dtype)
    y = run_a16_abi(f"asrq_w{bits}a16_gemm", case, dtype=dtype)
    y2 = run_a16_abi(f"asrq_w{bits}a16_gemm", case, dtype=dtype)
    assert torch.equal(y, y2)
    if dtype == torch.float16:
        assert_close_rows(y, ref, what=f"mid-M w{bits} m{m} {k}x{n}")
    else:
        wd = O.dequantize_weight(case["weight"], case["scales"], case["zeros"], bits, g, k, torch.float32)
        xf = case["x"].float()
        w_round = 6.0 * 2.0 ** -9 / 3 ** 0.5 * torch.sqrt((xf * xf) @ (wd * wd).t())
        assert_close_rows(y, ref, rel=2e-3, extra=bf16_half_ulp(ref) + w_round, what=f"mid-M bf16 w{bits} m{m} {k}x{n}")
    if m >= 32:
        with lib_option("mid_kernel", 1):
            y_old = run_a16_abi(f"asrq_w{bits}a16_gemm", case, dtype=dtype)
        scale = ref.abs().max(dim=-1, keepdim=True).values
        assert float(((y.float().cpu() - y_old.float().cpu()).abs() / scale).max()) < 4e-3


@pytest.mark.parametrize("m", [20, 64])
def test_mid_kernel_takes_the_qwen3_down_projection(m):
    """K = 6144 is 96 K blocks: eight parts of twelve.  Against the fp32 oracle and, bit for bit, two runs of itself."""
    case = O.make_c3(seed=11, m=m, k=6144, n=2048, bits=4, group_size=128)
    y = run_a16_abi("asrq_w4a16_gemm", case)
    assert_close_rows(y, _ref32(case), what=f"down projection m{m}")
    assert torch.equal(y, run_a16_abi("asrq_w4a16_gemm", case))
    with lib_option("mid_kernel", 1):
        y_old = run_a16_abi("asrq_w4a16_gemv" if m <= 32 else "asrq_w4a16_gemm", case)
    assert_close_rows(y_old, _ref32(case), what=f"down projection m{m}, other kernels")


@pytest.mark.parametrize("bits,dtype", [(4, torch.float16), (2, torch.float16), (4, torch.bfloat16), (2, torch.bfloat16)])
@pytest.mark.parametrize("m,k,n", [(17, 128, 128), (33, 192, 256), (64, 448, 128), (97, 2048, 128), (128, 2048, 12288), (193, 1280, 1280), (257, 5120, 256)])
def test_one_wave_kernel_tensor_memory_slots(m, k, n, bits, dtype):
    """Weights unpacked into tensor memory: fewer, as many and more K blocks than slots (three or six), rings of stages that go round,
    token tiles of 32 to 256 columns (half of tensor memory and all of it)."""
    gen = torch.Generator().manual_seed(m + k + n)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, 64, False)
    case = dict(x=torch.randn(m, k, generator=gen).to(dtype), weight=O.pack_codes(codes, bits), scales=scales.half(), zeros=zeros.half(),
                bias=(torch.randn(n, generator=gen) * 0.02).half(), bits=bits, group_size=64)
    y = run_a16_abi(f"asrq_w{bits}a16_gemm", case, dtype=dtype)
    ref = _ref32(case, dtype)
    extra = None
    if dtype == torch.bfloat16:  # the MMA takes weights rounded to bf16 (2^-9 of each): six standard deviations of that, and half an output ulp
        wd = codes.float() * scales.half().float().repeat_interleave(64, dim=1) + zeros.half().float().repeat_interleave(64, dim=1)
        extra = bf16_half_ulp(ref) + 6 * 2.0 ** -9 / 3 ** 0.5 * ((case["x"].float() ** 2) @ (wd ** 2).t()).sqrt()
    assert_close_rows(y, ref, extra=extra, what=f"one wave w{bits} m{m} {k}->{n}")
