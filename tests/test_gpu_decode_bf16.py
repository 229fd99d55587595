"""bf16 activations in the decode kernel (csrc/gemv_a16.cu): the fp32 sums are those of the exact codes, and nothing rides along."""
import pytest
import torch

from gpu_util import DEV, bf16_half_ulp, run_a16_abi
from oracle import linearq_oracle as O

pytestmark = pytest.mark.gpu


# every steps-per-warp and groups-per-step class: 128, 64 and 32 per group (4-bit), 256, 128 and 64 (2-bit); one wave and more
@pytest.mark.parametrize("bits,group,k,n", [(4, 128, 1280, 1280), (4, 64, 2048, 6144), (4, 32, 512, 256), (4, 128, 2048, 2048), (4, 128, 4096, 8192),
                                            (2, 256, 1280, 1280), (2, 64, 6144, 2048), (2, 128, 2048, 12288)])
@pytest.mark.parametrize("m", [1, 3, 8, 16])
@pytest.mark.parametrize("mean,scale", [(0.0, 1.0), (4.0, 1.0), (0.0, 1e5)])  # the last: beyond the range of fp16
def test_bf16_decode(bits, group, k, n, m, mean, scale):
    gen = torch.Generator().manual_seed(k + n + m)
    w = torch.randn(n, k, generator=gen) * 0.02
    codes, scales, zeros, _ = O.rtn_codes(w, bits, group, False)
    x = ((torch.randn(m, k, generator=gen) + mean) * scale).bfloat16()
    case = dict(x=x, weight=O.pack_codes(codes, bits), scales=scales.half(), zeros=zeros.half(), bias=None, bits=bits, group_size=group)
    y = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=torch.bfloat16).double().cpu()
    s, z = (t.half().double().repeat_interleave(group, dim=1) for t in (scales, zeros))
    wd = codes.double() * s + z
    ref = x.double() @ wd.t()
    assert_within(y, ref, x, codes, s, z)


def assert_within(y, ref, x, codes, s, z):
    # half an output ulp, and the fp32 sums of the terms code * scale * x and zero * x: fewer than 256 roundings, which add up like sixteen, each of
    # a last place (2^-24) of a partial sum; that is at most a quarter of all terms' magnitudes, since signs alternate
    bound = bf16_half_ulp(ref.float()).double() * 1.01 + 2.0 ** -22 * (x.double().abs() @ ((codes.double() * s).abs() + z.abs()).t())
    err = (y - ref).abs()
    assert bool((err <= bound).all()), float((err / bound.clamp_min(1e-300)).max())


@pytest.mark.parametrize("bits,group,k,n", [(4, 128, 1280, 1280), (4, 64, 2048, 2048), (4, 32, 512, 256), (2, 256, 1280, 1280), (2, 64, 6144, 2048), (2, 128, 2048, 2048)])
@pytest.mark.parametrize("m", [1, 2, 3, 8, 9, 16])
def test_large_activations_of_zero_weights_leave_the_sums_alone(bits, group, k, n, m):
    """Every other activation is 2^14 as large and meets a weight of exactly zero (code 0, zero point 0): no bit of the result is lost
    to it.  A sum that carried a multiple of sum(x) would lose ten and more."""
    gen = torch.Generator().manual_seed(k + n + m)
    codes = torch.randint(0, 2 ** bits, (n, k), generator=gen)
    x = torch.randn(m, k, generator=gen)
    large = torch.randperm(k, generator=gen)[:k // 2]
    codes[:, large] = 0
    x[:, large] *= 2.0 ** 14
    x = x.bfloat16()
    scales, zeros = torch.rand(n, k // group, generator=gen) * 0.01 + 0.005, torch.zeros(n, k // group)
    case = dict(x=x, weight=O.pack_codes(codes, bits), scales=scales.half(), zeros=zeros.half(), bias=None, bits=bits, group_size=group)
    y = run_a16_abi(f"asrq_w{bits}a16_gemv", case, dtype=torch.bfloat16).double().cpu()
    s = scales.half().double().repeat_interleave(group, dim=1)
    assert_within(y, x.double() @ (codes.double() * s).t(), x, codes, s, torch.zeros_like(s))
