"""bf16 activations in the decode kernel (csrc/gemv_a16.cu): codes ride on 128.0's mantissa, so a group's sum carries 128 * sum(x),
which its zero's term takes away again."""
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
    # half an output ulp, and fp32 sums of terms as large as (128 + code) * scale * |x|: 2^-22 of their sum in two's exponents
    bound = bf16_half_ulp(ref.float()).double() * 1.01 + 2.0 ** -22 * (x.double().abs() @ (((128 + codes.double()) * s).abs() + z.abs()).t())
    assert bool(((y - ref).abs() <= bound).all()), float(((y - ref).abs() / bound).max())
