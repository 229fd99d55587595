"""The one-wave tensor-core kernel at its edges: token tiles of 32 to 256 columns, one to eight K parts, parts longer than its ring
of stages, and tokens that divide neither among the parts nor into tiles."""
import pytest
import torch

from oracle import linearq_oracle as O
from tests.gpu_util import assert_close_rows, make_layer
from tests.test_gpu_a16 import _ref32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,bits", [
    (17, 1280, 1280, 4),   # eight parts of two or three K blocks
    (33, 2048, 4096, 4),   # four parts
    (64, 1280, 5120, 2),   # three parts
    (65, 1280, 1280, 4), (96, 2048, 2048, 4), (97, 1280, 3840, 2), (128, 1280, 5120, 4), (128, 64, 128, 4),
    (20, 6144, 2048, 4), (64, 6144, 2048, 4),   # six parts of sixteen
    (31, 8192, 128, 4),    # eight parts of sixteen
    (24, 2048, 12288, 4),  # one part, 32 K blocks through a ring of sixteen stages
    (65, 2048, 12288, 4), (128, 2048, 12288, 2),   # of eleven and of eight
    (24, 256, 19200, 4), (128, 128, 19072, 2),     # 150 and 149 feature tiles, more than one wave: the other kernels
    (129, 1280, 1280, 4), (257, 5120, 1280, 4), (300, 6144, 2048, 2),   # several token tiles; stages used many times
    (511, 2048, 2048, 4), (1000, 5120, 1280, 4), (1300, 6144, 256, 4), (2048, 5120, 256, 2),
])
def test_one_wave_kernel(m, k, n, bits):
    case = O.make_c3(seed=m + k, m=m, k=k, n=n, bits=bits, group_size=64 if k == 64 else 128)
    layer = make_layer(case)
    x = case["x"].cuda()
    y = layer(x)
    assert_close_rows(y.cpu(), _ref32(case), what=f"w{bits} m{m} {k}x{n}")
    assert torch.equal(y, layer(x))
    res = torch.randn_like(y)
    assert torch.equal(layer.forward_fused(x, residual=res), res + y)
