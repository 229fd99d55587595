"""The elementwise steps of a Conformer block (csrc/conformer.cu) are the sequence of modules, bit for bit."""
import pytest
import torch
import torch.nn.functional as F

from asrq_b200 import linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,C,T,dtype", [(1, 2, 1, torch.float16), (2, 64, 63, torch.float16), (1, 66, 65, torch.bfloat16), (3, 1024, 126, torch.float16),
                                         (2, 130, 250, torch.bfloat16), (2, 6, 7, torch.float16)])
def test_steps(B, C, T, dtype):
    g = torch.Generator().manual_seed(B * C + T)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()  # noqa: E731
    u, b2 = 2 * r(B, 2 * C, T), r(2 * C)
    assert torch.equal(linear.bias_glu(u, b2), F.glu(u + b2.view(1, -1, 1), dim=1))
    c, b, sc, sh = r(B, C, T), r(C), r(C), r(C)
    assert torch.equal(linear.bias_affine_silu(c, b, sc, sh), F.silu((c + b.view(1, -1, 1)) * sc.view(1, -1, 1) + sh.view(1, -1, 1)))
    x = r(B, T, C)
    assert torch.equal(linear.bias_add_transposed(x, c, b), x + (c + b.view(1, -1, 1)).transpose(1, 2))
    y, z = r(B, T, 8), r(B, T, 8) * 1e-6
    assert torch.equal(linear.half_step(y, z), y + 0.5 * z)
