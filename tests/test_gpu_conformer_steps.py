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


def test_operands_the_kernels_cannot_check():
    """The kernels get addresses and sizes: the wrappers refuse what does not fit them and lay out what is not contiguous."""
    x, c, b = (torch.randn(*s, device="cuda").half() for s in ((2, 5, 16), (2, 16, 5), (16,)))
    assert torch.equal(linear.bias_add_transposed(x, x.transpose(1, 2), b), linear.bias_add_transposed(x, x.transpose(1, 2).contiguous(), b))
    assert torch.equal(linear.bias_glu(x.transpose(1, 2), b), linear.bias_glu(x.transpose(1, 2).contiguous(), b))
    assert torch.equal(linear.half_step(c.transpose(1, 2), x), linear.half_step(c.transpose(1, 2).contiguous(), x))
    tok, scratch, pos = (torch.zeros(n, dtype=torch.long, device="cuda") for n in (2, 4, 1))
    kv, kc, q = (torch.zeros(*s, dtype=torch.half, device="cuda") for s in ((2, 2, 1, 8, 64), (2, 1, 8, 128), (2, 512)))
    w, t = torch.ones(128, device="cuda").half(), torch.ones(8, 128, device="cuda").half()
    for call in (lambda: linear.bias_add_transposed(x, c[:, :8], b), lambda: linear.bias_glu(c, b[:8]), lambda: linear.bias_glu(c, b.float()),
                 lambda: linear.bias_affine_silu(c, b, b, b[:8]), lambda: linear.half_step(x, x[:1]),
                 lambda: linear.argmax_rows(x[0], tok, scratch), lambda: linear.argmax_rows(q.t()[:2], tok, scratch),
                 lambda: linear.argmax_rows(q, tok, scratch[:3]), lambda: linear.argmax_rows(q, tok.int(), scratch),
                 lambda: linear.decode_self_attention(q[:, :192], kv.float(), pos), lambda: linear.decode_self_attention(q[:, :192], kv[..., ::2], pos),
                 lambda: linear.decode_cross_attention(q[:, :64], c.reshape(2, 5, 16), 1),
                 lambda: linear.decode_grouped_attention(q, w, w, t, t, kc, kc[:1], pos, 2, 1e-6, 1.0),
                 lambda: linear.decode_grouped_attention(q, w, w, t[:4], t, kc, kc.clone(), pos, 2, 1e-6, 1.0),
                 lambda: linear.decode_grouped_attention(q, w, w, t, t, kc, kc.clone(), pos.int(), 2, 1e-6, 1.0)):
        with pytest.raises(ValueError):
            call()
    with pytest.raises(RuntimeError):                              # torch.matmul's own refusal
        linear.dense_head(q, q[:, :256])
