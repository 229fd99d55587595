"""What lies between a Conformer block's layers (csrc/conformer.cu) against the sequence of modules it replaces."""
import pytest
import torch
import torch.nn.functional as F

from asrq_b200 import conformer as C, linear

pytestmark = pytest.mark.gpu


def _ulps(y, ref, dtype, n=2):
    eps = 2.0 ** (-10 if dtype == torch.float16 else -7)
    err = (y.float() - ref.float()).abs() - n * eps * ref.float().abs().clamp(min=0.25)
    assert float(err.max()) <= 0, float(err.max())


@pytest.mark.parametrize("rows,dim,dtype", [(1, 256, torch.float16), (3, 512, torch.bfloat16), (7, 768, torch.float16), (250, 1024, torch.float16),
                                            (5, 1280, torch.bfloat16), (4, 1536, torch.float16), (9, 1792, torch.float16), (513, 2048, torch.float16)])
def test_residual_norms(rows, dim, dtype):
    g = torch.Generator().manual_seed(rows + dim)
    x, d = (torch.randn(rows, dim, generator=g).to(dtype).cuda() for _ in range(2))
    n1, n2 = (((1 + 0.1 * torch.randn(dim, generator=g)).to(dtype).cuda(), torch.randn(dim, generator=g).to(dtype).cuda()) for _ in range(2))
    s = x + 0.5 * d
    got, h = linear.residual_norms(x, d, 0.5, n1)
    assert torch.equal(got, s)
    _ulps(h, F.layer_norm(s, (dim,), *n1), dtype)
    same, h = linear.residual_norms(x, None, 1.0, n1)
    assert same is x
    _ulps(h, F.layer_norm(x, (dim,), *n1), dtype)
    y, none = linear.residual_norms(x, d, 0.5, n1, write_h=False)
    assert none is None
    y2, z = linear.residual_norms(x, d, 0.5, n1, n2)
    assert torch.equal(y, y2)
    _ulps(y, F.layer_norm(s, (dim,), *n1), dtype)
    _ulps(z, F.layer_norm(y, (dim,), *n2), dtype)


@pytest.mark.parametrize("B,T,d,dtype", [(1, 1, 64, torch.float16), (2, 15, 256, torch.bfloat16), (1, 16, 6, torch.float16), (3, 17, 258, torch.float16),
                                         (2, 250, 1024, torch.float16), (1, 33, 2050, torch.bfloat16)])
def test_glu_dwconv(B, T, d, dtype):
    g = torch.Generator().manual_seed(B + T + d)
    x = torch.randn(B, T, 2 * d, generator=g).to(dtype).cuda()
    w, b = (0.3 * torch.randn(d, 1, 9, generator=g)).to(dtype).cuda(), torch.randn(d, generator=g).to(dtype).cuda()
    sc, sh = (torch.randn(d, generator=g).to(dtype).cuda() for _ in range(2))
    y = linear.glu_dwconv(x, w, b, sc, sh)
    u = F.glu(x, dim=-1)
    c = F.conv1d(u.transpose(1, 2).double(), w.double(), b.double(), padding=4, groups=d).to(dtype).transpose(1, 2)
    ref = F.silu(c * sc + sh)
    assert float((y.float() - ref.float()).abs().max()) <= (1e-2 if dtype == torch.float16 else 8e-2)


def test_joined_layers_follow_their_parts():
    """The fused blocks give what :meth:`block` gives (up to 4-bit code flips), and step aside for replaced buffers."""
    enc = C.FastConformerStandIn("cuda", n_layers=2, d_model=256, ffn=512, heads=4, mel=80, sub_channels=64, seed=4)
    feats = torch.randn(2, 80, 600, generator=torch.Generator().manual_seed(5)).half()
    assert enc._blocks_covered()
    a, b = enc.encode(feats).float(), enc.encode(feats, hook=lambda *_: None).float()
    assert float((a - b).abs().mean()) <= 0.02 * float(b.abs().max())
    q = enc.layers[1]["q"]
    q.load_quantized_params(q.scales * 2, q.zeros, q.weight.clone())
    assert not enc._blocks_covered()
    assert torch.equal(enc.encode(feats), enc.encode(feats, hook=lambda *_: None))
