"""Attention of one decoding step (csrc/decode_attn.cu) against fp32 PyTorch at the edges of its splits: a warp's batch is 32
keys (head of 64) or 16 (head of 128), a block has 2, 4 or 8 warps, an item 1 to 8 blocks."""
import pytest
import torch

from asrq_b200 import linear

pytestmark = pytest.mark.gpu


def _softmax_attention(q, k, v, scale):  # q (B, H, hd), k / v (B, H, T, hd)
    p = torch.softmax(torch.einsum("bhd,bhtd->bht", q.double(), k.double()) * scale, -1)
    return torch.einsum("bht,bhtd->bhd", p, v.double())


@pytest.mark.parametrize("B,H,hd,keys,dtype", [
    (1, 1, 64, 1, torch.float16), (1, 20, 64, 1500, torch.float16), (2, 3, 128, 17, torch.bfloat16), (3, 20, 64, 257, torch.bfloat16),
    (5, 20, 64, 1500, torch.float16), (32, 20, 64, 100, torch.float16), (40, 8, 128, 33, torch.float16), (16, 20, 64, 1500, torch.float16), (28, 20, 64, 191, torch.bfloat16),
])
@pytest.mark.parametrize("settled", [False, True])
def test_cross(B, H, hd, keys, dtype, settled):
    g = torch.Generator().manual_seed(B * keys)
    q = torch.randn(B, H * hd, generator=g).to(dtype).cuda()
    kv = torch.randn(B, keys, 2 * H * hd, generator=g).to(dtype).cuda()
    y = linear.decode_cross_attention(q, kv, H, hd ** -0.5, settled=settled)
    k, v = (t.reshape(B, keys, H, hd).transpose(1, 2) for t in kv.split(H * hd, -1))
    ref = _softmax_attention(q.view(B, H, hd), k, v, hd ** -0.5).reshape(B, H * hd)
    assert (y.double() - ref).abs().max() < (2e-3 if dtype == torch.float16 else 1.6e-2)


@pytest.mark.parametrize("B,H,hd,pos", [(1, 2, 64, 0), (1, 20, 64, 31), (2, 20, 64, 32), (3, 4, 128, 447), (16, 20, 64, 300), (40, 20, 64, 129)])
def test_self(B, H, hd, pos):
    g = torch.Generator().manual_seed(B + pos)
    qkv = torch.randn(B, 3 * H * hd, generator=g).half().cuda()
    kv = torch.randn(2, B, H, 448, hd, generator=g).half().cuda()
    kv[:, :, :, pos + 1:] = float("nan")  # nothing past the position is read
    y = linear.decode_self_attention(qkv, kv, torch.tensor([pos], device="cuda"), hd ** -0.5)
    q, k, v = (t.reshape(B, H, hd) for t in qkv.split(H * hd, -1))
    assert torch.equal(kv[0, :, :, pos], k) and torch.equal(kv[1, :, :, pos], v)
    ref = _softmax_attention(q, kv[0, :, :, :pos + 1], kv[1, :, :, :pos + 1], hd ** -0.5).reshape(B, H * hd)
    assert (y.double().view_as(ref) - ref).abs().max() < 2e-3


@pytest.mark.parametrize("B,nkv,pos,dtype", [(1, 8, 0, torch.float16), (1, 2, 15, torch.bfloat16), (2, 8, 16, torch.float16),
                                             (3, 8, 511, torch.bfloat16), (40, 8, 260, torch.float16)])
def test_grouped(B, nkv, pos, dtype):
    """Against qk_norm_rope (same cache bits) and fp32 attention over its cache."""
    g = torch.Generator().manual_seed(B * 1000 + pos)
    hd, nq, max_len = 128, 2 * nkv, 512
    qkv = torch.randn(B, (nq + 2 * nkv) * hd, generator=g).to(dtype).cuda()
    qn, kn = ((1 + 0.1 * torch.randn(hd, generator=g)).to(dtype).cuda() for _ in range(2))
    ang = torch.rand(max_len, hd // 2, generator=g) * 6.3
    cos, sin = (torch.cat([f(ang)] * 2, -1).to(dtype).cuda() for f in (torch.cos, torch.sin))
    kc, vc = (torch.randn(B, nkv, max_len, hd, generator=g).to(dtype).cuda() for _ in range(2))
    p = torch.tensor([pos], device="cuda")
    kc2, vc2 = kc.clone(), vc.clone()
    y = linear.decode_grouped_attention(qkv, qn, kn, cos, sin, kc, vc, p, nq, 1e-6, hd ** -0.5)
    q = linear.qk_norm_rope(qkv, qn, kn, cos, sin, kc2, vc2, p, B, 1, nq, nkv, 1e-6).view(B, nq, hd)
    assert torch.equal(kc, kc2) and torch.equal(vc, vc2)
    k, v = (t[:, :, :pos + 1].repeat_interleave(2, 1) for t in (kc, vc))
    ref = _softmax_attention(q, k, v, hd ** -0.5).reshape(B, nq * hd)
    assert (y.double() - ref).abs().max() < (2e-3 if dtype == torch.float16 else 1.6e-2)


@pytest.mark.parametrize("hd", [64, 128])
def test_self_behind_the_kernel_that_wrote_the_cache(hd):
    """A prompt's keys and values written by the library's own kernel, some waves of blocks long, directly ahead: the call waits
    for them.  (With ``settled`` the caller says that it need not; the same bits when that is so.)"""
    B, H, T, max_len = 32, 16, 200, 256
    g = torch.Generator().manual_seed(hd)
    prompt = torch.randn(B * T, 3 * H * hd, generator=g).half().cuda()
    qkv = torch.randn(B, 3 * H * hd, generator=g).half().cuda()
    w, pos = torch.ones(hd, dtype=torch.half, device="cuda"), torch.tensor([T], device="cuda")
    cos = torch.randn(max_len, hd, generator=g).half().cuda()
    kv = torch.zeros(2, B, H, max_len, hd, dtype=torch.half, device="cuda")
    want = None
    for _ in range(10):
        kv.zero_()
        linear.qk_norm_rope(prompt, w, w, cos, cos, kv[0], kv[1], 0, B, T, H, H, 1e-6)
        y = linear.decode_self_attention(qkv, kv, pos, hd ** -0.5)
        if want is None:
            torch.cuda.synchronize()
            want = linear.decode_self_attention(qkv, kv, pos, hd ** -0.5, settled=True)
        assert torch.equal(y, want)
