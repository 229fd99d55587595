"""The step's argmax kernel against torch.argmax: ties, NaN, infinities, odd widths, fewer columns than blocks."""
import pytest
import torch

from asrq_b200 import linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,dtype", [(1, 51866, torch.float16), (3, 151936, torch.bfloat16), (2, 7, torch.float16), (64, 1025, torch.float16),
                                       (5, 4098, torch.bfloat16)])
def test_argmax_rows(B, N, dtype):
    g = torch.Generator().manual_seed(B * N)
    scratch = torch.zeros(2 * B, dtype=torch.long, device="cuda")
    tok, ids, pos = torch.empty(B, dtype=torch.long, device="cuda"), torch.zeros(4, B, dtype=torch.long, device="cuda"), torch.tensor([2], device="cuda")
    base = torch.randn(B, N, generator=g).to(dtype)
    few = (base * 2).round()                                   # many equals: the first counts
    odd = base.clone()
    odd[:, N // 2], odd[0, N // 3] = float("inf"), float("nan")
    for y in (base, few, odd, torch.full_like(base, float("-inf")), -base.abs(), torch.zeros_like(base) * torch.where(base > 0, -1.0, 1.0).to(dtype)):
        y = y.cuda()
        linear.argmax_rows(y, tok, scratch, ids, pos)
        top = y.isnan().float().argmax(-1) if bool(y[0].isnan().any()) else None
        want = (y.float().cpu() == y.float().cpu().amax(-1, keepdim=True)).int().argmax(-1)  # the first of the largest
        if top is not None:
            want[0] = int(top[0])
        assert torch.equal(tok.cpu(), want) and torch.equal(ids[2].cpu(), want)
        assert not bool(scratch.any())
    assert not bool(ids[[0, 1, 3]].any())
