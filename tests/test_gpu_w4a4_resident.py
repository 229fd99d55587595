"""The W4A4 GEMM with its weights kept in shared memory over a worker's token tiles gives the bits of the tile-by-tile form."""
import pytest
import torch

from asrq_b200 import LinearQQ, packing
from tests.gpu_util import lib_option

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,g", [
    (4100, 1024, 1024, 128),   # two tiles for most workers, a ragged last token tile
    (6000, 1024, 4096, 128),   # workers that change the feature tile
    (16000, 1024, 3072, 128),
    (9001, 512, 2048, 256), (5000, 256, 4096, 128), (3000, 1024, 4096, 512),
])
def test_resident_weights(m, k, n, g):
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    weight, scales = packing.pack_w4a4_cuda(torch.randn(n, k, generator=gen, device="cuda") * 0.02, g, True)
    layer = LinearQQ(k, n, 4, 4, g, bias=True, hadamard=True).cuda()
    layer.load_quantized_params(scales, torch.zeros_like(scales), weight)
    layer.bias = (torch.randn(n, generator=gen, device="cuda") * 0.1).half()
    x = torch.randn(m, k, generator=gen, device="cuda").half()
    y = layer(x)
    with lib_option("w4a4_bt", 96):
        ref = layer(x)
    assert torch.equal(y, ref)
    assert all(torch.equal(layer(x), y) for _ in range(5))
