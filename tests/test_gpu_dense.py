"""Large W{2,4}A16 calls that dequantise the weights once (csrc/gemm_a16_dense.cu): the same bits as the kernels that unpack inside
the GEMM, at the edges of its tiles and of its shares of a round."""
import pytest
import torch

import asrq_b200
from asrq_b200 import _lib, packing
from gpu_util import DEV, lib_option

pytestmark = pytest.mark.gpu


def _layer(k, n, bits, group, bias):
    gen = torch.Generator(device=DEV).manual_seed(k + n + bits)
    layer = asrq_b200.LinearQ(k, n, bits, group, bias=bias).to(DEV)
    w, s, z = packing.rtn_pack_cuda((torch.randn(n, k, generator=gen, device=DEV) * 0.02).half(), bits, group)
    layer.load_quantized_params(s, z, w)
    if bias:
        layer.bias = (torch.randn(n, generator=gen, device=DEV) * 0.02).half()
    return layer, gen


# one K block; a single narrow tile; tiles of 256 with half a one left; more than one round with a ragged rest; 128 features beyond 256s
@pytest.mark.parametrize("k,n,group", [(64, 128, 64), (128, 256, 64), (640, 1408, 128), (1280, 5120, 128), (2048, 2048, 64)])
@pytest.mark.parametrize("m", [17, 31, 128, 257, 1500, 6001])
@pytest.mark.parametrize("bits,dtype", [(4, torch.float16), (2, torch.bfloat16), (4, torch.bfloat16), (2, torch.float16)])
def test_same_bits_as_unpacking_inside(m, k, n, group, bits, dtype):
    layer, gen = _layer(k, n, bits, group, bias=m != 31)
    asrq_b200.linear._workspace(torch.device(DEV), _lib.workspace_bytes(_lib.WS_LINEARQ, 1 << 14, n, k))
    x = torch.randn(m, k, generator=gen, device=DEV).to(dtype)
    r = torch.randn(m, n, generator=gen, device=DEV).to(dtype)
    times = -(-512 // m)  # few tokens go to other kernels: the reference takes the rows several times over
    for kw in ({}, {"gelu": True}, {"residual": r}, {"gelu": True, "residual": r}):
        with lib_option("tc_pair", 0), lib_option("mid_kernel", 1), lib_option("tc_split", 1):
            rep = {q: v.repeat(times, 1) if q == "residual" else v for q, v in kw.items()}
            want = layer.forward_fused(x.repeat(times, 1), **rep)[:m]
        with lib_option("tc_pair", 2):
            got = layer.forward_fused(x, **kw)
        assert torch.equal(got, want), kw
    asrq_b200.check_status()


def test_a_small_workspace_unpacks_inside():
    """A workspace without room for the 16-bit weights runs the call as before, with the same bits."""
    layer, gen = _layer(1280, 5120, 4, 128, True)
    x = torch.randn(6000, 1280, generator=gen, device=DEV).half()
    want = layer(x)
    assert _lib.workspace_bytes(_lib.WS_LINEARQ, 6000, 5120, 1280) > 2 * 5120 * 1280
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device=DEV)
    got = torch.empty_like(want)
    _lib.call("asrq_linearq_a16", 4, x.data_ptr(), layer.weight.data_ptr(), layer.scales.data_ptr(), layer.zeros.data_ptr(), layer.bias.data_ptr(),
              got.data_ptr(), 6000, 5120, 1280, 128, _lib.F16, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert torch.equal(got, want)
