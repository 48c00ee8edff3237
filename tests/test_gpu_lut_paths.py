"""Edges of the table-lookup kernels on the GPU: the vector forms of the dequantizers against the arithmetic they stand for.

Oracle: the dense weights of the packed tensors; compared bit by bit.
"""
import numpy as np
import pytest
import torch

from tests import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from decdec_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("bits", [3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("N,K", [(1, 32), (37, 1056), (300, 2048)])
def test_anyprec_dequant_forms(ops, dtype, bits, N, K):
    L = P.lut_layer(N, K, bits, seed=N + K + bits, dtype=dtype, real=False)
    held = torch.zeros(L["lut"].numel() + 1, dtype=L["lut"].dtype, device="cuda")
    shifted = held[1:].view_as(L["lut"]).copy_(L["lut"])                       # a table that is not 16-byte aligned
    for lut in (L["lut"].cuda(), shifted):
        assert np.array_equal(P.to_np(ops.anyprec_dequant(L["qweight"].cuda(), lut, bits)), L["w_hat"])


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("bits", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K,group", [(4, 32, 32), (36, 96, 32), (30, 96, 32), (2052, 1024, 128)])
def test_lutgemm_dequant_forms(ops, dtype, bits, N, K, group):
    """Four outputs per thread (N a multiple of 4) and the general form, with scales among them that cancel."""
    L = P.random_bcq_layer(N, K, bits, group, seed=N + bits, dtype=dtype)
    alpha = L["alpha"].clone()
    alpha[..., ::3] = alpha[..., :1, ::3]                                       # equal scales: sums of zero
    bias = L["q_bias"].clone()
    bias[..., ::2] = -0.0
    out = ops.lutgemm_dequant(L["qweight"].cuda(), alpha.cuda(), bias.cuda(), bits, group).cpu()
    words = L["qweight"].numpy().view(np.uint32)
    bit = ((words[:, None] >> np.arange(32, dtype=np.uint32)[None, :, None, None]) & 1).reshape(K, bits, N)
    gidx = torch.arange(K) // group
    total = torch.zeros(K, N)
    for p in range(bits):
        total = total + torch.from_numpy(bit[:, p].astype(np.float32) * 2 - 1) * alpha.float()[gidx, p]
    expected = total.to(P.TORCH_DT[dtype]) + bias[gidx]
    assert torch.equal(out.view(torch.int16), expected.view(torch.int16))
