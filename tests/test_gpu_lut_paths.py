"""Edges of the table-lookup kernels on the GPU: ragged layers (binary-coded), pair tables (SqueezeLLM), row
pairs (any-precision), vector dequantizers.

Oracle: the dense weights of the packed tensors in float64.  Tolerances of the GEMVs: products and sums are fp32, and the output is rounded once; with y = 0 before the call the error of an output is at most
half an ulp of it (2^-11 or 2^-8 of its size in fp16 and bf16) plus the fp32 sum's, K * 2^-24 of the sum of magnitudes, which
the bound below takes at its worst.  Dense weights are compared exactly.
"""
import numpy as np
import pytest
import torch

from oracle import formats, forward
from tests import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from decdec_b200 import ops as _ops
    return _ops


HALF_ULP = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8, "fp32": 2.0 ** -24}


def _assert_sums(y, w_hat, x, dtype):
    xd = P.to_np(x).reshape(-1)
    ref = w_hat @ xd
    mags = np.abs(w_hat) @ np.abs(xd)
    bound = HALF_ULP[dtype] * np.abs(ref) + w_hat.shape[1] * 2.0 ** -24 * mags + 2.0 ** -24
    worst = (np.abs(P.to_np(y).reshape(-1) - ref) / bound).max()
    assert worst <= 1.0, f"error up to {worst:.2f} of its bound"


@pytest.mark.parametrize("dtype", ["fp16", "bf16", "fp32"])
@pytest.mark.parametrize("N,K,bits,group", [
    (8, 32, 2, 32),          # a box larger than the tensor in every direction
    (120, 480, 3, 32),       # one short tile, one short slice
    (136, 544, 4, 32),       # one output tile and one slice, each with a remainder
    (2776, 1184, 4, 32),
    (3000, 4224, 3, 128),    # many tiles, the last slice a quarter full
])
def test_lutgemm_ragged_layers(ops, dtype, N, K, bits, group):
    L = P.random_bcq_layer(N, K, bits, group, seed=N + K, dtype=dtype)
    x = P.make_activation(K, seed=11, dtype=dtype)
    big = torch.zeros(N + 256, dtype=P.TORCH_DT[dtype], device="cuda")
    y = big[:N].view(1, 1, N)
    for _ in range(2):                                   # the second call finds the workspace as the first left it
        y.zero_()
        ops.lutgemm_gemv(x.cuda(), y, L["qweight"].cuda(), L["alpha"].cuda(), L["q_bias"].cuda(), bits, group)
        _assert_sums(y, L["w_hat"], x, dtype)
        assert not big[N:].any()                         # nothing beyond the last output


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("N,K", [
    (2, 32),            # one pair of columns, one group
    (64, 416),          # one tile, groups that do not fill the warps evenly
    (66, 1024),         # a tile of two columns
    (63, 256),          # odd: general kernel
    (190, 8192),        # tiles cut over several thread blocks
    (9600, 768),        # many tiles of few groups
    (9600, 1024),       # small layers above take the general kernel
    (2, 2336),
    (66, 2400),
])
def test_sqllm_pair_tables(ops, dtype, bits, N, K):
    L = P.lut_layer(N, K, bits, seed=N + K + bits, dtype=dtype, fmt="sqllm", real=False)
    x = P.make_activation(K, seed=7, dtype=dtype)
    for _ in range(2):                                   # the second call finds the workspace as the first left it
        y = torch.zeros(1, 1, N, dtype=P.TORCH_DT[dtype], device="cuda")
        ops.sqllm_gemv(x.cuda(), y, L["qweight"].cuda(), L["lut"].cuda(), bits)
        _assert_sums(y, L["w_hat"], x, dtype)


@pytest.mark.parametrize("K", [1024, 2400])      # general kernel, pair tables
@pytest.mark.parametrize("bits", [3, 4])
def test_sqllm_values_that_are_not_finite_stay_in_their_column(ops, bits, K):
    N = 256
    L = P.lut_layer(N, K, bits, seed=9, fmt="sqllm", real=False)
    lut = L["lut"].clone()
    lut[5, 1], lut[70, 2], lut[133, 0] = float("inf"), float("nan"), float("-inf")
    x = P.make_activation(K, seed=7).abs() + 1
    y = torch.zeros(1, 1, N, dtype=torch.float16, device="cuda")
    ops.sqllm_gemv(x.cuda(), y, L["qweight"].cuda(), lut.cuda(), bits)
    got = P.to_np(y).reshape(-1)
    assert got[5] == np.inf and np.isnan(got[70]) and got[133] == -np.inf
    rest = np.ones(N, bool)
    rest[[5, 70, 133]] = False
    _assert_sums(torch.from_numpy(got[rest]), L["w_hat"][rest], x, "fp16")


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("N,K,bits", [
    (1, 128, 3), (17, 128, 4), (33, 2048, 3), (33, 2048, 4), (47, 2176, 3), (47, 2176, 8), (300, 6272, 3), (31, 6272, 6),
    (3, 32768, 3), (3, 32768, 8), (2999, 1152, 3), (2999, 1152, 5), (2999, 1152, 7),
])
def test_anyprec_row_pairs(ops, dtype, N, K, bits):
    L = P.lut_layer(N, K, bits, seed=N + K + bits, dtype=dtype, real=False)
    x = P.make_activation(K, seed=8, dtype=dtype)
    held = torch.zeros(K + 1, dtype=x.dtype, device="cuda")
    for xd in (x.cuda(), held[1:].copy_(x.reshape(-1)).view(1, 1, K)):        # aligned, and one element into a buffer
        y = torch.zeros(1, 1, N, dtype=P.TORCH_DT[dtype], device="cuda")
        ops.anyprec_gemv(xd, y, L["qweight"].cuda(), L["lut"].cuda(), bits)
        _assert_sums(y, L["w_hat"], x, dtype)


@pytest.mark.parametrize("bits", [3, 4])
def test_anyprec_values_that_are_not_finite_stay_in_their_row(ops, bits):
    """Lanes without a plane word (K = 1152: a tail block of four words) add nothing, whatever their row's table holds."""
    N, K = 64, 1152
    L = P.lut_layer(N, K, bits, seed=10, real=False)
    codes, lut = L["codes"].copy(), L["lut"].clone()
    codes[codes == 0] = 1
    lut[:, 0] = float("inf")                              # an entry that no weight uses
    lut[9, 1] = float("nan")
    x = P.make_activation(K, seed=8)
    y = torch.zeros(1, 1, N, dtype=torch.float16, device="cuda")
    ops.anyprec_gemv(x.cuda(), y, torch.from_numpy(formats.anyprec_pack(codes, bits).copy()).cuda(), lut.cuda(), bits)
    got = P.to_np(y).reshape(-1)
    w_hat = np.take_along_axis(P.to_np(lut), codes.astype(np.int64), 1)
    assert np.isnan(got[9])
    rest = np.arange(N) != 9
    _assert_sums(torch.from_numpy(got[rest]), w_hat[rest], x, "fp16")


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


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("N,K,bits,n_tb", [
    (2050, 320, 4, 0),         # two columns in the last tile
    (4096, 4096, 3, 0),        # every tile in several parts
    (19200, 2336, 4, 0),       # whole tiles and cut ones in one thread block
    (2056, 2400, 4, 16),       # beside a compensation, eight columns in the last tile
    (9536, 2336, 4, 148),
])
def test_sqllm_parts_of_a_tile(ops, dtype, N, K, bits, n_tb):
    """Sums of parts meet in a fixed order: repeated calls give the same bits, on top of outputs that are not zero."""
    L = P.lut_layer(N, K, bits, seed=N + K, dtype=dtype, fmt="sqllm", real=False)
    x = P.make_activation(K, seed=7, dtype=dtype)
    y0 = (torch.randn(1, 1, N, generator=torch.Generator().manual_seed(3)) * 2).to(P.TORCH_DT[dtype])
    qw, lut, xd = L["qweight"].cuda(), L["lut"].cuda(), x.cuda()
    ref = L["w_hat"] @ P.to_np(x).reshape(-1) + P.to_np(y0).reshape(-1)
    mags = np.abs(L["w_hat"]) @ np.abs(P.to_np(x).reshape(-1)) + np.abs(P.to_np(y0).reshape(-1))
    outs = []
    for _ in range(8):
        y = y0.clone().cuda()
        ops.sqllm_gemv(xd, y, qw, lut, bits)
        outs.append(y)
    assert all(torch.equal(y, outs[0]) for y in outs)
    if n_tb:
        cs, rs = P.random_residual(N, K, seed=5, dtype=dtype)
        thr = P.make_thresholds(K, dtype, n_calib=32)
        k = 4 * K // 1024
        rows, acts = torch.zeros(k, dtype=torch.int32, device="cuda"), torch.zeros(k, dtype=P.TORCH_DT[dtype], device="cuda")
        ctx = ops.create_dec_context(n_tb, rows, acts)
        cfg = ops.create_dec_config(ctx, 4, cs, rs, thr)
        exp_rows, exp_acts, _ = P.expected_selection(x, thr, 4, dtype)
        delta = forward.dec_delta(P.to_np(x), exp_rows, cs.numpy(), P.to_np(rs), exp_acts)
        for _ in range(2):                               # the second call finds the workspace as the first left it
            y = y0.clone().cuda()
            ops.dec_sqllm(cfg, xd, y, qw, lut, bits)
            bound = HALF_ULP[dtype] * np.abs(ref + delta) + K * 2.0 ** -24 * (mags + np.abs(delta)) + 2.0 ** -24
            assert (np.abs(P.to_np(y).reshape(-1) - ref - delta) <= bound).all()
        ops.destroy_dec_config(cfg)
    bound = HALF_ULP[dtype] * np.abs(ref) + K * 2.0 ** -24 * mags + 2.0 ** -24
    assert (np.abs(P.to_np(outs[0]).reshape(-1) - ref) <= bound).all()


def _overlapped_producer(ops):
    """A GEMV that lets the next launch start before its own outputs are written: [28672] values of about 0.02."""
    N, K = 28672, 4096
    g = torch.Generator(device="cuda").manual_seed(2)
    qw = torch.randint(-2**31, 2**31 - 1, (K // 32, 3, N), dtype=torch.int32, device="cuda", generator=g)
    alpha = (torch.rand((K // 128, 3, N), device="cuda", generator=g) * 0.01).half()
    bias = torch.zeros((K // 128, N), device="cuda").half()
    x = (torch.randn((1, 1, K), device="cuda", generator=g) * 0.02).half()
    y = torch.zeros(1, 1, N, device="cuda").half()

    def produce():
        y.zero_()
        ops.lutgemm_gemv(x, y, qw, alpha, bias, 3, 128)
    return y.view(-1), produce


def test_ragged_scales_may_come_from_the_launch_before(ops):
    N, K, bits, group = 136, 544, 4, 32
    made, produce = _overlapped_producer(ops)
    alpha = made[: K // group * bits * N].view(K // group, bits, N)
    L = P.random_bcq_layer(N, K, bits, group, seed=21)
    x, qw, bias = P.make_activation(K, seed=22).cuda(), L["qweight"].cuda(), L["q_bias"].cuda()
    produce()
    w_hat = formats.bcq_dequant(L["qweight"].numpy(), P.to_np(alpha), P.to_np(L["q_bias"]), group)
    for _ in range(20):
        y = torch.zeros(1, 1, N, device="cuda").half()
        produce()
        ops.lutgemm_gemv(x, y, qw, alpha, bias, bits, group)
        _assert_sums(y, w_hat, x, "fp16")


def test_sqllm_tables_may_come_from_the_launch_before(ops):
    N, K, bits = 1792, 2336, 4
    made, produce = _overlapped_producer(ops)
    lut = made[: N * 2 ** bits].view(N, 2 ** bits)
    L = P.lut_layer(N, K, bits, seed=23, fmt="sqllm", real=False)
    x, qw = P.make_activation(K, seed=24).cuda(), L["qweight"].cuda()
    produce()
    w_hat = formats.lut_dequant(P.to_np(lut), L["codes"])
    for _ in range(20):
        y = torch.zeros(1, 1, N, device="cuda").half()
        produce()
        ops.sqllm_gemv(x, y, qw, lut, bits)
        _assert_sums(y, w_hat, x, "fp16")
