"""The pipelined binary-coded GEMV with tiles of more stages than its shared memory has slots, from two slots (4 bits with a
scale every 32 channels, the widest fp32 formats) to eight, alone, fused with compensation and through the entry point
without allocation.

Oracle: the packed tensors in float64 on a seeded subset of the outputs, twelve of every 128; all outputs are compared with
the register-staged kernel.  Bounds as in test_gpu_lut_paths.py: fp32 sums, one rounding of the output.
"""
import numpy as np
import pytest
import torch

from oracle import formats
from oracle import forward as ofw
from tests import problems as P

pytestmark = pytest.mark.gpu

HALF_ULP = {"fp16": 2.0 ** -11, "bf16": 2.0 ** -8, "fp32": 2.0 ** -24}


@pytest.fixture(scope="module")
def ops():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from decdec_b200 import ops as _ops
    return _ops


def _layer(N, K, bits, group, dtype):
    g = torch.Generator(device="cuda").manual_seed(N + K + bits)
    dt = P.TORCH_DT[dtype]
    qw = torch.randint(-2**31, 2**31 - 1, (K // 32, bits, N), dtype=torch.int32, device="cuda", generator=g)
    alpha = (torch.rand((K // group, bits, N), device="cuda", generator=g) * 0.01).to(dt)
    bias = ((torch.rand((K // group, N), device="cuda", generator=g) - 0.5) * 0.01).to(dt)
    return qw, alpha, bias


def _subset(N):
    rng = np.random.default_rng(N)
    return np.unique(np.concatenate([np.minimum(at + rng.choice(128, 12, replace=False), N - 1) for at in range(0, N, 128)]))


def _oracle(layer, group, x, idx):
    qw, alpha, bias = (t[..., torch.from_numpy(idx).cuda()].cpu() for t in layer)
    w = formats.bcq_dequant(qw.numpy(), P.to_np(alpha), P.to_np(bias), group)
    xd = P.to_np(x).reshape(-1)
    return w @ xd, np.abs(w) @ np.abs(xd)


def _bound(ref, mags, K, dtype):
    # the packed accumulator words round every partial sum to 2^-20; two of them per 512 channels, and the compensation's
    return HALF_ULP[dtype] * np.abs(ref) + K * 2.0 ** -24 * mags + (2 * (K // 512 + 1) + 64) * 2.0 ** -20


SHAPES = [
    # two slots
    (28672, 4096, 4, 32, "fp16"), (28672, 4096, 4, 32, "bf16"),
    (8192, 4128, 4, 32, "fp16"), (8192, 4128, 4, 32, "bf16"),          # a K slice of 32 channels
    (4096, 11008, 4, 32, "fp16"), (4096, 11008, 4, 32, "bf16"),        # six stages, half a K slice left over
    (4096, 11008, 3, 32, "fp32"), (4096, 11008, 4, 64, "fp32"),
    # three, four and eight slots, which do not always belong to one consumer group
    (4096, 11008, 4, 64, "fp16"), (4096, 11008, 3, 64, "fp16"), (28672, 4096, 3, 64, "bf16"), (28672, 4096, 2, 128, "fp16"),
]


@pytest.mark.parametrize("N,K,bits,group,dtype", SHAPES)
def test_tiles_of_more_stages_than_slots(ops, monkeypatch, N, K, bits, group, dtype):
    layer = _layer(N, K, bits, group, dtype)
    x = P.make_activation(K, seed=3, dtype=dtype)
    idx = _subset(N)
    ref, mags = _oracle(layer, group, x, idx)
    bound = _bound(ref, mags, K, dtype)
    xd = x.cuda()

    def run():
        y = torch.zeros(1, 1, N, dtype=P.TORCH_DT[dtype], device="cuda")
        ops.lutgemm_gemv(xd, y, *layer, bits, group)
        return y

    outs = [run() for _ in range(6)]                       # launches that follow each other: copies land at other times
    monkeypatch.setenv("DECDEC_BCQ_PIPE", "0")
    staged = P.to_np(run()).reshape(-1)
    worst = np.interp(np.arange(N), idx, bound)            # a bound for every output: the subset's, spread over its neighbours
    for y in outs:
        got = P.to_np(y).reshape(-1)
        assert (np.abs(got[idx] - ref) <= bound).all()
        # each side is within its bound of the exact sum; magnitudes differ little between neighbours: four of them
        assert (np.abs(got - staged) <= 4 * worst + 2 * HALF_ULP[dtype] * np.abs(staged)).all()
    assert ops.stream_status() == 0


@pytest.mark.parametrize("N,K,bits,group,dtype,k_chunk,n_tb", [
    (4104, 11008, 4, 32, "fp16", 4, 16),        # ragged outputs and channels, tickets
    (8192, 4128, 4, 32, "bf16", 8, 64),
    (4096, 11264, 4, 32, "fp16", 8, 96),        # whole slices: packed words
    (4096, 11008, 3, 64, "fp16", 4, 24),
])
def test_fused_tiles_of_more_stages_than_slots(ops, N, K, bits, group, dtype, k_chunk, n_tb):
    layer = _layer(N, K, bits, group, dtype)
    x = P.make_activation(K, seed=4, dtype=dtype)
    cs, rs = P.random_residual(N, K, seed=5, dtype=dtype)
    thr = P.make_thresholds(K, dtype, n_calib=32)
    k = k_chunk * K // 1024
    rows = torch.full((k,), -1, dtype=torch.int32, device="cuda")
    acts = torch.zeros(k, dtype=P.TORCH_DT[dtype], device="cuda")
    ctx = ops.create_dec_context(n_tb, rows, acts)
    cfg = ops.create_dec_config(ctx, k_chunk, cs, rs, thr)
    exp_rows, exp_acts, _ = P.expected_selection(x, thr, k_chunk, dtype)
    delta = ofw.dec_delta(P.to_np(x), exp_rows, cs.numpy(), P.to_np(rs), exp_acts)
    idx = _subset(N)
    ref, mags = _oracle(layer, group, x, idx)
    ref = ref + delta[idx]
    bound = _bound(ref, mags + np.abs(delta[idx]), K, dtype)
    xd = x.cuda()
    for _ in range(4):
        y = torch.zeros(1, 1, N, dtype=P.TORCH_DT[dtype], device="cuda")
        ops.dec_lutgemm(cfg, xd, y, *layer, bits, group)
        assert np.array_equal(rows.cpu().numpy(), exp_rows)
        assert (np.abs(P.to_np(y).reshape(-1)[idx] - ref) <= bound).all()
    assert ops.stream_status() == 0
    ops.destroy_dec_config(cfg)


def test_noalloc_tiles_of_more_stages_than_slots(ops):
    from decdec_b200 import capi
    N, K, bits, group, dtype = 4096, 11008, 4, 32, "fp16"
    layer = _layer(N, K, bits, group, dtype)
    x = P.make_activation(K, seed=6, dtype=dtype)
    idx = _subset(N)
    ref, mags = _oracle(layer, group, x, idx)
    xd = x.cuda()
    for _ in range(3):
        y = torch.zeros(1, 1, N, dtype=torch.float16, device="cuda")
        capi.call("decdec_lutgemm_gemv_noalloc", xd.data_ptr(), y.data_ptr(), *(t.data_ptr() for t in layer), N, K, bits, group,
                  capi.FP16, torch.cuda.current_stream().cuda_stream)
        assert (np.abs(P.to_np(y).reshape(-1)[idx] - ref) <= _bound(ref, mags, K, dtype)).all()
