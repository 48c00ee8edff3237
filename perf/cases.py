"""The work that is timed when the library's speed is compared between two versions.

A case is one pass of what a model's code does with the library: the quantized linears of one decoded token (every
entry point ACCUMULATES, so the outputs are cleared first, as the model's modules do), or the dense operands of a prefill.
All calls go through the public functions of `decdec_ext` (and `decdec_b200.ops.lutgemm_dequant`, which has no name there).

Fields of a case
  op       "decode": batch-1 linears; "prefill": the dense weights of the linears, for the GEMM of the host framework
  fmt      "bcq" (binary-coded planes, `group` channels per scale), "anyprec" (bit planes + per-row LUT), "sqllm" (dense
           codes + per-column LUT)
  bits, group, dtype
  hidden, qkv, ffn, blocks   the four projections of a transformer block: qkv x hidden, hidden x hidden, 2 ffn x hidden,
           hidden x ffn (out x in features), `blocks` times, every block with weights of its own; or
  n, k     a single linear of n outputs and k inputs
  comp     True: fused with error compensation, `n_tb` thread blocks for it, and channels per 1024 `kc_qkv`, `kc_o`, `kc_up`,
           `kc_down` per projection (`kc` for a single linear); False: the base GEMV
  graph    True: the pass is one CUDA graph, as decoding loops capture it; False: eager calls
Data are synthetic: N(0,1) activations with a fixed 1 % of the channels scaled by 20, random codes, sorted LUTs of
N(0,0.02) centroids, packed 4-bit residuals in host memory.
"""
from __future__ import annotations

import math

import torch

import decdec_ext as ext
from decdec_b200 import ops

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
PROJECTIONS = ("qkv", "o", "up", "down")


def listed():
    llama8b = dict(hidden=4096, qkv=6144, ffn=14336)
    return [
        # one eager call on a rank of eight: the smallest call there is, latency and host work only
        dict(name="bcq3_shard_eager", op="decode", fmt="bcq", bits=3, group=128, dtype="fp16", n=768, k=4096, comp=False, graph=False),
        # a ragged layer, called eagerly with compensation (evaluation code does not capture): neither side is a tile multiple
        dict(name="bcq4_ragged_eager", op="decode", fmt="bcq", bits=4, group=32, dtype="bf16", n=2776, k=1184, comp=True, kc=16, n_tb=16,
             graph=False),
        # the base token of an 8B model, compensation off
        dict(name="bcq3_8b_off", op="decode", fmt="bcq", bits=3, group=128, dtype="fp16", blocks=4, comp=False, graph=True, **llama8b),
        # the default workload: 32 channels of each 1024 compensated in every projection
        dict(name="bcq3_8b_kc32", op="decode", fmt="bcq", bits=3, group=128, dtype="fp16", blocks=2, comp=True, kc_qkv=32, kc_o=32, kc_up=32,
             kc_down=32, n_tb=96, graph=True, **llama8b),
        # the tuner's operating point: only the wide projections are compensated, and a little
        dict(name="bcq3_8b_tuned", op="decode", fmt="bcq", bits=3, group=128, dtype="fp16", blocks=2, comp=True, kc_qkv=0, kc_o=0, kc_up=5,
             kc_down=3, n_tb=32, graph=True, **llama8b),
        # a 14B model whose feed-forward width is not a whole number of selection chunks
        dict(name="bcq3_phi3_kc16", op="decode", fmt="bcq", bits=3, group=128, dtype="fp16", hidden=5120, qkv=7680, ffn=17920, blocks=1,
             comp=True, kc_qkv=16, kc_o=16, kc_up=16, kc_down=16, n_tb=40, graph=True),
        # one block of a 70B model on one GPU: the largest pass
        dict(name="bcq3_70b_off", op="decode", fmt="bcq", bits=3, group=128, dtype="fp16", hidden=8192, qkv=10240, ffn=28672, blocks=1,
             comp=False, graph=True),
        # non-uniform 3-bit weights, compensation off
        dict(name="lut3_8b_off", op="decode", fmt="anyprec", bits=3, group=0, dtype="fp16", blocks=2, comp=False, graph=True, **llama8b),
        # non-uniform 4-bit weights in bf16 with a little compensation
        dict(name="lut4_8b_kc8", op="decode", fmt="anyprec", bits=4, group=0, dtype="bf16", blocks=2, comp=True, kc_qkv=8, kc_o=8, kc_up=8,
             kc_down=8, n_tb=48, graph=True, **llama8b),
        # dense 4-bit codes with per-column centroids
        dict(name="sqllm4_8b_off", op="decode", fmt="sqllm", bits=4, group=0, dtype="fp16", blocks=2, comp=False, graph=True, **llama8b),
        # prefill: the dense weights of one block, from each of the two formats that have a dequantizer
        dict(name="lut3_8b_prefill", op="prefill", fmt="anyprec", bits=3, group=0, dtype="fp16", blocks=1, **llama8b),
        dict(name="bcq3_8b_prefill", op="prefill", fmt="bcq", bits=3, group=128, dtype="fp16", blocks=1, **llama8b),
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], spread evenly over the logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step
    return max(lo, min(hi, v))


def draw(rng):
    """One more case; drawn again while it would move more bytes, or more of them over the host link, than any listed case."""
    most = max(work(c)["bytes"] for c in listed())
    most_host = max(_host_bytes(c) for c in listed())
    while True:
        c = _draw(rng)
        if work(c)["bytes"] <= most and _host_bytes(c) <= most_host:
            return c


def _draw(rng):
    fmt = rng.choice(("bcq", "bcq", "bcq", "anyprec", "anyprec", "sqllm"))
    c = dict(fmt=fmt, dtype=rng.choice(("fp16", "fp16", "bf16")))
    if fmt == "bcq":
        c.update(bits=rng.choice((2, 3, 3, 3, 4, 4)), group=rng.choice((32, 64, 128, 128, 128)))
    elif fmt == "anyprec":
        c.update(bits=rng.choice((3, 3, 3, 4, 4, 5, 6, 8)), group=0)
    else:
        c.update(bits=rng.choice((3, 4)), group=0)
    kind = rng.choice(("block", "block", "block", "linear", "linear", "prefill"))
    if kind == "prefill" and fmt == "sqllm":
        kind = "linear"
    c["op"] = "prefill" if kind == "prefill" else "decode"
    if kind == "linear":
        # a single layer, whole or a shard, sides of any size that the format takes: multiples of the scale group, of 32
        # channels, of 8 outputs; half of them multiples of 128 as most layers are
        step_n, step_k = rng.choice(((128, 512), (128, 512), (8, max(c["group"], 32)), (32, 256)))
        c.update(n=_log(rng, 512, 16384, step_n), k=_log(rng, 1024, 14336, step_k))
    else:
        hidden = _log(rng, 2048, 6144, rng.choice((512, 512, 128)))
        c.update(hidden=hidden, qkv=rng.choice((hidden * 3 // 2 // 64 * 64, hidden * 3, hidden * 5 // 4 // 64 * 64)),
                 ffn=max(1, round(hidden * rng.uniform(2.5, 3.6) / 256)) * 256, blocks=1)
    if c["op"] == "decode":
        c["graph"] = rng.random() < (0.8 if kind == "block" else 0.4)
        c["comp"] = rng.random() < 0.5
        if c["comp"]:
            c["n_tb"] = rng.choice((8, 16, 24, 32, 40, 64, 96))
            kc = _log(rng, 2, 64, 1)
            if kind == "linear":
                c["kc"] = kc
            else:
                attn = rng.choice((kc, kc, 0))
                c.update(kc_qkv=attn, kc_o=attn, kc_up=kc, kc_down=kc)
    return c


# ---- shapes and bytes ---------------------------------------------------------------------------------------------

def _linears(case):
    """[(name, n, k, channels compensated per 1024)] of one block, and how many blocks."""
    if "n" in case:
        return [("linear", case["n"], case["k"], case.get("kc", 0))], 1
    h, f = case["hidden"], case["ffn"]
    dims = {"qkv": (case["qkv"], h), "o": (h, h), "up": (2 * f, h), "down": (h, f)}
    return [(p, *dims[p], case.get("kc_" + p, 0)) for p in PROJECTIONS], case["blocks"]


def _weight_bytes(case, n, k):
    b = case["bits"] * n * k / 8
    return b + (n * k / case["group"] * (case["bits"] + 1) * 2 if case["fmt"] == "bcq" else n * 2 ** case["bits"] * 2)


def _host_bytes(case):
    linears, blocks = _linears(case)
    return blocks * sum(kc * k // 1024 * n / 2 for _, n, k, kc in linears)


def work(case):
    linears, blocks = _linears(case)
    nbytes = flops = 0.0
    for _, n, k, kc in linears:
        nbytes += _weight_bytes(case, n, k)
        if case["op"] == "prefill":
            nbytes += 2 * n * k
            flops += 2 * n * k
            continue
        rows = kc * k // 1024
        nbytes += 2 * k + 2 * n                                   # activations in, outputs out
        nbytes += rows * (n / 2 + 6) + (2 * n if rows else 0)     # residual rows over the host link, selection, scales
        flops += 2 * n * (k + rows)
    return {"bytes": nbytes * blocks, "flops": flops * blocks}


def tolerance(case):
    """Measured against the dense weights in 64 bits over thirty shapes: 2.1e-4 (fp16) and 1.7e-3 (bf16) in the 2-norm, which is the
    one rounding of the output, and 4.5e-4 for 3-bit LUT weights in fp16, whose products may be summed in fp16 over four
    weights; the largest single difference was 2.3e-3 and 3.9e-3.  About four times that is allowed.  The dense weights of a
    prefill are looked up, or rounded twice in a fixed order: exact."""
    if case["op"] == "prefill":
        return "exact"
    return {"rel": 1.5e-3, "max": 0.01} if case["dtype"] == "fp16" else {"rel": 7e-3, "max": 0.03}


# ---- data ----------------------------------------------------------------------------------------------------------

class _State:
    """What a decoding program keeps: packed weights, outputs, compensation handles, and the captured graph."""

    def __init__(self, case):
        self.case, self.layers, self.configs, self.graph = case, [], [], None

    def __del__(self):
        self.graph = None
        if self.configs:
            torch.cuda.synchronize()
            for cfg in self.configs:
                ext.destroy_dec_config(cfg)


def _activation(k, dt, gen):
    x = torch.randn(k, device="cuda", generator=gen)
    outliers = torch.randperm(k, generator=torch.Generator().manual_seed(1234 + k))[: max(1, k // 100)]
    x[outliers.cuda()] *= 20.0
    return x.to(dt).reshape(1, 1, k)


def _thresholds(k, dt, gen):
    """Mean of the sorted |activation| of eight calibration samples."""
    samples = torch.stack([_activation(k, dt, gen).float().abs().reshape(-1) for _ in range(8)])
    return samples.sort(dim=1, descending=True).values.mean(dim=0).to(dt).cpu()


def _words(shape, gen):
    return torch.randint(-2**31, 2**31 - 1, shape, dtype=torch.int32, device="cuda", generator=gen)


def _weights(case, n, k, dt, gen):
    bits, fmt = case["bits"], case["fmt"]
    if fmt == "bcq":
        groups = k // case["group"]
        alpha = (torch.rand((groups, bits, n), device="cuda", generator=gen) * 0.01 + 1e-4).to(dt)
        bias = ((torch.rand((groups, n), device="cuda", generator=gen) - 0.5) * 0.01).to(dt)
        return _words((k // 32, bits, n), gen), alpha, bias
    lut = (torch.randn((n, 2 ** bits), device="cuda", generator=gen) * 0.02).sort(dim=1).values.to(dt)
    return _words((bits, n, k // 32) if fmt == "anyprec" else (k * bits // 32, n), gen), lut


def _inputs(case, seed):
    """(n, k, channels compensated per 1024), activations, (residual, scales, thresholds) or None, weights: of every linear of a pass."""
    dt = DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    linears, blocks = _linears(case)
    xs = {k: _activation(k, dt, gen) for k in sorted({k for _, _, k, _ in linears})} if case["op"] == "decode" else {}
    for _ in range(blocks):
        for _, n, k, kc in linears:
            compensation = None
            if case["op"] == "decode" and case["comp"]:
                residual = _words((k, n // 8), gen).cpu()
                scales = (torch.rand(n, device="cuda", generator=gen) * 1e-3 + 2e-4).to(dt).cpu()
                compensation = residual, scales, _thresholds(k, dt, gen)
            yield (n, k, kc), xs.get(k), compensation, _weights(case, n, k, dt, gen)


def prepare(case, seed):
    dt = DTYPES[case["dtype"]]
    s = _State(case)
    linears, blocks = _linears(case)
    if case["op"] == "prefill":
        s.layers = [weights for _, _, _, weights in _inputs(case, seed)]
        return s
    comp = case["comp"]
    if comp:
        s.rows = torch.zeros(32 * 1024, dtype=torch.int32, device="cuda")
        s.acts = torch.zeros(32 * 1024, dtype=dt, device="cuda")
        ctx = ext.create_dec_context(case["n_tb"], s.rows, s.acts)
        s.selected = linears[-1][3] * linears[-1][2] // 1024     # the last call's selection is in the buffers after a pass
    # one buffer for all outputs, so that one memset clears them; offsets keep each output 256-byte aligned
    pad = [(n + 127) // 128 * 128 for _, n, _, _ in linears]
    s.y = torch.zeros(blocks * sum(pad), dtype=dt, device="cuda")
    at = 0
    for (n, k, kc), x, compensation, weights in _inputs(case, seed):
        cfg = None
        if comp:
            cfg = ext.create_dec_config(ctx, kc, *compensation)
            s.configs.append(cfg)
        s.layers.append((cfg, x, s.y[at:at + n].view(1, 1, n), weights))
        at += (n + 127) // 128 * 128
    if case["graph"]:
        stream = torch.cuda.Stream() if prepare.stream is None else prepare.stream
        prepare.stream = stream
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            _decode(s)                                           # the first call of a stream makes its workspace
            stream.synchronize()
            s.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s.graph, stream=stream):
                _decode(s)
        torch.cuda.current_stream().wait_stream(stream)
    return s


prepare.stream = None      # graphs are captured on one stream, as a program with one decoding loop does


def _decode(s):
    fmt, bits, group, comp = s.case["fmt"], s.case["bits"], s.case["group"], s.case["comp"]
    s.y.zero_()
    for cfg, x, y, w in s.layers:
        if fmt == "bcq":
            if comp:
                ext.dec_lutgemm(cfg, x, y, *w, bits, group)
            else:
                ext.lutgemm_gemv(x, y, *w, bits, group)
        elif fmt == "anyprec":
            if comp:
                ext.dec_anyprec(cfg, x, y, *w, bits)
            else:
                ext.anyprec_gemv(x, y, *w, bits)
        elif comp:
            ext.dec_sqllm(cfg, x, y, *w, bits)
        else:
            ext.sqllm_gemv(x, y, *w, bits)


def run(s):
    if s.case["op"] == "prefill":
        if s.case["fmt"] == "bcq":
            return [ops.lutgemm_dequant(*w, s.case["bits"], s.case["group"]) for w in s.layers]
        return [ext.anyprec_dequant(*w, s.case["bits"]) for w in s.layers]
    if s.graph is not None:
        s.graph.replay()
    else:
        _decode(s)
    out = [layer[2] for layer in s.layers]
    if s.case["comp"] and s.selected:
        out += [s.rows[: s.selected], s.acts[: s.selected]]
    return out


# ---- the same results in 64 bits, without the library ----------------------------------------------------------------

def _dense(case, n, k, w):
    """[n, k] weights in 64 bits, from the packed tensors as their formats are documented."""
    bits, dev = case["bits"], "cuda"
    if case["fmt"] == "bcq":                       # words [k / 32, bits, n], bit i = channel i of the word: sum of +-alpha, plus the bias
        words, alpha, bias = w
        shifts = torch.arange(32, device=dev).view(1, 32, 1)
        dense = bias.double().repeat_interleave(case["group"], 0)
        for p in range(bits):
            signs = (((words[:, p].unsqueeze(1) >> shifts) & 1) * 2 - 1).view(k, n)
            dense += signs * alpha[:, p].double().repeat_interleave(case["group"], 0)
        return dense.t()
    words, lut = w
    if case["fmt"] == "anyprec":                   # planes [bits, n, k / 32], most significant first, channels interleaved within 1024
        channel = torch.empty(k, dtype=torch.long)
        for at in range(0, k, 1024):
            e = min(1024, k - at) // 32
            t, j, r = torch.meshgrid(torch.arange(e), torch.arange(4), torch.arange(8), indexing="ij")
            channel[at:at + 32 * e] = (at + 8 * e * j + 8 * t + r).reshape(-1)
        shifts = torch.arange(31, -1, -1, device=dev)
        codes = torch.zeros((n, k), dtype=torch.long, device=dev)
        for p in range(bits):
            codes = codes * 2 + ((words[p].unsqueeze(-1) >> shifts) & 1).view(n, k)
        dense = torch.empty((n, k), dtype=torch.float64, device=dev)
        dense[:, channel.to(dev)] = lut.double().gather(1, codes)
        return dense
    # 32 channels are one little-endian string of codes in `bits` words of a column
    string = ((words.view(k // 32, bits, 1, n) >> torch.arange(32, device=dev).view(1, 1, 32, 1)) & 1).view(k, bits, n)
    codes = (string.long() << torch.arange(bits, device=dev).view(1, bits, 1)).sum(1)
    return lut.double().gather(1, codes.t())


def _selection(x, thresholds, kc):
    """Channels that are compensated: per 1024 the kc of the highest buckets, the lowest indices of the last bucket."""
    k, dt = x.numel(), x.dtype
    a, b = thresholds[0], thresholds[max(0, kc * k // 1024 - 1)]
    level = torch.arange(32)
    upper = a + ((b - a).float() * level / 15).to(dt)
    lower = (b.float() * (31 - level) / 16).to(dt)
    floors = torch.where(level < 16, upper, lower).float()
    rows = []
    for at in range(0, k, 1024):
        mag = x[at:at + 1024].float().abs().cpu()
        over = mag.unsqueeze(1) >= floors
        bucket = torch.where(over.any(1), over.int().argmax(1), 32)
        rows.append(at + bucket.sort(stable=True).indices[: kc * mag.numel() // 1024])
    return torch.cat(rows).cuda()


def exact(case, seed):
    """The outputs of `run`; nothing for the selection that is returned beside them (whole numbers and copies), nor for the
    dense weights of a prefill, which are compared bit by bit."""
    if case["op"] == "prefill":
        return None
    out = []
    for (n, k, kc), x, comp, w in _inputs(case, seed):
        xd = x.reshape(-1).double()
        step = max(8, (1 << 27) // k // 8 * 8)
        parts = []
        for n0 in range(0, n, step):
            n1 = min(n, n0 + step)
            if case["fmt"] == "bcq":
                piece = (w[0][:, :, n0:n1], w[1][:, :, n0:n1], w[2][:, n0:n1])
            else:
                piece = (w[0][:, n0:n1], w[1][n0:n1])
            parts.append(_dense(case, n1 - n0, k, piece) @ xd)
        y = torch.cat(parts)
        if comp is not None and kc * k // 1024:
            residual, scales, thresholds = comp
            rows = _selection(x.reshape(-1), thresholds, kc)
            nibbles = (residual.cuda()[rows].unsqueeze(-1) >> (4 * torch.arange(8, device="cuda"))) & 15
            by_output = scales.cuda().double().view(8, n // 8).t().reshape(-1)      # stored [output % 8][output / 8]
            y += (xd[rows] @ (nibbles.double() - 8).view(-1, n)) * by_output
        out.append(y.view(1, 1, n))
    if case["comp"] and _linears(case)[0][-1][3] * _linears(case)[0][-1][2] // 1024:
        out += [None, None]
    return out
