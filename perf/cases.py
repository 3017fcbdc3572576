"""The work a user of this framework has it do, as measurable cases.

A case is a dict of plain values; its ``kind`` says which public entry point it goes through:

  gemv, gemv_f32          one eager call of ``ops.gemv_f16`` / ``ops.gemv_f32``: the smallest calls, where launch
                          latency counts as much as the weights' trip through HBM
  decode                  the linear layers of decoder blocks for a handful of tokens (fused QKV, output projection,
                          FFN up, FFN down): prepared launches queued in order with ``ops.run``, as a token loop does
  prefill                 the same four layers for a long prompt: one eager ``ops.gemm_f16`` each
  gemm                    one eager ``ops.gemm_f16``
  bert, resnet            the model-level sweep of the benchmark (``sweep.Sweep`` on four lanes), captured once in a
                          CUDA graph and replayed, which is how the benchmark and a sweep driver run it
  conv_stage              a stage of bottleneck blocks (1x1, 3x3, 1x1), every layer reading the one before it
  conv, conv_f32          one eager NHWC convolution, fp16 or true fp32
  gemm_f32                one eager true-fp32 GEMM

Sizes are those of the benchmark configurations and of the op-level shape suites (scripts/utils), and draws spread over
the ranges these suites span.
"""
import math

import torch

from helix_b200 import ops, sweep, workloads
from helix_b200._lib import LAUNCH_STATIC_A


def listed():
    return [
        # one token against one square projection: the smallest call there is
        {"name": "gemv_4096", "kind": "gemv", "rows": 4096, "k": 4096, "m": 1},
        # true-fp32 product of one vector with a square matrix (268 MB of weights)
        {"name": "gemv_f32_8192", "kind": "gemv_f32", "rows": 8192, "k": 8192, "m": 1},
        # one-token decode step through four decoder blocks; weights are static while the loop runs
        {"name": "decode_1", "kind": "decode", "hidden": 4096, "ffn": 11008, "tokens": 1, "layers": 4},
        # the same step for a batch of 16 requests: skinny tensor-core GEMMs
        {"name": "decode_16", "kind": "decode", "hidden": 4096, "ffn": 11008, "tokens": 16, "layers": 4},
        # prompt of an odd length (the longest of the sequence-length sweep) through one decoder block
        {"name": "prefill_1949", "kind": "prefill", "hidden": 4096, "ffn": 11008, "tokens": 1949},
        # the largest dense GEMM of the benchmark
        {"name": "gemm_8192", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192},
        # encoder half of the model-level sweep: six layers at batch 16, sequence 512, attention GEMMs batched
        {"name": "bert_b16_s512", "kind": "bert", "batch": 16, "seq": 512, "hidden": 768, "heads": 12, "layers": 6},
        # convolution half of the model-level sweep: all 53 layers at batch 32
        {"name": "resnet_b32", "kind": "resnet", "batch": 32, "image": 224},
        # a CNN's second stage run layer after layer: what inference does, one layer waiting for the previous one
        {"name": "conv_stage_28", "kind": "conv_stage", "batch": 32, "size": 28, "width": 128, "blocks": 4},
        # a 5 x 5 layer whose channel count is not a multiple of 64, on an image of 26 x 26
        {"name": "conv_5x5_c96", "kind": "conv", "batch": 20, "c": 96, "h": 26, "w": 26, "ko": 256, "r": 5, "stride": 1,
         "pad": 2},
        # the fp32 GEMM the reference's CPU template is quoted on
        {"name": "gemm_f32_1024", "kind": "gemm_f32", "m": 1024, "n": 1024, "k": 1024},
        # the same 3 x 3 layer as in the stage above, in true fp32
        {"name": "conv_f32_28", "kind": "conv_f32", "batch": 32, "c": 128, "h": 28, "w": 28, "ko": 128, "r": 3,
         "stride": 1, "pad": 1},
    ]


def _spread(rng, lo, hi, step=1):
    """A size of [lo, hi], spread over its logarithm, a multiple of `step`."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["gemv", "gemv_f32", "decode", "decode", "prefill", "gemm", "bert", "resnet", "conv_stage", "conv",
                       "conv", "gemm_f32", "conv_f32"])
    if kind == "gemv":
        return {"kind": kind, "rows": _spread(rng, 256, 16384), "k": _spread(rng, 256, 16384, 8), "m": rng.randint(1, 8)}
    if kind == "gemv_f32":
        return {"kind": kind, "rows": _spread(rng, 256, 12000), "k": _spread(rng, 256, 12000, 4), "m": rng.randint(1, 8)}
    if kind == "decode":
        hidden = 128 * rng.randint(8, 40)
        return {"kind": kind, "hidden": hidden, "ffn": 8 * int(hidden * rng.uniform(2.6, 4.0) / 8),
                "tokens": _spread(rng, 1, 128), "layers": rng.randint(1, 4)}
    if kind == "prefill":
        hidden = 128 * rng.randint(6, 32)
        return {"kind": kind, "hidden": hidden, "ffn": 8 * int(hidden * rng.uniform(2.6, 4.0) / 8),
                "tokens": _spread(rng, 129, 2048)}
    if kind == "gemm":
        return {"kind": kind, "m": _spread(rng, 128, 8192), "n": _spread(rng, 128, 8192, rng.choice([1, 8, 64])),
                "k": _spread(rng, 128, 8192, 8)}
    if kind == "bert":
        heads = rng.choice([12, 16])
        return {"kind": kind, "batch": rng.randint(1, 12), "seq": 8 * rng.randint(8, 64), "hidden": 64 * heads,
                "heads": heads, "layers": rng.randint(1, 4)}
    if kind == "resnet":
        return {"kind": kind, "batch": rng.randint(1, 28), "image": rng.choice([160, 192, 224])}
    if kind == "conv_stage":
        size, width = rng.choice([(56, 64), (28, 128), (14, 256), (7, 512)])
        return {"kind": kind, "batch": rng.randint(1, 64), "size": size, "width": width, "blocks": rng.randint(2, 6)}
    if kind == "conv":
        r = rng.choice([1, 3, 3, 5])
        h = rng.randint(7, 57)
        return {"kind": kind, "batch": _spread(rng, 1, 64), "c": _spread(rng, 16, 512, 8), "h": h,
                "w": max(7, h + rng.randint(-3, 3)), "ko": _spread(rng, 16, 512, 8), "r": r,
                "stride": rng.choice([1, 1, 2]), "pad": r // 2}
    if kind == "gemm_f32":
        return {"kind": kind, "m": _spread(rng, 96, 2048), "n": _spread(rng, 96, 2048, rng.choice([1, 4, 32])),
                "k": _spread(rng, 96, 2048, rng.choice([1, 4, 32]))}
    r = rng.choice([1, 3, 3, 5])
    h = rng.randint(7, 29)
    return {"kind": kind, "batch": rng.randint(1, 32), "c": _spread(rng, 16, 160, rng.choice([1, 4])), "h": h, "w": h,
            "ko": _spread(rng, 16, 160, rng.choice([1, 4])), "r": r, "stride": rng.choice([1, 1, 2]), "pad": r // 2}


def _decode_layers(case):
    """(out features, in features) of one decoder block: fused QKV, output projection, FFN up, FFN down."""
    h, f = case["hidden"], case["ffn"]
    return [(3 * h, h), (h, h), (f, h), (h, f)]


def _stage_layers(case):
    """(C, KO, filter, pad) of the stage's convolutions in order: blocks of 1x1 down, 3x3, 1x1 up."""
    w = case["width"]
    return [(4 * w, w, 1, 0), (w, w, 3, 1), (w, 4 * w, 1, 0)] * case["blocks"]


def _units(case):
    if case["kind"] == "bert":
        return workloads.bert_base_gemms(case["batch"], case["seq"], case["hidden"], case["heads"], 4 * case["hidden"],
                                         case["layers"])
    return workloads.resnet50_convs(case["batch"], case["image"])


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    kind = case["kind"]

    def normal(shape, scale, dtype=torch.float16):
        return torch.empty(shape, dtype=dtype, device=dev).normal_(0.0, scale, generator=gen)

    def uniform(shape, dtype=torch.float16):
        return torch.empty(shape, dtype=dtype, device=dev).uniform_(-1.0, 1.0, generator=gen)

    if kind == "gemv":
        return {"kind": kind, "w": normal((case["rows"], case["k"]), 0.02), "x": normal((case["m"], case["k"]), 1.0)}
    if kind == "gemv_f32":
        return {"kind": kind, "w": uniform((case["rows"], case["k"]), torch.float32),
                "x": uniform((case["m"], case["k"]), torch.float32)}
    if kind == "decode":
        t, launches, outs = case["tokens"], [], []
        for _ in range(case["layers"]):
            for n, k in _decode_layers(case):
                w, x = normal((n, k), 0.02), normal((t, k), 1.0)
                out = torch.empty((t, n), dtype=torch.float16, device=dev)
                if t <= 8:
                    l = ops.launch_gemv_f16(w, x, out)
                    l.flags = LAUNCH_STATIC_A
                else:
                    l = ops.launch_gemm_f16(x, w, out)
                launches.append(l)
                outs.append(out)
        return {"kind": kind, "launches": launches, "outs": outs}
    if kind == "prefill":
        return {"kind": kind, "pairs": [(normal((case["tokens"], k), 1.0), normal((n, k), 0.02))
                                        for n, k in _decode_layers(case)]}
    if kind == "gemm":
        s = 1.0 / math.sqrt(case["k"])
        return {"kind": kind, "a": normal((case["m"], case["k"]), s), "b": normal((case["n"], case["k"]), s)}
    if kind in ("bert", "resnet"):
        sw = sweep.Sweep(_units(case), seed=int(seed), lanes=4)
        sw.step()                       # outside the capture, as the benchmark does
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            sw.step()
        return {"kind": kind, "sweep": sw, "graph": graph, "outs": [t[2] for t in sw.tensors]}
    if kind == "conv_stage":
        b, s = case["batch"], case["size"]
        x = normal((b, s, s, 4 * case["width"]), 1.0)
        state = {"kind": kind, "x": x, "launches": [], "outs": []}
        for c, ko, r, pad in _stage_layers(case):
            w = normal((ko, r, r, c), 1.0 / math.sqrt(c * r * r))
            out = torch.empty((b, s, s, ko), dtype=torch.float16, device=dev)
            state["launches"].append(ops.launch_conv2d_f16(x, w, out, 1, pad))
            state["outs"].append(out)
            x = out
        return state
    if kind in ("conv", "conv_f32"):
        dtype = torch.float16 if kind == "conv" else torch.float32
        fan = case["c"] * case["r"] * case["r"]
        return {"kind": kind, "x": uniform((case["batch"], case["h"], case["w"], case["c"]), dtype),
                "w": normal((case["ko"], case["r"], case["r"], case["c"]), math.sqrt(2.0 / fan), dtype),
                "stride": case["stride"], "pad": case["pad"]}
    return {"kind": kind, "a": uniform((case["m"], case["k"]), torch.float32),
            "b": uniform((case["k"], case["n"]), torch.float32)}


def run(state):
    kind = state["kind"]
    if kind == "gemv":
        return ops.gemv_f16(state["w"], state["x"])
    if kind == "gemv_f32":
        return ops.gemv_f32(state["w"], state["x"])
    if kind in ("decode", "conv_stage"):
        for l in state["launches"]:
            ops.run(l)
        return state["outs"]
    if kind == "prefill":
        return [ops.gemm_f16(x, w) for x, w in state["pairs"]]
    if kind == "gemm":
        return ops.gemm_f16(state["a"], state["b"])
    if kind in ("bert", "resnet"):
        state["graph"].replay()
        return state["outs"]
    if kind == "conv":
        return ops.conv2d_f16_nhwc(state["x"], state["w"], state["stride"], state["pad"])
    if kind == "conv_f32":
        return ops.conv2d_f32_nhwc(state["x"], state["w"], state["stride"], state["pad"])
    return ops.gemm_f32(state["a"], state["b"])


def work(case):
    """Every input read once, every output written once; two operations per multiply-add."""
    kind = case["kind"]

    def gemm(m, n, k, size):
        return size * (m * k + n * k + m * n), 2 * m * n * k

    def conv(b, h, w, c, ko, r, stride, pad, size):
        ho, wo = ops.conv_out_hw(h, w, r, r, stride, pad)
        return size * (b * h * w * c + ko * r * r * c + b * ho * wo * ko), 2 * b * ho * wo * ko * c * r * r

    if kind == "gemv":
        parts = [gemm(case["m"], case["rows"], case["k"], 2)]
    elif kind == "gemv_f32":
        parts = [gemm(case["m"], case["rows"], case["k"], 4)]
    elif kind == "decode":
        parts = [gemm(case["tokens"], n, k, 2) for n, k in _decode_layers(case)] * case["layers"]
    elif kind == "prefill":
        parts = [gemm(case["tokens"], n, k, 2) for n, k in _decode_layers(case)]
    elif kind == "gemm":
        parts = [gemm(case["m"], case["n"], case["k"], 2)]
    elif kind == "gemm_f32":
        parts = [gemm(case["m"], case["n"], case["k"], 4)]
    elif kind in ("bert", "resnet"):
        parts = [(workloads.unit_bytes(u), workloads.unit_flops(u)) for u in _units(case)]
    elif kind == "conv_stage":
        parts = [conv(case["batch"], case["size"], case["size"], c, ko, r, 1, pad, 2)
                 for c, ko, r, pad in _stage_layers(case)]
    else:
        parts = [conv(case["batch"], case["h"], case["w"], case["c"], case["ko"], case["r"], case["stride"], case["pad"],
                      2 if kind == "conv" else 4)]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    # Measured against the same path in 64 bits, four times what was seen: one rounding to fp16 on top of fp32 sums is
    # 2.1e-4; a stage rounds once per layer and the errors of twelve to eighteen layers add up to 9e-4; true-fp32 sums
    # over 1024 to 8192 products are off by up to 6e-7.
    if case["kind"] in ("gemv_f32", "gemm_f32", "conv_f32"):
        return {"rel": 2.5e-6}
    return {"rel": 3.6e-3} if case["kind"] == "conv_stage" else {"rel": 8e-4}


def _matmul64(a, b_nk):
    return torch.matmul(a.double(), b_nk.double().transpose(-1, -2))


def _conv64(x, w, stride, pad):
    """NHWC convolution in 64 bits, one matrix product per filter tap."""
    x, w = x.double(), w.double()
    n, h, wd, c = x.shape
    ko, r, s, _ = w.shape
    ho, wo = (h + 2 * pad - r) // stride + 1, (wd + 2 * pad - s) // stride + 1
    xp = torch.zeros((n, h + 2 * pad, wd + 2 * pad, c), dtype=torch.float64, device=x.device)
    xp[:, pad:pad + h, pad:pad + wd] = x
    out = torch.zeros((n * ho * wo, ko), dtype=torch.float64, device=x.device)
    for i in range(r):
        for j in range(s):
            tap = xp[:, i:i + (ho - 1) * stride + 1:stride, j:j + (wo - 1) * stride + 1:stride]
            out.addmm_(tap.reshape(-1, c), w[:, i, j].t())
    return out.view(n, ho, wo, ko)


def exact(case, seed):
    """What `run` returns on the inputs of (case, seed), in 64 bits.  A stage's layers read each other unrounded."""
    state = prepare(case, seed)
    kind = state["kind"]
    if kind in ("gemv", "gemv_f32"):
        return _matmul64(state["x"], state["w"])
    if kind == "decode":
        out = []
        for l in state["launches"]:
            a, b, _ = l._refs
            out.append(_matmul64(b, a) if case["tokens"] <= 8 else _matmul64(a, b))
        return out
    if kind == "prefill":
        return [_matmul64(x, w) for x, w in state["pairs"]]
    if kind == "gemm":
        return _matmul64(state["a"], state["b"])
    if kind in ("bert", "resnet"):
        return [_matmul64(a, b) if u["kind"] == "gemm" else _conv64(a, b, u["shape"][7], u["shape"][8])
                for u, (a, b, _) in zip(state["sweep"].units, state["sweep"].tensors)]
    if kind == "conv_stage":
        x, out = state["x"], []
        for l, (_, _, _, pad) in zip(state["launches"], _stage_layers(case)):
            x = _conv64(x, l._refs[1], 1, pad)
            out.append(x)
        return out
    if kind in ("conv", "conv_f32"):
        return _conv64(state["x"], state["w"], state["stride"], state["pad"])
    return torch.matmul(state["a"].double(), state["b"].double())
