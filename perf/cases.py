"""Performance cases of the INT8 attention forward path: what programs built on this package ask of it.

A program that serves an INT8-quantised transformer calls, through the package's public functions,
  self      FMHAInferI8          encoder layers and prefill, q/k/v/o int8 [B,H,S,D] with a padding mask [B,S]
  cross     FMHAInferI8Cross     decoding against a cache (one query row), chunked prefill, encoder-decoder attention
  policy    FMHAInferI8Policy    the whole-row scales for the 8-bit probabilities (per-row or one static scale)
  quantize  quantize_f32         per-tensor symmetric quantisation of an fp32 activation, in front of the attention
  host      FMHAInferI8Host      buffers in (pinned) host memory in, host memory out

Sizes are those of `workloads.py` (C1..C5), of the test suite, or generic ones between them.  Activations are drawn
from a normal distribution and quantised symmetrically per tensor, as in `workloads.py`; where a batch is padded,
every sequence has its own length.  Inputs, output buffers, scratch and the descriptors live across calls.
"""
import importlib
import math

import torch

fmha = importlib.import_module("int8-flash-attention-fmha-quantization_b200")

# Lengths of a padded batch: uniform in [valid_min, S], rounded up to a multiple of `valid_step`.  valid_min == S: no padding.


def listed():
    return [
        # the smallest call: one short request, two heads (workload C1): latency of a call
        dict(name="self_smallest", kind="self", B=1, H=2, S=64, D=64, valid_min=64, valid_step=1),
        # one request through an encoder layer of 12 heads; ragged: 320 is no multiple of the 128-key tile, the text is shorter still
        dict(name="self_one_request", kind="self", B=1, H=12, S=320, D=64, valid_min=259, valid_step=1),
        # a batch of padded texts through an encoder layer (workload C2)
        dict(name="self_encoder_batch", kind="self", B=32, H=12, S=512, D=64, valid_min=256, valid_step=64),
        # many short sequences (workload C5)
        dict(name="self_many_short", kind="self", B=256, H=16, S=256, D=64, valid_min=64, valid_step=64),
        # prefill of a batch of prompts (workload C3)
        dict(name="self_prefill", kind="self", B=8, H=32, S=2048, D=128, valid_min=2048, valid_step=1, v_std=0.5),
        # long-context prefill with outliers in Q and K (workload C4)
        dict(name="self_long", kind="self", B=1, H=32, S=16384, D=128, valid_min=15360, valid_step=1024, outliers=0.01),
        # one decoding step of a batch: one query row per head against caches of different lengths
        dict(name="cross_decode", kind="cross", B=16, H=32, Sq=1, S=4096, D=128, valid_min=1025, valid_step=1),
        # a chunk of a prompt against what is cached already, unsigned probabilities; neither length a multiple of 128
        dict(name="cross_chunk", kind="cross", B=2, H=16, Sq=200, S=1984, D=128, valid_min=1201, valid_step=1, uint8_p=True),
        # per-row probability scales on an encoder batch
        dict(name="policy_row", kind="policy", B=4, H=16, S=1024, D=64, valid_min=512, valid_step=1, policy=1),
        # quantisation of one activation of a single request, odd size
        dict(name="quantize_request", kind="quantize", n=12 * 333 * 64 + 5),
        # quantisation of one activation of the prefill batch
        dict(name="quantize_prefill", kind="quantize", n=8 * 32 * 2048 * 128),
        # the encoder batch for a program whose activations live in host memory
        dict(name="host_encoder_batch", kind="host", B=32, H=12, S=512, D=64, valid_min=256, valid_step=64),
    ]


# The most that a drawn case asks for: bytes of one of q, k, v, o, and operations of one call (those of workload C4 are 4.4e12).
MOST_TENSOR = 1 << 26
MOST_FLOPS = 2.0e12


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("self", "self", "self", "self", "cross", "cross", "cross", "policy", "quantize", "quantize", "host"))
    if kind == "quantize":
        return dict(kind=kind, n=_log_int(rng, 4001, 1 << 26))
    D = rng.choice((64, 128))
    S = 64 * _log_int(rng, 1, 16384 // 64 if kind != "host" else 4096 // 64)
    H = rng.choice((2, 4, 8, 12, 16, 24, 32))
    Sq = S
    if kind == "cross":
        # half of the cross calls are decoding steps, the others chunks of a prompt
        S = max(S, 256)
        Sq = 1 if rng.random() < 0.5 else _log_int(rng, 2, 2048)
    most_b = min(MOST_TENSOR // (H * max(S, Sq) * D), MOST_FLOPS / (4.0 * H * Sq * S * D), 256)
    B = _log_int(rng, 1, max(1, int(most_b)))
    case = dict(kind=kind, B=B, H=H, S=S, D=D, valid_min=S, valid_step=1)
    if rng.random() < 0.6:
        case["valid_min"] = rng.randint(max(1, S // 4), S)
        case["valid_step"] = rng.choice((1, 64))
    if kind == "cross":
        case["Sq"] = Sq
    if kind == "policy":
        case["policy"] = rng.choice((fmha.POLICY_ROW, fmha.POLICY_STATIC))
    elif rng.random() < 0.2:
        case["uint8_p"] = True
    if kind == "self" and rng.random() < 0.2:
        case["outliers"] = 0.01
    return case


def _round_length(case, n):
    return min(case["S"], -(-n // case["valid_step"]) * case["valid_step"])


def _logit_variance(case):
    # of q.k/sqrt(D) when a share `outliers` of the entries of both is 8 times as large
    return (1.0 + 63.0 * case.get("outliers", 0.0)) ** 2


def _mean_keys(case):
    """Mean number of unpadded keys per sequence."""
    lo, hi = case["valid_min"], case["S"]
    return sum(_round_length(case, n) for n in range(lo, hi + 1)) / (hi - lo + 1)


def _quantised(shape, std, outliers, seed):
    """One activation: normal values, a few of them larger, quantised symmetrically with its own largest magnitude."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(shape, generator=g, device="cuda")
    if std != 1.0:
        x.mul_(std)
    if outliers:
        x = torch.where(torch.rand(shape, generator=g, device="cuda") < outliers, x * 8.0, x)
    amax = float(x.abs().max())
    return x.mul_(127.0 / amax).round_().clamp_(-127, 127).to(torch.int8), amax


def prepare(case, seed):
    if case["kind"] == "quantize":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        x = torch.randn(case["n"], generator=g, device="cuda")
        return dict(kind="quantize", x=x, out=torch.empty(case["n"], dtype=torch.int8, device="cuda"), amax=torch.empty(1, device="cuda"))
    B, H, S, D = case["B"], case["H"], case["S"], case["D"]
    Sq = case.get("Sq", S)
    outliers, v_std = case.get("outliers", 0.0), case.get("v_std", 1.0)
    q, q_amax = _quantised((B, H, Sq, D), 1.0, outliers, 4 * seed)
    k, k_amax = _quantised((B, H, S, D), 1.0, outliers, 4 * seed + 1)
    v, v_amax = _quantised((B, H, S, D), v_std, 0.0, 4 * seed + 2)
    g = torch.Generator()
    g.manual_seed(4 * seed + 3)
    lengths = torch.randint(case["valid_min"], S + 1, (B,), generator=g)
    lengths = torch.tensor([_round_length(case, int(n)) for n in lengths])
    mask = (torch.arange(S)[None, :] >= lengths[:, None]).to(torch.int8).cuda()     # non-zero = padding
    # The calibrated output range: six standard deviations of an average over that many normal values.
    # The calibrated s_max of the static policy: a probability that few rows exceed.
    var = _logit_variance(case)
    spread = math.sqrt(min(1.0, math.exp(min(var, 50.0)) / case["valid_min"]))
    param = fmha.FMHAParamI8(q_amax, k_amax, v_amax, min(v_amax, 6.0 * v_std * spread), min(1.0, spread))
    s = dict(kind=case["kind"], param=param, q=q, k=k, v=v, mask=mask, o=torch.empty_like(q), uint8_p=case.get("uint8_p", False))
    if case["kind"] in ("self", "host"):
        s["desc"] = fmha.AttnDataDescriptor(B, S, H, D)
    else:
        s["desc"] = fmha.AttnDataDescriptorX(B, Sq, S, H, D)
    if case["kind"] == "policy":
        s["policy"] = case["policy"]
        s["scratch"] = torch.empty(2 * B * H * Sq, device="cuda")
    if case["kind"] == "host":
        for name in ("q", "k", "v", "mask", "o"):
            on_gpu = s[name]
            s[name] = torch.empty(on_gpu.shape, dtype=on_gpu.dtype, pin_memory=True)
            s[name].copy_(on_gpu)
    return s


def run(s):
    kind = s["kind"]
    if kind == "quantize":
        fmha.quantize_f32(None, s["x"], s["out"], s["amax"])
        return s["out"], s["amax"]
    if kind == "self":
        fmha.FMHAInferI8(None, s["param"], s["desc"], s["q"], s["k"], s["v"], s["mask"], s["o"], True, uint8_p=s["uint8_p"])
    elif kind == "cross":
        fmha.FMHAInferI8Cross(None, s["param"], s["desc"], s["q"], s["k"], s["v"], s["mask"], s["o"], uint8_p=s["uint8_p"])
    elif kind == "policy":
        fmha.FMHAInferI8Policy(None, s["param"], s["desc"], s["q"], s["k"], s["v"], s["mask"], s["o"], s["policy"], s["scratch"])
    else:
        fmha.FMHAInferI8Host(s["param"], s["desc"], s["q"], s["k"], s["v"], s["mask"], s["o"], uint8_p=s["uint8_p"])
    return s["o"]


def work(case):
    if case["kind"] == "quantize":
        n = case["n"]
        return {"bytes": 5.0 * n + 4, "flops": 3.0 * n}
    B, H, S, D = case["B"], case["H"], case["S"], case["D"]
    Sq = case.get("Sq", S)
    keys = _mean_keys(case)
    # q in, o out, the unpadded keys and values in, the mask in; two contractions over the unpadded keys
    return {"bytes": B * H * D * (2.0 * Sq + 2.0 * keys) + B * S, "flops": 4.0 * B * H * Sq * keys * D}


def tolerance(case):
    if case["kind"] == "quantize":
        return "exact"
    # int8 results of fp32 arithmetic: a probability or an output that lies at a rounding boundary may fall on either
    # side of it in another order of summation or with another exp2 of the same accuracy
    return {"rel": 0.0, "differ": 2e-3}
