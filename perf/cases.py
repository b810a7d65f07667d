"""The calls whose speed counts for a user of this framework: training steps (forward and backward) and forward passes
of block-diffusion attention through the public functions, from one short sequence to batches that fill the GPU.

Imported with the repository's root as the working folder. Every function takes a case, a dict of plain values:

  op             "step": forward, then the gradients of q, k and v; "forward": forward only
  dtype          "bf16", "fp16" or "e4m3" (e4m3: forward only)
  layout         "batched": `batch` samples of `n` tokens a half; "varlen": packed samples of the half lengths `lengths`
                 (a text, comma separated); "qkv": like varlen, q, k and v in one packed projection
  heads, heads_k, dim, block, softcap, deterministic
"""

import math
import os
import sys

import torch

_PACKAGE = os.path.abspath("fast-diffusion-attention_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from fast_diffusion_attention import diffusion_attn_func, diffusion_attn_varlen_func  # noqa: E402
from fast_diffusion_attention.interface import diffusion_attn_varlen_qkvpacked_func  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "e4m3": torch.float8_e4m3fn}
_E4M3_MAX = 448.0


def _case(name, op, heads, heads_k, dim, block, *, batch=0, n=0, lengths="", layout="batched", dtype="bf16",
          softcap=0.0, deterministic=False):
    c = dict(op=op, dtype=dtype, layout=layout, batch=batch, n=n, lengths=lengths, heads=heads, heads_k=heads_k,
             dim=dim, block=block, softcap=softcap, deterministic=deterministic)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest training step: two short samples of a small model, where latency and launches count
        _case("step_small_d64", "step", 4, 4, 64, 64, batch=2, n=256),
        # scoring one sequence: a single forward call with hardly enough work for the chip
        _case("forward_one_sequence", "forward", 16, 16, 128, 32, batch=1, n=512),
        # ragged everything: odd length, a block size that divides nothing, a padded head dimension, fp16
        _case("step_ragged_fp16_d96", "step", 12, 4, 96, 20, batch=3, n=333, dtype="fp16"),
        # the headline training step: multi-head attention, 4K tokens a sample, blocks of 256
        _case("step_mha_block256", "step", 16, 16, 128, 256, batch=8, n=2048),
        # grouped-query training with the small blocks that block-diffusion language models use
        _case("step_gqa_block16", "step", 32, 8, 128, 16, batch=4, n=2048),
        # the same model family at head dimension 64
        _case("step_gqa_d64_block64", "step", 32, 8, 64, 64, batch=4, n=2048),
        # one long sequence, forward only (evaluation of a 16K-token sample)
        _case("forward_gqa_16k", "forward", 32, 8, 128, 64, batch=1, n=8192),
        # large blocks, bitwise reproducible gradients
        _case("step_gqa_deterministic", "step", 32, 8, 128, 1024, batch=4, n=4096, deterministic=True),
        # packed samples of odd lengths out of one projection tensor, blocks of 4
        _case("step_qkv_varlen_block4", "step", 32, 8, 128, 4, layout="qkv",
              lengths="517,4095,1203,2750,611,3391,1876,2049"),
        # a large packed batch, samples of very different lengths, capped scores
        _case("step_varlen_softcap_d64", "step", 32, 32, 64, 256, layout="varlen", softcap=30.0,
              lengths="7424,3584,6656,7680,3840,768,2560,8192,4608,4352,3584,7936,6912,7168,2816,8192"),
        # the widest heads
        _case("step_d256_16k", "step", 8, 8, 256, 256, batch=2, n=8192),
        # quantised inference: e4m3 inputs with a scale for each sample and head
        _case("forward_fp8_d256_16k", "forward", 8, 8, 256, 256, batch=2, n=8192, dtype="e4m3"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["step", "step", "forward"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "e4m3"] if op == "forward" else ["bf16", "bf16", "bf16", "fp16"])
    layout = rng.choice(["batched", "batched", "batched", "varlen"] if dtype == "e4m3"
                        else ["batched", "batched", "batched", "varlen", "qkv"])
    dim = rng.choice([64, 128, 128, 128, 96, 256, 192] if dtype == "e4m3" else [64, 64, 128, 128, 128, 96, 80, 256, 192])
    heads_k, group = rng.choice([(4, 1), (16, 1), (32, 1), (2, 4), (8, 4), (8, 2), (4, 3), (1, 8)])
    block = rng.choice([4, 16, 32, 64, 256, 1024, rng.randint(3, 300)])
    n = _log_int(rng, 64, 8192)
    if rng.random() < 0.5:
        n = max(64, n // 64 * 64)   # half of the lengths are round, half as they fall
    tokens = _log_int(rng, 512, 65536)
    samples = max(1, min(64, tokens // (2 * n)))
    c = _case("", op, heads_k * group, heads_k, dim, block, dtype=dtype, layout=layout,
              softcap=rng.choice([0.0, 0.0, 0.0, 0.0, 30.0]), deterministic=op == "step" and rng.random() < 0.2)
    lengths = [n] * samples
    if layout != "batched":
        lengths = [max(1, _log_int(rng, max(1, n // 8), n)) for _ in range(samples)] + [n]
    # no larger than the largest listed step: fewer tokens until it fits
    while True:
        if layout == "batched":
            c["batch"], c["n"] = len(lengths), lengths[0]
        else:
            c["lengths"] = ",".join(str(x) for x in lengths)
        w = work(c)
        if w["flops"] <= 3e12 and w["bytes"] <= 3e9:
            return c
        lengths = lengths[1:] if len(lengths) > 1 else [lengths[0] // 2]


def _lengths(case):
    if case["layout"] == "batched":
        return [case["n"]] * case["batch"]
    return [int(x) for x in case["lengths"].split(",")]


def prepare(case, seed):
    """Activations as the projections deliver them (unit normal in the compute type), gradients of the output likewise,
    what the autograd graph needs, and for packed samples the offsets."""
    device = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=device).manual_seed(seed)
    heads, heads_k, dim = case["heads"], case["heads_k"], case["dim"]
    lengths = _lengths(case)
    step = case["op"] == "step"
    fp8 = case["dtype"] == "e4m3"
    dtype = torch.bfloat16 if fp8 else _DTYPES[case["dtype"]]
    packed = case["layout"] != "batched"
    lead = (2 * sum(lengths),) if packed else (case["batch"], 2 * case["n"])

    def normal(*shape):
        return torch.randn(*lead, *shape, device=device, dtype=dtype, generator=gen)

    s = {"case": case, "kw": {"softcap": case["softcap"], "deterministic": case["deterministic"]}}
    if case["layout"] == "qkv":
        s["qkv"] = normal(heads + 2 * heads_k, dim).requires_grad_(step)
    else:
        s["q"], s["k"], s["v"] = (normal(h, dim) for h in (heads, heads_k, heads_k))
        if fp8:
            # a scale for each (sample, KV head) maps its largest magnitude to the largest e4m3 number
            offsets = [0]
            for x in lengths:
                offsets.append(offsets[-1] + 2 * x)
            for name in "qkv":
                x = s[name]
                scale = torch.empty(len(lengths), heads_k, device=device)
                y = torch.empty_like(x, dtype=torch.float8_e4m3fn)
                for b in range(len(lengths)):
                    at = slice(offsets[b], offsets[b + 1]) if packed else b
                    part = x[at].float().unflatten(-2, (heads_k, -1))
                    scale[b] = part.abs().amax(dim=(0, 2, 3)) / _E4M3_MAX
                    y[at] = (part / scale[b][:, None, None]).flatten(-3, -2).to(torch.float8_e4m3fn)
                s[name], s["kw"][name + "_descale"] = y, scale
        elif step:
            for name in "qkv":
                s[name].requires_grad_(True)
    if step:
        s["dout"] = normal(heads, dim)
    if packed:
        starts = [0]
        for x in lengths:
            starts.append(starts[-1] + 2 * x)
        s["cu"] = torch.tensor(starts, dtype=torch.int32, device=device)
        s["max"] = 2 * max(lengths)
    return s


def run(state):
    case, kw = state["case"], state["kw"]
    if case["layout"] == "qkv":
        inputs = (state["qkv"],)
        out = diffusion_attn_varlen_qkvpacked_func(state["qkv"], state["cu"], state["max"], case["block"],
                                                   num_heads_q=case["heads"], **kw)
    else:
        inputs = (state["q"], state["k"], state["v"])
        if case["layout"] == "varlen":
            out = diffusion_attn_varlen_func(*inputs, state["cu"], state["cu"], state["max"], state["max"],
                                             case["block"], **kw)
        else:
            out = diffusion_attn_func(*inputs, case["block"], **kw)
    if case["op"] == "forward":
        return out
    return (out,) + torch.autograd.grad(out, inputs, state["dout"])


def _visible_pairs(n, block):
    """(query, key) pairs of one sample and head: a noisy block sees itself and the clean blocks before it, a clean
    block the clean blocks up to itself."""
    full, rest = divmod(n, block)
    one_half = block * block * full * (full + 1) // 2 + rest * n
    return 2 * one_half


def work(case):
    lengths = _lengths(case)
    rows, pairs = 2 * sum(lengths), sum(_visible_pairs(n, case["block"]) for n in lengths)
    size = 1 if case["dtype"] == "e4m3" else 2
    q, kv = rows * case["heads"] * case["dim"], rows * case["heads_k"] * case["dim"]
    flops = 4.0 * pairs * case["heads"] * case["dim"]
    nbytes = (q + 2 * kv) * size + q * 2          # q, k, v in, out
    if case["op"] == "step":
        nbytes += q * 2 + (q + 2 * kv) * 2        # dout in, dq, dk, dv out
        flops *= 3.5                              # the backward's five products against the forward's two
    return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
    # probabilities and results are rounded to the compute type: 8, 11 and 4 significant bits
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "e4m3": 3e-2}[case["dtype"]]}
