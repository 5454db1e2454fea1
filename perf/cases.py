"""The attention calls whose speed is watched: what a model's training step, prompt or decoding step asks
of this library, made through the public Python entry points (`aotriton_b200.autograd`).

A case is a dict of plain values:

  api      "attention"   autograd.attention, dense (batch, heads, tokens, head dim) tensors
           "sdpa"        autograd.scaled_dot_product_attention, the torch.library operators
           "varlen"      autograd.varlen_attention, token-packed sequences
  train    True: forward and backward, gradients of every input returned; False: forward only, no autograd
  dtype    "bf16", "fp16" or "fp32"
  b hq hk sq sk d        sizes (varlen: b sequences of lengths drawn from lo..hi by the case's `lens` seed, sq = sk)
  mask     "none", "causal" (top-left), "tail" (causal, the queries being the last of the keys' positions) or
           "window" (`left` keys back, none ahead)
  p        dropout probability
  bias     True: additive (b, hq, sq, sk) bias in the inputs' type; its gradient is returned when training

Inputs are N(0, 1), as activations behind a normalisation are, and follow from the seed alone.
"""
import math
import random

import torch

from aotriton_b200 import autograd, flash

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(name, api, train, dtype, b, hq, hk, sq, sk, d, mask="none", left=0, p=0.0, bias=False, lo=0, hi=0, lens=0):
    c = dict(api=api, train=train, dtype=dtype, b=b, hq=hq, hk=hk, sq=sq, sk=sk, d=d, mask=mask, left=left, p=p, bias=bias,
             lo=lo, hi=hi, lens=lens)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest training step: one launch's latency and the host's work per call are all there is
        _case("train_tiny", "attention", True, "fp16", 2, 4, 4, 128, 128, 64),
        # single precision, as a reference run or a small model uses it
        _case("train_fp32", "attention", True, "fp32", 2, 8, 8, 500, 500, 64, mask="causal"),
        # one token of four sequences against a long key/value cache (decoding)
        _case("decode_gqa", "attention", False, "bf16", 4, 32, 8, 1, 6007, 128),
        # a prompt of odd length, grouped heads (prefill)
        _case("prefill_gqa", "attention", False, "bf16", 1, 32, 8, 3001, 3001, 128, mask="causal"),
        # cross attention of image tokens to a short text
        _case("train_cross", "sdpa", True, "fp16", 4, 8, 8, 1024, 77, 80),
        # an encoder layer with dropout, ragged batch length
        _case("train_encoder", "sdpa", True, "fp16", 16, 12, 12, 391, 391, 64, p=0.1),
        # decoder pretraining, packed batches: the benchmark's headline configuration
        _case("train_causal", "attention", True, "bf16", 4, 32, 32, 4096, 4096, 128, mask="causal"),
        # long context, grouped heads, sliding window
        _case("train_window_gqa", "attention", True, "bf16", 1, 64, 8, 16384, 16384, 128, mask="window", left=4096),
        # sequences of very different lengths packed together, with dropout
        _case("train_packed_dropout", "varlen", True, "fp16", 16, 32, 8, 0, 0, 128, mask="causal", p=0.1, lo=64, hi=8192, lens=42),
        # additive bias with its gradient and dropout: the widest head dim of the tensor-core kernels, and one that is padded
        _case("train_bias_d256", "attention", True, "fp16", 8, 16, 16, 2048, 2048, 256, p=0.2, bias=True),
        _case("train_bias_d72", "attention", True, "fp16", 8, 16, 16, 2048, 2048, 72, p=0.2, bias=True),
        # a batch of prompts of different lengths packed together (serving)
        _case("prefill_packed", "varlen", False, "bf16", 24, 32, 8, 0, 0, 128, mask="causal", lo=32, hi=2048, lens=7),
    ]


def _log(rng, lo, hi):
    """A whole number from lo..hi, even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _length(rng, lo, hi):
    """A sequence length: odd as often as a multiple of 128."""
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.6 else max(lo, min(hi, (n + 64) // 128 * 128 or 128))


def _heads(rng):
    hk = rng.choice([1, 2, 4, 8])
    return hk * rng.choice([1, 2, 4, 8]), hk


# the most floating-point operations a drawn case may ask for (below the largest listed case's)
_MOST_FLOPS = 3.0e12


def draw(rng):
    while True:
        kind = rng.choice(["tiny", "fp32", "decode", "prefill", "cross", "encoder", "causal", "window", "packed", "packed_dropout", "bias"])
        half = rng.choice(["bf16", "fp16"])
        if kind == "tiny":
            h, s = rng.choice([1, 2, 4, 8]), _length(rng, 16, 256)
            c = _case(None, rng.choice(["attention", "sdpa"]), True, half, _log(rng, 1, 4), h, h, s, s, rng.choice([32, 64, 128]),
                      mask=rng.choice(["none", "causal"]))
        elif kind == "fp32":
            h, s = rng.choice([2, 4, 8]), _length(rng, 100, 1024)
            c = _case(None, "attention", True, "fp32", _log(rng, 1, 4), h, h, s, s, rng.choice([32, 64, 80, 128]), mask=rng.choice(["none", "causal"]))
        elif kind == "decode":
            hq, hk = rng.choice([(8, 8), (16, 4), (32, 8), (64, 8), (32, 4), (16, 16)])
            c = _case(None, rng.choice(["attention", "attention", "sdpa"]), False, half, _log(rng, 1, 32), hq, hk, rng.choice([1, 1, 1, 2, 5]),
                      _length(rng, 200, 32768), rng.choice([64, 128, 128]))
            if c["sq"] > 1:
                c["api"], c["mask"] = "attention", "tail"
            if c["sq"] > 1 or c["b"] * c["hk"] * c["sk"] > 8 << 20:
                c["b"] = min(c["b"], 4)
            if c["api"] == "sdpa":
                c["b"] = min(c["b"], 8)
        elif kind == "prefill":
            hq, hk = _heads(rng)
            s = _length(rng, 256, 16384)
            c = _case(None, "attention", False, half, _log(rng, 1, 4), hq, hk, s, s, rng.choice([64, 128, 128, 96]), mask="causal")
        elif kind == "cross":
            h = rng.choice([5, 8, 10, 16])
            c = _case(None, "sdpa", True, half, _log(rng, 1, 8), h, h, _length(rng, 256, 4096), rng.choice([77, 128, 154, 257]), rng.choice([40, 64, 80, 128]))
        elif kind == "encoder":
            h, s = rng.choice([8, 12, 16]), _length(rng, 128, 1024)
            c = _case(None, rng.choice(["sdpa", "attention"]), True, half, _log(rng, 1, 32), h, h, s, s, 64, p=rng.choice([0.0, 0.1, 0.1]))
        elif kind == "causal":
            hq, hk = _heads(rng)
            s = _length(rng, 512, 8192)
            c = _case(None, "attention", True, half, _log(rng, 1, 4), hq, hk, s, s, rng.choice([64, 128, 128, 256]), mask="causal")
        elif kind == "window":
            hq, hk = _heads(rng)
            s = _length(rng, 2048, 16384)
            c = _case(None, "attention", True, half, 1, hq, hk, s, s, 128, mask="window", left=rng.choice([512, 1000, 1024, 2048, 4096]))
        elif kind == "packed":
            hq, hk = rng.choice([(16, 16), (32, 8), (64, 8), (16, 4)])
            c = _case(None, "varlen", False, half, _log(rng, 2, 48), hq, hk, 0, 0, 128, mask="causal", lo=_log(rng, 1, 128),
                      hi=_log(rng, 256, 4096), lens=rng.randrange(1 << 20))
        elif kind == "packed_dropout":
            hq, hk = rng.choice([(8, 8), (16, 4), (32, 8)])
            c = _case(None, "varlen", True, half, _log(rng, 2, 16), hq, hk, 0, 0, rng.choice([64, 128]), mask="causal", p=0.1,
                      lo=_log(rng, 16, 128), hi=_log(rng, 512, 8192), lens=rng.randrange(1 << 20))
        else:
            h, s = rng.choice([4, 8, 16]), _length(rng, 256, 2048)
            c = _case(None, "attention", True, half, _log(rng, 1, 8), h, h, s, s, rng.choice([64, 72, 128, 256]), p=rng.choice([0.0, 0.2]), bias=True)
        # (the fp32 kernels run on the ordinary arithmetic units)
        if work(c)["flops"] <= (1.0e11 if c["dtype"] == "fp32" else _MOST_FLOPS):
            return c


def _lengths(c):
    r = random.Random(c["lens"])
    return [r.randint(c["lo"], c["hi"]) for _ in range(c["b"])]


class State:
    pass


def prepare(case, seed):
    c, s = case, State()
    dt = DTYPES[c["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dt)

    s.case = c
    s.seed = 1 + seed % 1000003      # of the dropout
    s.mask = {"none": False, "causal": True, "tail": flash.CausalType.BOTTOM_RIGHT, "window": (c["left"], 0)}[c["mask"]]
    s.bias = None
    if c["api"] == "varlen":
        lens = _lengths(c)
        cu = [0]
        for n in lens:
            cu.append(cu[-1] + n)
        s.cu = torch.tensor(cu, dtype=torch.int32, device="cuda")
        s.most = max(lens)
        # (tokens, heads, head dim) storage, handed over as the (1, heads, tokens, head dim) view
        s.q, s.k, s.v, s.dout = (rand(1, cu[-1], h, c["d"]).transpose(1, 2) for h in (c["hq"], c["hk"], c["hk"], c["hq"]))
    else:
        s.q, s.dout = rand(c["b"], c["hq"], c["sq"], c["d"]), rand(c["b"], c["hq"], c["sq"], c["d"])
        s.k, s.v = rand(c["b"], c["hk"], c["sk"], c["d"]), rand(c["b"], c["hk"], c["sk"], c["d"])
        if c["bias"]:
            s.bias = rand(c["b"], c["hq"], c["sq"], c["sk"])
    if c["train"]:
        for t in (s.q, s.k, s.v) + ((s.bias,) if c["bias"] else ()):
            t.requires_grad_()
    return s


def _forward(s):
    c = s.case
    if c["api"] == "attention":
        return autograd.attention(s.q, s.k, s.v, s.bias, causal=s.mask, dropout_p=c["p"], philox_seed=s.seed)
    if c["api"] == "sdpa":
        return autograd.scaled_dot_product_attention(s.q, s.k, s.v, s.bias, dropout_p=c["p"], is_causal=s.mask,
                                                     enable_gqa=c["hq"] != c["hk"], philox_seed=s.seed)
    return autograd.varlen_attention(s.q, s.k, s.v, s.cu, s.cu, s.most, s.most, causal=s.mask, dropout_p=c["p"])


def run(state):
    s = state
    if not s.case["train"]:
        with torch.no_grad():
            return _forward(s)
    out = _forward(s)
    inputs = (s.q, s.k, s.v) + ((s.bias,) if s.bias is not None else ())
    return (out.detach(),) + torch.autograd.grad(out, inputs, s.dout)


def _pairs(c):
    """Scores per head that are not masked, over the whole batch."""
    if c["api"] == "varlen":
        return sum(n * (n + 1) // 2 if c["mask"] == "causal" else n * n for n in _lengths(c))
    sq, sk = c["sq"], c["sk"]
    if c["mask"] == "causal":
        return c["b"] * sum(min(i + 1, sk) for i in range(sq))
    if c["mask"] == "tail":
        return c["b"] * sum(max(0, i + 1 + sk - sq) for i in range(sq))
    if c["mask"] == "window":
        return c["b"] * sum(max(0, min(i, sk - 1) - max(0, i - c["left"]) + 1) for i in range(sq))
    return c["b"] * sq * sk


def work(case):
    c = case
    size = 4 if c["dtype"] == "fp32" else 2
    tokens_q, tokens_k = (sum(_lengths(c)),) * 2 if c["api"] == "varlen" else (c["b"] * c["sq"], c["b"] * c["sk"])
    q, kv = tokens_q * c["hq"] * c["d"], 2 * tokens_k * c["hk"] * c["d"]
    bias = c["b"] * c["hq"] * c["sq"] * c["sk"] if c["bias"] else 0
    forward = 4 * c["d"] * c["hq"] * _pairs(c)
    if not c["train"]:
        return {"bytes": size * (2 * q + kv + bias), "flops": forward}
    # q, k, v, bias and the output's gradient read; the output and the gradients of q, k, v, bias written
    return {"bytes": size * (4 * q + 2 * kv + 2 * bias), "flops": 3.5 * forward}


def tolerance(case):
    # Probabilities and score gradients are rounded to the inputs' type before the second products, outputs after
    # them (half an ulp is 2^-9 of a value in bf16, 2^-12 in fp16).  Against the same arithmetic in 64 bits the path
    # shows, over the cases' masks, head dims, bias and dropout: bf16 2.6e-3 (largest 0.18 of the root mean square,
    # where a causal gradient is small), fp16 3.1e-4 (1.3e-2), fp32 8e-7 (6e-6); stated is about four times that.
    rel, most = {"bf16": (1e-2, 0.6), "fp16": (1.25e-3, 6e-2), "fp32": (5e-6, 5e-5)}[case["dtype"]]
    return {"rel": rel, "max": most}
