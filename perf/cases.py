"""The work that performance is measured on: attention forward passes and training steps
through the public entry points, as a model's layer calls them.

A case is a dict of plain values:
  B, M, N, H, D   batch, query length, key length, heads, head dimension
  dtype           "bf16" or "fp16"
  bias            "none"
                  "float"  (B, H, M, N) in q's dtype, ~ 0.5 N(0, 1)
                  "f32"    the same in fp32 next to 16-bit q, k, v (a bias kept out of autocast)
                  "shared" (1, H, M, N) in q's dtype, expanded over the batch (a relative position table)
                  "mask"   (B, H, M, N) bool, each True with p = 0.9, diagonal True
                  "pad"    (B, N) key padding as bool, expanded over heads and query rows
  grad            the bias is trained: its gradient is asked for too
  causal          top-left aligned causal mask
  train           forward + backward (else the forward alone, without autograd)
  packed          q, k, v come as one (B, S, 3, H, D) tensor
"""
import math

import torch

from triton_flashattn_b200 import flash_attention_fn, flash_attention_qkvpacked_fn

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(B, M, N, H, D, dtype="bf16", bias="none", grad=False, causal=False, train=False, packed=False):
    return dict(B=B, M=M, N=N, H=H, D=D, dtype=dtype, bias=bias, grad=grad, causal=causal, train=train, packed=packed)


def listed():
    cases = {
        # the smallest training step that the tests name: launches and host work are all there is
        "step_small": _case(2, 128, 128, 4, 64, "fp16", "float", grad=True, train=True),
        # one new token for each of eight sequences against their key / value caches
        "decode_batch": _case(8, 1, 4096, 32, 128),
        # one new token of a single long sequence of odd length: few heads, many keys
        "decode_long": _case(1, 1, 20011, 32, 128),
        # the prompt of an inference request
        "prefill": _case(2, 4096, 4096, 32, 128, causal=True),
        # inference of an encoder with a trained position table shared by the batch
        "encode_shared_bias": _case(16, 512, 512, 12, 64, "fp16", "shared"),
        # causal self-attention training, head dimension 64
        "train_causal": _case(4, 1024, 1024, 16, 64, causal=True, train=True),
        # the headline configuration: a trained (B, H, M, N) bias
        "train_bias": _case(8, 2048, 2048, 16, 128, bias="float", grad=True, train=True),
        # packed projections, random bool mask, causal
        "train_mask_packed": _case(4, 4096, 4096, 32, 128, bias="mask", causal=True, train=True, packed=True),
        # a long sequence with a trained bias (a share of the sharded long-sequence configuration)
        "train_bias_long": _case(1, 8192, 8192, 32, 128, bias="float", grad=True, causal=True, train=True),
        # cross-attention over padded sequences, odd lengths
        "train_cross_padded": _case(4, 1000, 777, 12, 64, "fp16", "pad", train=True),
        # many short windows with a trained table: D below the tile width, N no multiple of anything
        "train_windows": _case(256, 49, 49, 6, 32, "fp16", "shared", grad=True, train=True),
        # the widest head dimension
        "train_wide_head": _case(4, 2048, 2048, 8, 256, bias="float", grad=True, train=True),
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6.5e12, w["flops"] / 1.4e15)


def _round_some(rng, n):
    """Half of the lengths are multiples of 64, as padded batches are; the others stay odd."""
    return max(64, n // 64 * 64) if n >= 64 and rng.random() < 0.5 else n


def draw(rng):
    most = max(_cost(c) for c in listed())
    heads = (1, 2, 3, 4, 6, 8, 12, 16, 24, 32)
    while True:
        dtype = rng.choice(("bf16", "bf16", "fp16"))
        kind = rng.choice(("decode", "forward", "plain", "masked", "bias", "cross", "windows", "wide"))
        if kind == "decode":
            c = _case(_log_int(rng, 1, 64), rng.choice((1, 1, 1, 2, 4, 8)), _log_int(rng, 128, 32768), rng.choice(heads[3:]),
                      rng.choice((64, 128, 128)), dtype, rng.choice(("none", "none", "pad", "float")))
        elif kind == "forward":
            s = _round_some(rng, _log_int(rng, 64, 8192))
            c = _case(_log_int(rng, 1, 32), s, s, rng.choice(heads), rng.choice((32, 64, 128, 128)), dtype,
                      rng.choice(("none", "float", "shared", "mask")), causal=rng.random() < 0.5)
        elif kind in ("plain", "masked"):
            s = _round_some(rng, _log_int(rng, 64, 8192))
            c = _case(_log_int(rng, 1, 16), s, s, rng.choice(heads), rng.choice((64, 128)), dtype,
                      "none" if kind == "plain" else rng.choice(("mask", "float")), causal=rng.random() < 0.7, train=True,
                      packed=rng.random() < 0.5)
        elif kind == "bias":
            s = _round_some(rng, _log_int(rng, 64, 8192))
            c = _case(_log_int(rng, 1, 16), s, s, rng.choice(heads), rng.choice((64, 128)), dtype,
                      rng.choice(("float", "float", "f32")), grad=True, causal=rng.random() < 0.5, train=True)
        elif kind == "cross":
            c = _case(_log_int(rng, 1, 16), _round_some(rng, _log_int(rng, 64, 4096)), _round_some(rng, _log_int(rng, 32, 4096)),
                      rng.choice(heads), rng.choice((64, 128)), dtype, rng.choice(("none", "pad")), train=True)
        elif kind == "windows":
            s = rng.randint(16, 144)
            c = _case(_log_int(rng, 16, 1024), s, s, rng.choice((3, 4, 6, 8, 12)), rng.choice((16, 32, 64)), dtype, "shared",
                      grad=True, train=True)
        else:
            s = _round_some(rng, _log_int(rng, 64, 4096))
            bias = rng.choice(("none", "float"))
            c = _case(_log_int(rng, 1, 8), s, s, rng.choice(heads[:8]), 256, dtype, bias, grad=bias == "float",
                      causal=rng.random() < 0.5, train=rng.random() < 0.7)
        if c["B"] * c["H"] <= 65535 and _cost(c) <= most:
            return c


def _pairs(case):
    """(query, key) pairs that take part, per (batch, head)."""
    M, N = case["M"], case["N"]
    if not case["causal"]:
        return M * N
    full = min(M, N)  # rows whose visible keys grow by one each; the rows below see all N keys
    return full * (full + 1) // 2 + (M - full) * N


def work(case):
    """Products: 4 D operations a pair forward, 10 D more backward.  Bytes: q, k, v, the bias and
    the upstream gradient read once, the result and the gradients written once."""
    B, M, N, H, D = (case[x] for x in ("B", "M", "N", "H", "D"))
    pairs = _pairs(case)
    qd, kd = B * M * H * D * 2, B * N * H * D * 2
    bias = {"none": 0, "float": 2 * B * H * pairs, "f32": 4 * B * H * pairs, "shared": 2 * H * pairs, "mask": B * H * pairs,
            "pad": B * N}[case["bias"]]
    bytes_ = 2 * qd + 2 * kd + bias
    if case["train"]:
        bytes_ += 2 * qd + 2 * kd
        if case["grad"]:  # the gradient is dense, its masked part zeros
            bytes_ += {"float": 2 * B, "f32": 4 * B, "shared": 2}[case["bias"]] * H * M * N
    return {"bytes": bytes_, "flops": (14 if case["train"] else 4) * B * H * pairs * D}


def tolerance(case):
    # P, dS and the results are rounded to 16 bits (2^-9 / 2^-12 relative); the differences of two
    # correct results add up over these roundings and through rowsum(o * do), which cancels
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}


def prepare(case, seed):
    B, M, N, H, D = (case[x] for x in ("B", "M", "N", "H", "D"))
    dt = _DTYPES[case["dtype"]]
    train, kind = case["train"], case["bias"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0, dtype=dt):
        t = torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=g)
        return t.mul_(scale) if scale != 1.0 else t

    bias = param = None
    if kind in ("float", "f32"):
        bias = param = normal(B, H, M, N, scale=0.5, dtype=torch.float32 if kind == "f32" else dt)
    elif kind == "shared":
        param = normal(1, H, M, N, scale=0.5)
    elif kind == "mask":
        bias = torch.empty((B, H, M, N), dtype=torch.uint8, device="cuda").random_(0, 10, generator=g).bool()
        bias.diagonal(dim1=2, dim2=3).fill_(True)
    elif kind == "pad":
        lens = torch.randint((N + 1) // 2, N + 1, (B, 1), generator=g, device="cuda")
        bias = (torch.arange(N, device="cuda")[None] < lens)[:, None, None].expand(B, H, M, N)
    if case["grad"]:
        param.requires_grad_()
    if case["packed"]:
        inputs = [normal(B, M, 3, H, D)]
    else:
        inputs = [normal(B, M, H, D), normal(B, N, H, D), normal(B, N, H, D)]
    if train:
        inputs = [t.requires_grad_() for t in inputs]
    return {"inputs": inputs, "bias": bias, "param": param, "shape": (B, H, M, N), "kind": kind, "causal": case["causal"],
            "wrt": inputs + ([param] if case["grad"] else []), "do": normal(B, M, H, D) if train else None}


def run(state):
    bias = state["bias"]
    if state["do"] is None:
        with torch.no_grad():
            return _forward(state, bias)
    out = _forward(state, bias)
    return (out, *torch.autograd.grad(out, state["wrt"], state["do"]))


def _forward(state, bias):
    if state["kind"] == "shared":
        bias = state["param"].expand(state["shape"])
    fn = flash_attention_qkvpacked_fn if len(state["inputs"]) == 1 else flash_attention_fn
    return fn(*state["inputs"], bias, state["causal"])
