"""Workloads by which the speed of this framework is followed: single passes through its public entry points.

A case is a dict of plain values.  ``kind`` names the entry point and the direction:

* ``decode``  one token for every sequence of a batch on a carried latent state (``flare_autoregressive_decode_triton``)
* ``prefill`` a prompt into a latent state, outputs and state returned (``flare_autoregressive_prefill_triton``);
  ``carry``: on top of a state from earlier text; ``padded``: prompts of different lengths, left-padded, with a mask
* ``forward`` the plain causal operator without gradients (``flare_autoregressive_triton``)
* ``train``   forward and backward of the causal operator, softmax or stablemax encoder
* ``block``   the block-causal operator (``flare_semi_autoregressive_trition``); ``grad``: with its backward

B sequences of N tokens, H heads of width D, M latents per head.
"""

import math
import os
import sys

import torch

_PACKAGE = os.path.abspath("causal-flare_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import causal_flare as cf  # noqa: E402
from causal_flare.autoregressive import flare_autoregressive_stablemax_triton  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}


def listed():
    return [
        # one user at a prompt: the smallest call there is, once for every token and layer
        dict(name="decode_one", kind="decode", dtype="bf16", B=1, H=8, M=64, D=64),
        # a server's decode batch on large states: every step reads and writes all of them
        dict(name="decode_batch", kind="decode", dtype="bf16", B=64, H=32, M=256, D=128),
        # one short prompt of an odd length
        dict(name="prompt", kind="prefill", dtype="bf16", B=1, N=777, H=16, M=64, D=64),
        # a batch of prompts of different lengths, left-padded to the longest
        dict(name="prompts_padded", kind="prefill", dtype="bf16", B=8, N=2000, H=16, M=128, D=64, padded=True),
        # one long document on top of the state of the text before it: few lanes, many tokens
        dict(name="document", kind="prefill", dtype="bf16", B=1, N=32768, H=16, M=128, D=128, carry=True),
        # the chunked causal prefill benchmark
        dict(name="forward", kind="forward", dtype="bf16", B=8, N=8192, H=16, M=128, D=64),
        # inference in half precision
        dict(name="forward_fp16", kind="forward", dtype="fp16", B=4, N=4096, H=16, M=64, D=128),
        # single precision, the small shape that results are checked against the reference with
        dict(name="forward_fp32", kind="forward", dtype="fp32", B=1, N=256, H=8, M=64, D=32),
        # the training step benchmark
        dict(name="train", kind="train", dtype="bf16", B=4, N=4096, H=16, M=64, D=128),
        # a small training step with the stablemax encoder, sequences of an odd length
        dict(name="train_stablemax", kind="train", dtype="bf16", B=2, N=1000, H=8, M=64, D=64, stablemax=True),
        # a training step of a model with narrow heads
        dict(name="train_narrow", kind="train", dtype="bf16", B=8, N=2048, H=16, M=64, D=32),
        # block-causal long context
        dict(name="block_long", kind="block", dtype="bf16", B=2, N=65536, H=32, M=256, D=128, block=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "forward", "train", "train", "block"])
    c = dict(kind=kind, dtype="bf16", B=1, H=rng.choice([4, 8, 12, 16, 32]), M=rng.choice([32, 64, 64, 96, 128, 128, 192, 256]),
             D=rng.choice([64, 128]))
    if kind == "decode":
        c["dtype"] = rng.choice(["bf16", "bf16", "fp16"])
        c["B"] = _log_int(rng, 1, 64)
        return c
    if kind == "prefill":
        c["B"] = _log_int(rng, 1, 8)
        c["N"] = _log_int(rng, 48, 32768)
        option = rng.choice(["", "carry", "padded"])
        if option == "padded":
            c["B"] = max(2, c["B"])
        if option:
            c[option] = True
    elif kind == "forward":
        c["dtype"] = rng.choice(["bf16", "fp16", "fp32"])
        c["B"] = _log_int(rng, 1, 8)
        c["N"] = _log_int(rng, 64, 16384)
        if c["dtype"] == "fp32":  # checks of results: small
            c.update(B=min(c["B"], 2), N=min(c["N"], _log_int(rng, 64, 1024)), H=min(c["H"], 8), M=rng.choice([32, 64]),
                     D=rng.choice([32, 64]))
    elif kind == "train":
        c["B"] = _log_int(rng, 1, 8)
        c["N"] = _log_int(rng, 128, 8192)
        c["D"] = rng.choice([32, 64, 64, 128, 128])
        if c["D"] == 32:  # narrow heads: moderate contexts and latent banks
            c.update(N=min(c["N"], 4096), M=min(c["M"], 128))
        elif rng.random() < 0.4:
            c["stablemax"] = True
    else:
        c["block"] = rng.choice([16, 32, 64, 128])
        c["B"] = _log_int(rng, 1, 4)
        c["N"] = max(1, _log_int(rng, 256, 65536) // c["block"]) * c["block"]
        if rng.random() < 0.5:
            c["grad"] = True
            c["N"] = min(c["N"], 16384)
    largest = listed()[-1]
    budget = largest["B"] * largest["N"] * largest["H"] / (4 if kind == "train" or c.get("grad") else 1)
    while c["B"] * c["N"] * c["H"] > budget and c["B"] > 1:
        c["B"] -= 1
    return c


class _State:
    pass


def prepare(case, seed):
    """What a program holds before the call: N(0, 1) queries, keys and values (activations after a normalisation), the
    state of the text so far, the mask of a padded batch, the upstream gradient."""
    s = _State()
    s.case = case
    s.scale = case["D"] ** -0.5
    B, H, M, D = case["B"], case["H"], case["M"], case["D"]
    N = case.get("N", 1)
    dt = _DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda").to(dt)

    s.q, s.k, s.v = normal(H, M, D), normal(B, N, H, D), normal(B, N, H, D)
    s.state = s.mask = None
    if case["kind"] == "decode" or case.get("carry"):
        # the statistics of a few thousand N(0, 1) tokens: a maximum of about 3.5, a denominator to match, and a
        # numerator whose quotient is a mean of values
        m = 3.5 + 0.3 * torch.randn(B, H, M, generator=g, device="cuda")
        d = 100.0 * torch.exp(0.2 * torch.randn(B, H, M, generator=g, device="cuda"))
        u = 0.1 * torch.randn(B, H, M, D, generator=g, device="cuda") * d[..., None]
        s.state = {"m": m, "d": d, "u": u}
    if case.get("padded"):
        lengths = torch.randint(N // 4, N + 1, (B, 1), generator=g, device="cuda")
        lengths[0] = N
        s.mask = torch.arange(N, device="cuda")[None, :] >= N - lengths
    if case["kind"] == "train" or case.get("grad"):
        s.dy = normal(B, N, H, D)
        for t in (s.q, s.k, s.v):
            t.requires_grad_()
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "decode":
        y, s.state = cf.flare_autoregressive_decode_triton(s.q, s.k, s.v, s.state, scale=s.scale)
        return y, s.state
    if kind == "prefill":
        return cf.flare_autoregressive_prefill_triton(s.q, s.k, s.v, state=s.state, scale=s.scale, attention_mask=s.mask)
    if kind == "forward":
        return cf.flare_autoregressive_triton(s.q, s.k, s.v)
    if kind == "train":
        op = flare_autoregressive_stablemax_triton if case.get("stablemax") else cf.flare_autoregressive_triton
        y = op(s.q, s.k, s.v)
        return y, torch.autograd.grad(y, (s.q, s.k, s.v), s.dy)
    y, aux = cf.flare_semi_autoregressive_trition(s.q, s.k, s.v, block_size=case["block"], chunk_size=min(case["block"], 64))
    if case.get("grad"):
        return y, aux, torch.autograd.grad(y, (s.q, s.k, s.v), s.dy)
    return y, aux


def work(case):
    """Every input read once, every output written once; per token and head 2 M D operations for the scores, as many for
    the state and for the read-out, and two and a half times that in the backward."""
    B, H, M, D = case["B"], case["H"], case["M"], case["D"]
    N = case.get("N", 1)
    e = _BYTES[case["dtype"]]
    row, bank = B * N * H * D * e, H * M * D * e
    state = B * H * M * (D + 2) * 4
    size, flops = 3 * row + bank, 6 * M * D * B * N * H
    if case["kind"] == "decode":
        size += 2 * state
    elif case["kind"] == "prefill":
        size += state * (2 if case.get("carry") else 1) + (B * N if case.get("padded") else 0)
    elif case["kind"] == "block":
        size += B * H * N * 4 + B * H * (N // case["block"]) * M * 4
    if case["kind"] == "train" or case.get("grad"):
        size += 3 * row + bank  # upstream gradient in, dK and dV and dQ out
        flops += 15 * M * D * B * N * H
    return {"bytes": size, "flops": flops}


def tolerance(case):
    # 16-bit inputs and outputs, sums in 32 bits; a single entry (of a gradient summed over few latents) may be off by a
    # few roundings of its largest term
    return {"rel": 1e-5, "max": 4e-4} if case["dtype"] == "fp32" else {"rel": 1e-2, "max": 0.4}
