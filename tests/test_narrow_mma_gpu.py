"""Narrow heads on the tensor cores (bf16, softmax): as close to 64 bits as the fp32 kernels, sharp scores, values that are not finite."""
import pytest
import torch

import causal_flare as cf
from causal_flare import _lib, _ops
from oracle import flare_oracle as orc
from util import to_dev

pytestmark = pytest.mark.gpu


def step(monkeypatch, path, q, k, v, dy):
    monkeypatch.setenv("FLARE_B200_PATH", path)
    ql, kl, vl = (t.detach().requires_grad_() for t in (q, k, v))
    y = cf.flare_autoregressive_triton(ql, kl, vl)
    return (y.detach(),) + torch.autograd.grad(y, (ql, kl, vl), dy)


# one token; a tile of 16 and its neighbours; a block of 32 and its neighbours; the second segment's first token; a ragged end of
# many segments; one warp, an odd number of warps and eight of them; unequal widths; more lanes than are cut into segments
SHAPES = [(1, 1, 1, 16, 16, 16), (2, 15, 2, 32, 32, 32), (1, 16, 3, 48, 16, 32), (1, 17, 1, 64, 32, 16), (2, 31, 1, 128, 32, 32),
          (1, 33, 2, 96, 32, 32), (1, 65, 2, 64, 32, 32), (1, 1999, 2, 80, 32, 32), (2, 1024, 2, 128, 32, 16), (40, 130, 16, 32, 32, 32)]


@pytest.mark.parametrize("shape", SHAPES)
def test_no_further_from_64_bits_than_the_fp32_kernels(monkeypatch, shape):
    # Both round the same sums to bf16, so the two distances differ by what roundings that fall the other way make of it: below
    # 1 % of the distance plus, for outputs of few entries, a fraction of one rounding.
    B, N, H, M, Dk, Dv = shape
    q, k, v, dy = orc.make_inputs(B, N, H, M, Dk, Dv, seed0=21, dtype=torch.bfloat16, with_dy=True)
    n = min(B, 2)
    if B > 2:  # equal batch rows: the oracle looks at the first ones
        k, v, dy = (t.clone() for t in (k, v, dy))
        k[1:], v[1:], dy[1:] = k[:1], v[:1], dy[:1]
    y_ref = orc.ar_forward(q, k[:n], v[:n])
    ref = orc.ar_backward_closed_form(q, k[:n], v[:n], dy[:n])
    want = (y_ref, ref["dQ"], ref["dK"], ref["dV"])
    got = {path: step(monkeypatch, path, *to_dev(q, k, v, dy)) for path in ("auto", "exact")}
    for i, name in enumerate(("y", "dQ", "dK", "dV")):
        err = {}
        for path, out in got.items():
            x = out[i].float().cpu()
            x = x * (n / B) if name == "dQ" else x[:n]
            # (a single token has no gradient but dV: what is left there are differences of equal fp32 numbers)
            err[path] = orc.rel_l2(x, want[i]) if N > 1 or name in ("y", "dV") else orc.max_abs(x, want[i])
        assert err["auto"] <= 1.01 * err["exact"] + 2.0 ** -9 / want[i].numel() ** 0.5 + 1e-5, f"{name}: {err}"


def test_roundings_are_those_of_the_exact_values():
    # A relative error e of a sum moves its rounding to bf16 with the probability 2 e / 2^-8 on average.  fp32 sums of terms that
    # cancel (dK, dQ) stay within 2^-20: 2^-11, and twice that for the spread over the entries.  Operands of 16 bits (2^-17 per
    # factor) move five times as many.
    B, N, H, M, D = 2, 1024, 4, 64, 32
    q, k, v, dy = orc.make_inputs(B, N, H, M, D, seed0=25, dtype=torch.bfloat16, with_dy=True)
    ql, kl, vl = (t.detach().cuda().requires_grad_() for t in (q, k, v))
    got = torch.autograd.grad(cf.flare_autoregressive_triton(ql, kl, vl), (ql, kl, vl), dy.cuda())
    ref = orc.ar_backward_closed_form(q, k, v, dy)
    for x, name in zip(got[1:], ("dK", "dV")):
        moved = (x.cpu() != ref[name].to(torch.bfloat16)).float().mean().item()
        assert moved <= 2.0 ** -10, f"{name}: {moved}"


def test_dq_in_fp32_is_that_of_the_fp32_kernels():
    # B N terms summed in fp32: one rounding each, 2^-24, which add up like their square root
    B, N, H, M, D = 2, 1000, 4, 64, 32
    q, k, v, dy = orc.make_inputs(B, N, H, M, D, seed0=26, dtype=torch.bfloat16, with_dy=True)
    auto, exact = (_ops.backward(*to_dev(q, k, v, dy), scale=D ** -0.5, path=path) for path in (_lib.PATH_AUTO, _lib.PATH_EXACT))
    for x, y in zip(auto[:3], exact[:3]):
        assert torch.equal(x, y)
    assert auto[0].dtype == torch.float32
    want = orc.ar_backward_closed_form(q, k, v, dy)["dQ"]
    assert orc.rel_l2(auto[0].cpu(), want) <= 2.0 ** -24 * (B * N) ** 0.5


@pytest.mark.parametrize("shape", [(2, 300, 4, 64, 32), (1, 33, 2, 32, 16)])
def test_every_entry_point_that_rounds_dq_takes_these_kernels(shape):
    # the autograd functions in Python and the recurrent operator give the gradients of the native layer, bit for bit
    B, N, H, M, D = shape
    q, k, v, dy = to_dev(*orc.make_inputs(B, N, H, M, D, seed0=29, dtype=torch.bfloat16, with_dy=True))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    want = torch.autograd.grad(cf.flare_autoregressive_triton(*leaves), leaves, dy)
    y, _ = cf.flare_autoregressive_triton(*leaves, profile=True)
    for x, ref in zip(torch.autograd.grad(y, leaves, dy), want):
        assert x.dtype == torch.bfloat16 and torch.equal(x, ref)
    y = cf.flare_recurrent_triton(*leaves)
    for x, ref in zip(torch.autograd.grad(y, leaves, dy.permute(0, 2, 1, 3)), want):
        assert torch.equal(x, ref)


@pytest.mark.parametrize("std", [4.0, 24.0])
def test_sharp_scores(monkeypatch, std):
    # at 24 the running maximum grows by hundreds of powers of two inside tiles, which are taken in several windows
    B, N, H, M, D = 2, 200, 4, 32, 32
    q, k, v, dy = to_dev(*orc.make_inputs(B, N, H, M, D, seed0=22, dtype=torch.bfloat16, with_dy=True))
    a, b = (step(monkeypatch, path, q * std, k, v, dy) for path in ("auto", "exact"))
    for name, x, y in zip(("y", "dQ", "dK", "dV"), a, b):
        assert torch.isfinite(x.float()).all(), name
        assert orc.rel_l2(x.float().cpu(), y.float().cpu()) <= 2.0 ** -8, name


@pytest.mark.parametrize("where", ["v", "k"])
def test_a_value_that_is_not_finite_reaches_no_earlier_token(monkeypatch, where):
    B, N, H, M, D = 1, 100, 2, 64, 32
    q, k, v, dy = to_dev(*orc.make_inputs(B, N, H, M, D, seed0=23, dtype=torch.bfloat16, with_dy=True))
    (v if where == "v" else k)[0, 43, 1, 5] = float("inf")
    a, b = (step(monkeypatch, path, q, k, v, dy)[0] for path in ("auto", "exact"))
    assert torch.isfinite(a[:, :43].float()).all() and torch.isfinite(a[:, :, 0].float()).all()
    assert torch.equal(torch.isfinite(a), torch.isfinite(b))


def test_head_slices(monkeypatch):
    B, N, H, M, D = 2, 300, 3, 64, 32
    q, k, v, dy = to_dev(*orc.make_inputs(B, N, H, M, D, seed0=24, dtype=torch.bfloat16, with_dy=True))
    k2, v2, dy2 = (torch.cat([t, t], dim=2)[:, :, :H] for t in (k, v, dy))
    for x, y in zip(step(monkeypatch, "auto", q, k, v, dy), step(monkeypatch, "auto", q, k2, v2, dy2)):
        assert torch.equal(x, y)


@pytest.mark.parametrize("shape, sharp", [((2, 77, 2, 32, 32, 32), 1.0), ((1, 300, 2, 128, 32, 32), 20.0), ((1, 16, 1, 16, 16, 32), 20.0)])
def test_windows(monkeypatch, shape, sharp):
    # One latent's score rises by 60 nats at ten tokens: next to one another, at edges of tiles, two in one tile; the others are
    # sharp by themselves or not.  (600 nats in all: 64 bits hold 700.)  As close to 64 bits as the fp32 kernels.
    B, N, H, M, Dk, Dv = shape
    q, k, v, dy = orc.make_inputs(B, N, H, M, Dk, Dv, seed0=27, dtype=torch.bfloat16, with_dy=True)
    q = (q.float() * sharp).bfloat16()
    steps = torch.zeros(N)
    steps[[t for t in (1, 2, 9, 15, 16, 31, 33, 47, 60, 70) if t < N]] = 1
    q[:, 0], q[:, 1:, 0], k[..., 0] = 0, 0, steps.cumsum(0).bfloat16()[None, :, None]
    q[:, 0, 0] = 60 * Dk ** 0.5
    want = (orc.ar_forward(q, k, v),) + tuple(orc.ar_backward_closed_form(q, k, v, dy)[n] for n in ("dQ", "dK", "dV"))
    got = {path: step(monkeypatch, path, *to_dev(q, k, v, dy)) for path in ("auto", "exact")}
    for i, name in enumerate(("y", "dQ", "dK", "dV")):
        err = {path: orc.rel_l2(out[i].float().cpu(), want[i]) for path, out in got.items()}
        assert err["auto"] <= 1.05 * err["exact"] + 2.0 ** -9 / want[i].numel() ** 0.5, f"{name}: {err}"


def test_sharp_scores_stay_on_the_tensor_cores():
    # (the kernels standing by walk a lane with one CTA: 20 times the call's time)
    q, k, v = to_dev(*orc.make_inputs(2, 1000, 4, 64, 32, seed0=28, dtype=torch.bfloat16))
    def best(q):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                cf.flare_autoregressive_triton(q, k, v)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)
    assert best(q * 200) <= 4 * best(q)
