"""GPU parity of the exact kernels for narrow heads (widths up to 32, at most 128 latents): against the CPU oracle and, for
the same numbers through separate (equal-valued) decode weights, against the general exact kernels."""
import pytest
import torch

import causal_flare as cf
from causal_flare.autoregressive import flare_autoregressive_stablemax_triton
from oracle import flare_oracle as orc
from util import assert_bf16_gate, assert_close, to_dev

pytestmark = pytest.mark.gpu

F32 = dict(atol=1e-5, rtol=1e-4)
GRAD32 = dict(atol=1e-3, rtol=1e-2)

# edges: one token, a tile of 16 and its neighbours, half-filled warps (M = 16, 48), one to four warps, several segments, a
# segment that ends inside a tile, unequal widths, more lanes than are cut into segments
SHAPES = [(1, 1, 1, 16, 16, 16), (2, 15, 2, 32, 32, 32), (1, 16, 3, 48, 16, 32), (1, 17, 1, 64, 32, 16), (2, 33, 2, 96, 32, 32),
          (1, 500, 2, 128, 32, 32), (1, 1991, 2, 64, 32, 32), (64, 130, 16, 16, 16, 16)]


@pytest.mark.parametrize("stablemax", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_forward_and_gradients(shape, stablemax):
    B, N, H, M, Dk, Dv = shape
    q, k, v, dy = orc.make_inputs(B, N, H, M, Dk, Dv, seed0=11, dtype=torch.float32, with_dy=True)
    if B > 2:  # equal batch rows: the oracle looks at the first ones
        q, k, v, dy = (t.clone() for t in (q, k, v, dy))
        k[1:], v[1:], dy[1:] = k[:1], v[:1], dy[:1]
    ql, kl, vl = (t.requires_grad_() for t in to_dev(q, k, v))
    op = flare_autoregressive_stablemax_triton if stablemax else cf.flare_autoregressive_triton
    y = op(ql, kl, vl)
    dq, dk, dv = torch.autograd.grad(y, (ql, kl, vl), dy.cuda())
    variant = dict(variant="stablemax", power=2.0) if stablemax else {}
    n = min(B, 2)
    ref = orc.ar_backward_closed_form(q, k[:n], v[:n], dy[:n], **variant)
    y_ref = orc.ar_forward(q, k[:n], v[:n], **variant)
    assert_close(y[:n], y_ref, what=f"{shape} y", **F32)
    assert_close(dk[:n], ref["dK"], what=f"{shape} dK", **GRAD32)
    assert_close(dv[:n], ref["dV"], what=f"{shape} dV", **GRAD32)
    # (dQ sums over the batch: with equal batch rows it is B / n of the oracle's, to the same relative bound)
    assert_close(dq * (n / B), ref["dQ"], what=f"{shape} dQ", **GRAD32)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", ["dense", "head_slice", "bhnd"])
def test_same_results_as_the_general_kernels(dtype, layout):
    # equal-valued decode weights are separate tensors: the general kernels.  Same arithmetic in fp32, sums in another
    # order: about sqrt(64) roundings of 2^-24 relative to the row; 16-bit outputs may differ by one ulp
    B, N, H, M, D = 2, 700, 4, 64, 32
    q, k, v, dy = to_dev(*orc.make_inputs(B, N, H, M, D, seed0=5, dtype=dtype, with_dy=True))
    if layout == "head_slice":
        k, v, dy = (torch.cat([t, t], dim=2)[:, :, :H] for t in (k, v, dy))
    elif layout == "bhnd":
        k, v, dy = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (k, v, dy))
    q = 6.0 * q  # sharp scores: the running maximum moves late in the sequence

    def run(separate):
        ql, kl, vl = (t.detach().requires_grad_() for t in (q, k, v))
        kw = dict(Q_dec=kl.detach().clone().requires_grad_(), K_dec=ql.detach().clone().requires_grad_()) if separate else {}
        y = cf.flare_autoregressive_triton(ql, kl, vl, **kw)
        leaves = (ql, kl, vl) + tuple(kw.values())
        g = torch.autograd.grad(y, leaves, dy)
        if separate:
            return y, g[0].float() + g[4].float(), g[1].float() + g[3].float(), g[2]
        return (y,) + g

    tol = dict(atol=1e-4, rtol=1e-3) if dtype == torch.float32 else dict(atol=3e-2, rtol=2e-2)
    for name, a, b in zip(("y", "dQ", "dK", "dV"), run(False), run(True)):
        assert_close(a.float(), b.float().cpu(), what=f"{dtype} {layout} {name}", **tol)


def test_mask_and_state():
    B, N, H, M, D = 3, 200, 2, 48, 32
    q, k, v = orc.make_inputs(B, N, H, M, D, seed0=7, dtype=torch.float32)
    mask = torch.ones(B, N, dtype=torch.bool)
    mask[0, :77] = False
    mask[1, 100:117] = False
    qc, kc, vc = to_dev(q, k, v)
    y, st = cf.flare_autoregressive_prefill_triton(qc, kc[:, :90], vc[:, :90], scale=D ** -0.5, attention_mask=mask[:, :90].cuda())
    y2, st2 = cf.flare_autoregressive_prefill_triton(qc, kc[:, 90:], vc[:, 90:], state=st, scale=D ** -0.5,
                                                     attention_mask=mask[:, 90:].cuda())
    whole, st_all = cf.flare_autoregressive_prefill_triton(qc, kc, vc, scale=D ** -0.5, attention_mask=mask.cuda())
    for i in range(B):
        keep = mask[i]
        ref = orc.ar_forward(q, k[i:i + 1, keep], v[i:i + 1, keep], scale=D ** -0.5)
        got = torch.cat([y, y2], dim=1)[i:i + 1].cpu()
        assert_close(got[:, keep], ref, what=f"row {i}", **F32)
        assert_close(whole[i:i + 1].cpu()[:, keep], ref, what=f"row {i} in one call", **F32)
        assert not got[:, ~keep].any()
    assert_close(st2["u"] / st2["d"][..., None], (st_all["u"] / st_all["d"][..., None]).cpu(), what="state", atol=2e-5, rtol=2e-4)


def test_bf16_gradients_against_the_oracle():
    q, k, v, dy = orc.make_inputs(2, 600, 2, 64, 32, seed0=8, dtype=torch.bfloat16, with_dy=True)
    ql, kl, vl = (t.requires_grad_() for t in to_dev(q, k, v))
    y = cf.flare_autoregressive_triton(ql, kl, vl)
    g = torch.autograd.grad(y, (ql, kl, vl), dy.cuda())
    ref = orc.ar_backward_closed_form(q, k, v, dy)
    for name, x in zip(("dQ", "dK", "dV"), g):
        assert_bf16_gate(x, ref[name], name, max_abs=max(2e-2, float(ref[name].abs().max()) * 2.0 ** -7), rel_l2=5e-3)
