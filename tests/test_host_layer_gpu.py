"""GPU: calls that the native host layer must leave to the Python layer (what it would lose, refuse or word differently)."""
from fractions import Fraction

import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as fwAD

import causal_flare as cf
from causal_flare.autoregressive import flare_autoregressive_stablemax_triton
from oracle import flare_oracle as orc
from util import to_dev

pytestmark = pytest.mark.gpu

OPS = {
    "softmax": lambda q, k, v: cf.flare_autoregressive_triton(q, k, v),
    "stablemax": lambda q, k, v: flare_autoregressive_stablemax_triton(q, k, v),
    "block": lambda q, k, v: cf.flare_semi_autoregressive_trition(q, k, v, block_size=32, chunk_size=32)[0],
}


def inputs(dtype=torch.bfloat16):
    return to_dev(*orc.make_inputs(1, 64, 2, 32, 64, seed0=21, dtype=dtype))


@pytest.mark.parametrize("requires_grad", [False, True])
@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("op", sorted(OPS))
def test_a_forward_mode_tangent_is_refused_not_dropped(op, which, requires_grad):
    args = [t.requires_grad_(requires_grad) for t in inputs()]
    with fwAD.dual_level():
        args[which] = fwAD.make_dual(args[which], torch.ones_like(args[which]))
        with pytest.raises((NotImplementedError, RuntimeError), match="jvp|forward mode"):
            OPS[op](*args)


@pytest.mark.parametrize("op", ["softmax", "stablemax"])
def test_a_traced_call_computes_when_it_is_replayed(op):
    q, k, v = inputs()
    traced = torch.jit.trace(lambda *a: OPS[op](*a) * 1, (q, k, v), check_trace=False)
    q2, k2, v2 = (t.flip(0).contiguous() * 0.5 for t in (q, k, v))
    want = OPS[op](q2, k2, v2)
    poison = [torch.full_like(want, float("nan")) for _ in range(8)]  # what a fresh output buffer would show
    del poison
    assert torch.equal(traced(q2, k2, v2), want)


def test_backward_of_the_block_causal_operator_allocates_no_gradients_of_the_log_sum_exps():
    def allocations(op):
        leaves = [t.requires_grad_() for t in inputs()]
        y = OPS[op](*leaves)
        dy = torch.ones_like(y)
        torch.autograd.grad(y, leaves, dy, retain_graph=True)
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        torch.autograd.grad(y, leaves, dy)
        return torch.cuda.memory_stats()["allocation.all.allocated"] - before

    assert allocations("block") == allocations("softmax")  # three gradients and the workspace


@pytest.mark.parametrize("op", sorted(OPS))
def test_an_undefined_gradient_of_y_stands_for_zeros(op):
    class Drop(torch.autograd.Function):
        @staticmethod
        def forward(ctx, y):
            return y.sum()

        @staticmethod
        def backward(ctx, g):
            return None

    leaves = [t.requires_grad_() for t in inputs()]
    for t, g in zip(leaves, torch.autograd.grad(Drop.apply(OPS[op](*leaves)), leaves)):
        assert g.shape == t.shape and g.dtype == t.dtype and not g.any()


@pytest.mark.parametrize("scale", ["0.125", Fraction(1, 8), np.float32(0.125), torch.tensor(0.125), True])
def test_scale_is_what_float_makes_of_it(scale):
    q, k, v = inputs()
    st = cf.flare_autoregressive_prefill_triton(q, k, v)[1]
    calls = [lambda s: cf.flare_autoregressive_triton(q, k, v, scale=s),
             lambda s: cf.flare_semi_autoregressive_trition(q, k, v, block_size=32, chunk_size=32, scale=s)[0],
             lambda s: cf.flare_autoregressive_prefill_triton(q, k, v, scale=s)[0],
             lambda s: cf.flare_autoregressive_decode_triton(q, k[:, 0], v[:, 0], {n: t.clone() for n, t in st.items()}, scale=s)[0]]
    for call in calls:
        assert torch.equal(call(scale), call(float(scale)))
        with pytest.raises((TypeError, ValueError)):
            call("wide")
