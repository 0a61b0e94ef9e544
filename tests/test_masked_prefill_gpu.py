"""Masked prefill on the tensor kernels: packing and unpacking of the valid tokens, and an fp16 read-out."""
import pytest
import torch

import causal_flare as cf
from oracle import flare_oracle as orc
from util import assert_bf16_gate, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,M,Dk,Dv", [(1, 64, 64, 64), (31, 192, 64, 128), (128, 64, 64, 64), (1025, 64, 64, 64)])
def test_packed_rows(N, M, Dk, Dv, dtype):
    # one token, part of a warp, a chunk, just beyond one tile of the ranks
    B, H = 5, 1
    q, k, v = orc.make_inputs(B, N, H, M, Dk, Dv, seed0=3, dtype=dtype)
    g = torch.Generator().manual_seed(N)
    mask = torch.rand(B, N, generator=g) < 0.6
    mask[0] = True
    mask[1] = False
    mask[2, : N // 2] = False  # left-padded
    mask[3, N // 2 + 1:] = False  # right-padded
    qc, kc, vc = to_dev(q, k, v)
    kc[~mask.cuda()] = float("nan")  # what stands at a masked position must not matter
    vc[~mask.cuda()] = float("inf")
    kc = torch.cat([kc, kc], dim=2)[:, :, :H]  # head-sliced storage: strides other than the dense ones
    y, st = cf.flare_autoregressive_prefill_triton(qc, kc, vc, scale=Dk ** -0.5, attention_mask=mask.cuda())
    assert y.dtype == dtype and not y.cpu()[~mask].any()
    assert torch.isinf(st["m"][1]).all() and not st["d"][1].any() and not st["u"][1].any()
    for b in (0, 2, 3, 4):
        keep = mask[b]
        if not keep.any():
            continue
        ref, ref_st = orc.ar_forward(q, k[b:b + 1, keep], v[b:b + 1, keep], scale=Dk ** -0.5, return_state=True)
        assert_bf16_gate(y[b:b + 1].cpu()[:, keep], ref, f"row {b}")
        assert_bf16_gate((st["u"] / st["d"][..., None])[b:b + 1], ref_st["u"] / ref_st["d"][..., None], f"state {b}")


@pytest.mark.parametrize("shape", [(1, 300, 2, 64, 64, 64), (2, 700, 2, 192, 64, 128), (1, 384, 2, 256, 128, 128), (2, 130, 3, 48, 128, 128)])
def test_fp16_read_out_is_rounded_once(shape):
    # y leaves the kernels as fp16: against the same call on the bf16 copies only the last rounding differs, at most half a
    # bf16 ulp (2^-8 relative) and half an fp16 ulp (2^-11 relative, 2^-25 absolute)
    B, N, H, M, Dk, Dv = shape
    q, k, v = to_dev(*orc.make_inputs(B, N, H, M, Dk, Dv, seed0=4, dtype=torch.bfloat16))
    q, k, v = (t.half().bfloat16() for t in (q, k, v))  # values that both formats hold
    a = cf.flare_autoregressive_triton(q.half(), k.half(), v.half()).double()
    b = cf.flare_autoregressive_triton(q, k, v).double()
    assert ((a - b).abs() <= b.abs() * (2.0 ** -8 + 2.0 ** -11) + 2.0 ** -24).all()
