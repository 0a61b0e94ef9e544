"""Masked prefill on the tensor kernels: packing and unpacking of the valid tokens, and an fp16 read-out."""
import ctypes as C

import pytest
import torch

import causal_flare as cf
from causal_flare import _lib, _ops
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


WIDE = [None, "1", "1 merge kernel"]  # instance of (128, 128) heads: the planner's choice, the wide one, its groups in global memory


def choose(monkeypatch, wide):
    if wide:
        monkeypatch.setenv("FLARE_B200_WIDE", "1")
        monkeypatch.setenv("FLARE_B200_CLUSTER", "0" if "merge" in wide else "1")


@pytest.mark.parametrize("bhnd", [False, True])
@pytest.mark.parametrize("wide", WIDE)
@pytest.mark.parametrize("shape", [(1, 300, 2, 64, 64, 64), (2, 700, 2, 192, 64, 128), (1, 384, 2, 128, 128, 128), (1, 384, 2, 256, 128, 128),
                                   (1, 200, 1, 384, 128, 128), (2, 130, 3, 48, 128, 128)])
def test_fp16_read_out_is_rounded_once(monkeypatch, shape, wide, bhnd):
    # y leaves the kernels as fp16.  Against the same call on the bf16 copies only the last rounding differs, at most half a
    # bf16 ulp (2^-8 relative) and half an fp16 ulp (2^-11 relative, 2^-25 absolute); rounded to bf16 on the way, every
    # entry would be a bf16 value, of which there are one in eight.
    B, N, H, M, Dk, Dv = shape
    choose(monkeypatch, wide)
    q, k, v = to_dev(*orc.make_inputs(B, N, H, M, Dk, Dv, seed0=4, dtype=torch.bfloat16))
    q, k, v = (t.half().bfloat16() for t in (q, k, v))  # values that both formats hold
    a = _ops.forward(q.half(), k.half(), v.half(), scale=Dk ** -0.5, out_bhnd=bhnd)[0]
    b = _ops.forward(q, k, v, scale=Dk ** -0.5, out_bhnd=bhnd)[0].double()
    assert a.dtype == torch.float16
    bf16_values = (a.bfloat16().double() == a.double()).double().mean()
    assert bf16_values < 0.3, f"{bf16_values:.2f} of the entries are bf16 values"
    assert ((a.double() - b).abs() <= b.abs() * (2.0 ** -8 + 2.0 ** -11) + 2.0 ** -24).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("wide", WIDE)
@pytest.mark.parametrize("M, Dk", [(128, 128), (256, 128), (64, 64)])
def test_rows_beyond_a_length_are_left_alone(monkeypatch, M, Dk, wide, dtype):
    B, N, H = 3, 300, 2
    choose(monkeypatch, wide)
    q, k, v = orc.make_inputs(B, N, H, M, Dk, seed0=9, dtype=dtype)
    lens = [300, 129, 0]
    qc, kc, vc = to_dev(q, k, v)
    y = torch.full_like(vc, 1.2345)
    before = y.clone()
    lengths = torch.tensor(lens, dtype=torch.int32, device="cuda")
    args = _lib.make_fwd_args(qc, kc, vc, None, None, y, scale=Dk ** -0.5, lengths=lengths)
    _lib.run_forward(args, qc.device)
    for b, n in enumerate(lens):
        assert torch.equal(y[b, n:], before[b, n:]), f"row {b}"
        if n:
            assert_bf16_gate(y[b:b + 1, :n], orc.ar_forward(q, k[b:b + 1, :n], v[b:b + 1, :n], scale=Dk ** -0.5), f"row {b}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("wide", [None, "1 merge kernel"])
@pytest.mark.parametrize("B,N,H,M,D", [(3, 127, 2, 64, 64), (3, 128, 2, 128, 64), (3, 129, 1, 192, 64), (2, 513, 2, 128, 128),
                                       (2, 300, 2, 256, 128), (2, 5000, 1, 64, 64)])
def test_left_padded_rows_stay_where_they_are(monkeypatch, B, N, H, M, D, wide, dtype):
    # y of the valid tokens and the state agree with those of the unpadded prompts on their own, and the padding, whatever it
    # holds, is not touched.  Edges of a chunk, latent groups (their merge kernel moves the rows), wide heads, a carried
    # state, sequence segments, an output in another layout.
    choose(monkeypatch, wide)
    q, k, v = orc.make_inputs(B, N, H, M, D, seed0=13, dtype=dtype)
    pads = [0, N // 3, N - 1][:B]
    mask = (torch.arange(N)[None, :] >= torch.tensor(pads)[:, None]).cuda()
    qc, kc, vc = to_dev(q, k, v)
    _, st0 = cf.flare_autoregressive_prefill_triton(qc, kc[:, :40], vc[:, :40], scale=D ** -0.5)
    kc, vc = kc.masked_fill(~mask[..., None, None], float("nan")), vc.masked_fill(~mask[..., None, None], float("inf"))
    for bhnd in (False, True):
        if bhnd:
            kc, vc = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (kc, vc))
        y, st, _, _ = _ops.forward(qc, kc, vc, scale=D ** -0.5, mask=mask, state_in=st0, want_state=True, out_bhnd=bhnd)
        y = y.transpose(1, 2) if bhnd else y
        for b, pad in enumerate(pads):
            assert not y[b, :pad].any()
            one = {key: t[b:b + 1] for key, t in st0.items()}
            ref, ref_st = cf.flare_autoregressive_prefill_triton(qc, kc[b:b + 1, pad:].contiguous(), vc[b:b + 1, pad:].contiguous(),
                                                                 state=one, scale=D ** -0.5)
            # (another number of segments sums in another order, one rounding of the 16-bit outputs and operands apart)
            assert_bf16_gate(y[b:b + 1, pad:], ref, f"row {b}")
            assert_bf16_gate((st["u"] / st["d"][..., None])[b:b + 1], ref_st["u"] / ref_st["d"][..., None], f"state {b}")


def test_masked_fp16_with_a_bank_expanded_over_the_heads():
    # (a stride of zero, which no tiled copy can express: the bank is copied, the packed rows are not)
    B, N, H, M, D = 2, 200, 2, 64, 64
    q, k, v = to_dev(*orc.make_inputs(B, N, H, M, D, seed0=14, dtype=torch.float16))
    mask = torch.rand(B, N, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) < 0.7
    shared = q[:1].expand(H, M, D)
    a = cf.flare_autoregressive_prefill_triton(shared, k, v, scale=D ** -0.5, attention_mask=mask)
    b = cf.flare_autoregressive_prefill_triton(shared.contiguous(), k, v, scale=D ** -0.5, attention_mask=mask)
    assert_bf16_gate(a[0], b[0], "y")
    assert_bf16_gate(a[1]["u"] / a[1]["d"][..., None], b[1]["u"] / b[1]["d"][..., None], "state")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,N,H,Dk,Dv", [(1, 1, 1, 8, 8), (4, 127, 2, 64, 32), (4, 129, 3, 16, 128), (5, 1030, 1, 64, 64)])
def test_pack_and_unpack_on_their_own(B, N, H, Dk, Dv, dtype):
    # the two entry points for callers that run the kernels on lengths themselves: copies, so bit for bit
    g = torch.Generator().manual_seed(N)
    mask = torch.rand(B, N, generator=g) < 0.5
    for row, keep in enumerate((torch.ones(N), torch.zeros(N), torch.arange(N) >= N // 3, torch.arange(N) < N // 2)[:B]):
        mask[row] = keep.bool()
    k, v = (torch.randn(B, N, 2, H, D, generator=g).to(dtype).cuda()[:, :, 1] for D in (Dk, Dv))  # (strides of a fused projection)
    m = mask.int().cuda()
    slot, lens = torch.full((B, N), -7, dtype=torch.int32, device="cuda"), torch.empty(B, dtype=torch.int32, device="cuda")
    kp, vp = (torch.full((B, N, H, D), float("nan"), dtype=dtype, device="cuda") for D in (Dk, Dv))
    strides = lambda t: (C.c_int64 * 3)(*t.stride()[:3])  # noqa: E731
    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    assert lib.flare_mask_pack(m.data_ptr(), k.data_ptr(), strides(k), v.data_ptr(), strides(v), B, N, H, Dk, Dv, slot.data_ptr(),
                               lens.data_ptr(), kp.data_ptr(), vp.data_ptr(), stream) == 0
    assert torch.equal(lens.cpu(), mask.sum(1).int())
    assert torch.equal(slot.cpu(), torch.where(mask, mask.cumsum(1) - 1, -1).int())
    for b in range(B):
        n = int(mask[b].sum())
        for src, out in ((k, kp), (v, vp)):
            assert torch.equal(out[b, :n], src[b][mask[b].cuda()])
            assert not out[b, n:min(N, -(-n // 128) * 128)].any()
    y = torch.full((B, N, H, Dv), float("nan"), dtype=dtype, device="cuda")
    assert lib.flare_mask_unpack(slot.data_ptr(), vp.data_ptr(), y.data_ptr(), strides(y), B, N, H, Dv, stream) == 0
    assert torch.equal(y, torch.where(mask.cuda()[..., None, None], v, torch.zeros_like(v)))
