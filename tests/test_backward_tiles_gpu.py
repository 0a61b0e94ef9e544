"""GPU: dS, dV and dK of the tensor-core backward leave in tiles of 64 and 32 tokens that are clipped at the sequence's and the latent
bank's end.  Lengths and banks around the tiles' edges, against the oracle's closed form (not one token: its y is v whatever q and k
are, so that dQ = 0 has no relative error); nothing around dV and dK is touched."""
import ctypes as C

import pytest
import torch

from causal_flare import _lib
from oracle import flare_oracle as orc
from test_backward_tensor_gpu import SWEEP, check_gate
from util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,M,Dk,Dv,bs", [
    (1, 17, 2, 64, 128, 128, 1), (1, 31, 2, 64, 128, 128, 1), (2, 33, 2, 128, 64, 64, 1), (2, 129, 2, 16, 64, 128, 1),
    (1, 160, 3, 192, 64, 64, 32), (1, 257, 2, 80, 128, 128, 1), (1, 97, 1, 48, 64, 64, 1), (3, 127, 2, 112, 64, 128, 1),
])
def test_rows_that_leave_in_tiles(B, N, H, M, Dk, Dv, bs):
    q, k, v, dy = orc.make_inputs(B, N, H, M, Dk, Dv, seed0=11, dtype=torch.bfloat16, with_dy=True)
    ref = orc.ar_backward_closed_form(q, k, v, dy, block_size=bs)
    qc, kc, vc, dyc = to_dev(q, k, v, dy)
    guard, size = 4096, B * N * H * Dv
    ksize = B * N * H * Dk
    dv_all, dk_all = (torch.full((n + 2 * guard,), 7.0, dtype=torch.bfloat16, device="cuda") for n in (size, ksize))
    dq = torch.empty(q.shape, dtype=torch.bfloat16, device="cuda")
    a = _lib.BwdArgs()
    a.fwd = _lib.make_fwd_args(qc, kc, vc, None, None, None, scale=Dk ** -0.5, block_size=bs)
    a.dy = dyc.data_ptr()
    a.dy_stride_b, a.dy_stride_n, a.dy_stride_h = dyc.stride()[:3]
    a.dq, a.dk, a.dv = dq.data_ptr(), dk_all[guard:].data_ptr(), dv_all[guard:].data_ptr()
    a.dq_dtype = 1
    assert _lib.load().flare_backward_uses_tensor_path(C.byref(a)) == 1
    _lib.run_backward(a, dyc.device)
    got = dict(dQ=dq, dK=dk_all[guard:guard + ksize].view(B, N, H, Dk), dV=dv_all[guard:guard + size].view(B, N, H, Dv))
    check_gate(got, ref, f"tiles {(B, N, H, M, Dk, Dv, bs)}", rel_l2=SWEEP)
    for x, n in ((dv_all, size), (dk_all, ksize)):
        assert bool((x[:guard] == 7).all()) and bool((x[guard + n:] == 7).all())
