"""The single-token decode kernel in each of the forms that its launch chooses from, against the CPU oracle."""
import pytest
import torch

import causal_flare as cf
from oracle import flare_oracle as orc
from util import assert_close, to_dev

pytestmark = pytest.mark.gpu

# Widths above 128: eight slices, where a lane doubles to them and just below; as many as are allowed of wider ones, which would
# double further (512 and 1024 columns); few latents, or too few columns per slice, that stop earlier.
WIDE = [(1, 2, 256, 128, 256), (1, 3, 144, 64, 256), (2, 1, 128, 64, 256), (1, 2, 256, 128, 512), (1, 2, 144, 32, 512), (1, 1, 256, 64, 1024),
        (1, 2, 80, 64, 1024), (2, 1, 16, 64, 1024), (19, 1, 256, 64, 512)]
# Many lanes: a state of 8 KB at most, just above it, of 16 KB with more than eight lanes per SM and just above that, of 24 KB, whose last
# vectors are a batch of their own; one to eight rows of latents, an odd number of them; a key wider than a round of its columns.
MANY = [(38, 16, 32, 64, 64), (38, 16, 48, 64, 64), (75, 16, 64, 64, 64), (75, 16, 80, 64, 64), (38, 16, 96, 64, 64), (75, 16, 16, 512, 64),
        (38, 16, 128, 32, 16), (19, 16, 160, 64, 64), (19, 16, 176, 64, 32), (38, 16, 208, 64, 32), (1, 2, 96, 64, 64), (1, 3, 16, 96, 64)]
# four slices; four with a number of latents that they do not share evenly by 32; two (64 columns); too many latents to slice; a lane
# whose state just fits what is asked for ahead, and one latent group more; more lanes than two CTAs per SM, with and without a
# remainder of the streaming loop
SHAPES = [(1, 2, 256, 128, 128), (2, 3, 208, 128, 128), (1, 1, 144, 64, 64), (1, 2, 512, 128, 128), (2, 2, 64, 128, 128),
          (2, 2, 80, 128, 128), (20, 16, 64, 64, 128), (19, 16, 48, 128, 128)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("separate", [False, True])
@pytest.mark.parametrize("shape", SHAPES + WIDE + MANY)
def test_step(shape, separate, dtype):
    # fp32: about 2^8 terms summed in another order, exponentials of the fast unit: 1e-5.  bf16: one rounding of y.
    B, H, M, Dk, Dv = shape
    q, k, v = orc.make_inputs(B, 1, H, M, Dk, Dv, seed0=17, dtype=dtype)
    kd = torch.randn(H, M, Dk, generator=torch.Generator().manual_seed(3)).to(dtype) if separate else None
    g = torch.Generator().manual_seed(5)
    st = {"m": 3.5 + 0.3 * torch.randn(B, H, M, generator=g), "d": 100 * torch.exp(0.2 * torch.randn(B, H, M, generator=g))}
    st["u"] = 0.1 * torch.randn(B, H, M, Dv, generator=g) * st["d"][..., None]
    mask = torch.ones(B, dtype=torch.bool)
    mask[B // 2 + 1:] = False
    sc = Dk ** -0.5
    y_ref, st_ref = orc.decode_step(q, k[:, 0], v[:, 0], {a: t.double() for a, t in st.items()}, scale=sc, K_dec=kd, attention_mask=mask)
    qc, kc, vc = to_dev(q, k, v)
    stc = {a: t.cuda().clone() for a, t in st.items()}
    kw = dict(K_dec=kd.cuda()) if separate else {}
    y, out = cf.flare_autoregressive_decode_triton(qc, kc, vc, stc, scale=sc, attention_mask=mask.cuda(), **kw)
    tol = dict(atol=1e-5, rtol=1e-4)
    assert_close(y[:, 0], y_ref.reshape(B, H, Dv), what="y", **(tol if dtype == torch.float32 else dict(atol=1e-4, rtol=2.0 ** -8)))
    for key in ("m", "d", "u"):
        assert_close(out[key], st_ref[key], what=key, atol=1e-4, rtol=1e-4)
        assert torch.equal(out[key][~mask.cuda()].cpu(), st[key][~mask]), key
