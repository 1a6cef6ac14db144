"""Row and column sums of the backward passes: the per-sample sums of modulation and gate gradients, and O . dO per head."""
import pytest
import torch

from mlperf_training_b200.ops import _lib
from mlperf_training_b200.ops._lib import call, ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,D", [(1, 1, 256), (2, 7, 512), (3, 33, 768), (1, 129, 1280), (2, 501, 3072), (40, 9, 2048)])
def test_sample_sums(B, S, D):
    torch.manual_seed(S)
    T = B * S
    dy, x, scale = (torch.randn(n, D, device="cuda").bfloat16() for n in (T, T, B))
    mean, rstd = x.float().mean(1), x.float().var(1, unbiased=False).add(1e-6).rsqrt()
    dx, (da, db, dg) = torch.empty_like(x), (torch.empty(B, D, device="cuda") for _ in range(3))
    call("b200_ln_modulate_bwd", ptr(dy), ptr(x), ptr(scale), D, ptr(mean), ptr(rstd), ptr(dx), ptr(da), ptr(db), T, D, S, stream_ptr())
    call("b200_gate_residual_bwd", ptr(dy), ptr(x), ptr(scale), D, ptr(dx), ptr(dg), T, D, S, stream_ptr())
    g, xd = dy.double(), x.double()
    xhat = (xd - mean.double()[:, None]) * rstd.double()[:, None]
    for got, term in ((da, g * xhat), (db, g), (dg, g * xd)):
        term = term.view(B, S, D)
        # fp32: the normalised value rounds three times, the product once, and each of the at most S / 8 + 16 additions once
        bound = (S / 8 + 20) * 2 ** -24 * (term.abs().sum(1) + g.abs().view(B, S, D).sum(1)) + 1e-30
        assert ((got.double() - term.sum(1)).abs() <= bound).all()


@pytest.mark.parametrize("B,S,H,D", [(1, 1, 1, 64), (1, 5, 3, 128), (2, 77, 5, 64), (3, 129, 8, 128)])
@pytest.mark.parametrize("shift", [0, 2])
def test_delta(B, S, H, D, shift):
    """``shift``: elements that move every row off its 16-byte boundary."""
    torch.manual_seed(S)
    row = H * D + shift
    o, do = (torch.randn(B * S * row + 8, device="cuda").bfloat16() for _ in range(2))
    delta = torch.empty(B, H, S, device="cuda")
    call("b200_attn_delta", ptr(o[shift:]), ptr(do[shift:]), ptr(delta), B, S, H, D, row, row, S * row, S * row, stream_ptr())
    term = (o[shift:].double() * do[shift:].double())[:B * S * row].view(B, S, row)[..., :H * D].view(B, S, H, D)
    # fp32: a product and at most 8 + 4 additions of it
    assert ((delta.double() - term.sum(-1).permute(0, 2, 1)).abs() <= 14 * 2 ** -24 * term.abs().sum(-1).permute(0, 2, 1)).all()
    _lib.check_status("attn_delta")
