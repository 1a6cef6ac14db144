"""Norm kernels at the edges of their row splits (lane teams, whole-CTA rows, partly filled vectors, ragged row counts)."""
import pytest
import torch

from mlperf_training_b200.ops import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 5, 333])
@pytest.mark.parametrize("D", [8, 64, 72, 128, 136, 256, 264, 512, 520, 1024, 1032, 2880, 4096, 4104, 8192])
@pytest.mark.parametrize("layer_norm,swish", [(False, False), (False, True), (True, False), (True, True)])
def test_norm_matches_fp32(T, D, layer_norm, swish):
    g = torch.Generator().manual_seed(T * 10007 + D)
    x, dy, dres = (torch.randn(T, D, generator=g).bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(D, generator=g)).bfloat16()
    b = (0.1 * torch.randn(D, generator=g)).bfloat16() if layer_norm else None
    kw = dict(layer_norm=layer_norm, swish=swish)
    y_c, h_c, mean_c, rstd_c = kernels.norm_fwd(x, w, b, 1e-5, **kw)
    dx_c, dw_c, db_c = kernels.norm_bwd(dy, h_c, w, b, mean_c, rstd_c, dres=dres, **kw)
    c = lambda t: None if t is None else t.cuda()
    y, h, mean, rstd = kernels.norm_fwd(c(x), c(w), c(b), 1e-5, **kw)
    dx, dw, db = kernels.norm_bwd(c(dy), h, c(w), c(b), mean, rstd, dres=c(dres), **kw)
    # bf16 outputs of the same fp32 arithmetic in another order: half an ulp each (2^-8 together)
    for a, r in ((y, y_c), (dx, dx_c)):
        assert (a.float().cpu() - r.float()).abs().max() <= 2 ** -8 * r.float().abs().max()
    torch.testing.assert_close(rstd.cpu(), rstd_c, rtol=1e-5, atol=0)
    # fp32 sums over T rows: T * 2^-24 of the sum of magnitudes, and expf's few ulp with swish
    for a, r in ((dw, dw_c), (db, db_c)):
        if a is not None:
            torch.testing.assert_close(a.cpu(), r, rtol=1e-4, atol=1e-4 * T ** 0.5)


@pytest.mark.parametrize("T,D", [(5001, 512), (3001, 1016), (2501, 1032), (2500, 2880), (1301, 4096), (701, 8192)])
@pytest.mark.parametrize("layer_norm", [False, True])
@pytest.mark.parametrize("res", [False, True])
def test_norm_bwd_over_many_row_groups(T, D, layer_norm, res):
    """More rows than the ring of row groups in flight holds, with a remainder, against fp64."""
    g = torch.Generator(device="cuda").manual_seed(D)
    x, dy, dres = (torch.randn(T, D, device="cuda", generator=g).bfloat16() for _ in range(3))
    w, b = (torch.randn(D, device="cuda", generator=g).bfloat16() for _ in range(2))
    y, h, mean, rstd = kernels.norm_fwd(x, w, b if layer_norm else None, 1e-5, layer_norm=layer_norm)
    dx, dw, db = kernels.norm_bwd(dy, x, w, b if layer_norm else None, mean, rstd, layer_norm=layer_norm, dres=dres if res else None)
    xd, wd = x.double().requires_grad_(True), w.double().requires_grad_(True)
    xc = xd - xd.mean(1, keepdim=True) if layer_norm else xd
    (xc * (xc.square().mean(1, keepdim=True) + 1e-5).rsqrt() * wd).backward(dy.double())
    ref = xd.grad + (dres.double() if res else 0)
    # one rounding to bf16 (2^-9) of fp32 arithmetic on terms of the row's size
    assert ((dx.double() - ref).abs() <= ref.abs() * 2 ** -8 + 2 ** -18 * ref.abs().max()).all()
    # fp32 sums over T rows: each term is off by a few 2^-24, they add up like sqrt(T) at worst times the largest
    bound = T ** 0.5 * 2 ** -20 * (dy.double() * xc.detach()).abs().max()
    assert (dw.double() - wd.grad).abs().max() <= bound
    if layer_norm:
        assert (db.double() - dy.double().sum(0)).abs().max() <= T ** 0.5 * 2 ** -20 * dy.double().abs().max()
