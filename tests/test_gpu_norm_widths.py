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
