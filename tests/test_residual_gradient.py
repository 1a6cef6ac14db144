"""The residual branch's gradient added inside the norm's backward equals the sum autograd would make."""
import pytest
import torch

from mlperf_training_b200.ops import functional as F


@pytest.mark.parametrize("layer_norm", [False, True])
@pytest.mark.parametrize("use", ["both", "norm", "residual"])
def test_pass_x(layer_norm, use):
    torch.manual_seed(0)
    x0, w, nw = torch.randn(6, 16), torch.randn(8, 16), torch.randn(16)
    grads = []
    for fused in (False, True):
        x, wp, nwp = x0.clone().requires_grad_(True), w.clone().requires_grad_(True), nw.clone().requires_grad_(True)
        kw = dict(layer_norm=layer_norm, norm_b=torch.zeros(16) if layer_norm else None)
        y, r = F.norm_linear(x, nwp, wp, pass_x=True, **kw) if fused else (F.norm_linear(x, nwp, wp, **kw), x)
        loss = (y * torch.arange(y.numel()).view(y.shape)).sum() if use != "residual" else 0.0
        if use != "norm":
            loss = loss + (r ** 2).sum()
        loss.backward()
        grads.append([t.grad for t in (x, nwp, wp)])
    for a, b in zip(*grads):
        assert (a is None) == (b is None)
        if a is not None:
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)


def test_pass_x_without_grad():
    x = torch.randn(4, 16)
    with torch.no_grad():
        y, r = F.norm_linear(x, torch.ones(16), torch.ones(8, 16), pass_x=True)
    assert torch.equal(r, x) and not y.requires_grad
