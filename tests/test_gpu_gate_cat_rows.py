"""Gated concatenation of an HSTU layer at the edges of its row split: one row, rows that fill no team or CTA, more rows than the
resident warps, every width, with and without dropout."""
import pytest
import torch

from mlperf_training_b200.ops import _lib
from mlperf_training_b200.ops.hstu_ops import GateCatFn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [256, 512, 768])
@pytest.mark.parametrize("T,p", [(1, 0.0), (3, 0.3), (7, 0.0), (593, 0.2), (2369, 0.0), (4801, 0.5)])
def test_rows(T, D, p):
    torch.manual_seed(T + D)
    wide = torch.randn(T, 2 * D, device="cuda").bfloat16()
    attn, w, b, dcat = (torch.randn(*s, device="cuda").bfloat16() for s in ((T, D), (D,), (D,), (T, 3 * D)))
    leaves = [t.clone().requires_grad_(True) for t in (wide, attn, w, b)]
    cat = GateCatFn.apply(leaves[0][:, :D], *leaves[1:], 1e-6, p)
    cat.backward(dcat)
    _lib.check_status("gate_cat")
    ref = [t.detach().double().requires_grad_(True) for t in leaves]
    u = torch.nn.functional.silu(ref[0][:, :D])
    plain = torch.cat([u, ref[1], u * torch.nn.functional.layer_norm(ref[1], (D,), ref[2], ref[3], 1e-6)], 1)
    thr = round(p * 65536) / 65536
    keep = (cat != 0).double() / (1 - thr) if p else torch.ones_like(plain)
    want = torch.autograd.grad(plain * keep, ref, dcat.double())
    # bf16 roundings (2^-9 each) of u, of the normalised row and of the result
    for got, r in zip([cat] + [t.grad for t in leaves], [plain * keep] + list(want)):
        assert (got.double() - r).norm() <= 2 ** -7 * r.norm()
    if p:
        assert abs((cat != 0).double().mean() - (1 - thr)) <= 5 * (p * (1 - p) / cat.numel()) ** 0.5 + 1e-3
