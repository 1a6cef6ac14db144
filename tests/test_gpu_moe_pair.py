"""Expert MLP on the CTA-pair grouped kernels: experts without tokens, one token, ragged widths (partly filled tiles and
contraction stages), gradients as new tensors and into ``main_grad``."""
import pytest
import torch

from mlperf_training_b200.ops import _lib, moe_ops as M

pytestmark = pytest.mark.gpu


def _reference(x, idx, w, w1, w2):
    out = torch.zeros_like(x)
    for e in range(w1.shape[0]):
        t, s = torch.nonzero(idx == e, as_tuple=True)
        g, u = (x[t] @ w1[e].t()).chunk(2, 1)
        out = out.index_add(0, t, (torch.nn.functional.silu(g) * u) @ w2[e].t() * w[t, s][:, None])
    return out


@pytest.mark.parametrize("T,E,k,D,F,precision", [(1, 4, 1, 64, 64, "bf16"), (300, 8, 2, 320, 448, "bf16"), (700, 5, 4, 576, 192, "bf16"),
                                                 (515, 6, 2, 384, 384, "mxfp8")])
@pytest.mark.parametrize("main_grad", [False, True])
def test_expert_mlp(T, E, k, D, F, precision, main_grad):
    g = torch.Generator().manual_seed(T)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g) * std).bfloat16().cuda()
    x, w1, w2, dy = mk(T, D), mk(E, 2 * F, D, std=D ** -0.5), mk(E, D, F, std=F ** -0.5), mk(T, D)
    logits = torch.randn(T, E, generator=g).cuda()
    logits[:, E - 2] = -9.0                               # an expert nobody picks (unless k = E)
    wts, idx = torch.topk(logits, k)
    wts = torch.softmax(wts, -1)
    counts = torch.bincount(idx.reshape(-1), minlength=E).to(torch.int32)
    leaves = [t.clone().requires_grad_(True) for t in (x, w1, w2)]
    if main_grad:
        for p in leaves[1:]:
            p.main_grad = torch.ones(p.shape, device="cuda")
    assert M.pair_rows_ok(x, w1, w2)
    y = M.moe_experts(leaves[0], idx.to(torch.int32), wts, counts, leaves[1], leaves[2], precision)
    y.backward(dy)
    ref = [t.double().requires_grad_(True) for t in (x, w1, w2)]
    want = _reference(ref[0], idx, wts.double(), ref[1], ref[2])
    want.backward(dy.double())
    # bf16: a handful of roundings of 2^-9 each; block-scaled e4m3: 4 mantissa bits on either operand of three GEMMs
    tol = 0.02 if precision == "bf16" else 0.12
    got = [y, leaves[0].grad] + [(p.main_grad - 1 if main_grad else p.grad) for p in leaves[1:]]
    for a, b in zip(got, [want, ref[0].grad, ref[1].grad, ref[2].grad]):
        assert (a.double() - b).norm() <= tol * b.norm()
    empty = [e for e in range(E) if counts[e] == 0]
    for e in empty:
        for a in got[2:]:
            assert not a[e].any()
    _lib.check_status("grouped pair")
