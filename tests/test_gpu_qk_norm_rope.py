"""Fused split + head norm + rotary + concatenation, and the single-stream entry, against fp64: both head dims, ragged token
counts, one and two streams, a projection with a wider pitch."""
import pytest
import torch

from mlperf_training_b200.ops import functional as F

gpu = pytest.mark.gpu


def _oracle(parts, cos, sin, B, H, D):
    out = [[], [], []]
    for x, qs, ks in parts:
        q, k, v = x.reshape(B, -1, 3, H, D).unbind(2)
        rms = lambda t, w: t * torch.rsqrt((t * t).mean(-1, keepdim=True) + 1e-6) * w
        for o, t in zip(out, (rms(q, qs), rms(k, ks), v)):
            o.append(t)
    q, k, v = (torch.cat(o, 1) for o in out)
    c, s = cos[:q.shape[1], None], sin[:q.shape[1], None]
    rot = lambda t: torch.cat([t[..., :D // 2] * c - t[..., D // 2:] * s, t[..., D // 2:] * c + t[..., :D // 2] * s], -1)
    return rot(q), rot(k), v


def _close(a, b):
    # one rounding to bf16 of fp32 arithmetic (the scale gradients: fp32 sums, then one rounding)
    assert (a.double() - b).abs().max() <= 2 ** -8 * b.abs().max() + 1e-6
    assert (a.double() - b).norm() <= 2 ** -8 * b.norm()


@gpu
@pytest.mark.parametrize("B,sizes,H,D", [(1, [1], 1, 64), (2, [5, 3], 3, 128), (3, [37], 5, 64), (2, [256, 256], 24, 128)])
def test_streams(B, sizes, H, D):
    torch.manual_seed(sum(sizes))
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16().requires_grad_(True)
    S = sum(sizes)
    ang = torch.rand(S, D // 2, device="cuda") * 6
    cos, sin = ang.cos(), ang.sin()
    parts = [(mk(B * n, 3 * H * D), mk(D), mk(D)) for n in sizes]
    assert F.qkv_norm_rope_ok(cos, D, parts)
    got = F.qkv_norm_rope(parts, cos, sin, B, H, D)
    ref = [tuple(t.detach().double().requires_grad_(True) for t in p) for p in parts]
    want = _oracle(ref, cos.double(), sin.double(), B, H, D)
    gr = [torch.randn(B, S, H, D, device="cuda").bfloat16() for _ in range(3)]
    torch.autograd.backward(got, gr)
    torch.autograd.backward(want, [g.double() for g in gr])
    for a, b in zip(got, want):
        _close(a, b)
    for p, r in zip(parts, ref):
        for a, b in zip(p, r):
            _close(a.grad, b.grad)


@gpu
@pytest.mark.parametrize("B,S,H,D,m", [(2, 19, 2, 64, 72), (1, 130, 3, 128, 512)])
def test_single_stream(B, S, H, D, m):
    torch.manual_seed(S)
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16().requires_grad_(True)
    n = 3 * H * D
    ang = torch.rand(S, D // 2, device="cuda") * 6
    cos, sin = ang.cos(), ang.sin()
    y, qs, ks = mk(B * S, n + m), mk(D), mk(D)
    got = F.single_stream_in(y, qs, ks, cos, sin, B, H, D)
    ref = [t.detach().double().requires_grad_(True) for t in (y, qs, ks)]
    want = (*_oracle([(ref[0][:, :n], ref[1], ref[2])], cos.double(), sin.double(), B, H, D),
            torch.nn.functional.gelu(ref[0][:, n:], approximate="tanh"))
    wide = torch.randn(B * S, H * D + m, device="cuda").bfloat16()
    gr = [torch.randn(B, S, H, D, device="cuda").bfloat16() for _ in range(3)] + [wide[:, H * D:]]     # a pitched gradient
    torch.autograd.backward(got, gr)
    torch.autograd.backward(want, [g.double() for g in gr])
    for a, b in zip([*got, y.grad, qs.grad, ks.grad], [*want, *(r.grad for r in ref)]):
        _close(a, b)


@pytest.mark.parametrize("bad", ["narrow", "wide", "rows", "scale", "pitched_scale", "short_table", "table_width", "sin", "sin_dtype", "samples"])
@pytest.mark.parametrize("single", [False, True])
def test_sizes_that_do_not_fit_are_refused(monkeypatch, bad, single):
    """What the reshapes of the separate chain refused is refused before anything is launched."""
    monkeypatch.setattr(F, "call", lambda *a: pytest.fail("launched"))
    B, S, H, D = 2, 6, 3, 64
    extra = 64 if single else 0
    n = 3 * H * D + extra
    x = torch.zeros(B * S + (bad == "rows"), {"narrow": 3 * H * D - 8, "wide": n + (4 if single else 64)}.get(bad, n)).bfloat16()
    qs = ks = torch.ones(D).bfloat16()
    if bad == "scale":
        ks = torch.ones(2 * D).bfloat16()
    if bad == "pitched_scale":
        qs = torch.ones(2 * D).bfloat16()[::2]
    cos = torch.ones(S - (bad == "short_table"), D if bad == "table_width" else D // 2)
    sin = torch.ones(S + 1, D // 2) if bad == "sin" else cos.double() if bad == "sin_dtype" else cos
    B = 0 if bad == "samples" else B
    with pytest.raises(ValueError):
        F.single_stream_in(x, qs, ks, cos, sin, B, H, D) if single else F.qkv_norm_rope([(x, qs, ks)], cos, sin, B, H, D)
