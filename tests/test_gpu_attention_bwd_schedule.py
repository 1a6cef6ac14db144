"""Attention backward at the edges of its schedule: one step, odd step counts, ragged tiles, keys that no query sees, windows,
more keys than queries, grouped heads."""
import ctypes
import re
from pathlib import Path

import pytest
import torch

from mlperf_training_b200.ops import _lib, kernels as K

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,D,causal,window,sink", [
    (1, 1, 1, 1, 1, 128, True, 0, False), (1, 128, 128, 1, 1, 64, True, 0, False), (2, 129, 129, 3, 3, 128, True, 0, False),
    (1, 300, 300, 8, 2, 64, True, 50, True), (1, 500, 500, 4, 1, 128, False, 0, False), (1, 130, 700, 4, 2, 128, True, 0, False),
    (2, 200, 90, 2, 1, 64, False, 0, False), (1, 1000, 1000, 2, 2, 128, True, 128, False), (1, 383, 383, 6, 2, 64, True, 0, True),
    (1, 200, 1500, 4, 2, 128, True, 100, False), (2, 70, 900, 2, 1, 64, True, 1, False), (1, 130, 1300, 2, 2, 128, False, 300, True)])
def test_backward(B, Sq, Skv, Hq, Hkv, D, causal, window, sink):
    torch.manual_seed(Sq + D)
    q, k, v = (torch.randn(B, s, h, D, device="cuda").bfloat16() for s, h in ((Sq, Hq), (Skv, Hkv), (Skv, Hkv)))
    do = torch.randn(B, Sq, Hq, D, device="cuda").bfloat16()
    sk = torch.randn(Hq, device="cuda") if sink else None
    out, lse = K.attention_fwd(q, k, v, causal=causal, window=window, sink=sk)
    dq, dk, dv, ds = K.attention_bwd(do, q, k, v, out, lse, causal=causal, window=window, sink=sk)
    leaves = [t.double().requires_grad_(True) for t in ((q, k, v, sk) if sink else (q, k, v))]
    g = Hq // Hkv
    s = torch.einsum("bqhd,bkhd->bhqk", leaves[0], leaves[1].repeat_interleave(g, 2)) * D ** -0.5
    s = s.masked_fill(~K._attn_mask(Sq, Skv, causal, window, "cuda"), float("-inf"))
    if sink:
        s = torch.cat([s, leaves[3].view(1, Hq, 1, 1).expand(B, Hq, Sq, 1)], -1)
    p = torch.softmax(s, -1)[..., :Skv]
    want = torch.autograd.grad(torch.einsum("bhqk,bkhd->bqhd", p, leaves[2].repeat_interleave(g, 2)), leaves, do.double())
    # bf16 P and dS (2^-9 each per term) and delta from the rounded output.  dP - delta is the difference of two fp32 sums of D
    # products (a single visible key: exactly 0): D * 2^-24 of |dO| |v| <= 1e-5 of |dO| beside the relative part
    for a, b in zip((dq, dk, dv, ds) if sink else (dq, dk, dv), want):
        assert (a.double() - b).norm() <= 2 ** -7 * b.norm() + 1e-5 * do.double().norm()
    unseen = ~K._attn_mask(Sq, Skv, causal, window, "cuda").any(0)
    assert not dk[:, unseen].any() and not dv[:, unseen].any()
    _lib.check_status("attention_bwd")


@gpu
@pytest.mark.parametrize("Sq,D", [(128, 128), (320, 64)])
def test_equal_queries_have_equal_gradients(Sq, D):
    """Probabilities must not depend on where in its tile a query stands: equal rows of q and dO give bit-equal rows of dQ (one
    key tile, so every row is a single sum)."""
    torch.manual_seed(D)
    k, v = (torch.randn(1, 128, 2, D, device="cuda").bfloat16() for _ in range(2))
    q, do = (torch.randn(1, 1, 2, D, device="cuda").bfloat16().expand(1, Sq, 2, D).contiguous() for _ in range(2))
    out, lse = K.attention_fwd(q, k, v, causal=False)
    dq = K.attention_bwd(do, q, k, v, out, lse, causal=False)[0]
    assert dq.any() and torch.equal(dq, dq[:, :1].expand_as(dq))
    _lib.check_status("attention_bwd")


def test_copies_are_issued_only_where_they_are_awaited():
    """A key tile without queries (``n_iter == 0``) skips every wait of the kernel, so it may not start a copy either: read from
    the source, since a CTA that leaves with copies in flight corrupts its successor's shared memory."""
    text = (Path(__file__).resolve().parent.parent / "mlperf_training_b200/csrc/attention_bwd.cu").read_text()
    role = text[text.index("TMA producer -"):text.index("MMA issuer -")]
    assert role.index("n_iter > 0") < role.index("mbar_expect_tx(kv_full") and re.search(r"if \([^)]*n_iter > 0\) \{", role)


def test_scratch_of_cut_key_tiles_is_bounded():
    """The planner's scratch stays below four times the bf16 dK and dV, or 32 MB, over sizes, groups, head dims and masks; the
    sizes whose times are known keep their cut."""
    out = (ctypes.c_longlong * 2)()
    plan = _lib.load().b200_attn_bwd_plan
    cut = 0
    for S in (200, 777, 2000, 4096, 7168, 9000):
        for Hq, Hkv in ((2, 2), (16, 2), (64, 8), (256, 16), (32, 1)):
            for D in (64, 128):
                for B, causal, window in ((1, 1, 0), (1, 0, 0), (3, 0, 0), (1, 1, 300)):
                    plan(B, S, S, Hq, Hkv, D, causal, window, out)
                    assert out[1] <= max(32 << 20, 4 * 2 * B * S * Hkv * D * 2), (S, Hq, Hkv, D, B, causal, window, out[1])
                    assert (out[0] > 0) == (out[1] > 0)
                    cut += out[0] > 0
    assert cut > 20
    for shape in ((1, 2000, 2000, 64, 8, 64, 1, 0), (1, 3000, 3000, 64, 8, 128, 1, 0), (1, 1024, 1024, 32, 8, 128, 1, 0)):
        plan(*shape, out)
        assert 0 < out[0] and out[1] < 26 << 20
