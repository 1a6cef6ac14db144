"""tcgen05 flash attention forward / backward against eager fp32 softmax attention."""
import math

import pytest
import torch

from mlperf_training_b200.ops import _lib, kernels

pytestmark = pytest.mark.gpu

CASES = [
    # B, Sq, Skv, Hq, Hkv, D, causal, window, sink
    (1, 128, 128, 1, 1, 128, True, 0, False),
    (2, 256, 256, 4, 2, 128, True, 0, False),
    (1, 384, 384, 2, 1, 64, True, 0, False),
    (2, 200, 200, 2, 2, 128, True, 0, False),
    (1, 512, 512, 4, 1, 64, True, 128, True),
    (1, 640, 640, 2, 1, 128, True, 128, False),
    (2, 512, 512, 3, 3, 128, False, 0, False),
    (1, 1024, 1024, 8, 2, 128, True, 0, True),
]


def _mk(B, Sq, Skv, Hq, Hkv, D, seed):
    torch.manual_seed(seed)
    q = torch.randn(B, Sq, Hq, D, device="cuda").bfloat16()
    k = torch.randn(B, Skv, Hkv, D, device="cuda").bfloat16()
    v = torch.randn(B, Skv, Hkv, D, device="cuda").bfloat16()
    return q, k, v


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,D,causal,window,sink", CASES)
def test_attention_fwd(B, Sq, Skv, Hq, Hkv, D, causal, window, sink):
    q, k, v = _mk(B, Sq, Skv, Hq, Hkv, D, Sq + D)
    sk = torch.randn(Hq, device="cuda") if sink else None
    scale = 1 / math.sqrt(D)
    o, lse = kernels.attention_fwd(q, k, v, scale=scale, causal=causal, window=window, sink=sk)
    torch.cuda.synchronize()
    _lib.check_status("attn fwd")
    o_ref, lse_ref = kernels.attention_reference(q, k, v, scale=scale, causal=causal, window=window, sink=sk)
    err = (o.float() - o_ref).abs().max().item()
    assert err < 2e-2, f"out err {err}"
    assert (lse - lse_ref).abs().max().item() < 2e-2


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,D,causal,window,sink", CASES)
def test_attention_bwd(B, Sq, Skv, Hq, Hkv, D, causal, window, sink):
    q, k, v = _mk(B, Sq, Skv, Hq, Hkv, D, Sq + D + 1)
    sk = torch.randn(Hq, device="cuda") if sink else None
    scale = 1 / math.sqrt(D)
    do = torch.randn(B, Sq, Hq, D, device="cuda").bfloat16()
    o, lse = kernels.attention_fwd(q, k, v, scale=scale, causal=causal, window=window, sink=sk)
    dq, dk, dv, dsink = kernels.attention_bwd(do, q, k, v, o, lse, scale=scale, causal=causal, window=window, sink=sk)
    torch.cuda.synchronize()
    _lib.check_status("attn bwd")
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    sf = None if sk is None else sk.clone().requires_grad_(True)
    o_ref, _ = kernels.attention_reference(qf, kf, vf, scale=scale, causal=causal, window=window, sink=sf)
    o_ref.backward(do.float())
    for name, got, ref in (("dq", dq, qf.grad), ("dk", dk, kf.grad), ("dv", dv, vf.grad)):
        err = (got.float() - ref).abs().max().item()
        sc = ref.abs().max().item()
        assert err < 3e-2 * max(sc, 1.0), f"{name}: err {err} scale {sc}"
    if sink:
        assert (dsink - sf.grad).abs().max().item() < 3e-2 * max(sf.grad.abs().max().item(), 1.0)


def test_attention_packed_qkv_views():
    """q/k/v as views into one [B*S, (Hq+2Hkv)*D] buffer, the layout the GPT block uses."""
    torch.manual_seed(9)
    B, S, Hq, Hkv, D = 2, 256, 4, 2, 128
    row = (Hq + 2 * Hkv) * D
    qkv = torch.randn(B * S, row, device="cuda").bfloat16()
    v4 = qkv.view(B, S, row)
    q = v4[:, :, :Hq * D].unflatten(-1, (Hq, D))
    k = v4[:, :, Hq * D:(Hq + Hkv) * D].unflatten(-1, (Hkv, D))
    v = v4[:, :, (Hq + Hkv) * D:].unflatten(-1, (Hkv, D))
    o, lse = kernels.attention_fwd(q, k, v, causal=True)
    torch.cuda.synchronize()
    o_ref, _ = kernels.attention_reference(q, k, v, scale=1 / math.sqrt(D), causal=True)
    assert (o.float() - o_ref).abs().max().item() < 2e-2
    _lib.check_status("attn packed")


@pytest.mark.parametrize("B,S,Hq,Hkv,D,causal,window", [(1, 530, 16, 2, 64, True, 0), (2, 700, 8, 1, 128, True, 0), (1, 1000, 16, 4, 64, False, 0),
                                                        (1, 900, 16, 2, 128, True, 200), (1, 1500, 32, 8, 128, True, 0)])
def test_attention_bwd_with_shared_key_tiles(monkeypatch, B, S, Hq, Hkv, D, causal, window):
    """Key tiles whose steps several CTAs share (few tiles on many SMs) against one CTA per tile: the same products in another
    order of fp32 additions."""
    q, k, v = _mk(B, S, S, Hq, Hkv, D, S)
    do = torch.randn(B, S, Hq, D, device="cuda").bfloat16()
    o, lse = kernels.attention_fwd(q, k, v, causal=causal, window=window)
    assert _lib.attn_bwd_plan((B, S, S, Hq, Hkv, D, int(causal), window), q.device)[0] > 0
    shared = kernels.attention_bwd(do, q, k, v, o, lse, causal=causal, window=window)
    monkeypatch.setattr(_lib, "attn_bwd_plan", lambda *a: (0, None))
    alone = kernels.attention_bwd(do, q, k, v, o, lse, causal=causal, window=window)
    _lib.check_status("attn bwd shared")
    for a, b in zip(shared[:3], alone[:3]):
        a, b = a.float(), b.float()
        # fp32 sums of at most 16 terms of 128 products each in another order, then one rounding to bf16 (dK, dV)
        assert ((a - b).abs() <= b.abs() * 2 ** -7 + 2 ** -15 * b.abs().max()).all()
