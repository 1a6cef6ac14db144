"""Attention forward at the edges of its work schedule: odd tile counts, more and fewer items than CTAs, windows that skip
a pair's first key tile, more keys than queries, a second, smaller L2 group of heads."""
import pytest
import torch

from mlperf_training_b200.ops import _lib, kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,D,causal,window,sink", [
    (1, 1, 1, 1, 1, 128, True, 0, False), (1, 129, 129, 2, 1, 64, True, 1, True), (2, 257, 257, 4, 2, 128, True, 128, False),
    (1, 640, 640, 8, 8, 64, True, 200, True), (3, 384, 511, 4, 1, 128, True, 0, False), (2, 300, 1000, 6, 3, 64, False, 0, False),
    (5, 513, 513, 8, 2, 128, True, 0, True), (1, 200, 1500, 4, 4, 128, True, 100, False),
    (3, 130, 2048, 24, 24, 128, False, 0, False)])      # 64 + 8 heads: two L2 groups
def test_forward(B, Sq, Skv, Hq, Hkv, D, causal, window, sink):
    torch.manual_seed(Sq)
    q, k, v = (torch.randn(B, s, h, D, device="cuda").bfloat16() for s, h in ((Sq, Hq), (Skv, Hkv), (Skv, Hkv)))
    sk = torch.randn(Hq, device="cuda") if sink else None
    out, lse = K.attention_fwd(q, k, v, causal=causal, window=window, sink=sk)
    ref, ref_lse = K.attention_reference(q, k, v, scale=D ** -0.5, causal=causal, window=window, sink=sk)
    # bf16 probabilities and output: 2^-9 each per term, at most 2^-7 of the largest value
    assert (out.float() - ref).abs().max() <= 2 ** -7 * ref.abs().max()
    assert (lse - ref_lse).abs().max() <= 2e-3       # a quarter of the exponentials carry up to 7e-4
    _lib.check_status("attention_fwd")


@pytest.mark.parametrize("key", [0, 6, 7, 134, 255])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_non_finite_keys_are_not_lost(key, value):
    """A NaN or infinity in one key makes the rows that see it non-finite and leaves the others alone (keys 6 and 7 of 8 have
    their exponentials on the FMA pipe)."""
    torch.manual_seed(key)
    q, k, v = (torch.randn(1, 256, 2, 64, device="cuda").bfloat16() for _ in range(3))
    clean, _ = K.attention_fwd(q, k, v, causal=True)
    k[0, key, 1, 5] = value
    q[..., 5] = q[..., 5].abs() + 0.5
    clean2, _ = K.attention_fwd(q[:, :, :1], k[:, :, :1], v[:, :, :1], causal=True)
    out, _ = K.attention_fwd(q, k, v, causal=True)
    assert not out[0, key:, 1].isfinite().any() and out[0, :key].isfinite().all()
    assert torch.equal(out[:, :, :1], clean2) and clean.isfinite().all()
    _lib.check_status("attention_fwd")
