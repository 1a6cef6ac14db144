"""Jagged attention beyond a few sequences: more (sequence, head) pairs than a grid axis holds."""
import pytest
import torch

from mlperf_training_b200.ops import _lib
from mlperf_training_b200.ops.hstu_ops import hstu_attention

pytestmark = pytest.mark.gpu


def _grads(q, k, v, lengths, do, max_len):
    offs = torch.cat([lengths.new_zeros(1), lengths.cumsum(0)]).to(torch.int32).cuda()
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = hstu_attention(*leaves, offs, max_len, 0.125)
    return [out.detach(), *torch.autograd.grad(out, leaves, do)]


def test_more_pairs_than_a_grid_axis():
    """16,400 sequences of 4 heads are 65,600 pairs: the same bits as the two halves of the batch by themselves."""
    B, H, D, N = 16400, 4, 64, 64
    g = torch.Generator().manual_seed(0)
    lengths = torch.randint(0, 4, (B,), generator=g)
    L = int(lengths.sum())
    q, k, v, do = (torch.randn(L, H, D, generator=g).bfloat16().cuda() for _ in range(4))
    whole = _grads(q, k, v, lengths, do, N)
    _lib.check_status("hstu attention")
    half = int(lengths[:B // 2].sum())
    for part, sel in ((slice(0, half), lengths[:B // 2]), (slice(half, L), lengths[B // 2:])):
        for a, b in zip(whole, _grads(q[part], k[part], v[part], sel, do[part], N)):
            assert b.any() and torch.equal(a[part], b)
