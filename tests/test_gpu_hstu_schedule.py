"""Jagged attention over its grid orders and head dims: few and many (sequence, head) pairs, sequences at the edges of a tile,
targets and contextual rows, more pairs than a grid axis holds."""
import pytest
import torch

from mlperf_training_b200.ops import _lib
from mlperf_training_b200.ops.hstu_ops import hstu_attention, valid_mask

pytestmark = pytest.mark.gpu


def _grads(q, k, v, lengths, do, max_len):
    offs = torch.cat([lengths.new_zeros(1), lengths.cumsum(0)]).to(torch.int32).cuda()
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = hstu_attention(*leaves, offs, max_len, 0.125)
    return [out.detach(), *torch.autograd.grad(out, leaves, do)]


def _oracle(q, k, v, lengths, max_len, alpha, nt, ctx):
    out, lo = [], 0
    for b, n in enumerate(lengths.tolist()):
        qb, kb, vb = (t[lo:lo + n].transpose(0, 1) for t in (q, k, v))
        p = torch.nn.functional.silu(qb @ kb.transpose(1, 2) * alpha) * valid_mask(n, int(nt[b]), ctx, q.device)
        out.append((p @ vb / max_len).transpose(0, 1))
        lo += n
    return torch.cat(out)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,ctx", [(7, 0), (7, 3), (110, 0), (110, 5)])
def test_grid_orders(B, ctx, D):
    """4 heads: 28 pairs (key tiles slowest) and 440 (pairs slowest, past two chips of CTAs)."""
    H, N, alpha = 4, 512, D ** -0.5
    g = torch.Generator().manual_seed(B + ctx + D)
    edges = torch.tensor([0, 1, 127, 128, 129, 257, 400, 3, 64])
    lengths = torch.cat([edges, edges[torch.randint(0, len(edges), (B,), generator=g)]])[:B].clamp(min=2 * ctx)
    nt = torch.minimum(torch.randint(0, 4, (B,), generator=g), lengths - ctx).to(torch.int32)
    L = int(lengths.sum())
    q, k, v, do = (torch.randn(L, H, D, generator=g).bfloat16().cuda() for _ in range(4))
    offs = torch.cat([lengths.new_zeros(1), lengths.cumsum(0)]).to(torch.int32).cuda()
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = hstu_attention(*leaves, offs, N, alpha, nt.cuda(), ctx)
    got = [out, *torch.autograd.grad(out, leaves, do)]
    _lib.check_status("hstu attention")
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    want = _oracle(*ref, lengths, N, alpha, nt, ctx)
    want = [want, *torch.autograd.grad(want, ref, do.double())]
    # bf16 P, dS and results (2^-9 each a term) and tanh to 2^-11; a row of one key is off by as much as its only term
    for a, b in zip(got, want):
        assert (a.double() - b).norm() <= 2 ** -7 * b.norm()
        assert (a.double() - b).abs().max() <= 2 ** -6 * b.abs().max()


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
