"""Bounded-key radix sort, run bookkeeping and the deterministic segment reduction against the CPU path."""
import pytest
import torch

from mlperf_training_b200.ops import _lib, sort
from mlperf_training_b200.parallel.embedding import ShardedEmbedding

gpu = pytest.mark.gpu


@gpu
@pytest.mark.parametrize("n,rows", [(1, 10), (1000, 50), (200_003, 400_000_000), (65_536, 3)])
def test_sort_unique_and_segment_sum(n, rows):
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(0, rows, (n,), generator=g)
    src = torch.randn(n, 64, generator=g).bfloat16()
    c = sort.sort_unique(ids, sort.key_bits_for(rows))
    d = sort.sort_unique(ids.cuda(), sort.key_bits_for(rows))
    torch.cuda.synchronize()
    _lib.check_status("sort")
    cnt = int(c.count)
    assert int(d.count.item()) == cnt
    assert torch.equal(d.keys.cpu(), c.keys) and torch.equal(d.perm.cpu(), c.perm)          # stable: same permutation
    assert torch.equal(d.uniq[:cnt].cpu(), c.uniq[:cnt]) and torch.equal(d.seg[:cnt + 1].cpu(), c.seg[:cnt + 1])
    assert torch.equal(d.inverse.cpu(), c.inverse) and bool((d.uniq[cnt:] == -1).all())
    for out_dtype in (torch.float32, torch.bfloat16):
        a = sort.segment_sum(src, c, out_dtype)[:cnt].float()
        b = sort.segment_sum(src.cuda(), d, out_dtype)[:cnt].float().cpu()
        assert (a - b).abs().max() <= 1e-2 * max(a.abs().max().item(), 1.0)
    b2 = sort.segment_sum(src.cuda(), d, torch.float32)
    assert torch.equal(b2, sort.segment_sum(src.cuda(), d, torch.float32))                  # run twice: bit-identical


@gpu
def test_segment_sum_long_runs():
    """Skewed ids: runs longer than one warp's share (summed through per-block partial sums), runs that start in the
    middle of a block, a run of exactly the block size, next to ordinary short runs."""
    g = torch.Generator().manual_seed(5)
    ids = torch.cat([torch.full((1000,), 7), torch.full((65,), 3), torch.full((64,), 11), torch.full((129,), 2),
                     torch.randint(100, 5000, (3000,), generator=g), torch.full((300,), 99)])
    ids = ids[torch.randperm(ids.numel(), generator=g)]
    for D, dt in ((256, torch.bfloat16), (72, torch.float32)):
        src = torch.randn(ids.numel(), D, generator=g).to(dt)
        c = sort.sort_unique(ids, 13)
        d = sort.sort_unique(ids.cuda(), 13)
        cnt = int(c.count)
        a = sort.segment_sum(src, c, torch.float32)[:cnt]
        b = sort.segment_sum(src.cuda(), d, torch.float32)
        torch.cuda.synchronize()
        _lib.check_status("segment sum long runs")
        assert (a - b[:cnt].cpu()).abs().max() <= 2e-4 * max(a.abs().max().item(), 1.0)
        assert torch.equal(b, sort.segment_sum(src.cuda(), d, torch.float32))               # bit-identical when repeated


@gpu
def test_embedding_backward_is_deterministic_and_matches_cpu():
    torch.manual_seed(0)
    ids = torch.randint(0, 500, (4000,))
    upstream = torch.randn(4000, 64)
    res = []
    for dev in ("cpu", "cuda", "cuda"):
        t = ShardedEmbedding(500, 64, device=dev, dtype=torch.float32, lr=0.1, seed=3)
        w0 = t.weight.clone()
        out = t.lookup(ids.to(dev))
        (out * upstream.to(dev)).sum().backward()
        res.append((t.weight - w0).cpu())
    torch.cuda.synchronize()
    assert torch.equal(res[1], res[2])
    assert (res[0] - res[1]).abs().max() < 1e-5


def test_sorts_in_flight_share_no_scratch(monkeypatch):
    """Two sorts that are in flight together (here: the second one starts inside the first one's launch) work in buffers of
    their own."""
    seen = []

    class Lib:
        @staticmethod
        def b200_sort_scratch_bytes(n):
            return 16 * n + 256

    def call(name, *args):
        seen.append((name, args[6] if name == "b200_unique_segments" else args[5]))
        if len(seen) == 1:
            sort.sort_unique(torch.arange(50))

    monkeypatch.setattr(sort, "use_kernels", lambda t: True)
    monkeypatch.setattr(sort, "load", lambda: Lib)
    monkeypatch.setattr(sort, "call", call)
    monkeypatch.setattr(sort, "stream_ptr", lambda: 0)
    sort.sort_unique(torch.arange(100))
    outer, inner = {seen[0][1]}, {p for _, p in seen[1:3]}
    assert len(seen) == 4 and not outer & inner


@gpu
def test_sorts_on_two_streams():
    """Sorts issued on two streams without a host read between them: each gives what it gives alone."""
    g = torch.Generator(device="cuda").manual_seed(0)
    ids = [torch.randint(0, 50_000, (300_000,), generator=g, device="cuda") for _ in range(8)]
    want = [sort.sort_unique(i, 16) for i in ids]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = [None] * len(ids)
    for i, t in enumerate(ids):
        with torch.cuda.stream(streams[i % 2]):
            got[i] = sort.sort_unique(t, 16)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        n = int(b.count)
        assert int(a.count) == n and torch.equal(a.keys, b.keys) and torch.equal(a.perm, b.perm)
        assert torch.equal(a.inverse, b.inverse) and torch.equal(a.seg[:n + 1], b.seg[:n + 1]) and torch.equal(a.uniq[:n], b.uniq[:n])
    _lib.check_status("sort")


@gpu
@pytest.mark.parametrize("entries", ["perm", "inverse"])
def test_entries_outside_their_range_are_skipped(entries):
    """Positions of the permutation outside the source (at the ends of blocks, where the partial sums look their runs up) are
    left out of the sums; a run index outside the runs is found by search instead."""
    ids = torch.cat([torch.full((200,), 3), torch.arange(10, 80), torch.full((100,), 5)])
    src = torch.randn(ids.numel(), 64, generator=torch.Generator().manual_seed(1)).bfloat16()
    d = sort.sort_unique(ids.cuda(), 7)
    want = d.perm.cpu().clone()
    at = torch.tensor([0, 63, 64, 127, 300, 369])
    if entries == "perm":
        want[at] = torch.tensor([-1, 370, 1 << 40, -(1 << 40), 371, 5000])
        d.perm.copy_(want)
    else:
        d.inverse[d.perm[at.cuda()]] = torch.tensor([-1, 72, 1 << 40, -(1 << 40), 1000, 73], device="cuda")
    out = sort.segment_sum(src.cuda(), d).cpu()
    keys, ok = d.keys.cpu(), (want >= 0) & (want < ids.numel())
    for j, key in enumerate(d.uniq[:int(d.count)].tolist()):
        rows = src[want[ok & (keys == key)]].double()
        # fp32 sums of up to 200 terms
        assert (out[j].double() - rows.sum(0)).abs().max() <= 200 * 2 ** -24 * max(rows.abs().sum(0).max().item() if len(rows) else 0, 1e-9)
