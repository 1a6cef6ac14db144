"""One-rank lookup without a host read: the same rows, table and optimizer sums as through an explicit plan; skewed ids (runs
far longer than a block of partial sums), ids outside the table, one id, no id."""
import pytest
import torch

from mlperf_training_b200.parallel import embedding
from mlperf_training_b200.parallel.embedding import ColumnShardedEmbedding, ShardedEmbedding

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["zipf", "single", "outside", "one", "none"])
def test_lookup_and_update(kind):
    rows, dim = 5000, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    n = {"one": 1, "none": 0}.get(kind, 20000)
    ids = (torch.rand(n, generator=g, device="cuda") ** 6 * rows).long().clamp(0, rows - 1)
    if kind == "single":
        ids[:] = 17
    if kind == "outside":
        ids[::7] = rows + 5
    dy = torch.randn(n, dim, generator=g, device="cuda").bfloat16()
    tabs = [ShardedEmbedding(rows, dim, device="cuda", seed=1) for _ in range(2)]
    outs = []
    for t, plan in zip(tabs, (None, tabs[1].input_dist(ids) if n else None)):
        o = t.lookup(ids, plan)
        o.backward(dy)
        outs.append(o)
    torch.cuda.synchronize()
    if n:
        ok = ids < rows
        fresh = ShardedEmbedding(rows, dim, device="cuda", seed=1).weight
        assert torch.equal(outs[0][ok], fresh[ids[ok]]) and not outs[0][~ok].any()
        uniq, inv = torch.unique(ids[ok], return_inverse=True)
        gsum = torch.zeros(len(uniq), dim, dtype=torch.float64, device="cuda").index_add_(0, inv, dy[ok].double())
        # fp32 sums of up to n terms
        torch.testing.assert_close(tabs[0].state[uniq].double(), (gsum * gsum).mean(-1), rtol=1e-4, atol=1e-6)
    assert torch.equal(outs[0], outs[1]) and torch.equal(tabs[0].weight, tabs[1].weight) and torch.equal(tabs[0].state, tabs[1].state)


@pytest.mark.parametrize("cls", [ShardedEmbedding, ColumnShardedEmbedding])
def test_repeated_ids_hold_no_row_per_position(cls, monkeypatch):
    """200,000 ids of 50 rows: the memory of a block of summed rows, not of one per id."""
    monkeypatch.setattr(embedding, "SUM_BLOCK_BYTES", 16 << 20)
    n, dim = 200_000, 256
    ids = torch.arange(n, device="cuda") % 50
    dy = torch.randn(n, dim, device="cuda").bfloat16()
    tabs = [cls(5000, dim, device="cuda", seed=1) for _ in range(2)]
    for t, plan in zip(tabs, (None, tabs[1].input_dist(ids))):
        o = t.lookup(ids, plan)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        base = torch.cuda.memory_allocated()
        o.backward(dy)
        torch.cuda.synchronize()
        # partial sums of long runs (two fp32 rows per 64 positions), a block of sums
        assert torch.cuda.max_memory_allocated() - base <= (2 * n // 64 + 2) * dim * 4 + (18 << 20)
    assert torch.equal(tabs[0].weight, tabs[1].weight) and torch.equal(tabs[0].state, tabs[1].state)


@pytest.mark.parametrize("rows_a_block", [1, 7, 999, 1000, 1001])
def test_blocks_of_rows(monkeypatch, rows_a_block):
    """The update in blocks: last block full, of one row, past the runs; long runs on either side of a block's edge."""
    dim, n = 64, 9000
    g = torch.Generator(device="cuda").manual_seed(2)
    ids = torch.cat([torch.arange(1000, device="cuda"), (torch.rand(n - 1000, generator=g, device="cuda") ** 4 * 1000).long()])
    if rows_a_block == 1:
        ids = ids % 40
    dy = torch.randn(n, dim, generator=g, device="cuda").bfloat16()
    tabs = [ShardedEmbedding(1000, dim, device="cuda", seed=1) for _ in range(2)]
    tabs[0].lookup(ids).backward(dy)
    monkeypatch.setattr(embedding, "SUM_BLOCK_BYTES", rows_a_block * dim * 4)
    tabs[1].lookup(ids, tabs[1].input_dist(ids) if rows_a_block == 1 else None).backward(dy)
    assert torch.equal(tabs[0].weight, tabs[1].weight) and torch.equal(tabs[0].state, tabs[1].state)


@pytest.mark.parametrize("n", [3000, 150_000])
def test_captured_step(n):
    """Forward and backward in a graph: nothing of a one-rank lookup waits for the host."""
    dim = 128
    ids = (torch.rand(n, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") * 900).long()
    dy = torch.randn(n, dim, device="cuda").bfloat16()
    tabs = [ShardedEmbedding(1000, dim, device="cuda", seed=1) for _ in range(2)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ShardedEmbedding(1000, dim, device="cuda", seed=1).lookup(ids).backward(dy)
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tabs[0].lookup(ids).backward(dy)
    for _ in range(2):
        graph.replay()
        tabs[1].lookup(ids).backward(dy)
    torch.cuda.synchronize()
    assert torch.equal(tabs[0].weight, tabs[1].weight) and torch.equal(tabs[0].state, tabs[1].state)
    del graph
