"""One-rank lookup without a host read: the same rows, table and optimizer sums as through an explicit plan; skewed ids (runs
far longer than a block of partial sums), ids outside the table, one id, no id."""
import pytest
import torch

from mlperf_training_b200.parallel.embedding import ShardedEmbedding

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
