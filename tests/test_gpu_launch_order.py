"""Kernels launched back to back see all of their predecessors' writes, eagerly and from a captured graph."""
import pytest
import torch

from mlperf_training_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,D", [(128, 512), (1337, 1024), (8192, 2048)])
def test_back_to_back_launches(T, D):
    """A chain in which each launch reads what the one before it wrote, over one input buffer that is rewritten between rounds: the
    values of the same chain with the device idle before every step, bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    w1, w2, nw, xs = rnd(2 * D, D) * D ** -0.5, rnd(D, D) * D ** -0.5, rnd(D), [rnd(T, D) for _ in range(3)]
    x = torch.empty_like(xs[0])

    def chain(sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        out = []
        with torch.no_grad():
            for src in xs:
                x.copy_(src)
                wait()
                y = x
                for _ in range(3):
                    y = F.rms_norm(y, nw)
                    wait()
                    y = F.linear(y, w1)
                    wait()
                    y = F.swiglu(y)
                    wait()
                    y = F.linear(y, w2)
                    wait()
                out.append(y)
        return out

    want = chain(True)
    for _ in range(5):
        for a, b in zip(chain(False), want):
            assert torch.equal(a, b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain(False)
    for _ in range(3):
        for o in out:
            o.zero_()
        graph.replay()
        for a, b in zip(out, want):
            assert torch.equal(a, b)
