"""Forwards without a gradient run past autograd's node, but not where a transform or a trace needs it."""
import pytest
import torch
from torch.autograd import forward_ad

from mlperf_training_b200.ops import functional as F

OPS = {"swiglu": F.swiglu, "gelu": F.gelu, "rms_norm": lambda x: F.rms_norm(x, torch.ones(16)),
       "linear": lambda x: F.linear(x, torch.ones(8, 16)), "norm_linear": lambda x: F.norm_linear(x, torch.ones(16), torch.ones(8, 16))}


@pytest.mark.parametrize("name", OPS)
def test_trace_records_the_operator(name):
    x, y = torch.randn(4, 16), torch.randn(4, 16)
    with torch.no_grad():
        traced = torch.jit.trace(OPS[name], (x,))
        assert any(n.kind() == "prim::PythonOp" for n in traced.graph.nodes())
        assert torch.equal(traced(y), OPS[name](y))


@pytest.mark.parametrize("name", OPS)
def test_transforms_meet_the_node(name):
    """An operator without a rule for them says so; it does not drop the tangent or run over a batch's wrapper."""
    x = torch.randn(4, 16)
    with torch.no_grad():
        with pytest.raises(RuntimeError):
            torch.func.vmap(OPS[name])(torch.randn(2, 4, 16))
        with forward_ad.dual_level():
            with pytest.raises(NotImplementedError):
                OPS[name](forward_ad.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("name", OPS)
def test_without_a_node_the_values_are_the_same(name):
    x = torch.randn(4, 16, requires_grad=True)
    want = OPS[name](x)
    with torch.no_grad():
        got = OPS[name](x)
    assert want.requires_grad and not got.requires_grad and torch.equal(got, want)
