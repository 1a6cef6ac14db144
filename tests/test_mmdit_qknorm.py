"""The head norms of an MMDiT block stay modules: whatever a user hangs on them is called, and only a plain one is fused."""
import pytest
import torch
from torch.nn.modules import module as nnm

from mlperf_training_b200.models import mmdit
from mlperf_training_b200.ops import functional as F


class Sub(mmdit.QKNorm):
    def forward(self, q, k):
        calls.append("sub")
        return super().forward(q, k)


calls: list = []


def _touch(*_):
    calls.append("hook")


def _attach(norm, kind):
    """Returns what takes it off again."""
    if kind == "none":
        pass
    elif kind == "subclass":
        norm.__class__ = Sub
    elif kind == "replaced":
        norm.forward = lambda q, k: (_touch(), mmdit.QKNorm.forward(norm, q, k))[1]
    elif kind == "eps":
        norm.eps = 1.0
    elif kind == "global":
        return nnm.register_module_forward_hook(lambda m, *_: _touch() if m is norm else None).remove
    else:
        getattr(norm, {"forward": "register_forward_hook", "pre": "register_forward_pre_hook",
                       "backward": "register_full_backward_hook"}[kind])(_touch)
    return lambda: None


@pytest.mark.parametrize("block", ["double", "single"])
@pytest.mark.parametrize("kind", ["none", "forward", "pre", "backward", "subclass", "replaced", "global", "eps"])
def test_norm_modules_are_called(monkeypatch, block, kind):
    fused = []

    def stop(parts, cos, sin, B, H, D, eps=None):
        fused.append(eps)
        raise StopIteration

    monkeypatch.setattr(F, "qkv_norm_rope_ok", lambda *a: True)
    monkeypatch.setattr(F, "qkv_norm_rope", stop)
    monkeypatch.setattr(F, "single_stream_in", lambda y, qs, ks, cos, sin, B, H, D, eps=None: stop(None, cos, sin, B, H, D, eps))
    calls.clear()
    cfg = mmdit.tiny_mmdit()
    torch.manual_seed(0)
    m = mmdit.MMDiT(cfg)
    blk = (m.double_blocks if block == "double" else m.single_blocks)[0]
    undo = _attach(blk.img_qknorm if block == "double" else blk.qknorm, kind)
    B, S = 2, 8
    x, t = (torch.randn(B * S, cfg.hidden, requires_grad=True) for _ in range(2))
    vec = torch.randn(B, cfg.hidden)
    n = 2 * S if block == "double" else S
    ang = torch.rand(n, cfg.head_dim // 2)
    try:
        out = blk(x, t, vec, ang.cos(), ang.sin(), B) if block == "double" else blk(x, vec, ang.cos(), ang.sin(), B)
        sum(o.sum() for o in (out if isinstance(out, tuple) else (out,))).backward()
    except StopIteration:
        pass
    finally:
        undo()
    if kind == "none":
        assert fused == [1e-6]
    elif kind == "eps":
        # one value for a fused launch: streams of different eps are not fused, a single stream takes its module's
        assert fused == ([] if block == "double" else [1.0])
    else:
        assert calls and not fused
