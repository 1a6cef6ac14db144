"""MoE kernels (router top-k, device-side plan, permutation, grouped tcgen05 GEMMs) against the
eager CPU bodies of the same operators."""
import pytest
import torch

from mlperf_training_b200.models.gpt import GPT, GPTConfig
from mlperf_training_b200.ops import _lib, moe_ops as M
from tests._tol import assert_tiles_close

pytestmark = pytest.mark.gpu


def test_router_and_plan_match_cpu():
    torch.manual_seed(0)
    T, E, k = 1000, 32, 4
    logits = torch.randn(T, E)
    idx_c, w_c, cnt_c = M.router_topk(logits, k)
    idx_g, w_g, cnt_g = M.router_topk(logits.cuda(), k)
    assert torch.equal(idx_g.cpu().sort(-1).values, idx_c.sort(-1).values)
    assert torch.equal(cnt_g.cpu(), cnt_c)
    assert torch.allclose(w_g.cpu().sort(-1).values, w_c.sort(-1).values, atol=1e-5)
    seg_c, te_c, dest_c, rows_c = M.plan(idx_g.cpu(), cnt_c, E)
    seg_g, te_g, dest_g, rows_g = M.plan(idx_g, cnt_g, E)
    assert rows_c == rows_g and torch.equal(seg_g.cpu(), seg_c) and torch.equal(te_g.cpu(), te_c)
    assert torch.equal(dest_g.cpu(), dest_c)
    x = torch.randn(T, 256).bfloat16()
    xp_c = M.permute_rows(x, dest_c, k, rows_c)
    xp_g = M.permute_rows(x.cuda(), dest_g, k, rows_g)
    assert torch.equal(xp_g.cpu(), xp_c)
    y_c = M.unpermute_sum(xp_c, dest_c, w_c, T, k)
    y_g = M.unpermute_sum(xp_g, dest_g, w_g, T, k)
    assert (y_g.float().cpu() - y_c.float()).abs().max() < 2e-2
    _lib.check_status("router")


@pytest.mark.parametrize("T,E,k,pad", [(1, 4, 1, 128), (300, 32, 4, 256), (128, 8, 1, 128)])
def test_permutation_clears_the_gaps_only_and_adds_the_residual(T, E, k, pad):
    """Buffers whose gap rows the kernels clear themselves (experts without rows among them) equal cleared ones."""
    torch.manual_seed(T)
    logits = torch.randn(T, E)
    logits[:, 0] = -50.0
    idx, w, cnt = M.router_topk(logits.cuda(), k)
    seg, te, dest, rows = M.plan(idx, cnt, E, pad=pad)
    x, res = torch.randn(T, 64, device="cuda").bfloat16(), torch.randn(T, 64, device="cuda").bfloat16()
    live = int(seg[-1])
    stale = torch.full((rows, 64), float("nan"), device="cuda", dtype=torch.bfloat16)
    del stale                                            # (what the allocator hands out next)
    xp = M.permute_rows(x, dest, k, rows, (seg, cnt))
    assert torch.equal(xp[:live], M.permute_rows(x, dest, k, rows)[:live])
    grads = []
    for gaps in ((), (seg, cnt)):
        yp, r, ww = xp.clone().requires_grad_(True), res.clone().requires_grad_(True), w.clone().requires_grad_(True)
        y = M.UnpermuteFn.apply(yp, dest, ww, T, k, r, *gaps)
        y.backward(x)
        grads.append((y.detach(), yp.grad[:live], r.grad, ww.grad))
    assert all(torch.equal(a, b) for a, b in zip(*grads)) and torch.equal(grads[0][2], x)
    ref = M.unpermute_sum(xp.cpu(), dest.cpu(), w.cpu(), T, k, res.cpu()).float()
    assert ((grads[0][0].float().cpu() - ref).abs() <= ref.abs() * 2 ** -7 + 1e-5).all()      # a flip of the one rounding
    _lib.check_status("gaps")


@pytest.mark.parametrize("T,E,k,D,Fh", [(512, 8, 2, 256, 512), (2048, 32, 4, 384, 320)])
def test_grouped_gemms(T, E, k, D, Fh):
    torch.manual_seed(1)
    logits = torch.randn(T, E)
    idx, w, cnt = M.router_topk(logits.cuda(), k)
    seg, te, dest, rows = M.plan(idx, cnt, E)
    x = (torch.randn(T, D) * 0.5).bfloat16().cuda()
    w1 = (torch.randn(E, Fh, D) * 0.05).bfloat16().cuda()
    xp = M.permute_rows(x, dest, k, rows)
    out = M.grouped_rows(xp, w1, te, seg)
    ref = M.grouped_rows(xp.cpu(), w1.cpu(), te.cpu(), seg.cpu())
    live = (te.cpu() >= 0).repeat_interleave(M.PAD)
    assert (out.float().cpu()[live] - ref.float()[live]).abs().max() < 3e-2
    # dgrad layout: b as [E, K, N]
    dg = M.grouped_rows(out.masked_fill(~live.cuda()[:, None], 0), w1, te, seg, b_mn_major=True)
    dg_ref = M.grouped_rows(ref, w1.cpu(), te.cpu(), seg.cpu(), b_mn_major=True)
    assert (dg.float().cpu()[live] - dg_ref.float()[live]).abs().max() < 3e-2 * max(dg_ref.abs().max().item(), 1)
    # wgrad, fp32 accumulate
    dy = out.masked_fill(~live.cuda()[:, None], 0)
    acc = torch.zeros(E, Fh, D, device="cuda")
    M.grouped_wgrad(dy, xp, seg, E, out=acc, accumulate=True)
    M.grouped_wgrad(dy, xp, seg, E, out=acc, accumulate=True)
    wg_ref = M.grouped_wgrad(dy.cpu(), xp.cpu(), seg.cpu(), E, out_dtype=torch.float32)
    assert (acc.cpu() - 2 * wg_ref).abs().max() < 2e-2 * max(wg_ref.abs().max().item(), 1)
    _lib.check_status("grouped gemm")


@pytest.mark.parametrize("T,E,k,D,Fh", [(1024, 8, 2, 256, 256), (4096, 32, 4, 960, 576)])
def test_grouped_mxfp8_mlp_matches_emulation(T, E, k, D, Fh):
    """Block-scaled grouped GEMMs against the eager emulation that rounds the same way; the second case has
    widths that are not multiples of 128 (partial K blocks, unfused dSwiGLU)."""
    torch.manual_seed(3)
    logits = torch.randn(T, E)
    logits[:, 1] -= 100.0                                   # an expert without tokens
    idx, w, cnt = M.router_topk(logits.cuda(), k)
    seg, te, dest, rows = M.plan(idx, cnt, E, pad=M.PAD_MX)
    x = (torch.randn(T, D) * 0.5).bfloat16().cuda()
    w1 = (torch.randn(E, 2 * Fh, D) * 0.05).bfloat16().cuda()
    w2 = (torch.randn(E, D, Fh) * 0.05).bfloat16().cuda()
    assert M.mx_supported(w1, w2)
    xp = M.permute_rows(x, dest, k, rows)
    live = (te.cpu() >= 0).repeat_interleave(M.PAD_MX)
    # forward / dgrad GEMM
    from mlperf_training_b200.ops import mxfp8
    a_g, at_g = mxfp8.quantize(xp, row_tile=128, col_tile=M.grouped_bn(D))
    b_g = M._stacked_weight_op(w1, False)
    out = M.grouped_rows_mx(a_g, b_g, te, E)
    torch.cuda.synchronize()
    _lib.check_status("grouped mx rows")
    a_c, at_c = mxfp8.quantize(xp.cpu(), row_tile=128, col_tile=M.grouped_bn(D))
    b_c, _ = mxfp8.quantize(w1.cpu().reshape(E * 2 * Fh, D), row_tile=M.grouped_bn(2 * Fh))
    ref = M.grouped_rows_mx(a_c, b_c, te.cpu(), E)
    assert_tiles_close(out.float().cpu()[live], ref.float()[live], rel=2e-2, what="grouped mx rows")
    # weight gradient: contraction over every expert's rows, accumulated twice into fp32
    dy = out.masked_fill(~live.cuda()[:, None], 0)
    _, dyt_g = mxfp8.quantize(dy, col_tile=128)
    acc = torch.zeros(E, 2 * Fh, D, device="cuda")
    M.grouped_wgrad_mx(dyt_g, at_g, seg, E, acc)
    M.grouped_wgrad_mx(dyt_g, at_g, seg, E, acc)
    torch.cuda.synchronize()
    _lib.check_status("grouped mx wgrad")
    _, dyt_c = mxfp8.quantize(dy.cpu(), col_tile=128)
    wg_ref = M.grouped_wgrad_mx(dyt_c, at_c, seg.cpu(), E, torch.zeros(E, 2 * Fh, D))
    assert acc[1].abs().max() == 0                            # the empty expert's gradient stays zero
    assert_tiles_close(acc.cpu().view(-1, D), 2 * wg_ref.view(-1, D), rel=1e-3, what="grouped mx wgrad")
    # the whole MLP with autograd against the bf16 grouped path
    def run(prec):
        xx = x.clone().requires_grad_()
        p1, p2 = w1.clone().requires_grad_(), w2.clone().requires_grad_()
        y = M.moe_experts(xx, idx, w, cnt, p1, p2, prec)
        (y.float() ** 2).sum().backward()
        return y.detach().float(), xx.grad.float(), p1.grad.float(), p2.grad.float()
    base, mx = run("bf16"), run("mxfp8")
    torch.cuda.synchronize()
    _lib.check_status("grouped mx mlp")
    for name, u, v in zip(("y", "dx", "dw1", "dw2"), base, mx):
        rel = ((u - v).norm() / u.norm()).item()
        assert rel < 0.12, (name, rel)


def test_moe_model_step_matches_cpu():
    cfg = GPTConfig(n_layers=2, hidden=256, n_heads=4, n_kv_heads=2, head_dim=64, ffn_hidden=512, vocab_size=1024,
                    seq_len=256, window=128, window_layers="even", sink=True, n_experts=8, top_k=2, moe_ffn_hidden=256)
    ref = GPT(GPTConfig(**{**cfg.to_dict(), "dtype": "fp32"}), "cpu", seed=2)
    dev = GPT(cfg, "cuda", seed=2)
    with torch.no_grad():
        for (n, p), (_, q) in zip(ref.named_parameters(), dev.named_parameters()):
            q.copy_(p.to(q.dtype))
            p.copy_(q.float().cpu())
    toks = torch.randint(0, cfg.vocab_size, (2, cfg.seq_len + 1))
    l_ref = ref(toks[:, :-1], toks[:, 1:]); l_ref.backward()
    d = toks.cuda()
    l_dev = dev(d[:, :-1], d[:, 1:]); l_dev.backward()
    torch.cuda.synchronize()
    _lib.check_status("moe step")
    assert abs(float(l_dev.detach()) - float(l_ref.detach())) < 5e-2
    bad = []
    for (n, p), (_, q) in zip(ref.named_parameters(), dev.named_parameters()):
        rel = (q.grad.float().cpu() - p.grad).norm().item() / (p.grad.norm().item() + 1e-9)
        if rel > (0.4 if n.endswith('router') else 0.15):   # top-k ties flip between fp32 and bf16 activations
            bad.append((n, rel))
    assert not bad, bad


@pytest.mark.parametrize("recipe", ["mxfp6", "mxfp4"])
def test_grouped_mlp_narrow_recipes(recipe):
    """The grouped expert MLP on operands rounded to 6- / 4-bit element grids (carried as e4m3 codes), forward and all
    three gradients against the bf16 grouped path, with an empty expert."""
    from mlperf_training_b200.ops import _lib
    from mlperf_training_b200.ops import moe_ops as M
    torch.manual_seed(0)
    T, k, E, D, F = 300, 2, 4, 384, 384
    x = torch.randn(T, D, device="cuda").bfloat16()
    logits = torch.randn(T, E, device="cuda")
    logits[:, 2] -= 100.0
    w1 = (torch.randn(E, 2 * F, D, device="cuda") * 0.05).bfloat16().requires_grad_()
    w2 = (torch.randn(E, D, F, device="cuda") * 0.05).bfloat16().requires_grad_()
    idx, w, counts = M.router_topk(logits, k)
    assert M.expert_precision(recipe, w1, w2) == recipe

    def run(prec):
        xx = x.clone().requires_grad_()
        w1.grad = w2.grad = None
        y = M.moe_experts(xx, idx, w, counts, w1, w2, prec)
        y.float().square().sum().backward()
        return y.detach().float(), xx.grad.float(), w1.grad.float().clone(), w2.grad.float().clone()

    ref = run("bf16")
    got = run(recipe)
    torch.cuda.synchronize()
    _lib.check_status("narrow grouped mlp")
    limit = 0.2 if recipe == "mxfp6" else 0.6
    for u, v in zip(ref, got):
        assert torch.isfinite(v).all() and ((u - v).norm() / u.norm()).item() < limit
    assert got[2][2].abs().max() == 0
