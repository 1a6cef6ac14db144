"""MXFP8 quantiser and block-scaled tcgen05 GEMM against the eager emulation (bit-exact codes and
scales; GEMM against an fp32 matmul of the dequantised operands)."""
import pytest
import torch

from mlperf_training_b200.ops import _lib, mxfp8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,C", [(128, 128), (256, 384), (896, 512)])
def test_quantize_matches_emulation(R, C):
    torch.manual_seed(R + C)
    x = (torch.randn(R, C) * torch.exp(torch.randn(R, 1) * 2)).bfloat16()
    x[3, 32:64] = 0  # an all-zero block
    x[5, 0] = 448.0 * 4  # amax exactly on a power-of-two boundary
    for row_tile, col_tile in ((128, 224), (224, 128)):
        r_c, c_c = mxfp8.quantize(x, row_tile=row_tile, col_tile=col_tile)
        r_g, c_g = mxfp8.quantize(x.cuda(), row_tile=row_tile, col_tile=col_tile)
        torch.cuda.synchronize()
        for cpu, gpu, what in ((r_c, r_g, "row"), (c_c, c_g, "col")):
            assert torch.equal(mxfp8.sf_plain(gpu).cpu(), cpu.sf), f"{what} scales"
            assert torch.equal(gpu.q.cpu(), cpu.q), f"{what} codes"
        # quantisation error is bounded by the e4m3 step
        err = (mxfp8.dequantize(r_g).cpu() - x.float()).abs()
        assert (err <= x.float().abs().view(R, C // 32, 32).amax(-1, keepdim=True).expand(-1, -1, 32).reshape(R, C) * 0.07 + 1e-30).all()


@pytest.mark.parametrize("R,C", [(256, 160), (384, 960), (2048, 2880)])
def test_quantize_partial_column_tile(R, C):
    """Widths that are multiples of 32 but not of 128 (the last 128-column tile is partial)."""
    torch.manual_seed(R + C)
    x = (torch.randn(R, C) * torch.exp(torch.randn(R, 1))).bfloat16()
    r_c, c_c = mxfp8.quantize(x, row_tile=128, col_tile=192)
    r_g, c_g = mxfp8.quantize(x.cuda(), row_tile=128, col_tile=192)
    torch.cuda.synchronize()
    _lib.check_status("quant partial")
    for cpu, gpu, what in ((r_c, r_g, "row"), (c_c, c_g, "col")):
        assert torch.equal(mxfp8.sf_plain(gpu).cpu(), cpu.sf), f"{what} scales"
        assert torch.equal(gpu.q.cpu(), cpu.q), f"{what} codes"
    gu = (torch.randn(R, 2 * C) * 2).bfloat16()
    a_c, at_c = mxfp8.quantize_swiglu(gu, row_tile=128, col_tile=192)
    a_g, at_g = mxfp8.quantize_swiglu(gu.cuda(), row_tile=128, col_tile=192)
    ref = mxfp8.dequantize(a_c)
    assert (mxfp8.dequantize(a_g).cpu() - ref).abs().max() <= 0.13 * ref.abs().max()      # SwiGLU rounding may flip a code
    assert (mxfp8.dequantize(at_g).cpu() - mxfp8.dequantize(at_c)).abs().max() <= 0.13 * ref.abs().max()


def test_quantize_scale_limits():
    """Blocks whose largest magnitude sits at the ends of the scale rule: 1.75 times a power of two and its bf16 neighbours,
    amax / 448 below the normal numbers, bf16 denormals, zero, the largest finite value."""
    x = torch.zeros(128, 256)
    amax = [1.75, 1.75 * (1 + 2 ** -7), 1.75 * (1 - 2 ** -7), 448.0, 450.0, 2.0 ** -118, 2.0 ** -119, 1.9 * 2.0 ** -118, 2.0 ** -126, 2.0 ** -130,
            0.0, 3.3e38, 1.75 * 2.0 ** 100, 1.0]
    for i, a in enumerate(amax):
        x[i] = a * torch.linspace(-1, 1, 256)
        x[i, ::32] = a
    x = x.bfloat16()
    for t, kw in ((x, dict(row_tile=128)), (x.t().contiguous(), dict(col_tile=128))):
        for cpu, gpu in zip(mxfp8.quantize(t, **kw), mxfp8.quantize(t.cuda(), **kw)):
            if cpu is not None:
                assert torch.equal(mxfp8.sf_plain(gpu).cpu(), cpu.sf)
                assert torch.equal(gpu.q.cpu(), cpu.q)


@pytest.mark.parametrize("R,F", [(128, 128), (256, 160), (384, 2880), (128, 96)])
def test_quantize_swiglu_bwd_equals_the_separate_kernels(R, F):
    """d gate | d up from one tile pair: codes and scales of quantising the stand-alone kernel's output, bit for bit, at widths
    whose halves start inside a scale word; with ``live`` the rows before it are the same."""
    from mlperf_training_b200.ops import kernels as K
    torch.manual_seed(R + F)
    gu, da = (torch.randn(R, 2 * F, device="cuda") * 3).bfloat16(), torch.randn(R, F, device="cuda").bfloat16()
    want = mxfp8.quantize(K.swiglu_bwd(da, gu), row_tile=128, col_tile=208)
    got = mxfp8.quantize_swiglu_bwd(da, gu, row_tile=128, col_tile=208)
    for a, b in zip(want, got):
        assert torch.equal(a.q, b.q) and torch.equal(mxfp8.sf_plain(a), mxfp8.sf_plain(b))
    assert torch.equal(want[0].sf, got[0].sf)            # (the padding of the last scale word, too)
    for w, g in zip(mxfp8.quantize(K.swiglu_fwd(gu), row_tile=128, col_tile=192), mxfp8.quantize_swiglu(gu, row_tile=128, col_tile=192)):
        assert torch.equal(w.q, g.q) and torch.equal(mxfp8.sf_plain(w), mxfp8.sf_plain(g))
    live = torch.tensor([128], dtype=torch.int32, device="cuda")
    part = mxfp8.quantize_swiglu_bwd(da, gu, row_tile=128, col_tile=208, live=live)
    assert torch.equal(part[0].q[:128], want[0].q[:128]) and torch.equal(part[1].q[:, :128], want[1].q[:, :128])


@pytest.mark.parametrize("live", [0, 128, 256, 384])
@pytest.mark.parametrize("F", [128, 160])
def test_quantisers_leave_rows_past_live_alone(live, F):
    """Codes and scales of the 128-row tiles behind ``live`` keep what the buffers held, those before it are the full run's."""
    from mlperf_training_b200.ops import _lib
    torch.manual_seed(live + F)
    R = 384
    gu, da = torch.randn(R, 2 * F, device="cuda").bfloat16(), torch.randn(R, F, device="cuda").bfloat16()
    n = torch.tensor([live], dtype=torch.int32, device="cuda")
    p, st = _lib.ptr, _lib.stream_ptr()
    for name, args, C in (("b200_quant_mxfp8", (p(gu), 2 * F, R, 2 * F), 2 * F), ("b200_quant_swiglu_mxfp8", (p(gu), 2 * F, R, F), F),
                          ("b200_quant_swiglu_bwd_mxfp8", (p(da), F, p(gu), 2 * F, R, F), 2 * F)):
        runs = []
        for fill, lv in ((0x5A, None), (0x5A, n)):
            size = (R * C, mxfp8.sf_bytes(R, C, 128), C * R, mxfp8.sf_bytes(C, R, 128))
            q_row, sf_row, q_col, sf_col = (torch.full((k,), fill, dtype=torch.uint8, device="cuda") for k in size)
            _lib.call(name, *args, p(q_row), p(sf_row), 128, p(q_col), p(sf_col), 128, p(lv), st)
            # rows tile by tile; the transposed copy's contraction in groups of 128 rows of the source
            runs.append((q_row.view(R // 128, -1), sf_row.view(R // 128, -1), q_col.view(C, R // 128, 128).transpose(0, 1),
                         sf_col.view(-1, R // 128, 512).transpose(0, 1)))
        for full, part in zip(*runs):
            assert torch.equal(part[:live // 128], full[:live // 128])
            assert (part[live // 128:] == 0x5A).all()
            if live < R:
                assert (full[live // 128:] != 0x5A).any()
    _lib.check_status("live")


def test_no_column_copies_without_grad_and_weight_copies_in_one_pass():
    from mlperf_training_b200.ops import functional as F
    w = torch.nn.Parameter((torch.randn(256, 384, device="cuda") * 0.05).bfloat16())
    x = torch.randn(128, 384, device="cuda").bfloat16()
    with torch.no_grad():
        y0 = F.linear(x, w, precision="mxfp8")
    assert w._mx_cache[2] is None
    row = w._mx_cache[1]
    y1 = F.linear(x.requires_grad_(True), w, precision="mxfp8")
    assert w._mx_cache[2] is not None and w._mx_cache[1] is row and torch.equal(y0, y1)
    y1.float().sum().backward()
    assert w.grad is not None and x.grad is not None


@pytest.mark.parametrize("K", [128, 384, 640])
def test_gemm_does_not_read_scales_past_an_odd_contraction(K):
    """The scales behind a contraction of an odd number of 128-blocks may be anything (here: NaN for every row tile's neighbour)."""
    torch.manual_seed(K)
    a, b = torch.randn(512, K, device="cuda").bfloat16(), torch.randn(416, K, device="cuda").bfloat16()
    b = torch.cat([b, torch.zeros(96, K, device="cuda").bfloat16()])
    qa, qb = mxfp8.quantize(a, row_tile=mxfp8.A_TILE)[0], mxfp8.quantize(b, row_tile=mxfp8.b_tile(512))[0]
    want = mxfp8.gemm(qa, qb)
    sf = qa.sf.clone()
    sf.view(4, -1)[1:] = 255                             # rows 128 .. of A: not a number
    got = mxfp8.gemm(mxfp8.MXOperand(qa.q, sf, qa.rows, qa.k, qa.tile_rows), qb)
    assert torch.equal(got[:128], want[:128])


@pytest.mark.parametrize("M,N,K", [(128, 128, 128), (256, 224, 256), (384, 448, 512), (512, 1000, 384),
                                   (1024, 4096, 1024), (136, 72, 128)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_mxfp8(M, N, K, out_dtype):
    torch.manual_seed(M + N + K)
    Mp, Np = (M + 127) // 128 * 128, (N + 127) // 128 * 128
    a = torch.randn(Mp, K, device="cuda").bfloat16()
    b = torch.randn(Np, K, device="cuda").bfloat16()
    a_op, _ = mxfp8.quantize(a, row_tile=mxfp8.A_TILE)
    b_op, _ = mxfp8.quantize(b, row_tile=mxfp8.b_tile(Np))
    d = mxfp8.gemm(a_op, b_op, out_dtype=out_dtype)
    torch.cuda.synchronize()
    _lib.check_status("gemm_mxfp8")
    ref = mxfp8.dequantize(a_op) @ mxfp8.dequantize(b_op).t()
    err = (d.float() - ref).abs().max().item()
    tol = (2e-2 if out_dtype == torch.bfloat16 else 1e-3) * ref.abs().max().item()
    assert err <= tol, f"err {err} tol {tol}"
    # and the quantised product is close to the bf16 product
    full = a.float() @ b.float().t()
    rel = (ref - full).norm() / full.norm()
    assert rel < 0.06


def test_gemm_mxfp8_epilogues():
    torch.manual_seed(0)
    M, N, K = 256, 512, 256
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    a_op, _ = mxfp8.quantize(a, row_tile=mxfp8.A_TILE)
    b_op, _ = mxfp8.quantize(b, row_tile=mxfp8.b_tile(N))
    ref = mxfp8.dequantize(a_op) @ mxfp8.dequantize(b_op).t()
    res = torch.randn(M, N, device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    d = mxfp8.gemm(a_op, b_op, residual=res, bias=bias, alpha=0.5)
    acc = torch.ones(M, N, device="cuda")
    mxfp8.gemm(a_op, b_op, out=acc, accumulate=True)
    mxfp8.gemm(a_op, b_op, out=acc, accumulate=True)
    torch.cuda.synchronize()
    sc = ref.abs().max().item()
    assert (d.float() - (0.5 * ref + res.float() + bias.float())).abs().max().item() < 2e-2 * sc
    assert (acc - (2 * ref + 1)).abs().max().item() < 2e-3 * sc
    _lib.check_status("gemm_mxfp8 epilogues")


def test_fused_mlp_matches_unfused_mxfp8_path():
    """The fused unit (quantisation folded into SwiGLU / dSwiGLU) computes exactly what the separate
    norm_linear + swiglu_linear MXFP8 path computes."""
    import torch
    from mlperf_training_b200.ops import functional as F
    torch.manual_seed(0)
    T, D, Fh = 512, 256, 512
    h0 = torch.randn(T, D, device="cuda").bfloat16()
    nw0 = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
    w1_0 = (torch.randn(2 * Fh, D, device="cuda") * 0.05).bfloat16()
    w2_0 = (torch.randn(D, Fh, device="cuda") * 0.05).bfloat16()
    dy = torch.randn(T, D, device="cuda").bfloat16()
    outs = []
    for fused in (False, True):
        h, nw, w1, w2 = (t.clone().requires_grad_(True) for t in (h0, nw0, w1_0, w2_0))
        assert F.fused_mlp_eligible(h, w1, w2)
        if fused:
            y = F.fused_mlp(h, nw, w1, w2, 1e-5)
        else:
            gu = F.norm_linear(h, nw, w1, eps=1e-5, precision="mxfp8")
            y = F.swiglu_linear(gu, w2, residual=h, precision="mxfp8")
        y.backward(dy)
        outs.append([t.detach().float() for t in (y, h.grad, nw.grad, w1.grad, w2.grad)])
    torch.cuda.synchronize()
    for name, a, b in zip(("y", "dh", "dnorm", "dw1", "dw2"), outs[0], outs[1]):
        if name == "dh":
            # the fused unit adds the residual gradient inside the norm backward (one rounding instead of two)
            assert (a - b).abs().max().item() <= 2.0 ** -6 * max(1.0, b.abs().max().item()), name
        else:
            assert torch.equal(a, b), (name, (a - b).abs().max().item())


@pytest.mark.parametrize("fmt", ["e2m1", "e2m3", "e3m2"])
def test_narrow_element_formats_match_the_cpu_oracle(fmt):
    """Operands rounded to a 4- / 6-bit element grid and carried as e4m3 codes: the same codes and scales as the CPU
    routine, and the block-scaled GEMM multiplies them like the dequantised matrices."""
    torch.manual_seed(0)
    x = (torch.randn(256, 384) * torch.logspace(-2, 1, 384)[None, :]).bfloat16()
    w = (torch.randn(256, 384) * 0.05).bfloat16()
    a_c = mxfp8.quantize(x, row_tile=mxfp8.A_TILE, fmt=fmt)[0]
    a_g = mxfp8.quantize(x.cuda(), row_tile=mxfp8.A_TILE, fmt=fmt)[0]
    assert torch.equal(a_g.q.cpu(), a_c.q) and torch.equal(mxfp8.sf_plain(a_g).cpu(), a_c.sf)
    bt = mxfp8.b_tile(256)
    b_c = mxfp8.quantize(w, row_tile=bt, fmt=fmt)[0]
    b_g = mxfp8.quantize(w.cuda(), row_tile=bt, fmt=fmt)[0]
    y_g = mxfp8.gemm(a_g, b_g, out_dtype=torch.float32)
    y_c = mxfp8.gemm(a_c, b_c, out_dtype=torch.float32)
    assert (y_g.cpu() - y_c).abs().max() <= 1e-3 * y_c.abs().max()
    _, col_g = mxfp8.quantize(x.cuda(), col_tile=bt, fmt="e4m3", col_fmt=fmt)
    _, col_c = mxfp8.quantize(x, col_tile=bt, fmt="e4m3", col_fmt=fmt)
    assert torch.equal(col_g.q.cpu(), col_c.q) and torch.equal(mxfp8.sf_plain(col_g).cpu(), col_c.sf)


@pytest.mark.parametrize("recipe", ["mxfp4", "a6w4"])
def test_narrow_recipes_through_the_linear_triple(recipe):
    from mlperf_training_b200.ops import functional as F
    torch.manual_seed(1)
    x = torch.randn(256, 256).bfloat16()
    w = (torch.randn(384, 256) * 0.05).bfloat16()
    g = torch.randn(256, 384).bfloat16()
    y_c = F.linear(x, w, None, None, recipe)
    xg, wg = x.cuda().requires_grad_(True), w.cuda().requires_grad_(True)
    y_g = F.linear(xg, wg, None, None, recipe)
    assert (y_g.float().cpu() - y_c.float()).abs().max() <= 2e-2 * y_c.float().abs().max()      # same operands, bf16 output
    y_g.backward(g.cuda())
    ref_dx, ref_dw = g.float() @ w.float(), g.float().t() @ x.float()
    rel = lambda a, b: float((a.float().cpu() - b).norm() / b.norm())
    assert rel(xg.grad, ref_dx) < 0.3 and rel(wg.grad, ref_dw) < 0.3        # stochastic 4-bit gradients: close, not equal
    _lib.check_status("narrow recipes")
