"""tcgen05 bf16 GEMM against a plain fp32 PyTorch matmul of the same bf16 operands."""
import pytest
import torch

from mlperf_training_b200.ops import _lib, kernels

pytestmark = pytest.mark.gpu


def _ref(a, b, a_mn, b_mn):
    am = a.float().t() if a_mn else a.float()
    bm = b.float() if b_mn else b.float().t()
    return am @ bm


def _check(d, ref, K, what):
    err = (d.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    tol = 2e-2 * scale if d.dtype == torch.bfloat16 else 2e-3 * scale
    _lib.check_status(what)
    assert err <= tol, f"{what}: max err {err} vs tol {tol} (scale {scale})"


SHAPES = [(128, 256, 64), (256, 256, 128), (128, 128, 256), (384, 512, 192), (300, 520, 136), (1024, 1024, 1024),
          (2048, 4096, 512), (136, 72, 64)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_layouts(M, N, K, a_mn, b_mn):
    torch.manual_seed(M * 7 + N * 3 + K)
    dev = "cuda"
    a = torch.randn((K, M) if a_mn else (M, K), device=dev).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=dev).bfloat16()
    d = kernels.gemm(a, b, a_mn_major=a_mn, b_mn_major=b_mn)
    torch.cuda.synchronize()
    _check(d, _ref(a, b, a_mn, b_mn), K, f"gemm {M}x{N}x{K} a_mn={a_mn} b_mn={b_mn}")


def test_gemm_fp32_out_and_accumulate():
    torch.manual_seed(1)
    M, N, K = 512, 768, 320
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    ref = _ref(a, b, False, False)
    d = kernels.gemm(a, b, out_dtype=torch.float32)
    torch.cuda.synchronize()
    _check(d, ref, K, "fp32 out")
    acc = torch.full((M, N), 0.5, device="cuda", dtype=torch.float32)
    kernels.gemm(a, b, out=acc, accumulate=True)
    kernels.gemm(a, b, out=acc, accumulate=True)
    torch.cuda.synchronize()
    _check(acc, 2 * ref + 0.5, K, "fp32 accumulate x2")
    accb = torch.zeros((M, N), device="cuda", dtype=torch.bfloat16)
    kernels.gemm(a, b, out=accb, accumulate=True)
    torch.cuda.synchronize()
    _check(accb, ref, K, "bf16 accumulate")


def test_gemm_bias_residual_alpha():
    torch.manual_seed(2)
    M, N, K = 300, 264, 128
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = torch.randn(N, K, device="cuda").bfloat16()
    bias = torch.randn(N, device="cuda").bfloat16()
    res = torch.randn(M, N, device="cuda").bfloat16()
    d = kernels.gemm(a, b, bias=bias, residual=res, alpha=0.5)
    torch.cuda.synchronize()
    ref = 0.5 * _ref(a, b, False, False) + bias.float() + res.float()
    _check(d, ref, K, "bias+residual+alpha")


def test_gemm_strided_views():
    torch.manual_seed(3)
    M, N, K = 256, 384, 128
    big_a = torch.randn(M, K + 64, device="cuda").bfloat16()
    a = big_a[:, 32:32 + K]  # pitch K+64, base offset 64 bytes
    b = torch.randn(N, K, device="cuda").bfloat16()
    out_big = torch.zeros(M, N + 128, device="cuda", dtype=torch.bfloat16)
    out = out_big[:, 64:64 + N]
    kernels.gemm(a, b, out=out)
    torch.cuda.synchronize()
    _check(out, _ref(a, b, False, False), K, "strided")
    assert out_big[:, :64].abs().max().item() == 0 and out_big[:, 64 + N:].abs().max().item() == 0


def test_gemm_deterministic():
    torch.manual_seed(4)
    a = torch.randn(1024, 512, device="cuda").bfloat16()
    b = torch.randn(768, 512, device="cuda").bfloat16()
    d1 = kernels.gemm(a, b)
    d2 = kernels.gemm(a, b)
    torch.cuda.synchronize()
    assert torch.equal(d1, d2)


def _forms():
    """Operands as callers hand them over: (name, arguments) of gemm, whose operands the native operator takes or leaves to the
    general path."""
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    out = []
    for M, N, K in ((1, 136, 64), (5, 72, 136), (129, 264, 136), (256, 2880, 320), (300, 520, 1000)):
        for a_mn in (False, True):
            for b_mn in (False, True):
                def ab(pad=0, off=0):
                    def t(r, c):
                        return rnd(r, c + pad + off)[:, off:off + c]
                    return (t(K, M) if a_mn else t(M, K)), (t(K, N) if b_mn else t(N, K))
                lay = dict(a_mn_major=a_mn, b_mn_major=b_mn)
                tag = f"{M}x{N}x{K} {int(a_mn)}{int(b_mn)}"
                a, b = ab()
                out.append((tag, a, b, lay))
                out.append((tag + " padded rows", *ab(pad=8), lay))
                out.append((tag + " odd pitch", *ab(pad=3), lay))
                out.append((tag + " off 16 bytes", *ab(pad=7, off=1), lay))
                out.append((tag + " fp32 out, alpha", a, b, dict(lay, out_dtype=torch.float32, alpha=0.5)))
                out.append((tag + " bias", a, b, dict(lay, bias=rnd(N))))
                out.append((tag + " fp32 strided bias", a, b, dict(lay, bias=rnd(2 * N).float()[::2])))
                out.append((tag + " residual of wider rows", a, b, dict(lay, residual=rnd(M, N + 8)[:, :N], bias=rnd(N))))
                out.append((tag + " fp32 residual", a, b, dict(lay, residual=rnd(M, N).float())))
                out.append((tag + " transposed residual", a, b, dict(lay, residual=rnd(N, M).t())))
                out.append((tag + " into wider rows", a, b, dict(lay, out=rnd(M, N + 16)[:, :N])))
                out.append((tag + " added to fp32", a, b, dict(lay, out=rnd(M, N).float(), accumulate=True)))
    a, b = rnd(16, 64), rnd(24, 64)
    out += [("expanded", rnd(1, 64).expand(16, 64), b, {}), ("one row", a[3:4], b, {}), ("transposed", rnd(64, 16).t(), b, {}),
            ("empty", a[:0], b, {}), ("widths", a, rnd(24, 72), {}), ("odd columns", a, b[:5], {}), ("fp32", a.float(), b, {}),
            ("fp16 out", a, b, dict(out_dtype=torch.float16)), ("nothing to add to", a, b, dict(accumulate=True)),
            ("other rows", a, b, dict(out=rnd(15, 24))), ("out in columns", a, b, dict(out=rnd(24, 16).t())),
            ("out off 16 bytes", a, b, dict(out=rnd(16, 32)[:, 1:25]))]
    return out


def test_native_operator_equals_the_general_path(monkeypatch):
    """Same results, bit for bit, and the same refusals, over the layouts, pitches, types and options of the operands."""
    if _lib.host is None:
        pytest.skip("no native operator in this build")

    def run(a, b, kw):
        if "out" in kw:
            base = kw["out"]
            kw = dict(kw, out=base.clone() if base.is_contiguous() else base._base.clone().as_strided(base.shape, base.stride(),
                                                                                                     base.storage_offset()))
        try:
            d = kernels.gemm(a, b, **kw)
            assert kw.get("out") is None or d is kw["out"]
            return d
        except (ValueError, TypeError, RuntimeError) as e:
            return type(e), str(e)
    forms = _forms()
    native = [run(a, b, kw) for _, a, b, kw in forms]
    monkeypatch.setattr(_lib, "host", None)
    refused = 0
    for (name, a, b, kw), got in zip(forms, native):
        want = run(a, b, kw)
        if isinstance(want, tuple):
            assert got == want, name
            refused += 1
        else:
            assert got.dtype == want.dtype and got.stride() == want.stride() and torch.equal(got, want), name
    assert refused >= 6
    _lib.check_status("native gemm")
