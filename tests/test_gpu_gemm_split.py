"""Dense GEMMs whose last wave is cut along K: ragged tiles, every epilogue option, both operand kinds."""
import pytest
import torch

from mlperf_training_b200.ops import _lib, kernels as K, mxfp8 as MX

pytestmark = pytest.mark.gpu

# one tile; ragged rows, columns and K; one full wave and a rest; N of one 128-wide tile
SHAPES = [(256, 256, 4096), (300, 520, 2056), (2048, 512, 8200), (1333, 3400, 8200), (5000, 1000, 2048), (4096, 120, 8192)]


def _rand(*shape):
    return torch.randn(*shape, device="cuda").bfloat16()


def _check(got, want, K_):
    # fp32 accumulation in another order, then one rounding to the output type
    eps = 2 ** -8 if got.dtype == torch.bfloat16 else 2 ** -24 * K_ ** 0.5 * 4
    assert (got.double() - want).abs().max() <= eps * want.abs().max() + 1e-6


@pytest.mark.parametrize("M,N,Kd", SHAPES)
@pytest.mark.parametrize("mode", ["plain", "bias_residual", "f32_accumulate", "bf16_accumulate", "wgrad", "dgrad"])
def test_bf16(M, N, Kd, mode):
    torch.manual_seed(M + N)
    assert _lib.gemm_workspace("b200_gemm_bf16_workspace", M, N, Kd, torch.device("cuda")) is not None
    kw, a, b = {}, _rand(M, Kd), _rand(N, Kd)
    want = a.double() @ b.double().t()
    if mode == "bias_residual":
        kw = dict(bias=_rand(N), residual=_rand(M, N), alpha=0.5)
        want = 0.5 * want + kw["bias"].double() + kw["residual"].double()
    elif mode == "f32_accumulate":
        kw = dict(out=torch.randn(M, N, device="cuda"), accumulate=True)
        want = want + kw["out"].double()
    elif mode == "bf16_accumulate":
        kw = dict(out=_rand(M, N), accumulate=True)
        want = want + kw["out"].double()
    elif mode == "wgrad":
        M8 = M // 8 * 8
        a, want, kw = a[:M8].t().contiguous(), want[:M8], dict(a_mn_major=True, b_mn_major=True, out_dtype=torch.float32)
        b = b.t().contiguous()
    elif mode == "dgrad":
        b, kw = b.t().contiguous(), dict(b_mn_major=True)
    first = K.gemm(a, b, **kw)
    if mode == "bf16_accumulate":      # whole tiles round the product before they add it: one more rounding
        assert (first.double() - want).abs().max() <= 2 ** -7 * want.abs().max()
    else:
        _check(first, want, Kd)
    if "accumulate" not in mode:
        assert torch.equal(first, K.gemm(a, b, **kw))      # no atomics: the same bits
    _lib.check_status("split gemm")


@pytest.mark.parametrize("M,N,Kd", [(256, 384, 4096), (1152, 512, 8192), (4096, 4096, 8192), (640, 128, 8192), (2176, 1920, 8320)])
@pytest.mark.parametrize("mode", ["bf16", "f32_accumulate"])
def test_mxfp8(M, N, Kd, mode):
    torch.manual_seed(M + N)
    assert _lib.gemm_workspace("b200_gemm_mxfp8_workspace", M, N, Kd, torch.device("cuda")) is not None
    qa, _ = MX.quantize(_rand(M, Kd), row_tile=MX.A_TILE)
    qb, _ = MX.quantize(_rand(N, Kd), row_tile=MX.b_tile(N))
    want = MX.dequantize(qa).double() @ MX.dequantize(qb).double().t()
    if mode == "bf16":
        res = _rand(M, N)
        _check(MX.gemm(qa, qb, residual=res), want + res.double(), Kd)
    else:
        out = torch.randn(M, N, device="cuda")
        want = want + out.double()
        _check(MX.gemm(qa, qb, out=out, accumulate=True), want, Kd)
    _lib.check_status("split gemm")


@pytest.mark.parametrize("M", [1, 8, 16, 100, 128])
@pytest.mark.parametrize("N,Kd", [(136, 4096), (512, 512), (3072, 9216), (4096, 4104), (38400, 64)])
@pytest.mark.parametrize("mode", ["plain", "dgrad", "wgrad", "bias_residual", "f32_accumulate", "bf16_accumulate"])
def test_few_rows(M, N, Kd, mode):
    """At most 128 rows: split over CTA pairs, 128- and 256-column tiles of one CTA."""
    torch.manual_seed(M + N)
    a, b, kw = _rand(M, Kd), _rand(N, Kd), {}
    want = a.double() @ b.double().t()
    if mode == "dgrad":
        b, kw = b.t().contiguous(), dict(b_mn_major=True)
    elif mode == "wgrad":
        a, b, kw = a.t().contiguous(), b.t().contiguous(), dict(a_mn_major=True, b_mn_major=True, out_dtype=torch.float32)
    elif mode == "bias_residual":
        kw = dict(bias=_rand(N), residual=_rand(M, N), alpha=0.5)
        want = 0.5 * want + kw["bias"].double() + kw["residual"].double()
    elif mode == "f32_accumulate":
        kw = dict(out=torch.randn(M, N, device="cuda"), accumulate=True)
        want = want + kw["out"].double()
    elif mode == "bf16_accumulate":
        kw = dict(out=_rand(M, N), accumulate=True)
        want = want + kw["out"].double()
    got = K.gemm(a, b, **kw)
    if mode == "bf16_accumulate":      # whole tiles round the product before they add it: one more rounding
        assert (got.double() - want).abs().max() <= 2 ** -7 * want.abs().max()
    else:
        _check(got, want, Kd)
    _lib.check_status("few rows")


@pytest.mark.parametrize("M,N,Kd", [(300, 520, 2056), (1333, 3400, 8200), (16, 512, 8192), (100, 3072, 9216)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("accumulate", [False, True])
def test_wide_output_and_residual(M, N, Kd, out_dtype, accumulate):
    """Column blocks of wider matrices: what stands beside the block stays as it was."""
    torch.manual_seed(M)
    assert _lib.gemm_workspace("b200_gemm_bf16_workspace", M, N, Kd, torch.device("cuda")) is not None
    a, b = _rand(M, Kd), _rand(N, Kd)
    wide, res = torch.randn(M, N + 48, device="cuda").to(out_dtype), _rand(M, N + 24)
    before, want = wide.clone(), a.double() @ b.double().t()
    if accumulate:
        want = want + wide[:, 16:16 + N].double()
        K.gemm(a, b, out=wide[:, 16:16 + N], accumulate=True)
    else:
        want = want + res[:, 8:8 + N].double()
        K.gemm(a, b, out=wide[:, 16:16 + N], residual=res[:, 8:8 + N])
    tol = 2 ** -7 if out_dtype == torch.bfloat16 else 2 ** -24 * Kd ** 0.5 * 4
    assert (wide[:, 16:16 + N].double() - want).abs().max() <= tol * want.abs().max() + 1e-6
    assert torch.equal(wide[:, :16], before[:, :16]) and torch.equal(wide[:, 16 + N:], before[:, 16 + N:])
    _lib.check_status("wide output")


@pytest.mark.parametrize("M,N,Kd", [(300, 520, 2056), (2048, 512, 8200), (16, 512, 8192), (128, 38400, 64)])
def test_infinities_and_nan(M, N, Kd):
    """An infinity in the first slice of K and a NaN in the last reach their own row and column and nothing else."""
    torch.manual_seed(M)
    a, b = _rand(M, Kd), _rand(N, Kd)
    a[3], a[M - 1] = 0, 0
    a[3, 0], a[M - 1, Kd - 1] = float("inf"), float("nan")
    b[:, 0] = b[:, 0].abs() + 0.5
    b[N - 2, Kd // 2] = float("-inf")
    a[:, Kd // 2] = a[:, Kd // 2].abs() + 0.5
    got = K.gemm(a, b)
    want = a.double() @ b.double().t()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()].double(), want[want.isinf()])
    fin = want.isfinite()
    _check(got[fin], want[fin], Kd)
    _lib.check_status("infinities")
