"""fp8 quantisation kernels and the scaled tcgen05 fp8 GEMM against fp32 PyTorch on the dequantised operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


@pytest.mark.parametrize("mode", [0, 1])
def test_quantise_rows_matches_torch(mode):
    from ghost_flow_b200.ops import fp8

    x = torch.randn(300, 512, device="cuda", dtype=torch.bfloat16) * 3
    q, s = fp8.quantize_rows(x, mode)
    qc, sc = fp8.quantize_rows(x.cpu(), mode)
    assert torch.allclose(s.cpu(), sc, rtol=1e-6)
    # bytes may differ by one code where x / scale sits on a rounding boundary; the values must agree closely
    d = fp8.dequantize(q.cpu(), s.cpu(), mode)
    assert _rel(d, fp8.dequantize(qc, sc, mode)) < 8e-3
    assert _rel(d, x.cpu()) < 4e-2


def test_quantise_block128_matches_torch():
    from ghost_flow_b200.ops import fp8

    w = torch.randn(320, 256, device="cuda", dtype=torch.bfloat16)
    q, s = fp8.quantize_block128(w)
    qc, sc = fp8.quantize_block128(w.cpu())
    assert torch.allclose(s.cpu(), sc, rtol=1e-6)
    assert _rel(fp8.dequantize(q.cpu(), s.cpu(), 1, weight=True), fp8.dequantize(qc, sc, 1, weight=True)) < 8e-3


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("M,N,K", [(256, 512, 256), (1000, 777 // 8 * 8, 1024), (4096, 4096, 4096)])
def test_fp8_gemm_matches_dequantised_reference(mode, M, N, K):
    from ghost_flow_b200.ops import _lib, fp8

    torch.manual_seed(0)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.05
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    aq, sa = fp8.quantize_rows(a, mode)
    bq, sb = fp8.quantize_rows(b, 0) if mode == 0 else fp8.quantize_block128(b)
    y = fp8.gemm_fp8(aq, sa, bq, sb, mode, bias)
    torch.cuda.synchronize()
    _lib.check_status(a.device)
    ref = fp8.dequantize(aq, sa, mode) @ fp8.dequantize(bq, sb, mode, weight=True).t() + bias.float()
    assert _rel(y, ref) < 6e-3
    # and the quantised product is close to the bf16 one
    assert _rel(y, a.float() @ b.float().t() + bias.float()) < 6e-2


@pytest.mark.parametrize("M,N,K", [(64, 5120, 8192), (16, 1280, 8192)])
def test_fp8_skinny_gemm_split_k(M, N, K):
    from ghost_flow_b200.ops import _lib, fp8

    torch.manual_seed(1)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.05
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    aq, sa = fp8.quantize_rows(a, 0)
    bq, sb = fp8.quantize_rows(b, 0)
    y = fp8.gemm_fp8(aq, sa, bq, sb, 0, bias)
    torch.cuda.synchronize()
    _lib.check_status(a.device)
    ref = fp8.dequantize(aq, sa, 0) @ fp8.dequantize(bq, sb, 0, weight=True).t() + bias.float()
    assert _rel(y, ref) < 6e-3


def test_fp8_training_linear_matches_the_emulation_and_fp32(kernel_status):
    """Forward, input gradient and weight gradient of the e4m3 training linear on the tcgen05 fp8 kernel against the
    same quantisation emulated in fp32 on the CPU, and against the unquantised layer."""
    from ghost_flow_b200.ops import fp8

    torch.manual_seed(0)
    T, K, N = 512, 256, 384
    x = torch.randn(T, K)
    w = 0.1 * torch.randn(N, K)
    b = torch.randn(N)
    g = torch.randn(T, N)
    outs = {}
    for dev in ("cpu", "cuda"):
        xd = x.to(dev, torch.bfloat16).requires_grad_()
        wd = w.to(dev, torch.bfloat16).requires_grad_()
        bd = b.to(dev, torch.bfloat16).requires_grad_()
        y = fp8.fp8_linear(xd, wd, bd)
        y.backward(g.to(dev, torch.bfloat16))
        outs[dev] = [t.detach().float().cpu() for t in (y, xd.grad, wd.grad, bd.grad)]
    xr, wr, br = x.clone().requires_grad_(), w.clone().requires_grad_(), b.clone().requires_grad_()
    yr = torch.nn.functional.linear(xr, wr, br)
    yr.backward(g)
    rel = lambda a, c: ((a - c).norm() / c.norm()).item()  # noqa: E731
    for got, emu, ref in zip(outs["cuda"], outs["cpu"], (yr.detach(), xr.grad, wr.grad, br.grad)):
        assert rel(got, emu) < 2e-2, rel(got, emu)          # same quantisation, different summation order
        assert rel(got, ref) < 7e-2, rel(got, ref)          # e4m3 against fp32


# columns around the steps of the row kernel (registers per thread, threads per row, the loop beyond 16384), rows that
# leave the last block part empty
@pytest.mark.parametrize("T,K", [(1, 8), (9, 256), (3, 264), (7, 1024), (5, 1032), (3, 2056), (2, 4096), (3, 4104), (2, 8200),
                                 (2, 12296), (3, 16384), (2, 16392)])
def test_quantise_rows_gives_the_oracle_bytes(T, K):
    from ghost_flow_b200.ops import fp8

    x = torch.randn(T, K, device="cuda", dtype=torch.bfloat16) * 3
    x[0] = 0                                           # an all-zero row keeps the smallest scale
    if T > 2:
        x[2, K // 2] = float("nan")                    # ignored by the maximum, kept as NaN
    q, s = fp8.quantize_rows(x, 0)
    f = x.float()
    amax = torch.nan_to_num(f.abs(), nan=0.0).amax(1)
    scale = amax.clamp_min(1e-12) / torch.full_like(amax, 448.0)     # a true division (by a number, torch multiplies)
    assert torch.equal(s, scale)
    want = (f * (torch.ones_like(scale) / scale)[:, None]).clamp(-448, 448).to(torch.float8_e4m3fn)
    # the same fp32 operations and one conversion: equal up to the sign of NaN
    assert torch.equal(torch.nan_to_num(q.view(torch.float8_e4m3fn).float(), nan=999.0), torch.nan_to_num(want.float(), nan=999.0))


@pytest.mark.parametrize("R,K", [(16, 16), (128, 64), (144, 80), (112, 528), (1040, 1008), (4096, 2048), (16, 5008)])
def test_transposed_quantisation_equals_quantising_the_transpose(R, K):
    from ghost_flow_b200.ops import fp8

    buf = torch.randn(R * K + 8, device="cuda", dtype=torch.bfloat16)
    x = buf[8:].view(R, K)
    x[0, 0], x[-1, -1], x[:, 3] = 300.0, -1e30, 0.0
    x[5, 7] = float("nan")
    q, s, qt, st = fp8.quantize_transposed(x, rows=True)
    q1, s1 = fp8.quantize_rows(x, 0)
    qt1, st1 = fp8.quantize_rows(x.t().contiguous(), 0)
    assert torch.equal(q, q1) and torch.equal(s, s1) and torch.equal(qt, qt1) and torch.equal(st, st1)
    qt2, st2 = fp8.quantize_transposed(x)
    assert torch.equal(qt2, qt1) and torch.equal(st2, st1)
    # a start off the 16-byte boundary is copied first; sizes the kernel does not take go through the plain transpose
    odd = buf[1:1 + R * K].view(R, K)
    assert torch.equal(fp8.quantize_transposed(odd)[0], fp8.quantize_rows(odd.clone().t().contiguous(), 0)[0])
    part = x[:, :8].contiguous()
    assert torch.equal(fp8.quantize_transposed(part)[0], fp8.quantize_rows(part.t().contiguous(), 0)[0])


# 256 x 256 tiles for 74 pairs and one fewer, ragged in every dimension, K of one block and of a part of one
@pytest.mark.parametrize("M,N,K", [(2048, 2368, 128), (2000, 2600, 528), (2560, 1800, 272), (2304, 2100, 1040), (256, 18944, 256),
                                   (257, 9500, 256), (384, 11000, 272), (400, 11008, 272), (700, 22000, 256)])
@pytest.mark.parametrize("with_bias", [True, False])
def test_large_products_with_row_and_column_scales(M, N, K, with_bias, kernel_status):
    from ghost_flow_b200.ops import fp8

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    N = N // 8 * 8
    aq, sa = fp8.quantize_rows(torch.randn(M, K, generator=g, device="cuda").bfloat16())
    bq, sb = fp8.quantize_rows(torch.randn(N, K, generator=g, device="cuda").bfloat16() * torch.linspace(0.01, 3, N, device="cuda").bfloat16()[:, None])
    bias = torch.randn(N, generator=g, device="cuda").bfloat16() if with_bias else None
    y = fp8.gemm_fp8(aq, sa, bq, sb, 0, bias)
    want = fp8.dequantize(aq, sa, 0).double() @ fp8.dequantize(bq, sb, 0).double().t() + (bias.double() if with_bias else 0)
    # e4m3 products are exact in fp32; fp32 sums of K of them, of size one times the scale of the column, and one bf16 rounding
    assert torch.allclose(y.double(), want, rtol=2 ** -8, atol=3 * K * 2 ** -20)
