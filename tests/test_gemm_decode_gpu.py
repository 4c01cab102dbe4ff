"""GEMM of decode steps (one tile, or share of one, per CTA) at the edges of tiles, shares and K blocks."""
import pytest
import torch

from ksanallm_b200.ops import native

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def close(y, want, sums):
    # fp32 sums (2^-24 of the magnitudes per K block and share), the result rounded to bf16 unless it is fp32
    err = (y.double() - want).abs()
    bound = (2 ** -8 if y.dtype == torch.bfloat16 else 2 ** -23) * want.abs() + 2 ** -18 * sums
    assert bool((err <= bound).all()), float((err - bound).max())


@pytest.mark.parametrize("M", [1, 3, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(8, 64), (32, 7168), (130, 520), (4096, 1032), (19000, 256), (1000, 4096)])
def test_bf16(M, N, K):
    torch.manual_seed(M + N)
    x = torch.randn(M, K + 8, device=DEV, dtype=torch.bfloat16)[:, :K]
    w = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    bias, res = torch.randn(N, device=DEV, dtype=torch.bfloat16), torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
    want, sums = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    close(native.gemm_bf16(x, w), want, sums)
    close(native.gemm_bf16(x, w, out_f32=torch.empty(M, N, device=DEV)), want, sums)
    out = res.clone()
    close(native.gemm_bf16(x, w, out=out, bias=bias, residual=out), want + bias.double() + res.double(), sums)
    odd = torch.zeros(M, N + 3, device=DEV, dtype=torch.bfloat16)[:, 1:N + 1]           # rows on no vector boundary
    close(native.gemm_bf16(x, w, out=odd), want, sums)
    native.check_err_flag(DEV)


@pytest.mark.parametrize("M", [1, 16, 30, 33, 64])
@pytest.mark.parametrize("N,K", [(128, 128), (136, 896), (4096, 7168), (20480, 640), (576, 4224)])
def test_block_scaled(M, N, K):
    torch.manual_seed(M + K)
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16) * torch.logspace(-2, 2, M, device=DEV).unsqueeze(1).to(torch.bfloat16)
    xq, xs = native.quant_fp8(x)
    wq = (torch.randn(N, K, device=DEV) * 64).clamp(-448, 448).to(torch.float8_e4m3fn)
    ws = 2.0 ** torch.randint(-9, -4, (-(-N // 128), K // 128), device=DEV).float()
    xd = xq.double() * xs[:, :M].t().repeat_interleave(128, 1).double()
    wd = wq.double() * ws.repeat_interleave(128, 0)[:N].repeat_interleave(128, 1).double()
    res = torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
    want, sums = xd @ wd.t(), xd.abs() @ wd.abs().t()
    close(native.gemm_fp8(xq, xs, wq, ws, hw_scale=True), want, sums)
    out = res.clone()
    close(native.gemm_fp8(xq, xs, wq, ws, out=out, residual=out, hw_scale=True), want + res.double(), sums)
    native.check_err_flag(DEV)


@pytest.mark.parametrize("M", [1, 5, 33, 64])
@pytest.mark.parametrize("N,K", [(10100, 2056), (5000, 4096)])
def test_three_and_six_shares(M, N, K):
    """K ranges cut in three (79 tiles) and six (40): shares of unequal length, fewer tokens than shares."""
    torch.manual_seed(M + N)
    x, w = torch.randn(M, K, device=DEV, dtype=torch.bfloat16), torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    close(native.gemm_bf16(x, w), x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t())
    K = K // 128 * 384
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    xq, xs = native.quant_fp8(x)
    wq = (torch.randn(N, K, device=DEV) * 64).clamp(-448, 448).to(torch.float8_e4m3fn)
    ws = 2.0 ** torch.randint(-9, -4, (-(-N // 128), K // 128), device=DEV).float()
    xd = xq.double() * xs[:, :M].t().repeat_interleave(128, 1).double()
    wd = wq.double() * ws.repeat_interleave(128, 0)[:N].repeat_interleave(128, 1).double()
    close(native.gemm_fp8(xq, xs, wq, ws, hw_scale=True), xd @ wd.t(), xd.abs() @ wd.abs().t())
    native.check_err_flag(DEV)
