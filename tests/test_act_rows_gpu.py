"""Activation and quantisation at odd sizes."""
import pytest
import torch

from ksanallm_b200.ops import native, reference as ref

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


@pytest.mark.parametrize("M,inter", [(1, 8), (3, 24), (5, 128), (129, 384), (64, 2048), (1000, 14336)])
@pytest.mark.parametrize("act", ["silu", "gelu", "relu"])
def test_act_mul_sizes(M, inter, act):
    torch.manual_seed(M)
    for gated in (True, False):
        x = torch.randn(M, inter * (2 if gated else 1), device=DEV, dtype=torch.bfloat16) * 3
        want = ref.act_mul(x.float(), act, gated)
        y = native.act_mul(x, act, gated)
        err = (y.float() - want).abs()
        # the approximate tanh (2^-11 of the activation) and the result's own rounding
        assert bool((err <= 2 ** -7 * want.abs() + 2 ** -10 * x.float().abs().amax()).all())
        if inter % 128 == 0:
            out, q, s = native.act_mul(x, act, gated, quant=True)
            bq, bs = native.quant_fp8(y)
            rq, rs = ref.quant_fp8(y.cpu())
            assert torch.equal(out, y) and torch.equal(q.view(torch.uint8), bq.view(torch.uint8)) and torch.equal(s[:, :M], bs[:, :M])
            assert torch.equal(bq.view(torch.uint8).cpu(), rq.view(torch.uint8)) and torch.equal(bs[:, :M].cpu(), rs[:, :M])


@pytest.mark.parametrize("M,H", [(1, 16), (3, 48), (5, 896), (2, 4096), (700, 4112), (333, 7168), (3000, 128), (1200, 8192), (7, 16384)])
def test_norm_rows(M, H):
    """Rows of a chunk, odd numbers of chunks, more rows than CTAs; with and without the fp8 copy."""
    torch.manual_seed(M + H)
    x = torch.randn(M, H, device=DEV, dtype=torch.bfloat16) * torch.logspace(-2, 2, M, device=DEV)[:, None].to(torch.bfloat16)
    w = 1 + 0.1 * torch.randn(H, device=DEV, dtype=torch.bfloat16)
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * w.double()
    y = native.norm(x, w, 1e-5)
    # one rounding to bf16 (2^-9 of the value), fp32 sums and an approximate root before it
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20).all())
    if H % 128 == 0:
        out, q, s = native.norm(x, w, 1e-5, quant=True)
        _, q2, s2 = native.norm(x, w, 1e-5, quant=True, want_out=False)
        rq, rs = ref.quant_fp8(out.cpu())
        assert torch.equal(out, y)
        for a, b in ((q, s), (q2, s2)):
            assert torch.equal(a.view(torch.uint8).cpu(), rq.view(torch.uint8)) and torch.equal(b[:, :M].cpu(), rs[:, :M])


@pytest.mark.parametrize("M,H", [(1, 4096), (7, 16), (700, 8192), (3, 24), (5, 16400)])
def test_norm_with_largest_magnitude(M, H):
    """The pass that also takes the result's largest magnitude: bits and scale of one pass after the other; NaN do not count."""
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.empty(M, H, device="cuda", dtype=torch.bfloat16).normal_(generator=g)
    w = torch.empty(H, device="cuda", dtype=torch.bfloat16).normal_(generator=g)
    x[M - 1, H - 1] = 60.0
    x[0, 0] = float("nan") if M > 1 else 1.0
    for _ in range(2):
        y, scale = native.norm_absmax(x, w, 1e-5, 7.0)
        want = native.norm(x, w, 1e-5)
        assert torch.equal(y.view(torch.int16), want.view(torch.int16))
        assert float(scale) == float(native.absmax_scale(want, 7.0)) > 0


@pytest.mark.parametrize("M,inter,gap,act", [(1, 4096, 0, "silu"), (300, 14336, 0, "silu"), (2001, 1552, 16, "gelu"), (2000, 1544, 0, "silu")])
def test_act_with_largest_magnitude(M, inter, gap, act):
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.empty(M, 2 * inter + gap, device="cuda", dtype=torch.bfloat16).normal_(generator=g)[:, :2 * inter]
    x[M - 1, inter - 1], x[M - 1, 2 * inter - 1] = 9.0, -50.0
    x[M // 2, 5] = float("nan")
    for _ in range(2):
        y, scale = native.act_mul_absmax(x, act, 7.0)
        want = native.act_mul(x, act, True)
        assert torch.equal(y.view(torch.int16), want.view(torch.int16))
        assert float(scale) == float(native.absmax_scale(want, 7.0)) > 0
