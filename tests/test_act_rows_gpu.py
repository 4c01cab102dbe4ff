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
