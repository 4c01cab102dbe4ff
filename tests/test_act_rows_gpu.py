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
