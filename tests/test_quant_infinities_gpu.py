"""FP8 operands of rows that hold infinities and NaN: quantisation, norm and activation."""
import pytest
import torch

from ksanallm_b200.ops import native

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"
NAN8 = 0x7F


def expect(values, q, s):
    """A group that holds an infinity has an infinite scale: its finite values are 0, the others NaN. Elsewhere NaN stays NaN and does
    not reach the scale."""
    M, K = values.shape
    v, q = values.view(M, K // 128, 128), q.view(torch.uint8).view(M, K // 128, 128)
    s = s[:, :M].t()
    inf = v.isinf().any(-1)
    assert torch.equal(s.isinf(), inf) and not bool(s.isnan().any())
    assert bool((q[inf][v[inf].isfinite()] & 0x7F == 0).all())
    assert bool((q[v.isnan()] & 0x7F == NAN8).all()) and bool((q[v.isinf()] & 0x7F == NAN8).all())
    rest = ~inf
    clean = torch.where(v.isfinite(), v, 0).reshape(M, K)
    cq, cs = native.quant_fp8(clean.contiguous())
    cq, cs = cq.view(torch.uint8).view(M, K // 128, 128), cs[:, :M].t()
    assert torch.equal(s[rest], cs[rest]) and torch.equal(q[rest][v[rest].isfinite()], cq[rest][v[rest].isfinite()])


def rows(M, K):
    torch.manual_seed(K)
    x = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    x[0, 5], x[1, K - 1], x[2, 130], x[2, 131] = float("inf"), float("-inf"), float("nan"), 3e38
    x[3, :128], x[4, 7], x[4, 8] = float("nan"), float("inf"), float("nan")
    return x


@pytest.mark.parametrize("K", [256, 2048])
def test_infinities(K):
    x = rows(7, K)
    expect(x, *native.quant_fp8(x))
    # not gated: relu keeps what is not negative (and gives 0 for NaN)
    y, q, s = native.act_mul(x, "relu", False, quant=True)
    expect(y, q, s)
    g = torch.cat([x, torch.ones_like(x)], 1)
    y, q, s = native.act_mul(g, "silu", True, quant=True)
    expect(y, q, s)


def test_norm_with_an_infinite_weight():
    x, w = torch.randn(5, 512, device=DEV, dtype=torch.bfloat16), torch.ones(512, device=DEV, dtype=torch.bfloat16)
    w[200] = float("inf")
    for layernorm in (False, True):
        y, q, s = native.norm(x, w, 1e-5, quant=True, layernorm=layernorm)
        expect(y, q, s)
