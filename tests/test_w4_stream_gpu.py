"""4-bit weight stream of decode-sized batches against the expanded weights in 64 bits."""
import pytest
import torch

from ksanallm_b200.ops import native, reference as ref

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K,group", [(16, 128, 128), (100, 640, 128), (4096, 1024, 256), (136, 14336, 128), (1000, 4224, 128)])
def test_against_expanded_weights(M, N, K, group):
    torch.manual_seed(M + N + K)
    w = torch.randn(N, K, device=DEV) * 0.05 + 0.02 * torch.randn(N, 1, device=DEV)
    packed, scale, zs = ref.quant_w4(w, group)
    dense = ref.dequant_w4(packed, scale, zs).double()
    x = torch.randn(M, K + 8, device=DEV, dtype=torch.bfloat16)[:, :K]
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    for b, add in ((None, False), (bias, True)):
        out = torch.randn(M, N, device=DEV, dtype=torch.bfloat16)
        want = x.double() @ dense.t()
        if b is not None:
            want = want + b.double()
        if add:
            want = want + out.double()
        y = native.linear_w4(x, packed, scale, zs, out=out, bias=b, residual=out if add else None)
        assert y.data_ptr() == out.data_ptr()
        # fp32 sums of (128 + level) x: 2^-24 of the terms' magnitudes for each of the K / 16 steps at most; the result in bf16
        sums = x.double().abs() @ (torch.repeat_interleave(scale.double(), group, 1) * 160).t()
        err = (y.double() - want).abs()
        assert bool((err <= 2 ** -8 * want.abs() + 2 ** -24 * (K / 16) * sums + 1e-6).all()), float(err.max())
