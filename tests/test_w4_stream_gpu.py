"""4-bit weight stream of decode-sized batches against the expanded weights in 64 bits."""
import pytest
import torch

from ksanallm_b200.ops import native, reference as ref

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K,group", [(16, 128, 128), (100, 640, 128), (4096, 1024, 256), (136, 14336, 128), (1000, 4224, 128)])
@pytest.mark.parametrize("offset", [0.0, 3.0])
def test_against_expanded_weights(M, N, K, group, offset, monkeypatch):
    real, name = native._load(), "ksana_w4_stream_wins"
    monkeypatch.setattr(real, name, lambda *args: 1)                      # this kernel, whatever is faster
    torch.manual_seed(M + N + K)
    w = torch.randn(N, K, device=DEV) * 0.05 + 0.02 * torch.randn(N, 1, device=DEV)
    packed, scale, zs = ref.quant_w4(w, group)
    dense = ref.dequant_w4(packed, scale, zs).double()
    x = (torch.randn(M, K + 8, device=DEV, dtype=torch.bfloat16) + offset)[:, :K]
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
        # A group of 128 is scale * sum((128 + level) x) - (zs + 128 scale) * sum(x), both up to 143 scale sum|x|: eight steps of 16 products and
        # two more roundings there, twelve additions of half a unit and two roundings here, 2^-23 each. Then the groups' sum, a rounding of
        # at most the weights' magnitudes per group. The result in bf16.
        groups = x.double().abs().unflatten(1, (-1, 128)).sum(-1) @ scale.double().repeat_interleave(group // 128, 1).t()
        total = x.double().abs() @ dense.abs().t()
        bound = 2 ** -8 * want.abs() + 2 ** -23 * (143 * 18 * groups + (K / 128 + 8) * total) + 1e-6
        err = (y.double() - want).abs()
        assert bool((err <= bound).all()), float((err / bound).max())
