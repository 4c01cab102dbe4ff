"""bf16 GEMM of more than 128 rows: CTA pairs or single CTAs, the faster of the two as measured (148 SMs)."""
import pytest

from ksanallm_b200.ops import native


# us with single CTAs and with pairs
@pytest.mark.parametrize("M,N,K,single,pair", [
    (2048, 1152, 896, 10.2, 11.8), (2048, 1152, 4096, 22.3, 26.0), (2048, 1152, 14336, 60.8, 76.4), (136, 4096, 256, 5.6, 6.7),
    (300, 1152, 128, 4.3, 5.6), (384, 1152, 512, 5.7, 6.5), (513, 896, 256, 4.9, 5.9), (1024, 1152, 512, 6.5, 7.1), (1100, 896, 512, 9.2, 10.0),
    (3103, 256, 128, 7.4, 8.2), (384, 4096, 512, 8.4, 7.4), (136, 6144, 512, 8.2, 7.1), (300, 4096, 256, 7.4, 6.5), (1100, 1152, 512, 8.6, 7.3),
    (2048, 896, 512, 9.9, 8.4), (136, 4096, 896, 8.0, 7.3), (1100, 6144, 4096, 50.7, 46.1), (300, 14336, 4096, 57.5, 45.9),
    (5000, 4608, 128, 38.4, 22.0)])
def test_the_faster_one(M, N, K, single, pair):
    assert native._pair_wins(M, N, K, 148) == (pair < single)
