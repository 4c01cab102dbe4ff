"""Prefill attention with one or two query tiles per CTA where the CTAs of one run at once and those of two need a second round."""
import pytest

from ksanallm_b200.ops import native


# sequences of n new tokens on so many cached ones, us with one tile and with two (148 SMs)
@pytest.mark.parametrize("Hq,Hkv,B,n,past,one,two", [
    (14, 2, 16, 150, 100, 15.1, 18.3), (14, 2, 16, 150, 300, 21.7, 26.3), (14, 2, 16, 150, 800, 35.8, 41.7), (14, 2, 8, 330, 0, 18.7, 20.6),
    (14, 2, 32, 150, 100, 26.9, 28.1), (14, 2, 32, 150, 300, 39.7, 38.5), (28, 4, 8, 150, 100, 18.0, 21.3), (28, 4, 24, 40, 300, 22.1, 25.6),
    (28, 4, 8, 330, 0, 38.2, 34.9), (16, 16, 6, 300, 300, 29.3, 32.7), (16, 16, 4, 600, 0, 34.6, 28.2), (40, 40, 2, 300, 300, 30.1, 33.8),
    (40, 40, 1, 850, 0, 35.7, 33.2), (40, 40, 1, 1000, 0, 47.2, 37.9), (40, 40, 2, 300, 2000, 82.8, 80.2), (64, 8, 12, 40, 300, 21.7, 25.0),
    (64, 8, 2, 300, 100, 24.6, 27.7), (64, 8, 2, 300, 300, 36.7, 31.4), (64, 8, 1, 600, 0, 27.9, 20.3), (64, 8, 4, 150, 100, 26.6, 23.8),
    (32, 8, 8, 150, 100, 27.0, 21.8), (32, 8, 16, 33, 200, 17.2, 11.8), (12, 2, 8, 400, 0, 30.0, 25.4)])
def test_the_faster_one(Hq, Hkv, B, n, past, one, two):
    rows = B * n
    pairs = B * (n * (n + past) - n * (n - 1) // 2)
    assert native.prefill_pair_wins(pairs, rows, B, Hq, Hkv, 148) == (two < one)
