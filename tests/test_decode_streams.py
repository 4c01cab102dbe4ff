"""Which decode calls share themselves out over the CTAs, and that the others are given a number of splits."""
import math

import pytest
import torch

from ksanallm_b200.ops import dispatch, native


def cache(D, bt=16, Hkv=2, fp8=False, blocks=4, device="cpu"):
    return torch.zeros(blocks, 2, Hkv, bt, D, device=device, dtype=torch.float8_e4m3fn if fp8 else torch.bfloat16)


def streams(c, B=4, Hq=8, Hkv=2, **kw):
    return native.decode_streams(c, None, c.stride(0), c.shape[3], B, Hq, Hkv, c.shape[4], **kw)


@pytest.mark.parametrize("D", [64, 72, 80, 88, 96, 104, 112, 120, 128, 136, 192, 256])
def test_head_sizes(D):
    assert streams(cache(D))
    assert streams(cache(D, fp8=True)) == (D % 16 == 0 and D <= 128)     # rows of whole 16-byte units


@pytest.mark.parametrize("bt,ok", [(8, True), (16, True), (64, True), (4, False), (24, False), (128, False)])
def test_block_sizes(bt, ok):
    assert streams(cache(128, bt)) == ok and streams(cache(128, bt, fp8=True)) == ok


def test_strides_and_panels():
    c = cache(128)
    assert not native.decode_streams(c, None, c.stride(0) + 4, 16, 4, 8, 2, 128)          # block stride off 16 bytes
    k, v = torch.zeros(4 * 16 * 2 * 128 + 8, dtype=torch.bfloat16), cache(128)[:, 1]
    odd = k[1:1 + 4 * 2 * 16 * 128].view(4, 2, 16, 128)
    assert native.decode_streams(cache(128)[:, 0], v, v.stride(0), 16, 4, 8, 2, 128)
    assert not native.decode_streams(odd, v, v.stride(0), 16, 4, 8, 2, 128)               # panel off 16 bytes
    assert not streams(c, B=60000)                                                        # the sequences' prefix sums do not fit


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")
@pytest.mark.parametrize("D,bt,fp8,split", [(72, 16, True, True), (120, 16, True, True), (128, 16, True, False), (72, 16, False, False),
                                            (128, 24, False, True)])
def test_long_contexts_are_split(D, bt, fp8, split, monkeypatch):
    torch.manual_seed(D)
    n, Hq, Hkv = 3001, 8, 2
    nb = -(-n // bt)
    c = torch.randn(nb, 2, Hkv, bt, D, device="cuda").to(torch.float8_e4m3fn if fp8 else torch.bfloat16)
    table, kvl = torch.arange(nb, device="cuda", dtype=torch.int32).view(1, nb), torch.tensor([n], device="cuda", dtype=torch.int32)
    q = torch.randn(1, (Hq + 2 * Hkv) * D, device="cuda", dtype=torch.bfloat16)
    seen, real = [], native.paged_decode
    monkeypatch.setattr(native, "paged_decode", lambda *a, **kw: (seen.append(a[16]), real(*a, **kw)))
    cu = torch.tensor([0, 1], device="cuda", dtype=torch.int32)
    out = dispatch.paged_attention(q, None, c, bt, table, cu, kvl, 0, 1, 0, 1, Hq, Hkv, D, 1 / math.sqrt(D), num_splits=0, max_kv_len=n)
    assert (seen[0] > 1) == split
    kv = c.double().permute(1, 0, 3, 2, 4).reshape(2, nb * bt, Hkv, D)[:, :n].repeat_interleave(Hq // Hkv, 2)
    w = torch.softmax(torch.einsum("hd,thd->ht", q[0, :Hq * D].view(Hq, D).double(), kv[0]) / math.sqrt(D), -1)
    want, room = torch.einsum("ht,thd->hd", w, kv[1]), torch.einsum("ht,thd->hd", w, kv[1].abs())
    # weights, keys (where they are dequantised to bf16) and the result rounded to bf16
    assert bool(((out.view(Hq, D).double() - want).abs() <= 2 ** -8 * (room + want.abs()) + 2 ** -20).all())
