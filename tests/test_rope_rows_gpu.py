"""Rotary embedding of whole heads with the cache append, the form that takes 8 pairs per thread, against a statement in 64 bits."""
import pytest
import torch

from ksanallm_b200.ops import native, reference as ref

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (5, 1), (8, 2), (28, 4), (40, 8), (64, 4)])      # 24 to 576 items of two half heads at D = 128
@pytest.mark.parametrize("D", [16, 64, 96, 128])
@pytest.mark.parametrize("turned", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn])
def test_bits(Hq, Hkv, D, turned, dtype):
    torch.manual_seed(Hq + D)
    T, bt, nblk = 19, 16, 3
    qkv = torch.randn(T, Hq + 2 * Hkv, D, device=DEV).to(torch.bfloat16)
    qkv[5, Hq:] *= 400.0                                            # beyond the range of e4m3
    was = qkv.clone()
    pos = torch.randint(0, 500, (T,), device=DEV, dtype=torch.int32)
    slots = torch.randperm(nblk * bt, device=DEV)[:T].to(torch.int32)
    slots[3] = slots[T - 1] = -1
    cs = ref.build_cos_sin_cache(D, 512, 10000.0, device=DEV)
    cache = torch.full((nblk, 2, Hkv, bt, D), 0.5, device=DEV).to(dtype)
    want = cache.clone()
    ks, vs = (0.5, 2.0) if dtype != torch.bfloat16 else (1.0, 1.0)
    native.rope_kv_append(qkv.view(T, -1), pos, slots, cs, cache, cache.stride(0), bt, Hq, Hkv, D, D, True, k_scale=ks, v_scale=vs, apply_rope=turned)
    if turned:
        x, (c, s) = was[:, :Hq + Hkv].double(), cs[pos.long()].double()[:, None].split(D // 2, -1)
        a, b = x.split(D // 2, -1)
        exact = torch.cat([a * c - b * s, b * c + a * s], -1)
        # what a product pair summed in 32 bits and rounded to bf16 once can be
        off = 2.0 ** -21 * torch.cat([a.abs() + b.abs()] * 2, -1)
        y = qkv[:, :Hq + Hkv].double()
        assert bool((((exact - off).to(torch.bfloat16).double() <= y) & (y <= (exact + off).to(torch.bfloat16).double())).all())
    else:
        assert torch.equal(qkv, was)
    assert torch.equal(qkv[:, Hq + Hkv:], was[:, Hq + Hkv:])
    # the cache holds what the rows hold now, in its type; nothing else of it has changed
    k, v = qkv[:, Hq:Hq + Hkv], qkv[:, Hq + Hkv:]
    for t in range(T):
        if slots[t] >= 0:
            at = int(slots[t]) // bt, int(slots[t]) % bt
            for i, (x, scale) in enumerate(((k, ks), (v, vs))):
                y = x[t].float() / scale
                want[at[0], i, :, at[1]] = (y.clamp(-448.0, 448.0) if dtype != torch.bfloat16 else y).to(dtype)
    bits = torch.uint8 if dtype != torch.bfloat16 else torch.int16
    assert torch.equal(cache.view(bits), want.view(bits))
