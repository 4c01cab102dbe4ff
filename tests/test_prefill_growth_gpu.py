"""Prefill attention with two query tiles per CTA where rows outgrow their reference maximum in a later, unmasked tile: exponentials taken ahead
of the tile's maximum are taken again, sums and outputs so far are rescaled."""
import math

import pytest
import torch

from ksanallm_b200.ops import native
from test_prefill_pair_gpu import DEV, attend64, check, shift_tiles

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

# keys of every 128 tokens lie this far along a direction that some queries have 6 of: steps of more than 2^8 in consecutive tiles, in tiles
# that are not adjacent, in one of 64 keys, and back to where they were
LEVELS = {"steps": [0, 14, 28, 42, 56, 70, 84, 98], "apart": [0, 0, 30, 0, 0, 60, 0, 90], "once": [0, 0, 0, 50, 50, 50, 50, 50]}


@pytest.fixture(autouse=True)
def this_kernel(monkeypatch):
    monkeypatch.setattr(native, "prefill_pair_wins", lambda *args: True)          # whatever is faster


def along(q, k, levels, half):
    """q [n, heads, D], k [tokens, kv heads, D] with the levels on them; rows that grow are a third of all, anywhere in a warp."""
    u = torch.nn.functional.normalize(torch.randn(q.shape[-1], device=DEV), dim=0)
    coef = 6.0 * (torch.rand(q.shape[:2], device=DEV) < 0.34).float()
    q32, k32 = q.float(), k.float()
    q.copy_(q32 + (coef - q32 @ u)[..., None] * u)
    at = torch.arange(k.shape[0], device=DEV)
    level = torch.tensor(levels, dtype=torch.float32, device=DEV)[at // 128]
    if half:
        level = level * (at // 64 % 2)
    k.copy_(k32 + level.view(-1, 1, 1) * u)


def outgrown(q, k, scale, tile):
    """Share of the (row, tile) pairs past the first tile whose maximum is more than 2^8 above all before."""
    s = torch.einsum("nhd,thd->nht", q.float(), k.float().repeat_interleave(q.shape[1] // k.shape[1], 1)) * (scale * math.log2(math.e))
    top = s[..., :s.shape[-1] // tile * tile].unflatten(-1, (-1, tile)).amax(-1)
    return float((top[..., 1:] > top.cummax(-1).values[..., :-1] + 8).float().mean())


@pytest.mark.parametrize("levels", LEVELS)
@pytest.mark.parametrize("n,kv,Hq,Hkv,D", [(40, 1000, 8, 2, 128), (300, 1024, 5, 1, 64), (129, 900, 16, 16, 128)])
@pytest.mark.parametrize("half", [False, True])
def test_paged(n, kv, Hq, Hkv, D, levels, half):
    torch.manual_seed(n + kv)
    bt, scale = 16, 1 / math.sqrt(D)
    nb = -(-kv // bt)
    qkv = torch.randn(n, (Hq + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16)
    q = qkv[:, :Hq * D].view(n, Hq, D)
    k, v = torch.randn(2, nb * bt, Hkv, D, device=DEV, dtype=torch.bfloat16)
    along(q, k, LEVELS[levels], half)
    shift_tiles(v)
    assert 0.005 < outgrown(q, k[:kv - n], scale, 128) < 0.5
    cache = torch.stack([k, v]).view(2, nb, bt, Hkv, D).permute(1, 0, 3, 2, 4).contiguous()
    table = torch.arange(nb, device=DEV, dtype=torch.int32)[None]
    cu = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    out = torch.full((n, Hq * D), float("nan"), device=DEV, dtype=torch.bfloat16)
    native.paged_prefill(qkv, qkv.stride(0), out, cache, cache.stride(0), bt, table, cu, torch.tensor([kv], dtype=torch.int32, device=DEV), 1, n,
                         Hq, Hkv, D, scale)
    native.check_err_flag(DEV)
    check(out.view(n, Hq, D), [attend64(q, k[:kv], v[:kv], scale)])


@pytest.mark.parametrize("levels", LEVELS)
@pytest.mark.parametrize("n,kv,heads", [(40, 1000, 16), (300, 1024, 3)])
@pytest.mark.parametrize("half", [False, True])
def test_expanded_latents(n, kv, heads, levels, half):
    torch.manual_seed(n + kv)
    scale = 1 / math.sqrt(192)
    q = torch.randn(n, heads, 192, device=DEV, dtype=torch.bfloat16)
    kx = torch.randn(kv, heads, 256, device=DEV, dtype=torch.bfloat16)
    lat = torch.randn(kv, 576, device=DEV, dtype=torch.bfloat16)
    along(q[..., :128], kx[..., :128], LEVELS[levels], half)
    shift_tiles(kx[..., 128:])
    k = torch.cat([kx[..., :128], lat[:, None, 512:].expand(-1, heads, -1)], -1)
    assert 0.005 < outgrown(q, k[:kv - n], scale, 64) < 0.5
    cu = [torch.tensor([0, m], dtype=torch.int32, device=DEV) for m in (n, kv)]
    out = native.mha_prefill(q, kx, lat[:, 512:], cu[0], cu[1], cu[1][1:], n, scale)
    native.check_err_flag(DEV)
    check(out, [attend64(q, k, kx[..., 128:], scale)])
