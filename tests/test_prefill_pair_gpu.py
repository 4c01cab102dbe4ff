"""Prefill attention with two query tiles per CTA: paged grouped queries, and latents expanded to keys and values of every head."""
import math

import pytest
import torch

from ksanallm_b200.ops import native

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


@pytest.fixture(autouse=True)
def this_kernel(monkeypatch):
    monkeypatch.setattr(native, "prefill_pair_wins", lambda *args: True)          # whatever is faster


def attend64(q, k, v, scale, slopes=None, sinks=None):
    """Causal attention of the last q.shape[0] positions in 64 bits: q [n, heads, D], k, v [tokens, kv heads, D / Dv]; the result and what
    a correct kernel may differ by."""
    n, hq, _ = q.shape
    total, rep = k.shape[0], hq // k.shape[1]
    q, k, v = q.double(), k.double().repeat_interleave(rep, 1), v.double().repeat_interleave(rep, 1)
    s = torch.einsum("nhd,thd->hnt", q, k) * scale
    size = torch.einsum("nhd,thd->hnt", q.abs(), k.abs()) * scale * (q.shape[-1] / 16)
    pos = torch.arange(total - n, total, device=q.device)[:, None]
    key = torch.arange(total, device=q.device)
    if slopes is not None:
        bias = slopes.double()[:, None, None] * (key - pos)
        s, size = s + bias, size + bias.abs()
    s = s.masked_fill(key > pos, float("-inf"))
    if sinks is not None:
        s = torch.cat([s, sinks.double()[:, None, None].expand(-1, n, 1)], -1)
    w = torch.softmax(s, -1)[..., :total]
    out = torch.einsum("hnt,thd->nhd", w, v)
    # the weights are rounded to bf16 (by 2^-8 of each at most) and so is the result; the fp32 sums of a score (2^-24 of its terms per step of
    # 16 columns, above and below the division) change a weight by as much as the score
    off = 2 ** -8 + size.masked_fill(key > pos, 0).amax(-1).t()[..., None] * 2 ** -23
    return out, off * torch.einsum("hnt,thd->nhd", w, v.abs()) + 2 ** -8 * out.abs() + 2 ** -20


def shift_tiles(v):
    """Another offset for every 64 values, so that a tile that is left out or taken twice shows."""
    n = v.shape[0]
    v += (4.0 * torch.randint(-1, 2, (n // 64 + 1,), device=v.device))[torch.arange(n, device=v.device) // 64].view(-1, 1, 1).to(v.dtype)


def check(out, parts):
    want, bound = (torch.cat(x) for x in zip(*parts))
    err = (out.double() - want).abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.parametrize("q_lens,kv_lens", [([256], [256]), ([1, 300, 33], [70, 300, 1000]), ([129, 64, 65, 7], [129, 640, 65, 2000]),
                                            ([2], [130]), ([700], [700])])
@pytest.mark.parametrize("Hq,Hkv,D,bt,extra", [(8, 2, 128, 16, ""), (8, 1, 128, 64, "sinks"), (5, 1, 64, 8, ""), (16, 16, 128, 32, "alibi"),
                                               (6, 2, 96, 16, "")])
def test_paged(q_lens, kv_lens, Hq, Hkv, D, bt, extra):
    torch.manual_seed(sum(q_lens) + Hq)
    B, nblk = len(q_lens), sum(-(-n // bt) for n in kv_lens) + 2
    cache = torch.randn(nblk, 2, Hkv, bt, D, device=DEV, dtype=torch.bfloat16)
    ids = torch.randperm(nblk, device=DEV).to(torch.int32)
    table = torch.zeros(B, max(-(-n // bt) for n in kv_lens), dtype=torch.int32, device=DEV)
    T = sum(q_lens)
    q = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, dtype=torch.bfloat16)
    slopes = torch.logspace(-1, -6, Hq, 2.0, device=DEV) if extra == "alibi" else None
    sinks = torch.randn(Hq, device=DEV) * 2 if extra == "sinks" else None
    scale, at, row, want = 1 / math.sqrt(D), 0, 0, []
    for s, (n, kv) in enumerate(zip(q_lens, kv_lens)):
        nb = -(-kv // bt)
        table[s, :nb] = ids[at:at + nb]
        at += nb
        if kv % bt:
            cache[table[s, nb - 1].long(), :, :, kv % bt:] = float("nan")       # past the end: not read
        k, v = cache[table[s, :nb].long()].permute(1, 0, 3, 2, 4).reshape(2, nb * bt, Hkv, D)[:, :kv]
        shift_tiles(v)
        for i in range(nb):
            cache[table[s, i].long(), 1, :, :min(bt, kv - i * bt)] = v[i * bt:(i + 1) * bt].transpose(0, 1)
        want.append(attend64(q[row:row + n, :Hq * D].view(n, Hq, D), k, v, scale, slopes, sinks))
        row += n
    cu = torch.tensor([0] + q_lens, device=DEV).cumsum(0).to(torch.int32)
    kvl = torch.tensor(kv_lens, dtype=torch.int32, device=DEV)
    out = torch.full((T, Hq * D), float("nan"), device=DEV, dtype=torch.bfloat16)
    native.paged_prefill(q, q.stride(0), out, cache, cache.stride(0), bt, table, cu, kvl, B, max(q_lens), Hq, Hkv, D, scale, alibi=slopes,
                         sinks=sinks)
    native.check_err_flag(DEV)
    check(out.view(T, Hq, D), want)


@pytest.mark.parametrize("q_lens,kv_lens", [([1], [1]), ([300], [300]), ([128, 257, 5], [128, 400, 69]), ([64, 1000], [64, 1000])])
@pytest.mark.parametrize("heads", [1, 16])
def test_expanded_latents(q_lens, kv_lens, heads):
    torch.manual_seed(sum(kv_lens))
    T, L = sum(q_lens), sum(kv_lens)
    q = torch.randn(T, heads, 192, device=DEV, dtype=torch.bfloat16)
    kx = torch.randn(L, heads, 256, device=DEV, dtype=torch.bfloat16)
    lat = torch.randn(L, 576, device=DEV, dtype=torch.bfloat16)
    scale, want, a, b = 1 / math.sqrt(192), [], 0, 0
    for n, kv in zip(q_lens, kv_lens):
        shift_tiles(kx[b:b + kv, :, 128:])
        k = torch.cat([kx[b:b + kv, :, :128], lat[b:b + kv, None, 512:].expand(-1, heads, -1)], -1)
        want.append(attend64(q[a:a + n], k, kx[b:b + kv, :, 128:], scale))
        a, b = a + n, b + kv
    cu = [torch.tensor([0] + n, device=DEV).cumsum(0).to(torch.int32) for n in (q_lens, kv_lens)]
    out = native.mha_prefill(q, kx, lat[:, 512:], cu[0], cu[1], torch.tensor(kv_lens, dtype=torch.int32, device=DEV), max(q_lens), scale)
    native.check_err_flag(DEV)
    check(out, want)
