"""Decode attention whose units are shared out over the CTAs by the device: ragged batches, items cut into many pieces, runs of whole
items, empty sequences, 8-bit caches."""
import math

import pytest
import torch

from ksanallm_b200.ops import native

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def attention64(q, k, v, scale):
    """q [heads, D], k [tokens, kv heads, D], v [tokens, kv heads, Dv] in 64 bits: the result and what a correct kernel may differ by."""
    group = q.shape[0] // k.shape[1]
    k, v = k.repeat_interleave(group, 1), v.repeat_interleave(group, 1)
    w = torch.softmax(torch.einsum("hd,thd->ht", q, k) * scale, -1)
    out = torch.einsum("ht,thd->hd", w, v)
    # the weights are rounded to bf16 (by 2^-8 of each at most) and so is the result; the fp32 sums of a score (2^-24 of its terms per step of
    # 16 columns, above and below the division) change a weight by as much as the score
    scores = torch.einsum("hd,thd->ht", q.abs(), k.abs()).amax(-1, keepdim=True) * scale * 2 ** -23 * (q.shape[1] / 16)
    return out, (2 ** -8 + scores) * torch.einsum("ht,thd->hd", w, v.abs()) + 2 ** -8 * out.abs() + 2 ** -20


@pytest.mark.parametrize("Hq,Hkv,D,bt,fp8", [(32, 8, 128, 16, False), (32, 8, 128, 16, True), (64, 8, 128, 64, True), (20, 1, 128, 8, False),
                                             (20, 1, 128, 8, True), (4, 4, 64, 16, True), (6, 2, 96, 32, True), (8, 2, 192, 16, False),
                                             (4, 2, 256, 16, False), (8, 8, 64, 16, False)])
@pytest.mark.parametrize("lens", [[0, 1, 63, 64, 65, 129, 3000, 16], [9000], [1], [500 + 7 * i for i in range(70)], [194] * 25,
                                  [3079, 3000, 2500, 60, 0], [1 + 37 * i % 190 for i in range(160)]],
                         ids=["ragged", "long", "one", "many", "short", "pieces", "runs"])
def test_ragged_batches(Hq, Hkv, D, bt, fp8, lens):
    torch.manual_seed(len(lens) + D)
    B, nblk, dtype = len(lens), sum(-(-n // bt) for n in lens) + 3, torch.float8_e4m3fn if fp8 else torch.bfloat16
    cache = torch.randn(nblk, 2, Hkv, bt, D, device=DEV).mul_(1.5)
    ids = torch.randperm(nblk, device=DEV).to(torch.int32)
    table = torch.zeros(B, max(1, max(-(-n // bt) for n in lens)), dtype=torch.int32, device=DEV)
    at, want, bound = 0, torch.zeros(B, Hq, D, dtype=torch.float64, device=DEV), torch.zeros(B, Hq, D, dtype=torch.float64, device=DEV)
    q = torch.randn(B, Hq * D + 8, device=DEV, dtype=torch.bfloat16)
    if B > 1:
        q *= torch.logspace(-3, 3, B, device=DEV).unsqueeze(1).to(torch.bfloat16)
    ks, vs, scale = (0.75, 1.25, 1 / math.sqrt(D)) if fp8 else (1.0, 1.0, 1 / math.sqrt(D))
    for s, n in enumerate(lens):
        nb = -(-n // bt)
        table[s, :nb] = ids[at:at + nb]
        at += nb
        shift = 4.0 * torch.randint(-1, 2, (nb * bt // 64 + 1,), device=DEV)         # a tile that is left out or taken twice shows
        cache[table[s, :nb].long(), 1] += shift[torch.arange(nb, device=DEV) * bt // 64].view(nb, 1, 1, 1)
    cache = cache.to(dtype)
    for s, n in enumerate(lens):
        nb = -(-n // bt)
        rows = cache.view(torch.uint8 if fp8 else torch.bfloat16)
        if n % bt:                                    # what lies past the end is not read: NaN there
            rows[table[s, nb - 1].long(), :, :, n % bt:] = 0x7F if fp8 else float("nan")
        if n:
            kv = cache[table[s, :nb].long()].double().permute(1, 0, 3, 2, 4).reshape(2, nb * bt, Hkv, D)[:, :n]
            want[s], bound[s] = attention64(q[s, :Hq * D].view(Hq, D).double(), kv[0] * ks, kv[1] * vs, scale)
    kvl = torch.tensor(lens, dtype=torch.int32, device=DEV)
    out = torch.full((B, Hq * D), float("nan"), device=DEV, dtype=torch.bfloat16)

    def run(dst):
        native.paged_decode(q, q.stride(0), dst, cache, cache.stride(0), bt, table, kvl, B, Hq, Hkv, D, scale, k_scale=ks, v_scale=vs)
        native.check_err_flag(DEV)

    run(out)
    err = (out.view(B, Hq, D).double() - want).abs()
    worst = (err / bound.clamp_min(1e-30)).amax((1, 2))
    assert bool((err <= bound).all()), [(n, round(float(r), 2)) for n, r in zip(lens, worst) if r > 1]
    again = torch.empty_like(out)
    run(again)                                        # counters are back at zero, sums do not depend on who comes last
    assert torch.equal(again, out)
    odd = torch.zeros(B, Hq * D + 2, device=DEV, dtype=torch.bfloat16)[:, 1:-1]     # rows that no vector store may touch
    run(odd)
    assert torch.equal(odd, out)
