"""Expert products with scales applied by the tensor cores, FP8 rows taken to their experts."""
import pytest
import torch

from ksanallm_b200.ops import native

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


@pytest.mark.parametrize("T,K,E,N,H", [(1, 2, 4, 256, 128), (7, 2, 3, 200, 384), (64, 8, 32, 512, 640), (700, 4, 8, 1032, 1152)])
def test_grouped_mxfp8(T, K, E, N, H):
    torch.manual_seed(T)
    x = torch.randn(T, H, device=DEV, dtype=torch.bfloat16)
    ids = torch.rand(T, E, device=DEV).topk(K, dim=1).indices.to(torch.int32)
    q, s = native.quant_fp8(x)
    dst, tile_expert, _, _, cap, tile_rows = native.moe_align(ids, E)
    pq, ps = native.moe_permute_fp8(q, s, dst, K, cap)
    rows = dst.long()
    # permuting quantised rows gives what quantising permuted rows does
    bq, bs = native.quant_fp8(native.moe_permute(x, dst, K, cap, zero=True))
    assert torch.equal(pq.view(torch.uint8)[rows], bq.view(torch.uint8)[rows]) and torch.equal(ps[:, rows], bs[:, rows])
    wq = (torch.randn(E * N, H, device=DEV) * 64).clamp(-448, 448).to(torch.float8_e4m3fn)
    ws = 2.0 ** torch.randint(-9, -5, (E * -(-N // 128), H // 128), device=DEV).float()
    token = torch.arange(T, device=DEV).repeat_interleave(K)
    xd = (q.float() * s[:, :T].t().repeat_interleave(128, 1)).double()
    full = ws.view(E, -1, H // 128).repeat_interleave(128, 1)[:, :N].repeat_interleave(128, 2).double()
    w = wq.double().view(E, N, H) * full
    want = torch.einsum("rh,rnh->rn", xd[token], w[ids.flatten().long()])
    for tr in (tile_rows, None):
        y = native.gemm_grouped(pq, wq, tile_expert, E, N, a_scale=ps, w_scale=ws, tile_rows=tr, hw_scale=True)
        native.check_err_flag(DEV)
        # fp32 sums of exact products, rounded to bf16
        err = (y[rows].double() - want).abs()
        assert bool((err <= 2 ** -8 * want.abs() + 2 ** -18 * want.abs().amax()).all()), float(err.max())
