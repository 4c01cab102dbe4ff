"""Activation and FP8 quantisation of launches that take chunks of 16 elements per thread: skipped rows, a last warp that is not full, strides."""
import pytest
import torch

from ksanallm_b200.ops import native, reference as ref

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def same(q, s, rq, rs, rows):
    return torch.equal(q.view(torch.uint8)[rows].cpu(), rq.view(torch.uint8)[rows]) and torch.equal(s[:, :q.shape[0]][:, rows].cpu(), rs[:, :q.shape[0]][:, rows])


@pytest.mark.parametrize("act", ["silu", "gelu", "relu"])
@pytest.mark.parametrize("M,inter", [(1280, 2048), (8192, 384)])
def test_skipped_rows(M, inter, act):
    torch.manual_seed(inter)
    x = torch.randn(M, 2 * inter, device=DEV, dtype=torch.bfloat16) * 3
    tile_rows = torch.tensor([0, 1, 127, 128, 64, 33] * (M // 128), dtype=torch.int32, device=DEV)[:M // 128]
    q = torch.full((M, inter), 0x55, device=DEV, dtype=torch.uint8)
    s = torch.full((inter // 128, M), -1.0, device=DEV)
    out = torch.full((M, inter), 7.0, device=DEV, dtype=torch.bfloat16)
    native.act_mul(x, act, True, out=out, quant=True, q=q.view(torch.float8_e4m3fn), s=s, tile_rows=tile_rows)
    y = native.act_mul(x, act, True)
    rq, rs = ref.quant_fp8(y.cpu())
    held = (torch.arange(M, device=DEV) % 128 < tile_rows.repeat_interleave(128)).cpu()
    assert torch.equal(out[held.to(DEV)], y[held.to(DEV)]) and same(q, s, rq, rs, held)
    skipped = ~held
    assert bool((q.cpu()[skipped] == 0x55).all()) and bool((s.cpu()[:, skipped] == -1).all()) and bool((out.cpu()[skipped] == 7).all())


@pytest.mark.parametrize("act", ["silu", "gelu", "relu"])
@pytest.mark.parametrize("M,inter", [(5001, 640), (2639, 1152)])          # 8 and 24 lanes in the last warp
def test_last_warp(M, inter, act):
    torch.manual_seed(M)
    assert M * inter // 16 % 32
    x = torch.randn(M, 2 * inter, device=DEV, dtype=torch.bfloat16) * torch.logspace(-3, 3, M, device=DEV)[:, None].to(torch.bfloat16)
    out, q, s = native.act_mul(x, act, True, quant=True)
    rq, rs = ref.quant_fp8(out.cpu())
    want = ref.act_mul(x.float(), act, True)
    # the approximate tanh (2^-11 of the activation) and the result's own rounding
    gate, up = x.float().split(inter, -1)
    assert bool(((out.float() - want).abs() <= 2 ** -7 * want.abs() + 2 ** -10 * gate.abs() * up.abs()).all())
    assert same(q, s, rq, rs, slice(None))


@pytest.mark.parametrize("M,K,ld", [(3001, 896, 1024), (3001, 896, 904), (2500, 1280, 1280)])
def test_quantised_view(M, K, ld):
    torch.manual_seed(ld)
    x = (torch.randn(M, ld, device=DEV) * torch.logspace(-3, 3, ld, device=DEV)).to(torch.bfloat16)[:, :K]
    q, s = native.quant_fp8(x)
    rq, rs = ref.quant_fp8(x.cpu().contiguous())
    assert same(q, s, rq, rs, slice(None))


def down_to_the_smallest(M, K):
    """Rows of every magnitude that bf16 has, subnormal ones among them, and ordinary ones."""
    x = (torch.randn(M, K, device=DEV) * 10.0 ** torch.randint(-39, 3, (M, 1), device=DEV)).to(torch.bfloat16)
    x[::2] = torch.randn(M, K, device=DEV)[::2].to(torch.bfloat16) * 3
    return x


@pytest.mark.parametrize("act", ["silu", "gelu", "relu"])
@pytest.mark.parametrize("M", [1390, 1850, 1900])
def test_activation_by_either_kernel(M, act):
    """The same bits as in pieces that are too small for chunks."""
    torch.manual_seed(M)
    x = down_to_the_smallest(M, 4096)
    parts = [x[m:m + 400] for m in range(0, M, 400)]
    assert torch.equal(native.act_mul(x, act), torch.cat([native.act_mul(p, act) for p in parts]))
    _, q, s = native.act_mul(x, act, quant=True)
    pieces = [native.act_mul(p, act, quant=True) for p in parts]
    assert torch.equal(q.view(torch.uint8), torch.cat([b.view(torch.uint8) for _, b, _ in pieces]))
    assert torch.equal(s[:, :M], torch.cat([c[:, :p.shape[0]] for p, (_, _, c) in zip(parts, pieces)], 1))


def test_quantised_by_either_kernel():
    torch.manual_seed(1)
    x = down_to_the_smallest(1900, 2048)
    q, s = native.quant_fp8(x)
    pieces = [(p, *native.quant_fp8(p)) for p in x.split(400)]
    assert torch.equal(q.view(torch.uint8), torch.cat([b.view(torch.uint8) for _, b, _ in pieces]))
    assert torch.equal(s[:, :1900], torch.cat([c[:, :p.shape[0]] for p, _, c in pieces], 1))


@pytest.mark.parametrize("residual", [False, True])          # the kernel whose CTAs stay, and the other one
def test_norm_of_subnormal_numbers(residual):
    x = torch.ones(3, 4096, device=DEV, dtype=torch.bfloat16)
    x[1, 7], x[2, 9] = 2.0 ** -130, 2.0 ** -100
    w = torch.ones(4096, device=DEV, dtype=torch.bfloat16)
    w[9] = 2.0 ** -30
    y = native.norm(x, w, 1e-5, residual=torch.zeros_like(x) if residual else None)
    assert float(y[1, 7]) == 0 and float(y[2, 9]) == 0 and float(y[0, 7]) == float(y[2, 7]) != 0
