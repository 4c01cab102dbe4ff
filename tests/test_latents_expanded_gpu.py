"""A model whose prompts attend expanded latents against the same model on the absorbed path."""
import pytest
import torch

from ksanallm_b200.ops import native

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]
DEV = "cuda"


def test_expanded_against_absorbed(monkeypatch):
    from ksanallm_b200.config import ModelConfig
    from ksanallm_b200.models.common import StepInput
    from ksanallm_b200.models.deepseek import DeepseekModel
    from ksanallm_b200.models.weights import RandomSource, build_model
    torch.manual_seed(3)
    cfg = ModelConfig(model_type="deepseek_v3", hidden_size=512, num_layers=2, num_heads=16, num_kv_heads=16, head_dim=192, intermediate_size=512,
                      vocab_size=640, rope_neox=False, max_position_embeddings=2048, max_token_len=2048, q_lora_rank=256, kv_lora_rank=512,
                      qk_nope_head_dim=128, qk_rope_head_dim=64, v_head_dim=128)
    model = build_model(cfg, RandomSource(seed=1, std=0.05), device=DEV, max_positions=2048)
    q_lens, kv_lens, bt = [600, 33, 250], [600, 97, 250], 16
    nb = [-(-n // bt) for n in kv_lens]
    table = torch.zeros(3, max(nb), dtype=torch.int32, device=DEV)
    for i in range(3):
        table[i, :nb[i]] = torch.arange(sum(nb[:i]), sum(nb[:i + 1]), device=DEV).to(torch.int32)
    pos = torch.cat([torch.arange(kv - n, kv) for n, kv in zip(q_lens, kv_lens)]).to(DEV)
    seq = torch.repeat_interleave(torch.arange(3), torch.tensor(q_lens)).to(DEV)
    slots = (table[seq, pos // bt] * bt + pos % bt).to(torch.int32)
    ids = torch.randint(0, 640, (sum(q_lens),), dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + q_lens, device=DEV).cumsum(0).to(torch.int32)
    step = StepInput(ids, pos.to(torch.int32), slots, cu, torch.tensor(kv_lens, dtype=torch.int32, device=DEV), table, num_multi=3,
                     num_tokens=sum(q_lens), num_multi_tokens=sum(q_lens), max_q_len=600, max_kv_len=600, total_kv_len=sum(kv_lens),
                     pairs=sum(n * kv - n * (n - 1) // 2 for n, kv in zip(q_lens, kv_lens)))
    got = []
    with torch.inference_mode():
        for expand in (True, False, None):
            monkeypatch.setattr(DeepseekModel, "_expands", lambda self, mw, st, T, e=expand: e is not False)
            if expand is None:                                               # no room for it: absorbed after all
                def full(*args, empty=torch.empty, **kw):
                    if args[0] == sum(kv_lens):
                        raise torch.cuda.OutOfMemoryError()
                    return empty(*args, **kw)
                monkeypatch.setattr(torch, "empty", full)
            model.allocate_kv_cache(sum(nb) + 1, bt)
            model.kv_cache.copy_(torch.randn(model.kv_cache.shape, generator=torch.Generator().manual_seed(5)).to(model.kv_cache))
            got.append((model.forward(step).float(), model.kv_cache.clone()))
            native.check_err_flag(DEV)
    assert torch.equal(got[1][0], got[2][0]) and torch.equal(got[1][1], got[2][1])
    assert torch.equal(got[0][1][:, 0], got[1][1][:, 0])                     # the first layer appends the same latents
    # two roundings of queries and keys to bf16 in other places
    assert float((got[0][0] - got[1][0]).norm() / got[1][0].norm()) < 2e-2
