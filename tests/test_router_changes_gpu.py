"""A router that a program changes after loading decides the next step."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def test_changed_router_is_seen():
    from ksanallm_b200.config import ModelConfig
    from ksanallm_b200.models.moe import route
    from ksanallm_b200.models.weights import RandomSource, build_model
    cfg = ModelConfig(model_type="mixtral", hidden_size=256, num_layers=1, num_heads=2, num_kv_heads=1, head_dim=128, intermediate_size=256,
                      moe_intermediate_size=128, vocab_size=64, num_experts=8, num_experts_per_tok=2, max_position_embeddings=64,
                      max_token_len=64)
    model = build_model(cfg, RandomSource(seed=5, std=0.05), device="cuda", dtype=torch.bfloat16)
    mw, x = model.layers[0].moe, torch.randn(20, 256, device="cuda", dtype=torch.bfloat16)
    first = route(model, mw, x)[0].sort(1).values.long()
    logits = x.double() @ mw.router.double().t()
    assert torch.equal(logits.topk(2).indices.sort(1).values, first)
    mw.router.neg_()
    assert torch.equal(logits.topk(2, largest=False).indices.sort(1).values, route(model, mw, x)[0].sort(1).values.long())
