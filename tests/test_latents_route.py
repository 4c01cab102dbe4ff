"""Which form of latent attention a step of prompts takes."""
from types import SimpleNamespace

import pytest

from ksanallm_b200.models.deepseek import DeepseekModel
from ksanallm_b200.ops import native


# heads of a rank, (new tokens, keys) of the sequences, whether keys and values of every head are the faster form (both measured, on 148 SMs)
@pytest.mark.parametrize("heads,batch,expands", [
    (16, [(128, 128)], False), (32, [(128, 128)], False), (16, [(200, 4000)], False), (32, [(200, 4000)], False), (16, [(512, 8000)], False),
    (16, [(33, 1000)] * 16, False), (128, [(64, 2000)], False), (128, [(10, 3000)] * 8, False), (128, [(33, 1000)] * 16, False),
    (16, [(2, 2)], True), (16, [(300, 300)], True), (16, [(2000, 2000)], True), (16, [(40, 40)] * 8, True), (16, [(300, 1500)] * 4, True),
    (16, [(1000, 12000)], True), (32, [(512, 8000)], True), (128, [(128, 128)], True), (128, [(200, 4000)], True),
    (128, [(300, 300)] * 8, True), (128, [(1000, 12000)], True), (128, [(300, 70000)], False)])
def test_expands(monkeypatch, heads, batch, expands):
    monkeypatch.setattr(native, "_sms", lambda device: 148)
    model = SimpleNamespace(nope=128, rope=64, vdim=128, lora=512, Hq=heads, device="cuda")
    step = SimpleNamespace(num_single=0, pairs=sum(n * kv - n * (n - 1) // 2 for n, kv in batch), total_kv_len=sum(kv for _, kv in batch),
                           max_kv_len=max(kv for _, kv in batch))
    T = sum(n for n, _ in batch)
    assert DeepseekModel._expands(model, SimpleNamespace(kv_b=object()), step, T) == expands
    assert not DeepseekModel._expands(model, SimpleNamespace(kv_b=None), step, T)
