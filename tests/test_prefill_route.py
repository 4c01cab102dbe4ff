"""Which prefill attention kernel a batch takes, and the totals that decide."""
import numpy as np
import pytest
import torch

from ksanallm_b200.models.common import StepInput
from ksanallm_b200.ops import native
from ksanallm_b200.parallel.pipeline import micro_step


class Calls:
    """Stands in for the kernel library: remembers the names of the calls."""

    def __init__(self):
        self.seen = []

    def __getattr__(self, name):
        return lambda *args: self.seen.append(name) or 0


# (new tokens, keys) of the sequences, heads, whether two query tiles per CTA are the faster form (both measured, on 148 SMs)
@pytest.mark.parametrize("Hq,Hkv,batch,pair", [
    (32, 8, [(200, 200)], False), (32, 8, [(512, 512)], False), (32, 8, [(50, 50)] * 32, False), (64, 8, [(300, 300)] * 8, False),
    (40, 40, [(300, 300)] * 8, False), (28, 4, [(64, 4000)], False), (14, 2, [(300, 8000)], False), (28, 4, [(33, 1000)] * 16, False),
    (32, 8, [(64, 4000)], True), (32, 8, [(1024, 1024)], True), (32, 8, [(33, 1000)] * 16, True), (64, 8, [(5000, 5000)], True),
    (28, 4, [(5000, 5000)], True), (160, 1, [(5000, 5000)], False), (16, 16, [(20, 20)] * 15 + [(2000, 2000)], True)])
@pytest.mark.parametrize("counted", [True, False])
def test_route(monkeypatch, Hq, Hkv, batch, pair, counted):
    calls = Calls()
    monkeypatch.setattr(native, "lib", lambda: calls)
    monkeypatch.setattr(native, "_st", lambda: 0)
    monkeypatch.setattr(native, "_sms", lambda device: 148)
    if not counted and len(set(batch)) > 1:
        pytest.skip("a full block table is only a bound where lengths differ")
    D, bt, rows = 128, 16, sum(n for n, _ in batch)
    cache = torch.zeros(1, 2, Hkv, bt, D, dtype=torch.bfloat16)
    q = torch.zeros(1, Hq * D, dtype=torch.bfloat16).expand(rows, -1)
    ints = torch.zeros(1, dtype=torch.int32)
    table = ints.expand(len(batch), -(-max(kv for _, kv in batch) // bt))
    totals = dict(rows=rows, pairs=sum(n * kv - n * (n - 1) // 2 for n, kv in batch)) if counted else {}
    native.paged_prefill(q, Hq * D, q, cache, cache.stride(0), bt, table, ints, ints, len(batch), max(n for n, _ in batch), Hq, Hkv, D, 1.0,
                         **totals)
    assert calls.seen == ["ksana_paged_prefill_pair" if pair else "ksana_paged_prefill_tc"]


@pytest.mark.parametrize("a,b,num_multi", [(0, 2, 3), (1, 4, 4), (2, 4, 3), (3, 4, 3)])
def test_pairs_of_a_micro_batch(a, b, num_multi):
    q, kv = np.array([5, 2, 7, 1]), np.array([5, 9, 20, 3])
    cu = np.concatenate([[0], np.cumsum(q)])
    z = torch.zeros(int(cu[-1]), dtype=torch.int64)
    step = StepInput(input_ids=z, positions=z, slots=z, cu_q=torch.tensor(cu), kv_lens=torch.tensor(kv),
                     block_table=torch.zeros(4, 2, dtype=torch.int32), num_multi=num_multi, num_single=4 - num_multi, num_tokens=int(cu[-1]),
                     num_multi_tokens=int(cu[num_multi]), max_q_len=7, max_kv_len=20, multi_pairs=77)
    want = sum(int(k) - int(n) + i + 1 for n, k in list(zip(q, kv))[a:min(b, num_multi)] for i in range(n))
    assert micro_step(step, cu, a, b, kv).multi_pairs == want
    assert micro_step(step, cu, a, b).multi_pairs == 0
