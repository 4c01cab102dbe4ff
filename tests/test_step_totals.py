"""Key and pair totals of a step and of its pipeline micro-batches, which choose the form of latent attention."""
import numpy as np
import pytest
import torch

from ksanallm_b200.models.common import StepInput
from ksanallm_b200.parallel.pipeline import micro_step


@pytest.mark.parametrize("a,b,num_multi", [(0, 2, 4), (1, 4, 4), (3, 4, 4), (0, 4, 4), (2, 4, 3)])
def test_micro_batch_totals(a, b, num_multi):
    q, kv = np.array([5, 1, 7, 3]), np.array([5, 9, 20, 3])
    cu = np.concatenate([[0], np.cumsum(q)])
    T = int(cu[-1])
    pairs = [sum(int(k) - int(n) + i + 1 for i in range(n)) for n, k in zip(q, kv)]
    z = torch.zeros(T, dtype=torch.int64)
    step = StepInput(input_ids=z, positions=z, slots=z, cu_q=torch.tensor(cu), kv_lens=torch.tensor(kv),
                     block_table=torch.zeros(4, 2, dtype=torch.int32), num_multi=num_multi, num_single=4 - num_multi, num_tokens=T,
                     num_multi_tokens=int(cu[num_multi]), max_q_len=7, max_kv_len=20, total_kv_len=int(kv.sum()), pairs=sum(pairs))
    sub = micro_step(step, cu, a, b, kv)
    whole = sub.num_single == 0
    assert sub.total_kv_len == (int(kv[a:b].sum()) if whole else 0)
    assert sub.pairs == (sum(pairs[a:b]) if whole else 0)
    assert micro_step(step, cu, a, b).pairs == 0
