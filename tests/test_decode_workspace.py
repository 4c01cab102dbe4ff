"""Decode attention launches that may overlap have no scratch in common."""
import math

import pytest
import torch

from ksanallm_b200.ops import native



def test_a_call_without_a_workspace_has_its_own(monkeypatch):
    seen = []

    class Lib:
        def ksana_paged_decode(self, *args):
            seen.append(args[-6:-2])
            return 0

    lib = Lib()
    monkeypatch.setattr(native, "lib", lambda: lib)
    monkeypatch.setattr(native, "_st", lambda: 0)
    monkeypatch.setattr(native, "_sms", lambda device: 148)
    monkeypatch.setattr(native, "err_flag", lambda device: torch.zeros(1, dtype=torch.int32))
    kept, real = [], native._p
    monkeypatch.setattr(native, "_p", lambda t: (kept.append(t), real(t))[1])       # nothing is freed: equal addresses are one tensor
    B, Hq, Hkv, D = 3, 40, 2, 64
    q, cache = torch.zeros(B, Hq * D, dtype=torch.bfloat16), torch.zeros(4, 2, Hkv, 16, D, dtype=torch.bfloat16)
    table, kvl = torch.zeros(B, 2, dtype=torch.int32), torch.ones(B, dtype=torch.int32)
    work = native.decode_workspace("cpu")

    def call(**kw):
        native.paged_decode(q, q.stride(0), q, cache, cache.stride(0), 16, table, kvl, B, Hq, Hkv, D, 1.0, **kw)

    call()
    call()
    call(work=work)
    (s0, n0, c0, l0), (s1, n1, c1, l1), (s2, n2, c2, l2) = seen
    assert s0 != s1 and c0 != c1 and (s2, c2) == (work[0].data_ptr(), work[1].data_ptr())
    assert n0 >= 2 * 3 * 148 * 16 * (D + 2) * 4 and l0 == B * Hkv * 2               # two pieces of 16 rows per CTA; 20 heads are two groups
    assert n2 >= 2 * 2 * 148 * 16 * (256 + 2) * 4 and l2 == native.DECODE_COUNTERS
    assert native.decode_workspace("cpu")[1].data_ptr() != work[1].data_ptr() and not bool(work[1].any())


def _inputs(seed, lens, Hq=32, Hkv=8, D=128, bt=16):
    torch.manual_seed(seed)
    nb = [-(-n // bt) for n in lens]
    cache = torch.randn(sum(nb), 2, Hkv, bt, D, device="cuda", dtype=torch.bfloat16)
    table = torch.zeros(len(lens), max(nb), dtype=torch.int32, device="cuda")
    for s in range(len(lens)):
        table[s, :nb[s]] = torch.arange(sum(nb[:s]), sum(nb[:s + 1]), device="cuda")
    q = torch.randn(len(lens), Hq * D, device="cuda", dtype=torch.bfloat16)
    kvl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    outs = torch.zeros(20, len(lens), Hq * D, device="cuda", dtype=torch.bfloat16)

    def run(i, **kw):
        native.paged_decode(q, q.stride(0), outs[i], cache, cache.stride(0), bt, table, kvl, len(lens), Hq, Hkv, D, 1 / math.sqrt(D), **kw)
    return run, outs


@pytest.mark.parametrize("capture", [False, True])
@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")
def test_two_streams(capture):
    """Batches that are cut, on two streams at once, in plain launches and in graphs captured one after the other."""
    sides = [_inputs(1, [5000, 300, 900]), _inputs(2, [100 + 41 * i for i in range(40)])]
    want = []
    for run, outs in sides:
        run(0)
        torch.cuda.synchronize()
        want.append(outs[0].clone())
    streams, graphs = [torch.cuda.Stream() for _ in sides], []
    if capture:
        for run, outs in sides:
            graphs.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(graphs[-1]):
                for i in range(20):
                    run(i)
    torch.cuda.synchronize()
    for turn in range(5):
        for k, (run, outs) in enumerate(sides):
            with torch.cuda.stream(streams[k]):
                outs.zero_()
                if capture:
                    graphs[k].replay()
                else:
                    for i in range(20):
                        run(i)
        torch.cuda.synchronize()
        native.check_err_flag("cuda")
        for k in range(2):
            assert bool((sides[k][1] == want[k]).all())


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")
def test_one_workspace_in_turn():
    run, outs = _inputs(3, [4000, 10, 2000])
    run(0)
    work = native.decode_workspace("cuda")
    for i in range(1, 20):
        run(i, work=work)
    torch.cuda.synchronize()
    assert bool((outs == outs[0]).all()) and not bool(work[1].any())
