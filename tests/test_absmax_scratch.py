"""Tensor scales of NVFP4 operands: calls that overlap, on other threads or streams, share no scratch."""
import pytest
import torch

from ksanallm_b200.ops import native


@pytest.mark.parametrize("call", [lambda x: native.absmax_scale(x, 7.0), lambda x: native.norm_absmax(x, x[0], 1e-5, 7.0),
                                  lambda x: native.act_mul_absmax(x, "silu", 7.0)])
def test_overlapping_calls(monkeypatch, call):
    x, scratch = torch.ones(4, 32, dtype=torch.bfloat16), []

    class Lib:
        def __getattr__(self, name):
            def f(*args):
                scratch.append((args[-4], args[-2]))        # the CTAs' maxima, the scale
                if len(scratch) < 3:
                    call(x)                          # another thread's call, while this one is still running
                return 0
            return f

    monkeypatch.setattr(native, "lib", lambda: Lib())
    monkeypatch.setattr(native, "_st", lambda: 0)
    monkeypatch.setattr(native, "_sms", lambda device: 148)
    call(x)
    places = [p.value if hasattr(p, "value") else p for pair in scratch for p in pair]
    assert len(places) == 6 == len(set(places))


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")
def test_two_streams():
    streams, sizes = [torch.cuda.Stream() for _ in range(2)], [1.0, 64.0]
    x = [torch.full((3000, 4096), v, device="cuda", dtype=torch.bfloat16) for v in sizes]
    w = torch.ones(4096, device="cuda", dtype=torch.bfloat16)
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(40):
        for s in (0, 1):
            with torch.cuda.stream(streams[s]):
                a = native.absmax_scale(x[s], 2.0)
                n = native.norm_absmax(x[s], w * sizes[s], 0.0, 2.0)[1]
                g = native.act_mul_absmax(x[s], "relu", 2.0)[1]
                got[s].append(torch.stack([a, n, g]))
    torch.cuda.synchronize()
    for s in (0, 1):
        # x / rms(x) is 1 but for the approximate root (2^-22): rounded to bf16, 1 times w
        want = torch.tensor([sizes[s], sizes[s], sizes[s] ** 2], device="cuda") / 2
        assert bool((torch.stack(got[s]) == want).all())
