"""GEMMs whose weight operand the launch before them writes: such a launch must not request it early."""
import pytest
import torch

from ksanallm_b200.ops import dispatch, native, reference as ref


class Calls:
    """Stands in for the kernel library: remembers every call."""

    def __init__(self):
        self.seen = []

    def __getattr__(self, name):
        def call(*args):
            self.seen.append((name, args))
            return 0
        return call


@pytest.fixture
def calls(monkeypatch):
    c = Calls()
    monkeypatch.setattr(native, "lib", lambda: c)
    monkeypatch.setattr(native, "_st", lambda: 0)
    monkeypatch.setattr(native, "err_flag", lambda device: torch.zeros(1, dtype=torch.int32))
    monkeypatch.setattr(native, "gemm_workspace", lambda device: (torch.zeros(4), torch.zeros(4, dtype=torch.int32)))
    return c


FIXED = {"ksana_gemm_decode": -3, "ksana_gemm_smallm": -3}       # place of the argument that vouches for the weights


@pytest.mark.parametrize("M", [33, 64, 65, 128])
def test_expanded_four_bit_weights_are_not_vouched_for(calls, M):
    N, K, group = 48, 64, 32                                      # groups of 32: expanded, then multiplied
    q4, scale, zs = ref.quant_w4(torch.randn(N, K), group)
    native.linear_w4(torch.randn(M, K).to(torch.bfloat16), q4, scale, zs)
    (first, a), (second, b) = calls.seen
    assert first == "ksana_w4_dequant" and second in FIXED
    assert a[3] == b[5]                                           # the GEMM reads what the launch before it writes
    assert b[FIXED[second]] == 0


@pytest.mark.parametrize("M", [1, 64, 100])
def test_only_the_caller_vouches(calls, M):
    x, w = torch.zeros(M, 64, dtype=torch.bfloat16), torch.zeros(32, 64, dtype=torch.bfloat16)
    native.gemm_bf16(x, w)
    native.gemm_bf16(x, w, fixed_w=True)
    assert [a[FIXED[n]] for n, a in calls.seen] == [0, 1]


def test_linear_layers_vouch_for_loaded_weights(calls, monkeypatch):
    monkeypatch.setattr(dispatch, "_is_cuda", lambda x: True)
    x = torch.zeros(4, 64, dtype=torch.bfloat16)
    dispatch.linear(x, dispatch.LinearWeight(w=torch.zeros(32, 64, dtype=torch.bfloat16)))
    dispatch.linear(x, dispatch.LinearWeight(w=torch.zeros(32, 64, dtype=torch.bfloat16)), out_f32=True)
    assert [a[FIXED[n]] for n, a in calls.seen] == [1, 1]


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")
@pytest.mark.parametrize("M", [33, 50, 64, 65, 128])
def test_layers_that_share_the_expanded_matrix(M):
    """Two layers of groups of 32 in turn, both expanded into the same scratch matrix."""
    N, K = 512, 2080
    torch.manual_seed(M)
    layers = [ref.quant_w4(torch.randn(N, K, device="cuda") * s, 32) for s in (0.05, 2.0)]
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    ys = [native.linear_w4(x, *layers[i % 2]) for i in range(8)]
    native.check_err_flag("cuda")
    for i, y in enumerate(ys):
        dense = ref.dequant_w4(*layers[i % 2]).to(torch.bfloat16).double()
        want, sums = x.double() @ dense.t(), x.double().abs() @ dense.abs().t()
        # fp32 sums (2^-24 of the magnitudes per K block and share) of exact products, the result rounded to bf16
        assert bool(((y.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -18 * sums).all())
        assert torch.equal(y, ys[i % 2])
