"""What a problem keeps alive, and which backward it calls, without a GPU: a fake library in the place of the kernels."""
import gc
import weakref

import pytest
import torch

from flex_attention_tpu_b200 import _binding as B
from flex_attention_tpu_b200.flex_attention import _FlexAttentionFn


class FakeLib:
    fused_status = 0

    def __init__(self):
        self.calls = []

    def flexattn_fwd(self, stream, ref):
        return 0

    def flexattn_bwd(self, stream, side, ref):
        self.calls.append("separate")
        return 0

    def flexattn_bwd_fused(self, stream, ref, scratch, nbytes):
        self.calls.append("fused")
        return self.fused_status

    def flexattn_status_string(self, code):
        return b"a status"


@pytest.fixture
def prob(monkeypatch):
    monkeypatch.setattr(B, "lib", FakeLib())
    monkeypatch.setattr(B, "_stream_ptr", lambda device: 7)
    monkeypatch.setattr(B, "TWO_STREAM_BACKWARD", False)
    p = object.__new__(B.Problem)
    monkeypatch.setattr(torch.Tensor, "get_device", lambda t: None)   # what a CPU device's index is
    p.device, p.dtype, p.shape_q, p.shape_k = torch.device("cpu"), torch.bfloat16, (1, 2, 8, 64), (1, 2, 8, 64)
    p.p, p._keep, p.ab = B.FlexAttnParams(), {}, None
    return p


def test_a_training_step_leaves_nothing_for_the_garbage_collector(prob):
    """The graph of an output holds the problem, so a problem that held the output (or the gradients) would keep both, step
    after step, until a collection happened to run."""
    q, k, v = (torch.randn(1, 2, 8, 64, dtype=torch.bfloat16, requires_grad=True) for _ in range(3))
    gc.disable()
    try:
        o = _FlexAttentionFn.apply(q, k, v, None, prob)
        grads = torch.autograd.grad(o, (q, k, v), torch.ones_like(o))
        gone = [weakref.ref(t) for t in (o, *grads)]
        del o, grads
        assert [r() is None for r in gone] == [True] * 4
    finally:
        gc.enable()


def _backward(prob):
    t = torch.zeros(1, 2, 8, 64, dtype=torch.bfloat16)
    r = torch.zeros(1, 2, 8)
    return prob.backward(t, t, t, t, t, r, r)


def test_a_backward_whose_scratch_does_not_fit_runs_the_separate_kernels(prob, monkeypatch):
    """A call fits where its operands and results do: those kernels take no scratch."""
    empty = torch.empty
    prob._bwd_scratch = 12345
    _backward(prob)

    def full(size, **kw):
        if size == 12345:
            raise torch.OutOfMemoryError("no room")
        return empty(size, **kw)
    monkeypatch.setattr(torch, "empty", full)
    assert [tuple(t.shape) for t in _backward(prob)] == [(1, 2, 8)] + 3 * [(1, 2, 8, 64)]
    assert B.lib.calls == ["fused", "separate"]


def test_a_fused_backward_that_was_not_built_for_the_call(prob):
    prob._bwd_scratch = 256
    B.lib.fused_status = 13                 # a user score function it cannot be compiled around
    assert len(_backward(prob)) == 4 and B.lib.calls == ["fused", "separate"]
    B.lib.fused_status = 8
    with pytest.raises(B.FlexAttnError):
        _backward(prob)
    assert B.lib.calls == ["fused", "separate", "fused"]
