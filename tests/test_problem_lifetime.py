"""What a problem keeps alive, without a GPU: a fake library in the place of the kernels."""
import gc
import weakref

import pytest
import torch

from flex_attention_tpu_b200 import _binding as B
from flex_attention_tpu_b200.flex_attention import _FlexAttentionFn


class FakeLib:
    def flexattn_fwd(self, stream, ref):
        return 0

    def flexattn_bwd(self, stream, side, ref):
        return 0


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
