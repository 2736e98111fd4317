"""The mask maps and ALiBi slopes the binding keeps between calls, without a GPU: a fake library that only notes on which
stream a map was built and into which buffer."""
import ctypes
from collections import OrderedDict

import pytest
import torch

from flex_attention_tpu_b200 import _binding as B


class FakeLib:
    def __init__(self):
        self.built = []      # (stream, buffer)

    def flexattn_build_mask_map(self, stream, ref):
        self.built.append((stream, ctypes.cast(ref, ctypes.POINTER(B.FlexAttnParams)).contents.workspace))
        return 0


@pytest.fixture
def host(monkeypatch):
    """What stands in for the GPU: `stream` is the current stream."""
    class Host:
        lib, stream = FakeLib(), 7
    h = Host()
    monkeypatch.setattr(B, "lib", h.lib)
    monkeypatch.setattr(B, "_stream_ptr", lambda device: h.stream)
    monkeypatch.setattr(B.Problem, "_map_cache", OrderedDict())
    monkeypatch.setattr(B.Problem, "_slope_cache", OrderedDict())
    return h


def _bound(seq=256, doc_ids=None):
    """A problem with its workspace bound (what the constructor does last)."""
    prob = object.__new__(B.Problem)
    prob.device, prob.doc_ids, prob.p = torch.device("cpu"), doc_ids, B.FlexAttnParams()
    prob.p.batch, prob.p.seq_q, prob.p.seq_k, prob.p.workspace_bytes = 1, seq, seq, 512
    prob.p.mask_kind = B.MASK_CAUSAL if doc_ids is None else B.MASK_DOCUMENT
    prob._bind_workspace()
    return prob


def test_a_stream_reads_only_the_map_that_was_built_on_it(host):
    """A map is built asynchronously: a call on another stream must not find a buffer whose builder may still run."""
    a = _bound()
    again = _bound()
    host.stream = 8
    other = _bound()
    assert host.lib.built == [(7, a.p.workspace), (8, other.p.workspace)]
    assert again.p.workspace == a.p.workspace != other.p.workspace
    host.stream = 7
    assert _bound().p.workspace == a.p.workspace and len(host.lib.built) == 2


def test_the_map_not_used_for_longest_goes_first(host):
    for n in range(B.Problem._MAP_CACHE_ENTRIES):
        _bound(seq=128 * (n + 1))
    _bound(seq=128)                                                     # used again
    _bound(seq=128 * 100)                                               # one more than there is room for: seq 256 leaves
    built = len(host.lib.built)
    _bound(seq=128)
    assert len(host.lib.built) == built
    _bound(seq=256)
    assert len(host.lib.built) == built + 1


def test_document_ids_changed_in_place_give_a_new_map(host):
    ids = torch.zeros(1, 256, dtype=torch.int32)
    first = _bound(doc_ids=ids)
    assert _bound(doc_ids=ids).p.workspace == first.p.workspace
    ids[0, 128:] = 1
    assert _bound(doc_ids=ids).p.workspace != first.p.workspace and len(host.lib.built) == 2


def test_slopes_belong_to_the_stream_they_were_uploaded_on(host):
    """An evicted copy goes back to the pool of its own stream, where nothing waits for the kernels of another."""
    prob, slopes = _bound(), (0.5, 0.25)
    a = prob._device_slopes(slopes, 2)
    assert prob._device_slopes(slopes, 2) is a and a.tolist() == [0.5, 0.25]
    host.stream = 8
    b = prob._device_slopes(slopes, 2)
    assert b is not a and b.tolist() == a.tolist() and prob._device_slopes([0.5, 0.25], 2) is b
