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
    """What stands in for the GPU: `stream` is the current stream, `capturing` whether it is being captured."""
    class Host:
        lib, stream, capturing = FakeLib(), 7, False
    h = Host()
    monkeypatch.setattr(B, "lib", h.lib)
    monkeypatch.setattr(B.Problem, "_graph_held", {})
    monkeypatch.setattr(B.Problem, "_map_cache", OrderedDict())
    monkeypatch.setattr(B.Problem, "_slope_cache", OrderedDict())
    return h


@pytest.fixture
def bound(host):
    def make(seq=256, doc_ids=None):
        """A problem with its workspace bound (what the constructor does last)."""
        prob = object.__new__(B.Problem)
        prob.device, prob.doc_ids, prob.p = torch.device("cpu"), doc_ids, B.FlexAttnParams()
        prob.p.workspace_bytes = 512
        kind = B.MASK_CAUSAL if doc_ids is None else B.MASK_DOCUMENT
        prob._bind_workspace(host.stream, host.capturing, (0, kind, 0, 0, 1, seq, seq))
        return prob
    return make


@pytest.fixture
def slopes_of(host, bound):
    return lambda values, heads: bound()._device_slopes(values, heads, host.stream, host.capturing)


def test_a_stream_reads_only_the_map_that_was_built_on_it(host, bound):
    """A map is built asynchronously: a call on another stream must not find a buffer whose builder may still run."""
    a = bound()
    again = bound()
    host.stream = 8
    other = bound()
    assert host.lib.built == [(7, a.p.workspace), (8, other.p.workspace)]
    assert again.p.workspace == a.p.workspace != other.p.workspace
    host.stream = 7
    assert bound().p.workspace == a.p.workspace and len(host.lib.built) == 2


def test_the_map_not_used_for_longest_goes_first(host, bound):
    for n in range(B.Problem._MAP_CACHE_ENTRIES):
        bound(seq=128 * (n + 1))
    bound(seq=128)                                                     # used again
    bound(seq=128 * 100)                                               # one more than there is room for: seq 256 leaves
    built = len(host.lib.built)
    bound(seq=128)
    assert len(host.lib.built) == built
    bound(seq=256)
    assert len(host.lib.built) == built + 1


def test_document_ids_changed_in_place_give_a_new_map(host, bound):
    ids = torch.zeros(1, 256, dtype=torch.int32)
    first = bound(doc_ids=ids)
    assert bound(doc_ids=ids).p.workspace == first.p.workspace
    ids[0, 128:] = 1
    assert bound(doc_ids=ids).p.workspace != first.p.workspace and len(host.lib.built) == 2


def test_slopes_belong_to_the_stream_they_were_uploaded_on(host, slopes_of):
    """An evicted copy goes back to the pool of its own stream, where nothing waits for the kernels of another."""
    a = slopes_of((0.5, 0.25), 2)
    assert slopes_of((0.5, 0.25), 2) is a and a.tolist() == [0.5, 0.25]
    host.stream = 8
    b = slopes_of((0.5, 0.25), 2)
    assert b is not a and b.tolist() == a.tolist() and slopes_of([0.5, 0.25], 2) is b


def test_a_map_recorded_in_a_graph_is_not_taken_for_a_finished_one(host, bound):
    """The builder of such a map runs at a replay, if there ever is one."""
    host.capturing = True
    recorded = bound()
    second_graph = bound()
    host.capturing = False
    eager = bound()
    assert [b for _, b in host.lib.built] == [recorded.p.workspace, second_graph.p.workspace, eager.p.workspace]
    assert len({b for _, b in host.lib.built}) == 3


def test_a_replay_reads_the_document_ids_it_finds(host, bound):
    """... so the builder of their map is part of every graph, also where a call before the capture has built one."""
    ids = torch.zeros(1, 256, dtype=torch.int32)
    eager = bound(doc_ids=ids)
    host.capturing = True
    recorded = bound(doc_ids=ids)
    assert recorded.p.workspace != eager.p.workspace and len(host.lib.built) == 2


def test_what_a_graph_reads_outlives_the_cache(host, bound, slopes_of, monkeypatch):
    eager, slopes = bound(), slopes_of((0.5, 0.25), 2)
    host.stream, host.capturing = 8, True                               # captured on a stream of its own
    assert bound().p.workspace == eager.p.workspace and len(host.lib.built) == 1
    assert slopes_of((0.5, 0.25), 2) is slopes
    host.capturing = False
    for n in range(2, 2 + max(B.Problem._MAP_CACHE_ENTRIES, B.Problem._SLOPE_CACHE_ENTRIES)):
        bound(seq=64 + 128 * n)
        slopes_of((float(n),), 1)
    held = [t for e in B.Problem._graph_held.values() for t in (e if isinstance(e, tuple) else (e,))]
    assert any(t is eager.workspace for t in held) and any(t is slopes for t in held)
    host.capturing = True
    assert bound().p.workspace == eager.p.workspace
    monkeypatch.setattr(B.Problem, "_GRAPH_HELD_ENTRIES", len(B.Problem._graph_held))
    host.capturing = False
    full = bound(seq=128 * 1000)
    host.capturing = True
    assert bound(seq=128 * 1000).p.workspace != full.p.workspace       # no room: the graph builds its own
