"""Calls captured into a CUDA graph: a replay reads its inputs, the document ids among them, and the mask map it was captured
with is still there after many other shapes have been run."""
import numpy as np
import pytest
import torch

from helpers import make_qkvdo

pytestmark = pytest.mark.gpu


def _step(fa, q, k, v, do, **kw):
    seg, causal = kw.get("segment_ids"), kw.get("causal", False)
    o, l, m = fa._flex_attention_impl(q, k, v, None, seg, True, causal, 0.125, 1, 128, 128, 128, False, None, None, None)
    return [o, *fa.flex_attention_bwd(q, k, v, o, l, m, do, segment_ids=seg, causal=causal, sm_scale=0.125)]


def _capture(fa, *args, **kw):
    for _ in range(2):
        _step(fa, *args, **kw)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = _step(fa, *args, **kw)
    return g, out


def test_a_replay_follows_document_ids_changed_in_place():
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), _ = make_qkvdo((2, 2, 900, 64), (2, 2, 900, 64), 41, torch.bfloat16)
    ids = torch.from_numpy(np.repeat(np.arange(3, dtype=np.int32), 300)[None].repeat(2, 0).copy()).cuda()
    g, out = _capture(fa, q, k, v, do, segment_ids=ids)
    for cut in (100, 640):
        ids.copy_((torch.arange(900, device="cuda") >= cut).to(torch.int32)[None].expand(2, -1))
        g.replay()
        want = _step(fa, q, k, v, do, segment_ids=ids.clone())
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, want)), cut


def test_a_replay_after_many_other_shapes():
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200 import _binding as B
    (q, k, v, do), _ = make_qkvdo((1, 2, 700, 64), (1, 2, 700, 64), 42, torch.bfloat16)
    g, out = _capture(fa, q, k, v, do, causal=True)
    want = [t.clone() for t in _step(fa, q, k, v, do, causal=True)]
    for n in range(1, B.Problem._MAP_CACHE_ENTRIES + 4):
        x = torch.zeros(1, 1, 64 * n, 64, device="cuda", dtype=torch.bfloat16)
        _step(fa, x, x, x, x, causal=True)
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want))


def test_a_replay_of_the_fused_backward():
    """... whose scratch belongs to the graph: other calls in between get other memory, and find none of theirs changed."""
    import flex_attention_tpu_b200 as fa
    g_ = torch.Generator(device="cuda").manual_seed(43)
    q, k, v, do = (torch.randn((16, 12, 300, 64), generator=g_, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    prob = fa._resolve.make_problem(q, k, ab=None, segment_ids=None, causal=True, sm_scale=0.125, mask_fn=None, block_mask_fn=None,
                                    score_fn=None)
    assert prob._bwd_scratch > 0
    g, out = _capture(fa, q, k, v, do, causal=True)
    want = [t.clone() for t in _step(fa, q, k, v, do, causal=True)]
    for _ in range(3):
        for t in out:
            t.fill_(float("nan"))
        other = _step(fa, do, v, k, q, causal=True)
        g.replay()
        again = _step(fa, do, v, k, q, causal=True)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, want))
        assert all(torch.equal(a, b) for a, b in zip(other, again))
