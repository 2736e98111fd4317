"""The two-query-tile forward where its CTAs take pair after pair: several hundred pairs a launch whose streams start and end
apart (odd tile counts, windows, documents, query tiles without a key, pairs without any), against the CUDA-core backend, twice
over; and that the library gives it these calls itself."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import workloads
from helpers import assert_close, make_qkvdo, run_hot_path
from oracle import mha_reference_cpu as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Sq,Sk,D,mask_kind,score_kind", [
    (8, 60, 129, 129, 64, "causal", "none"),            # pairs of a full tile and one row
    (6, 64, 640, 640, 128, "causal", "alibi"),          # five tiles: the last pair has one stream; keys from the last tile down
    (3, 200, 200, 50, 128, "none", "softcap"),          # one kv tile, partial
    (5, 90, 700, 700, 64, "sliding_window_causal", "none"),   # streams that start a tile apart
    (2, 140, 900, 300, 128, "sliding_window_causal", "none"),  # query tiles and whole pairs without keys: zeros
    (4, 70, 1000, 1000, 64, "document", "none"),        # ranges that end inside a pair
    (4, 70, 1000, 1000, 128, "document", "softcap"),
    (2, 30, 3100, 3100, 64, "sliding_window", "none"),  # long rows, groups of heads
])
def test_many_pairs(B, H, Sq, Sk, D, mask_kind, score_kind):
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), _ = make_qkvdo((B, H, Sq, D), (B, H, Sk, D), 40 + Sq, torch.bfloat16)
    kw = dict(window=150) if "window" in mask_kind else {}
    if mask_kind == "document":
        kw["doc_ids"] = workloads.draw_documents(np.random.default_rng(Sq), B, Sq, lo=30, hi=400)[0]
        kw["doc_ids"][0] = np.roll(kw["doc_ids"][0], Sq // 3)   # ids that come back
    slopes = oracle.alibi_slopes(H) if score_kind == "alibi" else None
    args = dict(sm_scale=1.0 / np.sqrt(D), mask_kind=mask_kind, score_kind=score_kind, cap=5.0 if score_kind == "softcap" else 0.0, slopes=slopes, **kw)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    hot = lambda: run_hot_path(fa, q, k, v, do, status=status, **args)
    got = hot()
    assert status.tolist() == [0, 0, 0, 0]
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        again = hot()
        torch.cuda.synchronize()
    assert any("fwd_pair" in e.name for e in prof.events())
    assert all(torch.equal(got[n], again[n]) for n in ("o", "l", "m"))
    simt = run_hot_path(fa, q, k, v, do, backend="simt", **args)
    rows = slice(None)
    if mask_kind == "sliding_window_causal" and Sq > Sk:   # fully masked rows are undefined, a tile of them is zero
        rows = slice(0, Sk + 149)
        assert not got["o"][:, :, (rows.stop + 127) // 128 * 128:].any()
    cut = lambda r: {n: r[n][:, :, rows] for n in ("o", "l", "m")}
    assert_close(cut(got), cut(simt), torch.bfloat16, names=("o",), what=f"pairs {mask_kind} {Sq}x{Sk}", roundings=2)
