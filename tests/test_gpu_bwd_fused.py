"""The fused backward (dQ, dK and dV in one pass over the tile pairs, dQ added up in an f32 scratch): every mask, both ways
dq is stored, ragged and rectangular sizes, groups and rings smaller than the problem, query tiles that no key sees, repeats."""
import ctypes
import os

import numpy as np
import pytest
import torch

import workloads

from helpers import assert_close, build_mods, make_qkvdo, oracle_hot_path, run_hot_path
from oracle import mha_reference_cpu as oracle

pytestmark = pytest.mark.gpu


def _fused(fa, q, k, v, do, l, m, o, *, sm, mods, status=None):
    """The C entry point itself, whatever the sizes: flexattn_bwd_fused with a scratch that starts as NaN."""
    from flex_attention_tpu_b200 import _binding as B
    from flex_attention_tpu_b200._resolve import make_problem
    mf, bf, sf, seg = mods
    prob = make_problem(q, k, ab=None, segment_ids=seg, causal=False, sm_scale=sm, mask_fn=mf, block_mask_fn=bf, score_fn=sf,
                        status=status)
    delta = torch.full(l.shape, float("nan"), device="cuda")
    dq, dk, dv = (torch.full_like(t, float("nan")) for t in (q, k, v))
    prob._bind(q=q, k=k, v=v, o=o, d_o=do, l=l, m=m, delta=delta, dq=dq, dk=dk, dv=dv)
    nbytes = B.lib.flexattn_bwd_scratch_bytes(ctypes.byref(prob.p)) or 64 << 20
    scratch = torch.full((nbytes // 4,), float("nan"), device="cuda")
    B.check(B.lib.flexattn_bwd_fused(B._stream_ptr(prob.device), ctypes.byref(prob.p), scratch.data_ptr(), nbytes), "flexattn_bwd_fused")
    torch.cuda.synchronize()
    return dict(dq=dq, dk=dk, dv=dv, delta=delta)


@pytest.mark.parametrize("B,H,Sq,Sk,D,mask_kind,score_kind", [
    (1, 1, 2, 3, 128, "none", "none"),                # two rows, three keys
    (1, 2, 128, 128, 64, "causal", "none"),           # one tile: its part is the first and the last
    (1, 3, 129, 257, 128, "none", "softcap"),         # remainders of one row and one key
    (2, 3, 777, 777, 64, "causal", "alibi"),          # short rows: dq stored with the last part
    (2, 3, 777, 777, 128, "causal", "softcap"),
    (1, 2, 1500, 1500, 128, "causal", "none"),        # longer rows: the finishing kernel
    (1, 2, 1500, 1500, 64, "none", "none"),
    (1, 3, 100, 1300, 128, "causal", "none"),         # kv tiles without any query: dK = dV = 0
    (1, 2, 1300, 300, 64, "sliding_window_causal", "none"),   # query tiles without any key: dq = 0
    (2, 3, 1411, 1411, 128, "sliding_window_causal", "alibi"),
    (1, 2, 900, 900, 128, "sliding_window", "none"),
    (2, 2, 1500, 1500, 128, "document", "softcap"),
    (2, 2, 1500, 1500, 64, "document", "none"),
    (1, 2, 1300, 1300, 64, "s2", "none"),
    (1, 2, 1300, 1300, 128, "s2", "alibi"),
])
def test_fused_backward(B, H, Sq, Sk, D, mask_kind, score_kind):
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), host = make_qkvdo((B, H, Sq, D), (B, H, Sk, D), 700 + Sq, torch.bfloat16)
    kw = dict(sliding_window=dict(window=300), sliding_window_causal=dict(window=200), s2=dict(window=100, stride=48)).get(mask_kind, {})
    if mask_kind == "document":
        kw["doc_ids"] = workloads.draw_documents(np.random.default_rng(Sq), B, Sq, lo=60, hi=500)[0]
    slopes = oracle.alibi_slopes(H) if score_kind == "alibi" else None
    cap = 4.0 if score_kind == "softcap" else None
    sm = 1.0 / np.sqrt(D)
    fw = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind=mask_kind, score_kind=score_kind, cap=cap or 0.0, slopes=slopes, **kw)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    mods = build_mods(fa, mask_kind, score_kind, slopes=slopes, cap=cap or 0.0, **kw)
    got = _fused(fa, q, k, v, do, fw["l"], fw["m"], fw["o"], sm=sm, mods=mods, status=status)
    assert status.tolist() == [0, 0, 0, 0]
    rows = slice(0, Sk + 199) if mask_kind == "sliding_window_causal" and Sq > Sk else slice(None)   # fully masked rows: undefined
    assert all(torch.isfinite(got[n]).all() for n in got)
    if rows.stop is not None:
        assert not got["dq"][:, :, (rows.stop + 127) // 128 * 128:].any()
        fw = {n: (t[:, :, rows] if n in ("o", "l", "m", "dq") else t) for n, t in fw.items()}
        got["dq"] = got["dq"][:, :, rows]
        # against the separate kernels: both are within one operand rounding of each other
        for n in ("dq", "dk", "dv"):
            assert float((got[n].float() - fw[n].float()).norm() / fw[n].float().norm()) < 1e-2, n
        return
    want = oracle_hot_path(*host, sm_scale=sm, mask_kind=mask_kind, score_kind=score_kind, cap=cap, slopes=slopes, **kw)
    got.update(o=fw["o"], l=fw["l"], m=fw["m"])
    assert_close(got, want, torch.bfloat16, what=f"fused {Sq}x{Sk}")
    assert torch.equal(got["delta"], fw["delta"])


@pytest.mark.parametrize("B,H,S,D,mask_kind,sums", [
    (16, 16, 640, 64, "none", 256),                   # hundreds of items a CTA walks through, dq with the last part
    (4, 70, 700, 128, "sliding_window_causal", 264),  # fewer sums than slices: a slice takes the place of one 264 before
    (1, 16, 16384, 128, "document", 9),               # ... of one nine before, in groups of three
    (4, 24, 1152, 128, "causal", 96),                 # the finishing kernel
    (5, 104, 8192, 64, "causal", 260),                # ... of two launches
])
def test_fused_backward_repeats_and_agrees(B, H, S, D, mask_kind, sums):
    """Larger problems, given to the fused backward by the library itself (sums: slices its scratch holds the f32 sums of dQ of):
    the same bits every time, and the separate kernels' results."""
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200 import _binding
    from flex_attention_tpu_b200._resolve import make_problem
    g = torch.Generator(device="cuda").manual_seed(31)
    q, k, v, do = (torch.randn((B, H, S, D), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    kw = dict(window=300) if mask_kind == "sliding_window_causal" else {}
    if mask_kind == "document":
        ids = workloads.draw_documents(np.random.default_rng(5), B, S, lo=100, hi=3000)[0]
        ids[0] = np.roll(ids[0], S // 3)              # ids that come back: compared one by one
        kw["doc_ids"] = ids
    sm = 1.0 / np.sqrt(D)
    mf, bf, _, seg = build_mods(fa, mask_kind, "none", **kw)
    prob = make_problem(q, k, ab=None, segment_ids=seg, causal=False, sm_scale=sm, mask_fn=mf, block_mask_fn=bf, score_fn=None)
    tiles = (S + 127) // 128
    launch = sums if mask_kind in ("none", "causal") else B * H   # the statistics of a launch: 1 KB a tile, and its flag
    assert prob._bwd_scratch == sums * tiles * 128 * D * 4 + launch * tiles * 1024 + -(-(launch * tiles + 1) * 4 // 256) * 256
    fw = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind=mask_kind, **kw)
    args = (q, k, v, fw["o"], fw["l"], fw["m"], do)
    outs = [fa.flex_attention_bwd(*args, segment_ids=seg, sm_scale=sm, mask_fns=None if mf is None else (mf, bf)) for _ in range(3)]
    torch.cuda.synchronize()
    _binding.raise_if_failed(q.device)
    for r in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(outs[0], r))
    assert not torch.equal(outs[0][0], fw["dq"])      # not those kernels themselves
    # dK, dV: the same operations in another order of q tiles at most; dQ: f32 sums of the same bf16 operands.  Slice by slice,
    # so that a single one that was left out cannot hide among the others.
    for n, t in zip(("dq", "dk", "dv"), outs[0]):
        for b in range(B):
            e = (t[b].float() - fw[n][b].float()).flatten(1).norm(dim=1) / fw[n][b].float().flatten(1).norm(dim=1)
            assert float(e.max()) < 2e-3, (n, b, int(e.argmax()))


@pytest.mark.parametrize("B,H,Sq,Sk,D,mask_kind,score_kind,fused", [
    (8, 16, 2048, 2048, 128, "causal", "none", True), (4, 32, 8192, 8192, 128, "sliding_window_causal", "alibi", True),
    (2, 16, 16384, 16384, 128, "document", "softcap", True), (16, 12, 512, 512, 64, "none", "none", True),
    (2, 16, 4096, 4096, 64, "s2", "none", True), (1, 12, 8192, 8192, 128, "none", "none", True), (1, 192, 1, 8192, 64, "none", "none", True),
    (1, 72, 445, 18173, 128, "causal", "alibi", True), (1, 96, 256, 256, 128, "none", "none", True),
    # one or a few query tiles against many kv tiles: every part of a query tile waits for the one before
    (1, 16, 128, 8192, 64, "none", "none", False), (1, 64, 128, 8192, 128, "none", "softcap", False),
    (1, 16, 2048, 2048, 64, "none", "none", False), (1, 16, 1280, 1280, 64, "causal", "none", False),
    # a few long rows at D = 128, short ones against shorter keys, a user function
    (1, 8, 16384, 16384, 128, "causal", "none", False), (1, 4, 32768, 32768, 128, "none", "none", False),
    (3, 24, 1277, 394, 128, "none", "none", False), (6, 32, 12544, 384, 128, "causal", "none", False), (2, 8, 1920, 1920, 128, "causal", "user", False),
    (1, 2, 384, 384, 128, "causal", "softcap", False),
])
def test_which_backward_serves_a_call(B, H, Sq, Sk, D, mask_kind, score_kind, fused):
    """The choice by sizes, on both sides of its lines, as measured on a GPU with 148 SMs."""
    from flex_attention_tpu_b200 import _binding
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines were drawn for 148 SMs")
    p = _binding.FlexAttnParams()
    p.batch, p.heads, p.seq_q, p.seq_k, p.head_dim, p.window, p.stride = B, H, Sq, Sk, D, 256, 64
    p.mask_kind, p.score_kind = _binding.MASK_KIND_IDS[mask_kind], _binding.SCORE_KIND_IDS[score_kind]
    assert (_binding.lib.flexattn_bwd_scratch_bytes(ctypes.byref(p)) > 0) == fused


def test_a_scratch_that_does_not_fit():
    """... leaves the call to the separate kernels: memory for the results, but not for the sums of dQ."""
    import flex_attention_tpu_b200 as fa
    B, H, S, D = 8, 16, 2048, 128
    (q, k, v, do), _ = make_qkvdo((B, H, S, D), (B, H, S, D), 8, torch.bfloat16)
    fw = run_hot_path(fa, q, k, v, do, sm_scale=0.09, mask_kind="causal")
    args, kw = (q, k, v, fw["o"], fw["l"], fw["m"], do), dict(sm_scale=0.09, mask_fns=fa.masks.make_causal_mask_fns(128, 128))
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.empty_cache()
    try:   # dq, dk, dv and delta take 194 MiB, the scratch 130
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (260 << 20)) / total)
        got = fa.flex_attention_bwd(*args, **kw)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    torch.cuda.synchronize()
    assert all(torch.equal(t, fw[n]) for n, t in zip(("dq", "dk", "dv"), got))
    assert not torch.equal(fa.flex_attention_bwd(*args, **kw)[0], fw["dq"])   # with room: sums in another order
