"""Forms of the kernels that larger calls reach and that the choice by sizes gives no small call of the other tests: dense S2 through the
fused backward (both ways dQ leaves) and through the split forward, the persistent forward with several items a CTA under every mask,
and gathered S2 over several launches and in the bounds-checked build."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest
import torch

from helpers import assert_close, build_mods, make_qkvdo, oracle_hot_path, run_hot_path
from kernel_names import forward_kernels
from oracle import mha_reference_cpu as oracle
from test_gpu_bwd_fused import _fused

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("B,H,S,D,window,stride,score_kind", [
    (1, 2, 1500, 64, 900, 64, "none"),       # twelve kv tiles: dQ left to the finishing kernel
    (1, 2, 1411, 128, 900, 48, "alibi"),
    (2, 2, 1000, 64, 700, 32, "softcap"),    # eight: dQ stored with the last part
    (1, 2, 900, 128, 500, 7, "none"),
])
def test_dense_s2_through_the_fused_backward(B, H, S, D, window, stride, score_kind):
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), host = make_qkvdo((B, H, S, D), (B, H, S, D), 80 + S, torch.bfloat16)
    slopes = oracle.alibi_slopes(H) if score_kind == "alibi" else None
    cap = 4.0 if score_kind == "softcap" else None
    kw, sm = dict(window=window, stride=stride), 1.0 / np.sqrt(D)
    fw = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind="s2", score_kind=score_kind, cap=cap or 0.0, slopes=slopes, **kw)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    mods = build_mods(fa, "s2", score_kind, slopes=slopes, cap=cap or 0.0, **kw)
    got = _fused(fa, q, k, v, do, fw["l"], fw["m"], fw["o"], sm=sm, mods=mods, status=status)
    assert status.tolist() == [0, 0, 0, 0]
    tiles = -(-S // 128)
    assert not 1.2 * (window / 128 + 2 + tiles / (2 * stride)) < 0.5 * (tiles + 1)   # (the line beyond which it would be gathered)
    want = oracle_hot_path(*host, sm_scale=sm, mask_kind="s2", score_kind=score_kind, cap=cap, slopes=slopes, **kw)
    got.update(o=fw["o"], l=fw["l"], m=fw["m"])
    assert_close(got, want, torch.bfloat16, what=f"dense S2, fused {S}")


@pytest.mark.parametrize("S,D,score_kind", [(3111, 128, "softcap"), (3300, 64, "none")])
def test_dense_s2_through_the_split_forward(S, D, score_kind):
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), _ = make_qkvdo((1, 1, S, D), (1, 1, S, D), 90 + S, torch.bfloat16)
    args = dict(sm_scale=1.0 / np.sqrt(D), mask_kind="s2", score_kind=score_kind, cap=4.0, window=1500, stride=48)
    hot = lambda backend: run_hot_path(fa, q, k, v, do, backend=backend, **args)
    (name,), = forward_kernels([(1, 1, S, S, D, "s2", score_kind, 1500, 48)])
    assert "fwd_split" in name
    assert_close(hot("tcgen05"), hot("simt"), torch.bfloat16, names=("o",), what=f"dense S2, split {S}", roundings=2)


CHILD = textwrap.dedent("""
    import sys
    sys.path.insert(0, %r); sys.path.insert(0, %r)
    import numpy as np, torch
    import flex_attention_tpu_b200 as fa
    from helpers import assert_close, make_qkvdo, run_hot_path
    from oracle import mha_reference_cpu as oracle
    # 160 to 960 query tiles of one to eight kv tiles: several items a CTA, which walks them as one stream
    cases = [("none", "none", 4, 64, 256, 640, 128), ("none", "softcap", 2, 80, 130, 300, 64), ("document", "softcap", 4, 48, 500, 500, 128),
             ("document", "none", 4, 40, 900, 900, 128), ("document", "none", 4, 30, 700, 700, 64), ("sliding_window_causal", "alibi", 4, 48, 500, 500, 128),
             ("sliding_window_causal", "none", 2, 60, 900, 400, 64), ("sliding_window", "none", 4, 48, 500, 500, 64), ("causal", "none", 5, 96, 384, 384, 64),
             ("causal", "alibi", 3, 50, 1000, 1000, 128), ("s2", "none", 4, 48, 500, 500, 128)]
    for mask, score, B, H, Sq, Sk, D in cases:
        (q, k, v, do), _ = make_qkvdo((B, H, Sq, D), (B, H, Sk, D), 21 + Sq, torch.bfloat16)
        doc = oracle.draw_documents(np.random.default_rng(3), B, Sq, lo=60, hi=300)[0] if mask == "document" else None
        if doc is not None:
            doc[0] = np.roll(doc[0], Sq // 3)      # ids that come back
        args = dict(sm_scale=1.0 / np.sqrt(D), mask_kind=mask, score_kind=score, doc_ids=doc, cap=6.0,
                    slopes=oracle.alibi_slopes(H) if score == "alibi" else None, window=200, stride=32)
        st = torch.zeros(4, dtype=torch.int32, device="cuda")
        got = run_hot_path(fa, q, k, v, do, backend="tcgen05", status=st, **args)
        assert st.tolist() == [0, 0, 0, 0], (mask, score, st.tolist())
        want = run_hot_path(fa, q, k, v, do, backend="simt", **args)
        rows = slice(0, Sk + 199) if mask == "sliding_window_causal" else slice(None)      # beyond: rows without a key, undefined
        cut = lambda r: {n: r[n][:, :, rows] for n in ("o", "l", "m")}
        assert_close(cut(got), cut(want), torch.bfloat16, names=("o",), what=f"persistent {mask}/{score} {Sq}x{Sk} D{D}", roundings=2)
        ok = torch.isfinite(want["m"][:, :, rows])
        lse = lambda r: (r["m"].double() + r["l"].double().log())[:, :, rows]
        # l sums f32 exponentials of f32 scores in both; tanh.approx, with softcap, is within 2^-10.9, times the cap of 6: 3e-3
        assert float((lse(got) - lse(want))[ok].abs().max()) < 4e-3, (mask, score)
    print("RARE_OK")
""")


def test_persistent_forward_with_several_items_a_cta():
    """Forced, as the library gives most such calls to the two-query-tile kernel."""
    r = subprocess.run([sys.executable, "-c", CHILD % (ROOT, os.path.join(ROOT, "tests"))], capture_output=True, text=True, timeout=900,
                       env=dict(os.environ, FLEXATTN_FWD_KERNEL="pipe"))
    assert r.returncode == 0 and "RARE_OK" in r.stdout, r.stdout[-3000:] + r.stderr[-3000:]


def test_gathered_s2_of_two_launches():
    """The sums of 128 slices, two a query tile, take 1 GiB, the limit of a launch, without the rows of the strided keys: the second launch's
    slices begin at 64.  Slice by slice against the separate kernels, which walk every tile below the diagonal."""
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200._resolve import make_problem
    B, H, S, D, sm = 4, 32, 8192, 128, 128 ** -0.5
    g = torch.Generator(device="cuda").manual_seed(32)
    q, k, v, do = (torch.randn((B, H, S, D), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    mf, bf = fa.masks.make_s2_mask_fns(128, 128, 128, 48)
    prob = make_problem(q, k, ab=None, segment_ids=None, causal=False, sm_scale=sm, mask_fn=mf, block_mask_fn=bf, score_fn=None)
    assert B * H * 2 * (S // 128) * 128 * D * 4 == 1 << 30 and 0 < prob._bwd_scratch < 1 << 30
    fw = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind="s2", window=128, stride=48)
    args = (q, k, v, fw["o"], fw["l"], fw["m"], do)
    backward = lambda: fa.flex_attention_bwd(*args, sm_scale=sm, mask_fns=(mf, bf))
    got = backward()
    assert all(torch.equal(a, b) for a, b in zip(got, backward()))
    for n, t in zip(("dq", "dk", "dv"), got):
        for b in range(B):   # (as in test_gpu_bwd_fused.py: f32 sums of the same bf16 operands)
            e = (t[b].float() - fw[n][b].float()).flatten(1).norm(dim=1) / fw[n][b].float().flatten(1).norm(dim=1)
            assert float(e.max()) < 2e-3, (n, b, int(e.argmax()))


DEBUG_CHILD = textwrap.dedent("""
    import sys
    sys.path.insert(0, %r); sys.path.insert(0, %r)
    import numpy as np, torch
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200 import _binding as B
    from helpers import assert_close, build_mods, make_qkvdo, oracle_hot_path, run_hot_path
    from oracle import mha_reference_cpu as oracle
    assert B.DEBUG_BUILD
    for score, H, Sq, Sk, D, window, stride in [("none", 2, 1300, 1300, 64, 100, 48), ("alibi", 2, 2049, 2049, 128, 257, 5), ("softcap", 1, 1411, 1411, 128, 1, 2),
                                                ("none", 2, 2000, 1100, 64, 150, 7), ("none", 2, 1100, 2000, 128, 150, 5000)]:
        (q, k, v, do), host = make_qkvdo((1, H, Sq, D), (1, H, Sk, D), 5, torch.bfloat16)
        slopes = oracle.alibi_slopes(H) if score == "alibi" else None
        kw, sm = dict(window=window, stride=stride), 1.0 / np.sqrt(D)
        st = torch.zeros(4, dtype=torch.int32, device="cuda")
        got = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind="s2", score_kind=score, backend="tcgen05", cap=6.0, slopes=slopes, status=st, **kw)
        mf, bf, sf, _ = build_mods(fa, "s2", score, cap=6.0, slopes=slopes, **kw)
        got["dq"], got["dk"], got["dv"] = fa.flex_attention_bwd(q, k, v, got["o"], got["l"], got["m"], do, sm_scale=sm, mask_fns=(mf, bf), score_fn=sf)
        torch.cuda.synchronize()
        assert st.tolist() == [0, 0, 0, 0] and B._mailbox(q.device).tolist() == [0, 0, 0, 0], (score, st.tolist(), B._mailbox(q.device).tolist())
        want = oracle_hot_path(*host, sm_scale=sm, mask_kind="s2", score_kind=score, cap=6.0, slopes=slopes, **kw)
        assert_close(got, want, torch.bfloat16, what=f"debug build, gathered S2 {score} {Sq}x{Sk}")
    print("RARE_OK")
""")


def test_gathered_s2_in_the_bounds_checked_build():
    r = subprocess.run([sys.executable, "-c", DEBUG_CHILD % (ROOT, os.path.join(ROOT, "tests"))], capture_output=True, text=True, timeout=900,
                       env=dict(os.environ, FLEXATTN_DEBUG="1", FLEXATTN_BWD_KERNEL="fused"))
    assert r.returncode == 0 and "RARE_OK" in r.stdout, r.stdout[-3000:] + r.stderr[-3000:]
