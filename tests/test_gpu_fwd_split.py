"""The split forward kernel (a cluster of CTAs per query tile, merged through distributed shared memory), which serves few
query tiles against many keys: one row to several tiles, every cluster size, chunks of unequal length, rows past the end,
masks whose chunks are partly or wholly outside a row's range, and the residuals l and m the backward rebuilds p from."""
import numpy as np
import pytest
import torch

from helpers import assert_close, make_qkvdo, oracle_hot_path, run_hot_path
from oracle import mha_reference_cpu as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,Sq,Sk,D,mask_kind,score_kind", [
    (1, 2, 1, 8191, 128, "none", "none"),             # one row, 64 kv tiles over 8 CTAs
    (2, 18, 1, 2050, 64, "none", "softcap"),          # 4 CTAs, last tile two columns wide
    (2, 30, 33, 1665, 128, "none", "none"),           # 2 CTAs, chunks of 7 and 7 tiles, a second warp with one row
    (5, 40, 6, 1640, 64, "none", "alibi"),            # more query tiles than clusters of two: one CTA each
    (5, 40, 32, 1640, 128, "none", "none"),           # ... and the most rows of a query tile that still takes it
    (5, 40, 128, 1640, 64, "none", "alibi"),          # ... a full query tile does not: the persistent kernel
    (1, 3, 300, 2500, 64, "none", "none"),            # three query tiles, the last one ragged
    (1, 2, 3200, 3200, 128, "causal", "none"),        # causal: chunks of 0 to 13 tiles per CTA and stream
    (1, 2, 3175, 3175, 64, "causal", "alibi"),
    (1, 2, 2499, 2499, 64, "sliding_window", "none"),
    (1, 1, 3111, 3111, 128, "s2", "softcap"),
    (1, 2, 2500, 2500, 64, "sliding_window_causal", "none"),
])
def test_split_forward(B, H, Sq, Sk, D, mask_kind, score_kind):
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), host = make_qkvdo((B, H, Sq, D), (B, H, Sk, D), 900 + Sq, torch.bfloat16)
    kw = dict(sliding_window=dict(window=700), sliding_window_causal=dict(window=1700), s2=dict(window=100, stride=48)).get(mask_kind, {})
    slopes = oracle.alibi_slopes(H) if score_kind == "alibi" else None
    cap = 4.0 if score_kind == "softcap" else None
    sm = 1.0 / np.sqrt(D)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    got = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind=mask_kind, score_kind=score_kind, cap=cap or 0.0, slopes=slopes,
                       status=status, **kw)
    assert status.tolist() == [0, 0, 0, 0]
    simt = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind=mask_kind, score_kind=score_kind, cap=cap or 0.0, slopes=slopes,
                        backend="simt", **kw)
    # what the forward returns (o, l, m) against the f32 kernels on the same inputs, both stored in bf16; where it is quick
    # the gradients rebuilt from l and m as well, against the oracle
    assert_close(got, simt, torch.bfloat16, names=("o",), what=f"split {Sq}x{Sk} vs simt", roundings=2)
    if Sq * Sk <= 3_000_000 and B * H <= 40:
        want = oracle_hot_path(*host, sm_scale=sm, mask_kind=mask_kind, score_kind=score_kind, cap=cap, slopes=slopes, **kw)
        assert_close(got, want, torch.bfloat16, what=f"split {Sq}x{Sk}")


@pytest.mark.parametrize("B,H,Sq,Sk,D,mask_kind,kernel", [
    (1, 2, 1, 8191, 128, "none", "fwd_split"), (5, 40, 6, 1640, 64, "none", "fwd_split"), (5, 40, 32, 1640, 128, "none", "fwd_split"),
    (1, 2, 3200, 3200, 128, "causal", "fwd_split"), (1, 2, 2500, 2500, 64, "sliding_window_causal", "fwd_split"),
    (5, 40, 128, 1640, 64, "none", "fwd_pipe"), (5, 40, 33, 1640, 64, "none", "fwd_pipe"), (1, 2, 1, 1024, 64, "none", "fwd_pipe"),
    (2, 16, 4096, 4096, 64, "causal", "fwd_pair"),
])
def test_which_forward_kernel_serves_a_call(B, H, Sq, Sk, D, mask_kind, kernel):
    """The cases above, and those of the other kernels, mean nothing if the choice moves: the name of what was launched."""
    import flex_attention_tpu_b200 as fa
    from helpers import build_mods
    from torch.profiler import ProfilerActivity, profile
    q, k = (torch.zeros(B, H, s, D, device="cuda", dtype=torch.bfloat16) for s in (Sq, Sk))
    mf, bf, _, _ = build_mods(fa, mask_kind, "none", window=1700)

    def call():
        fa._flex_attention_impl(q, k, k, None, None, False, False, 0.1, 1, 128, 128, 128, False, bf, mf, None)
        torch.cuda.synchronize()
    call()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
    names = [e.key for e in prof.key_averages() if "_sm100_kernel" in e.key]
    assert len(names) == 1 and kernel in names[0], names
