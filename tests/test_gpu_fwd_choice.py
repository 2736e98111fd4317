"""Which of the two forward kernels that work through a list of query tiles the library gives a call, on both sides of the lines that
were drawn from timings with either (148 SMs)."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import workloads
from helpers import build_mods

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Sq,Sk,D,mask_kind,score_kind,window,kernel", [
    # pairs that are half empty, in calls of three, five and seven query tiles; two-query-tile / persistent, us
    (192, 384, 384, 64, "causal", "softcap", 0, "fwd_pipe"),                   # 26.0 / 23.4
    (64, 777, 777, 64, "causal", "softcap", 0, "fwd_pipe"),                    # 33 / 30
    (64, 512, 512, 64, "sliding_window_causal", "softcap", 200, "fwd_pipe"),   # 17.8 / 16.1, less than a wave
    (8, 4096, 512, 128, "sliding_window_causal", "none", 256, "fwd_pipe"),     # 15.1 / 10.6, query tiles without keys
    (16, 2048, 512, 64, "sliding_window_causal", "none", 256, "fwd_pipe"),     # 13.6 / 9.9
    (16, 3001, 3001, 128, "causal", "none", 0, "fwd_pipe"),
    (32, 2048, 2048, 64, "causal", "none", 0, "fwd_pair"),                     # 36 / 42
    (24, 1024, 1024, 128, "none", "none", 0, "fwd_pair"),                      # 23 / 27
    (96, 1024, 1024, 64, "sliding_window", "none", 1000, "fwd_pair"),          # 49 / 62
    (64, 2048, 2048, 64, "s2", "none", 1900, "fwd_pair"),                      # (dense)
    # documents
    (96, 384, 384, 64, "document", "none", 0, "fwd_pipe"),                     # 23.9 / 22.5
    (22, 2048, 2048, 64, "document", "none", 0, "fwd_pipe"),                   # 44 / 41
    (128, 384, 384, 128, "document", "none", 0, "fwd_pipe"),                   # 29.5 / 28.3
    (128, 777, 777, 128, "document", "none", 0, "fwd_pipe"),                   # 66 / 62
    (24, 1536, 1536, 64, "document", "none", 0, "fwd_pair"),                   # 36 / 42
    (96, 1024, 1024, 128, "document", "none", 0, "fwd_pair"),                  # 49 / 54
])
def test_which_forward_kernel(H, Sq, Sk, D, mask_kind, score_kind, window, kernel):
    import flex_attention_tpu_b200 as fa
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines were drawn for 148 SMs")
    B = 2 if mask_kind == "document" else 1
    q, k = (torch.zeros(B, H // B, s, D, device="cuda", dtype=torch.bfloat16) for s in (Sq, Sk))
    ids = workloads.draw_documents(np.random.default_rng(1), B, Sq, lo=64, hi=1500)[0] if mask_kind == "document" else None
    mf, bf, sf, seg = build_mods(fa, mask_kind, score_kind, window=window, stride=64, cap=20.0, doc_ids=ids)

    def call():
        fa._flex_attention_impl(q, k, k, None, seg, False, False, 0.1, 1, 128, 128, 128, False, bf, mf, sf)
        torch.cuda.synchronize()
    call()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
    names = [e.key for e in prof.key_averages() if "_sm100_kernel" in e.key]
    assert len(names) == 1 and kernel in names[0], names


@pytest.mark.parametrize("H,S,D,window,stride,kernel,fused", [
    # S2, gathered (", 6>"), against the split kernel's dense form and the separate backward kernels
    (1, 4096, 64, 64, 2, "fwd_split", False),      # forward 25.4 / 20.3
    (1, 4096, 64, 512, 3, "fwd_split", False),     # 21.9 / 20.4
    (1, 4096, 64, 512, 4, ", 6>", False),          # 19.2 / 20.5
    (1, 5000, 64, 64, 2, ", 6>", False),           # 29.4 / 35.3
    (3, 8192, 64, 64, 2, ", 6>", False),           # backward 194 / 155
    (3, 8192, 64, 64, 4, ", 6>", True),
    (3, 8192, 128, 64, 4, ", 6>", False),          # 174 / 166
    (4, 8192, 64, 64, 2, ", 6>", True),            # 201 / 223
    (6, 4096, 128, 64, 4, ", 6>", True),           # 104 / 105
])
def test_where_s2_is_gathered(H, S, D, window, stride, kernel, fused):
    import ctypes
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200 import _binding
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines were drawn for 148 SMs")
    q = torch.zeros(1, H, S, D, device="cuda", dtype=torch.bfloat16)
    call = lambda: fa.flex_attention(q, q, q, mask_fns=fa.masks.make_s2_mask_fns(128, 128, window, stride))
    call()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages() if "_sm100_kernel" in e.key]
    assert len(names) == 1 and kernel in names[0], names
    p = _binding.FlexAttnParams()
    p.batch, p.heads, p.seq_q, p.seq_k, p.head_dim, p.window, p.stride, p.mask_kind = 1, H, S, S, D, window, stride, _binding.MASK_S2
    assert (_binding.lib.flexattn_bwd_scratch_bytes(ctypes.byref(p)) > 0) == fused
