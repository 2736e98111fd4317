"""Which of the two forward kernels that work through a list of query tiles the library gives a call, on both sides of the lines that
were drawn from timings with either (148 SMs), and where S2 is gathered."""
import ctypes

import pytest
import torch

from kernel_names import forward_kernels

pytestmark = pytest.mark.gpu

# slices (batch rows x heads where more than one; documents: two rows), queries, keys, head dimension, mask, score function, window, kernel
CALLS = [
    # pairs that are half empty, in calls of three, five and seven query tiles; two-query-tile / persistent, us
    (192, 384, 384, 64, "causal", "softcap", 0, "fwd_pipe"),                   # 26.0 / 23.4
    (64, 777, 777, 64, "causal", "softcap", 0, "fwd_pipe"),                    # 33 / 30
    (64, 512, 512, 64, "sliding_window_causal", "softcap", 200, "fwd_pipe"),   # 17.8 / 16.1, less than a wave
    (8, 4096, 512, 128, "sliding_window_causal", "none", 256, "fwd_pipe"),     # 15.1 / 10.6, query tiles without keys
    (16, 2048, 512, 64, "sliding_window_causal", "none", 256, "fwd_pipe"),     # 13.6 / 9.9
    (16, 3001, 3001, 128, "causal", "none", 0, "fwd_pipe"),
    ((3, 24), 1088, 1088, 64, "causal", "softcap", 0, "fwd_pair"),             # 52 / 74: the list begins anew with every row
    ((1, 72), 1088, 1088, 64, "causal", "softcap", 0, "fwd_pipe"),
    (96, 512, 512, 64, "causal", "user", 0, "fwd_pipe"),                       # 24.1 / 21.3
    (64, 2048, 2048, 64, "causal", "user", 0, "fwd_pair"),
    (32, 2048, 2048, 64, "causal", "none", 0, "fwd_pair"),                     # 36 / 42
    (24, 1024, 1024, 128, "none", "none", 0, "fwd_pair"),                      # 23 / 27
    (96, 1024, 1024, 64, "sliding_window", "none", 1000, "fwd_pair"),          # 49 / 62
    (64, 2048, 2048, 64, "s2", "none", 1900, "fwd_pair"),                      # (dense)
    # documents
    (96, 384, 384, 64, "document", "none", 0, "fwd_pipe"),                     # 23.9 / 22.5
    (22, 2048, 2048, 64, "document", "none", 0, "fwd_pipe"),                   # 44 / 41
    ((1, 24), 1472, 1472, 128, "document", "softcap", 0, "fwd_pipe"),          # 55 / 43
    ((7, 2), 2985, 2985, 64, "document", "none", 0, "fwd_pair"),               # 40 / 45
    (128, 384, 384, 128, "document", "none", 0, "fwd_pipe"),                   # 29.5 / 28.3
    (128, 777, 777, 128, "document", "none", 0, "fwd_pipe"),                   # 66 / 62
    (24, 1536, 1536, 64, "document", "none", 0, "fwd_pair"),                   # 36 / 42
    (96, 1024, 1024, 128, "document", "none", 0, "fwd_pair"),                  # 49 / 54
]
# heads, positions, head dimension, window, stride, forward kernel, whether the fused backward serves it
S2_CALLS = [
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
]


@pytest.fixture(scope="module")
def names():
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines were drawn for 148 SMs")
    rows = lambda H, mask: H if isinstance(H, tuple) else (2, H // 2) if mask == "document" else (1, H)
    calls = [(*rows(H, mask), Sq, Sk, D, mask, score, window, 64) for H, Sq, Sk, D, mask, score, window, _ in CALLS]
    calls += [(1, H, S, S, D, "s2", "none", window, stride) for H, S, D, window, stride, _, _ in S2_CALLS]
    return forward_kernels(calls)


@pytest.mark.parametrize("i", range(len(CALLS)), ids=["-".join(map(str, c)) for c in CALLS])
def test_which_forward_kernel(names, i):
    assert len(names[i]) == 1 and CALLS[i][-1] in names[i][0], names[i]


@pytest.mark.parametrize("i", range(len(S2_CALLS)), ids=["-".join(map(str, c)) for c in S2_CALLS])
def test_where_s2_is_gathered(names, i):
    from flex_attention_tpu_b200 import _binding
    H, S, D, window, stride, kernel, fused = S2_CALLS[i]
    got = names[len(CALLS) + i]
    assert len(got) == 1 and kernel in got[0], got
    p = _binding.FlexAttnParams()
    p.batch, p.heads, p.seq_q, p.seq_k, p.head_dim, p.window, p.stride, p.mask_kind = 1, H, S, S, D, window, stride, _binding.MASK_S2
    assert (_binding.lib.flexattn_bwd_scratch_bytes(ctypes.byref(p)) > 0) == fused
