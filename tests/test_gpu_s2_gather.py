"""S2, gathered (window tiles and tiles of the keys on the stride grid): forward and fused backward against the CPU oracle where the
index sets can go wrong: windows that end inside a tile, on its edge and beyond the keys, one and several strided tiles, grids
that do not divide the length, more queries than keys and the other way round; and which calls are gathered."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from helpers import assert_close, build_mods, make_qkvdo, oracle_hot_path, run_hot_path
from oracle import mha_reference_cpu as oracle
from test_gpu_bwd_fused import _fused

pytestmark = pytest.mark.gpu


def _kernels(fn):
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if "sm100_kernel" in e.name]


@pytest.mark.parametrize("B,H,Sq,Sk,D,window,stride,score_kind", [
    (1, 2, 1152, 1152, 64, 128, 16, "none"),      # window of one tile, grid and length multiples of the tile
    (1, 2, 1300, 1300, 128, 100, 48, "alibi"),    # window inside a tile, grid that does not divide the length
    (2, 2, 2049, 2049, 64, 257, 3, "none"),       # several strided tiles, the last one of one key; one row in the last query tile
    (1, 2, 1411, 1411, 128, 1, 2, "softcap"),     # a window of one key, the densest grid
    (1, 2, 1411, 1411, 64, 64, 5000, "alibi"),    # a grid of one key
    (1, 2, 2000, 1100, 128, 150, 7, "none"),      # more queries than keys: query tiles without a window tile
    (1, 2, 1100, 2000, 64, 150, 7, "softcap"),    # kv tiles without a query, strided ones too
])
def test_gathered_s2(B, H, Sq, Sk, D, window, stride, score_kind):
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), host = make_qkvdo((B, H, Sq, D), (B, H, Sk, D), 900 + Sq, torch.bfloat16)
    slopes = oracle.alibi_slopes(H) if score_kind == "alibi" else None
    cap = 4.0 if score_kind == "softcap" else None
    kw, sm = dict(window=window, stride=stride), 1.0 / np.sqrt(D)
    hot = lambda: run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind="s2", score_kind=score_kind, cap=cap or 0.0, slopes=slopes, **kw)
    fw = hot()
    assert any("fwd_pipe" in n and ", 6>" in n for n in _kernels(hot))   # 6: the gathered form
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    mods = build_mods(fa, "s2", score_kind, slopes=slopes, cap=cap, **kw)
    bwd = lambda: _fused(fa, q, k, v, do, fw["l"], fw["m"], fw["o"], sm=sm, mods=mods, status=status)
    got = bwd()
    assert status.tolist() == [0, 0, 0, 0]
    want = oracle_hot_path(*host, sm_scale=sm, mask_kind="s2", score_kind=score_kind, cap=cap, slopes=slopes, **kw)
    got.update(o=fw["o"], l=fw["l"], m=fw["m"])
    assert_close(got, want, torch.bfloat16, what=f"gathered S2 {Sq}x{Sk}")
    again = bwd()
    assert all(torch.equal(again[n], got[n]) for n in ("dq", "dk", "dv"))
    assert any("fused" in n and ", 6, 0>" in n for n in _kernels(bwd))


@pytest.mark.parametrize("S,window,stride", [(640, 64, 16), (2048, 900, 64), (2048, 64, 1)])
def test_dense_s2(S, window, stride):
    """Short rows, wide windows and the grid of every key stay on the kernels that walk all tiles below the diagonal."""
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), _ = make_qkvdo((1, 2, S, 64), (1, 2, S, 64), 5, torch.bfloat16)
    fns = fa.masks.make_s2_mask_fns(128, 128, window, stride)
    names = _kernels(lambda: fa.flex_attention(q, k, v, mask_fns=fns))
    assert names and not any(", 6>" in n for n in names), names
