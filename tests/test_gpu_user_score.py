"""User score functions on the GPU: a Python function traced by make_jax_score_fn, compiled into the tensor-core
forward, dQ and dK/dV kernels at run time, against the CPU oracle evaluating the SAME expression tree (and its
symbolic derivative) with NumPy."""
import numpy as np
import pytest
import torch

from helpers import assert_close, build_mods, errors, make_qkvdo, oracle_hot_path, run_hot_path
from oracle import mha_reference_cpu as oracle

pytestmark = pytest.mark.gpu


def _softcap(s, b, h, qi, ki):
    return 8.0 * np.tanh(s / 8.0)


def _distance_and_head(s, b, h, qi, ki):
    return s - 0.03 * (h + 1) * abs(qi - ki) + 0.25 * b


def _reference_form(q_tile, k_tile):
    from flex_attention_tpu_b200 import score_expr as se
    x = q_tile @ k_tile.T
    return se.where(x >= 0.0, x, 0.5 * x) + 0.1 * se.sigmoid(x)


# (all on the persistent forward kernel: the two-query-tile one takes long rows of many slices, and is forced around a user
# function in test_gpu_fwd_kernels.py)
CASES = [("softcap", _softcap, "causal", 128, 777), ("distance", _distance_and_head, "none", 128, 500),
         ("distance", _distance_and_head, "document", 64, 700), ("leaky", _reference_form, "sliding_window_causal", 128, 640),
         ("distance", _distance_and_head, "none", 128, 1700), ("softcap", _softcap, "causal", 64, 3300)]


@pytest.mark.parametrize("name,fn,mask_kind,D,S", CASES)
def test_user_score_matches_the_oracle(name, fn, mask_kind, D, S):
    import flex_attention_tpu_b200 as fa
    B, H = (2, 3) if S < 1500 else (1, 2)
    (q, k, v, do), host = make_qkvdo((B, H, S, D), (B, H, S, D), 1200 + S, torch.bfloat16)
    sf = fa.util.make_jax_score_fn(fn)
    doc = oracle.draw_documents(np.random.default_rng(5), B, S, lo=60, hi=300)[0] if mask_kind == "document" else None
    window = 200 if mask_kind == "sliding_window_causal" else 0
    sm = 1.0 / np.sqrt(D)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    got = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind=mask_kind, score_kind="user", user_fn=sf, backend="tcgen05",
                       window=window, doc_ids=doc, status=status)
    assert status.tolist() == [0, 0, 0, 0], status.tolist()
    want = oracle_hot_path(*host, sm_scale=sm, mask_kind=mask_kind, score_kind="user", user=(sf, sf.dscore),
                           window=window or None, doc_ids=doc)
    assert_close(got, want, torch.bfloat16, what=f"user score {name}/{mask_kind}/D{D}")


def test_user_softcap_agrees_with_the_built_in_functor():
    import flex_attention_tpu_b200 as fa
    (q, k, v, do), _ = make_qkvdo((1, 4, 512, 128), (1, 4, 512, 128), 1300, torch.bfloat16)
    sm = 1.0 / np.sqrt(128)
    a = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind="causal", score_kind="user", backend="tcgen05",
                     user_fn=lambda s, b, h, qi, ki: 8.0 * np.tanh(s / 8.0))
    b_ = run_hot_path(fa, q, k, v, do, sm_scale=sm, mask_kind="causal", score_kind="softcap", cap=8.0, backend="tcgen05")
    for n in ("o", "dq", "dk", "dv"):     # tanhf against tanh.approx: a few bf16 ulps at most
        assert float((a[n].float() - b_[n].float()).abs().max()) <= 2e-2, n


def test_user_score_needs_the_tensor_core_kernels():
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200._binding import FlexAttnError
    q = torch.randn(1, 1, 128, 64, device="cuda")
    sf = fa.util.make_jax_score_fn(_softcap)
    with pytest.raises(FlexAttnError):      # float32 inputs run on the CUDA-core kernels, which have no compiled user path
        fa._flex_attention_impl(q, q, q, None, None, True, True, 1.0, 1, 128, 128, 128, False, None, None, sf)


@pytest.mark.parametrize("mask_kind,Sq,Sk,D", [("causal", 500, 500, 64), ("none", 300, 433, 128)])
def test_user_score_with_a_dense_bias(mask_kind, Sq, Sk, D):
    """The forms of the three kernels that are compiled at run time with a dense bias, which joins the user's score."""
    import flex_attention_tpu_b200 as fa
    B, H, sm = 1, 2, 1.0 / np.sqrt(D)
    (q, k, v, do), host = make_qkvdo((B, H, Sq, D), (B, H, Sk, D), 1400 + Sq, torch.bfloat16)
    ab_h = (0.7 * np.random.default_rng(9).standard_normal((B, H, Sq, Sk))).astype(np.float32)
    ab = torch.from_numpy(ab_h).cuda()
    mf, bf, sf, _ = build_mods(fa, mask_kind, "user", user_fn=_distance_and_head)
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    o, l, m = fa._flex_attention_impl(q, k, v, ab, None, True, False, sm, 1, 128, 128, 128, False, bf, mf, sf, status=status)
    delta = fa.bwd_preprocess(o, do)
    dq, dab = fa.flex_attention_bwd_dq(q, k, v, ab, None, l, m, o, do, delta, sm_scale=sm, score_fn=sf, mask_fn=mf,
                                       block_mask_fn=bf, return_dab=True, status=status)
    dk, dv = fa.flash_attention_bwd_dkv(k, v, q, ab, None, l, m, delta, do, sm_scale=sm, score_fn=sf, mask_fn=mf,
                                        block_mask_fn=bf, status=status)
    torch.cuda.synchronize()
    assert status.tolist() == [0, 0, 0, 0], status.tolist()
    kw = dict(sm_scale=sm, mask_kind=mask_kind, score_kind="user", user=(sf, sf.dscore))
    qh, kh, vh, doh = host
    ro, rl, rm = oracle.mha_reference(qh, kh, vh, ab_h, save_residuals=True, **kw)
    rdq, rdk, rdv, rdab = oracle.mha_bwd_reference(qh, kh, vh, ro, doh, rl, rm, ab_h, return_dab=True, **kw)
    assert_close(dict(o=o, l=l, m=m, dq=dq, dk=dk, dv=dv), dict(o=ro, l=rl, m=rm, dq=rdq, dk=rdk, dv=rdv), torch.bfloat16,
                 what=f"user score with bias {mask_kind}/D{D}")
    e = errors(dab, rdab)   # float32, but delta comes from the bf16-rounded o: the relative bound of the bias tests
    assert e["max_rel"] <= 1e-2, e


def _call(S, spec=None):
    """A causal call at D = 64 that the library gives to the fused backward: its arguments and the separate kernels' gradients."""
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200._resolve import make_problem
    (q, k, v, do), _ = make_qkvdo((2, 8, S, 64), (2, 8, S, 64), 1500 + S, torch.bfloat16)
    sf = fa.util.make_jax_score_fn(_distance_and_head)
    if spec is not None:
        sf.spec = spec
    fns = fa.masks.make_causal_mask_fns(128, 128)
    want = run_hot_path(fa, q, k, v, do, sm_scale=0.125, mask_kind="causal", score_kind="user", user_fn=sf)
    prob = make_problem(q, k, ab=None, segment_ids=None, causal=False, sm_scale=0.125, mask_fn=fns[0], block_mask_fn=fns[1], score_fn=sf)
    assert prob._bwd_scratch > 0
    args = (q, k, v, want["o"], want["l"], want["m"], do)
    return (lambda: fa.flex_attention_bwd(*args, sm_scale=0.125, mask_fns=fns, score_fn=sf)), [want[n] for n in ("dq", "dk", "dv")], prob


def test_user_score_through_the_fused_backward():
    from flex_attention_tpu_b200 import _binding as B
    backward, want, prob = _call(2048)
    first, second = backward(), backward()
    torch.cuda.synchronize()
    B.raise_if_failed(prob.device)
    assert all(torch.equal(a, b) for a, b in zip(first, second))
    for got, ref in zip(first, want):   # the same operands in another order of summation
        assert float((got.float() - ref.float()).norm() / ref.float().norm()) < 2e-3
    assert not torch.equal(first[0], want[0])


def test_a_function_the_fused_backward_cannot_be_compiled_around():
    from test_user_score import only_the_fused_backward_fails
    from flex_attention_tpu_b200.scores import ScoreSpec
    backward, want, _ = _call(2050, ScoreSpec("user", expr=only_the_fused_backward_fails().decode(), dexpr="1.0f"))
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(backward(), want))


def test_a_captured_backward_whose_fused_kernel_is_not_loaded():
    """Nothing can be loaded during a capture: dQ and dK/dV, which an earlier call has loaded, are recorded."""
    from flex_attention_tpu_b200.scores import ScoreSpec
    backward, want, _ = _call(2060, ScoreSpec("user", expr="0.75f * s - 0.01f * fabsf((float)(i - j))", dexpr="0.75f"))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = backward()
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want))
    assert not torch.equal(backward()[0], want[0])   # outside: the fused kernel


@pytest.mark.parametrize("first,then", [((1, 2, 300), (4, 16, 2048)), ((4, 16, 2048), (1, 2, 300))])
def test_a_captured_forward_whose_kernel_is_not_loaded(first, then):
    """Which forward kernel serves a call depends on its size; under capture one that an earlier call of another size has loaded takes
    the place of one that cannot be loaded then."""
    import flex_attention_tpu_b200 as fa
    B, H, S = first
    sf = fa.util.make_jax_score_fn(lambda s, b, h, qi, ki: (0.5 + 0.125 * B) * s - 0.015 * abs(qi - ki))   # a function of this test's own
    mf, bf, _, _ = build_mods(fa, "causal", "none")

    def forward(B, H, S):
        (q, k, v, _), _ = make_qkvdo((B, H, S, 64), (B, H, S, 64), 1600 + S, torch.bfloat16)
        return lambda: fa._flex_attention_impl(q, k, v, None, None, True, False, 0.125, 1, 128, 128, 128, False, bf, mf, sf)
    forward(*first)()
    call = forward(*then)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = call()
    g.replay()
    torch.cuda.synchronize()
    for name, got, want in zip(("o", "l", "m"), out, call()):   # outside: the kernel of this size; p rounded to bf16 in both
        assert float((got.float() - want.float()).norm() / want.float().norm()) < 5e-3, name
