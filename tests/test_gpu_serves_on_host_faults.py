"""Host-side faults the kernels' launchers have to answer with another kernel, made on the host by the bounds-checked build
(FLEXATTN_HOST_FAULT, see csrc/common.cuh): nothing faulty ever runs on the GPU."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent("""
    import sys
    sys.path.insert(0, %r); sys.path.insert(0, %r)
    import numpy as np, torch
    import flex_attention_tpu_b200 as fa
    from flex_attention_tpu_b200 import _binding as B
    from helpers import assert_close, build_mods, make_qkvdo, run_hot_path
    from kernel_names import launched_kernels
    assert B.DEBUG_BUILD

    kernels = lambda fn: launched_kernels(fn)[1]

    def case(mask, score, Bn, H, Sq, Sk, D, fwd, bwd, user=None, **kw):
        (q, k, v, do), _ = make_qkvdo((Bn, H, Sq, D), (Bn, H, Sk, D), 11, torch.bfloat16)
        args = dict(sm_scale=D ** -0.5, mask_kind=mask, score_kind=score, cap=6.0, user_fn=user, **kw)
        got = run_hot_path(fa, q, k, v, do, **args)
        want = run_hot_path(fa, q, k, v, do, backend="simt", **dict(args, score_kind="none" if score == "user" else score))
        if user is None:
            assert_close(got, want, torch.bfloat16, what=f"{mask} {Sq}x{Sk}", roundings=2)
        mf, bf, sf, _ = build_mods(fa, mask, score, cap=6.0, user_fn=user, **kw)
        names = kernels(lambda: fa._flex_attention_impl(q, k, v, None, None, True, False, D ** -0.5, 1, 128, 128, 128, False, bf, mf, sf))
        assert len(names) == 1 and fwd in names[0], (fwd, names)
        back = lambda: fa.flex_attention_bwd(q, k, v, got["o"], got["l"], got["m"], do, sm_scale=D ** -0.5,
                                             mask_fns=None if mf is None else (mf, bf), score_fn=sf)
        names = kernels(back)
        assert any(bwd in n for n in names), (bwd, names)
        for n, t in zip(("dq", "dk", "dv"), back()):
            assert float((t.float() - got[n].float()).norm() / got[n].float().norm()) < 5e-3, n
        assert B._mailbox(q.device).tolist() == [0, 0, 0, 0]

    user = fa.util.make_jax_score_fn(lambda s, b, h, qi, ki: s - 0.02 * (h + 1) * abs(qi - ki))
    # the cases
    print("HOST_FAULT_OK")
""")


def _run(fault, body):
    env = dict(os.environ, FLEXATTN_DEBUG="1")
    if fault:
        env["FLEXATTN_HOST_FAULT"] = fault
    code = (CHILD % (ROOT, os.path.join(ROOT, "tests"))).replace("# the cases", textwrap.dedent(body))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=900, env=env)
    assert r.returncode == 0 and "HOST_FAULT_OK" in r.stdout, r.stdout[-3000:] + r.stderr[-3000:]


REGISTERS = """
    case("causal", "none", 8, 16, 2048, 2048, 128, "{pair}", "{fused}")
    case("none", "none", 1, 2, 1, 8191, 128, "{split}", "dq_sm100")
    case("causal", "user", 4, 16, 2048, 2048, 64, "{pair}", "{fused}", user=user)
"""


@pytest.mark.parametrize("fault,names", [("", dict(pair="fwd_pair", split="fwd_split", fused="fused_sm100")),
                                         ("registers", dict(pair="fwd_pipe", split="fwd_pipe", fused="dq_sm100"))])
def test_a_kernel_compiled_for_too_few_registers_is_not_launched(fault, names):
    """Its warpgroups raise their registers out of what the CTA was launched with, and would wait for good: the kernels that hand none
    round serve the call, ahead-of-time compiled and around a user function."""
    _run(fault, REGISTERS.format(**names))


STRIDED = """
    case("s2", "none", 1, 3, 2049, 2049, 64, "{fwd}", "{bwd}", window=257, stride=16)     # 2049 rows: no multiple of the stride
    case("s2", "softcap", 2, 8, 2048, 2048, 128, "{fwd}", "{bwd16}", window=128, stride=32)
"""


@pytest.mark.parametrize("fault,names", [("", dict(fwd=", 6>", bwd="dq_sm100", bwd16="fused_sm100")),   # mask kind 6: gathered
                                         ("strided_map", dict(fwd=", 5>", bwd="dq_sm100", bwd16="dq_sm100"))])
def test_a_refused_strided_tensor_map_leaves_s2_to_the_dense_form(fault, names):
    """The gathered form fetches the keys on the stride grid through a tensor map of that pitch; every S2 call has a form without."""
    _run(fault, STRIDED.format(**names))
