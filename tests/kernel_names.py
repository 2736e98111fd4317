"""The names of the tensor-core kernels a call launches, for tests of the choice among them.  The profiler's clock and the GPU's drift
apart over the minutes that a test process lives, until its windows miss the kernels in them: names are taken in a process of their own."""
import json
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import json, sys
sys.path.insert(0, %r); sys.path.insert(0, %r)
import numpy as np, torch
import flex_attention_tpu_b200 as fa, workloads
from helpers import build_mods
from kernel_names import launched_kernels
out = []
for B, H, Sq, Sk, D, mask, score, window, stride in json.loads(sys.argv[1]):
    q, k = (torch.zeros(B, H, s, D, device="cuda", dtype=torch.bfloat16) for s in (Sq, Sk))
    ids = workloads.draw_documents(np.random.default_rng(1), B, Sq, lo=64, hi=1500)[0] if mask == "document" else None
    mf, bf, sf, seg = build_mods(fa, mask, score, window=window, stride=stride, cap=20.0, doc_ids=ids,
                                 user_fn=lambda s, b, h, qi, ki: s - 0.03 * (h + 1) * abs(qi - ki))
    out.append(launched_kernels(lambda: fa._flex_attention_impl(q, k, k, None, seg, False, False, 0.1, 1, 128, 128, 128, False, bf, mf, sf))[1])
print("NAMES", json.dumps(out))
"""


def launched_kernels(fn):
    """(result of fn, names); in a young process."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    for _ in range(5):   # (a window that holds none, though every caller's fn launches one, is taken again)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            out = fn()
            torch.cuda.synchronize()
        names = [e.name for e in prof.events() if "_sm100_kernel" in e.name]
        if names:
            break
    return out, names


def forward_kernels(calls):
    """Names for each of the forward calls (B, H, Sq, Sk, D, mask kind, score kind, window, stride)."""
    r = subprocess.run([sys.executable, "-c", CHILD % (ROOT, os.path.join(ROOT, "tests")), json.dumps(calls)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.split("NAMES", 1)[1])
