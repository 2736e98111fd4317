"""Builds libflexattn.so (sm_100a only) in-tree with nvcc, and next to it libflexattn_debug.so, the same sources with
-DFLEXATTN_DEBUG (bounds checks on every direct global-memory access of the tensor-core kernels; selected at import
time with the environment variable FLEXATTN_DEBUG=1).  Usage: python flex_attention_tpu_b200/build.py [-v]"""
from __future__ import annotations

import concurrent.futures
import hashlib
import os
import re
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
BASE_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]
# extra compiler flags, e.g. FLEXATTN_NVCC_FLAGS="-DFLEXATTN_PAIR_EX2_FMA=1" to build another kernel configuration
BASE_FLAGS += os.environ.get("FLEXATTN_NVCC_FLAGS", "").split()
# the variant being built (set by build_variant): object directory, library path, compiler flags
OBJ = os.path.join(PKG, "build")
LIB = os.path.join(PKG, "libflexattn.so")
FLAGS = list(BASE_FLAGS)


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stamp(src):
    """Hash of a source plus every header it could include: objects are rebuilt only when it changes."""
    h = hashlib.sha256()
    headers = sorted(f for f in os.listdir(CSRC) if f.endswith((".cuh", ".h")))
    for path in [src if os.path.isabs(src) else os.path.join(CSRC, src)] + [os.path.join(CSRC, x) for x in headers] + \
            [os.path.join(PKG, "..", "include", "flexattn.h")]:
        with open(path, "rb") as f:
            text = f.read()
        h.update(text)
        for name in re.findall(rb'^#include "(\w+\.cu)"', text, re.M):   # a kernel file compiled in another form
            with open(os.path.join(CSRC, name.decode()), "rb") as f:
                h.update(f.read())
    h.update(" ".join(FLAGS).encode())
    return h.hexdigest()


# sources the library carries as text: a user score function is compiled into these kernels at run time (csrc/jit.cu)
EMBEDDED = ["fwd_pipe_sm100.cu", "bwd_dq_sm100.cu", "bwd_dkv_sm100.cu", "bwd_fused_sm100.cu", "fwd_pair_sm100.cu", "sched.cuh", "score_row.cuh", "sm100.cuh",
            "common.cuh",
            os.path.join("..", "..", "include", "flexattn.h")]


def _embed_sources():
    """Writes build/embedded_sources.cu: the files of EMBEDDED as string literals, looked up by base name."""
    out = os.path.join(OBJ, "embedded_sources.cu")
    parts = ["// generated by build.py from the kernel sources: do not edit\nnamespace flexattn {\n"]
    names = []
    for i, rel in enumerate(EMBEDDED):
        text = open(os.path.join(CSRC, rel)).read()
        assert ')FLEXSRC"' not in text
        names.append(os.path.basename(rel))
        # string literals are limited in length by some compilers: split into chunks and let them concatenate
        chunks = [text[j:j + 8000] for j in range(0, len(text), 8000)]
        parts.append(f"static const char kSrc{i}[] =\n" + "\n".join(f'R"FLEXSRC({c})FLEXSRC"' for c in chunks) + ";\n")
    parts.append("extern const char* const kEmbeddedNames[] = {" + ", ".join(f'"{n}"' for n in names) + "};\n")
    parts.append("extern const char* const kEmbeddedSources[] = {" + ", ".join(f"kSrc{i}" for i in range(len(names))) + "};\n")
    parts.append(f"extern const int kEmbeddedCount = {len(names)};\n}}  // namespace flexattn\n")
    text = "".join(parts)
    if not os.path.exists(out) or open(out).read() != text:
        with open(out, "w") as f:
            f.write(text)
    return out


def _compile(src, verbose):
    obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
    stamp_path = obj + ".stamp"
    stamp = _stamp(src)
    if os.path.exists(obj) and os.path.exists(stamp_path) and open(stamp_path).read() == stamp:
        return obj, ""
    cmd = [NVCC, *FLAGS, "-c", src if os.path.isabs(src) else os.path.join(CSRC, src), "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
    with open(stamp_path, "w") as f:
        f.write(stamp)
    return obj, r.stderr


def build(verbose: bool = False, jobs: int | None = None) -> str:
    """Both libraries; returns the path of the ordinary one."""
    global OBJ, LIB, FLAGS
    OBJ, LIB, FLAGS = os.path.join(PKG, "build_debug"), os.path.join(PKG, "libflexattn_debug.so"), BASE_FLAGS + ["-DFLEXATTN_DEBUG"]
    build_variant(verbose, jobs, extras=False)
    OBJ, LIB, FLAGS = os.path.join(PKG, "build"), os.path.join(PKG, "libflexattn.so"), list(BASE_FLAGS)
    return build_variant(verbose, jobs, extras=True)


def build_variant(verbose: bool = False, jobs: int | None = None, extras: bool = True) -> str:
    os.makedirs(OBJ, exist_ok=True)
    srcs = _sources() + [_embed_sources()]
    with concurrent.futures.ThreadPoolExecutor(jobs or os.cpu_count() or 4) as ex:
        results = list(ex.map(lambda s: _compile(s, verbose), srcs))
    objs = [o for o, _ in results]
    if verbose:
        for _, log in results:
            if log:
                print(log)
    newest = max(os.path.getmtime(o) for o in objs)
    # relink when an object is newer than the library or when the list of sources changed
    list_path, listing = os.path.join(OBJ, "sources.list"), "\n".join(srcs)
    same_list = os.path.exists(list_path) and open(list_path).read() == listing
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < newest or not same_list:
        # only the C ABI of include/flexattn.h is exported; the C++ launchers between the objects stay internal
        vs = os.path.join(OBJ, "exports.map")
        with open(vs, "w") as f:
            f.write("{ global: flexattn_*; local: *; };\n")
        cmd = [NVCC, "-shared", "-o", LIB, *objs, "-cudart", "shared", "-ldl", "-Xlinker", "--no-undefined",
               "-Xlinker", f"--version-script={vs}"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
        with open(list_path, "w") as f:
            f.write(listing)
    if extras:
        _build_driver()
        _build_xla_shim()
    return LIB


def _build_xla_shim():
    """libflexattn_xla.so: the XLA FFI handlers over the C ABI (csrc/xla_ffi_shim.cc).  Needs the headers that ship
    with jaxlib; where JAX is not installed the step is skipped and returns None (the jax.ffi binding is then
    unavailable, the library itself is unaffected)."""
    try:
        import jax
        inc = jax.ffi.include_dir()
    except Exception:
        return None
    src = os.path.join(CSRC, "xla_ffi_shim.cc")
    out = os.path.join(PKG, "libflexattn_xla.so")
    if os.path.exists(out) and os.path.getmtime(out) >= max(os.path.getmtime(src), os.path.getmtime(LIB)):
        return out
    cmd = [NVCC, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", inc, "-I", os.path.join(PKG, "..", "include"),
           src, "-o", out, "-L", PKG, "-lflexattn", "-cudart", "shared", "-Xlinker", "-rpath", "-Xlinker", "$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"XLA FFI shim build failed:\n{r.stdout}\n{r.stderr}")
    return out


def _build_driver():
    """flexattn_bench: the stand-alone C++ driver over the C ABI (csrc/flexattn_bench.cpp), linked against the
    library next to it."""
    src = os.path.join(CSRC, "flexattn_bench.cpp")
    exe = os.path.join(PKG, "flexattn_bench")
    if os.path.exists(exe) and os.path.getmtime(exe) >= max(os.path.getmtime(src), os.path.getmtime(LIB)):
        return exe
    cmd = [NVCC, "-O2", "-std=c++17", "-I", os.path.join(PKG, "..", "include"), src, "-o", exe, "-L", PKG, "-lflexattn",
           "-cudart", "shared", "-Xlinker", "-rpath", "-Xlinker", "$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"driver build failed:\n{r.stdout}\n{r.stderr}")
    return exe


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
