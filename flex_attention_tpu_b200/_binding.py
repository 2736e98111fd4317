"""ctypes binding of libflexattn.so (the C ABI declared in include/flexattn.h).

This is the only backend: there is no CPU or PyTorch fallback.  Importing the module without the built
library raises, and every call checks the returned status.
"""
from __future__ import annotations

import ctypes
import os
from collections import OrderedDict

import torch

# FLEXATTN_DEBUG=1 loads the bounds-checked build of the same library (every direct global-memory access of the
# tensor-core kernels guarded; an out-of-range index is reported through the status words as code 14 instead of
# faulting).  Slower; meant for bring-up and for the tests that run without a memory checker.
DEBUG_BUILD = os.environ.get("FLEXATTN_DEBUG", "0") not in ("", "0")
_LIB_PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)),
                         "libflexattn_debug.so" if DEBUG_BUILD else "libflexattn.so")

DTYPE_BF16, DTYPE_F32 = 0, 1
SCORE_NONE, SCORE_ALIBI, SCORE_SOFTCAP, SCORE_USER = 0, 1, 2, 3
MASK_NONE, MASK_CAUSAL, MASK_SLIDING_WINDOW, MASK_SLIDING_WINDOW_CAUSAL, MASK_DOCUMENT, MASK_S2 = range(6)
BACKEND_AUTO, BACKEND_SIMT, BACKEND_TCGEN05 = 0, 1, 2
TILE = 128
ABI_VERSION = 4   # FLEXATTN_ABI_VERSION of include/flexattn.h this binding was written against

MASK_KIND_IDS = {"none": MASK_NONE, "causal": MASK_CAUSAL, "sliding_window": MASK_SLIDING_WINDOW,
                 "sliding_window_causal": MASK_SLIDING_WINDOW_CAUSAL, "document": MASK_DOCUMENT, "s2": MASK_S2}
SCORE_KIND_IDS = {"none": SCORE_NONE, "alibi": SCORE_ALIBI, "softcap": SCORE_SOFTCAP, "user": SCORE_USER}
BACKEND_IDS = {"auto": BACKEND_AUTO, "simt": BACKEND_SIMT, "tcgen05": BACKEND_TCGEN05}


class FlexAttnParams(ctypes.Structure):
    _fields_ = [
        ("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("v", ctypes.c_void_p), ("o", ctypes.c_void_p),
        ("d_o", ctypes.c_void_p), ("dq", ctypes.c_void_p), ("dk", ctypes.c_void_p), ("dv", ctypes.c_void_p),
        ("l", ctypes.c_void_p), ("m", ctypes.c_void_p), ("delta", ctypes.c_void_p),
        ("doc_ids", ctypes.c_void_p), ("alibi_slopes", ctypes.c_void_p),
        ("batch", ctypes.c_int32), ("heads", ctypes.c_int32), ("seq_q", ctypes.c_int32),
        ("seq_k", ctypes.c_int32), ("head_dim", ctypes.c_int32),
        ("dtype", ctypes.c_int32), ("sm_scale", ctypes.c_float),
        ("score_kind", ctypes.c_int32), ("softcap", ctypes.c_float),
        ("mask_kind", ctypes.c_int32), ("window", ctypes.c_int32), ("stride", ctypes.c_int32),
        ("workspace", ctypes.c_void_p), ("workspace_bytes", ctypes.c_size_t),
        ("status", ctypes.c_void_p), ("backend", ctypes.c_int32), ("user_score", ctypes.c_int32),
        ("ab", ctypes.c_void_p), ("dab", ctypes.c_void_p),
    ]


class FlexAttnError(RuntimeError):
    def __init__(self, code, where):
        self.code = code
        super().__init__(f"{where}: {status_string(code)} (status {code})")


def _load():
    if not os.path.exists(_LIB_PATH):
        raise ImportError(
            f"{_LIB_PATH} is missing: build it with `python flex_attention_tpu_b200/build.py` "
            "(there is no fallback implementation)")
    lib = ctypes.CDLL(_LIB_PATH)
    P = ctypes.POINTER(FlexAttnParams)
    lib.flexattn_abi_version.restype = ctypes.c_int
    lib.flexattn_status_string.restype = ctypes.c_char_p
    lib.flexattn_status_string.argtypes = [ctypes.c_int]
    lib.flexattn_workspace_bytes.restype = ctypes.c_size_t
    lib.flexattn_workspace_bytes.argtypes = [P]
    for name in ("flexattn_build_mask_map", "flexattn_fwd", "flexattn_bwd_preprocess", "flexattn_bwd_dq",
                 "flexattn_bwd_dkv"):
        fn = getattr(lib, name)
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.c_void_p, P]
    lib.flexattn_bwd.restype = ctypes.c_int
    lib.flexattn_bwd.argtypes = [ctypes.c_void_p, ctypes.c_void_p, P]
    lib.flexattn_bwd_scratch_bytes.restype = ctypes.c_size_t
    lib.flexattn_bwd_scratch_bytes.argtypes = [P]
    lib.flexattn_bwd_fused.restype = ctypes.c_int
    lib.flexattn_bwd_fused.argtypes = [ctypes.c_void_p, P, ctypes.c_void_p, ctypes.c_size_t]
    lib.flexattn_fwd_noalloc.restype = ctypes.c_int
    lib.flexattn_fwd_noalloc.argtypes = [ctypes.c_void_p, P]
    lib.flexattn_noalloc_scratch_bytes.restype = ctypes.c_size_t
    lib.flexattn_read_mask_map.restype = ctypes.c_int
    lib.flexattn_read_mask_map.argtypes = [ctypes.c_void_p, P, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                           ctypes.POINTER(ctypes.c_int32)]
    lib.flexattn_selftest_umma.restype = ctypes.c_int
    lib.flexattn_selftest_umma.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p,
                                           ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p]
    lib.flexattn_selftest_timeout.restype = ctypes.c_int
    lib.flexattn_selftest_timeout.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p]
    lib.flexattn_reset_abort.restype = ctypes.c_int
    lib.flexattn_reset_abort.argtypes = [ctypes.c_void_p]
    lib.flexattn_user_score_create.restype = ctypes.c_int
    lib.flexattn_user_score_create.argtypes = [ctypes.c_char_p, ctypes.c_char_p, ctypes.POINTER(ctypes.c_int32)]
    lib.flexattn_user_score_destroy.restype = ctypes.c_int
    lib.flexattn_user_score_destroy.argtypes = [ctypes.c_int32]
    lib.flexattn_user_score_log.restype = ctypes.c_char_p
    lib.flexattn_user_score_log.argtypes = [ctypes.c_int32]
    lib.flexattn_user_score_compile.restype = ctypes.c_int
    lib.flexattn_user_score_compile.argtypes = [ctypes.c_int32, ctypes.c_int, ctypes.c_int32, ctypes.c_int32]
    if lib.flexattn_abi_version() != ABI_VERSION:
        raise ImportError("libflexattn.so ABI version mismatch: rebuild the library")
    return lib


lib = _load()


def status_string(code: int) -> str:
    return lib.flexattn_status_string(int(code)).decode()


def check(code: int, where: str):
    if code != 0:
        raise FlexAttnError(code, where)


_USER_SCORES = {}   # (score expression, derivative expression) -> handle of the library


def user_score_handle(score_expr: str, dscore_expr: str) -> int:
    """Registers a pair of CUDA expressions with the library (once per distinct pair) and returns its handle."""
    key = (score_expr, dscore_expr)
    h = _USER_SCORES.get(key)
    if h is None:
        out = ctypes.c_int32(0)
        check(lib.flexattn_user_score_create(score_expr.encode(), dscore_expr.encode(), ctypes.byref(out)),
              "flexattn_user_score_create")
        h = _USER_SCORES[key] = int(out.value)
    return h


def check_user(code: int, where: str, handle: int):
    """`check` that appends the run-time compiler's log when a user score function failed to compile."""
    if code == 13:
        log = lib.flexattn_user_score_log(handle).decode(errors="replace")
        raise FlexAttnError(code, f"{where}\n{log}")
    check(code, where)


def _device_index(device):
    return device.index if device.index is not None else torch.cuda.current_device()


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_capturing = torch.cuda.is_current_stream_capturing


def _stream_ptr(device):
    index = device.index
    return _raw_stream(torch.cuda.current_device() if index is None else index)


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


# ------------------------------------------------------------------------------------------ failure mailbox
# A device-side wait that gives up reports through four status words.  When the caller passes no `status`
# tensor the binding supplies one of its own per device, in pinned host memory the device writes through the
# bus: the host can then look at it at the start of every call WITHOUT synchronising, and raises on the first
# call after the failure became visible.  A time-out is sticky on its device until `reset_abort` has run.
_MAILBOX = {}


def _mailbox(device):
    key = _device_index(device)
    box = _MAILBOX.get(key)
    if box is None:
        box = _MAILBOX[key] = torch.zeros(4, dtype=torch.int32).pin_memory()
    return box


def raise_if_failed(device):
    """Raises FlexAttnError if an earlier launch on `device` reported a device-side time-out into the binding's
    own status words.  Never synchronises."""
    key = _device_index(device)
    box = _MAILBOX.get(key)
    # read through its address: indexing the tensor costs more than the rest of the check
    if box is not None and ctypes.c_int32.from_address(box.data_ptr()).value != 0:
        code, kernel, block, detail = (int(x) for x in box.tolist())
        raise FlexAttnError(code, f"an earlier launch on cuda:{key} (kernel id {kernel}, block {block}, detail {detail}; "
                                  "outputs of launches since then are not valid; call reset_abort() to re-arm)")


def reset_abort(device=None):
    """Clears the device's abort word (stream-ordered on the current stream) and the binding's status words."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    check(lib.flexattn_reset_abort(_stream_ptr(device)), "flexattn_reset_abort")
    torch.cuda.current_stream(device).synchronize()
    key = _device_index(device)
    if key in _MAILBOX:
        _MAILBOX[key].zero_()


# Debug switch for the test-suite: every output tensor the binding allocates is filled with NaN before the
# kernels run, so an element a kernel failed to write cannot pass for a result left over from an earlier call.
POISON_OUTPUTS = os.environ.get("FLEXATTN_POISON_OUTPUTS", "0") not in ("", "0")


class Problem:
    """One attention problem: shapes, score/mask spec and the tensors bound so far.  Owns the mask-map
    workspace (a torch buffer) and rebuilds the map only when the mask inputs or the stream change."""

    _map_cache: "OrderedDict[tuple, torch.Tensor]" = OrderedDict()
    _MAP_CACHE_ENTRIES = 16
    # maps and slopes that captured graphs read: one of each, a few KB, kept for good (nobody tells when a graph has gone).
    # Beyond this many a graph builds the map it reads.
    _graph_held = {}
    _GRAPH_HELD_ENTRIES = 256
    _bwd_scratch = 0   # bytes of scratch the fused backward takes; 0: the separate kernels serve the problem
    _images = {}   # sizes and options -> the parameter struct they give (no pointers in it): filling the fields one by one
                   # and asking for the sizes of workspace and scratch costs a short call more than its launches

    def __init__(self, q, k, *, sm_scale, mask_kind=MASK_NONE, window=0, stride=0, doc_ids=None,
                 score_kind=SCORE_NONE, softcap=0.0, alibi_slopes=None, backend=BACKEND_AUTO, status=None, ab=None,
                 user_score=0):
        if not q.is_cuda:
            raise ValueError("flex attention tensors must live on a CUDA device (no CPU path exists)")
        if q.dim() != 4 or k.dim() != 4:
            raise ValueError("expected [batch, heads, seq, head_dim] tensors")
        self.device, self.dtype, shape_q, shape_k = q.device, q.dtype, q.shape, k.shape
        device, dtype = self.device, self.dtype
        if dtype not in (torch.bfloat16, torch.float32):
            raise NotImplementedError(f"dtype {dtype} is not supported (bfloat16 or float32)")
        stream, capturing = _stream_ptr(device), _capturing()
        B, H, Sq, D = self.shape_q = tuple(shape_q)
        self.shape_k = tuple(shape_k)
        Sk = shape_k[2]
        sm_scale, softcap, window, stride = float(sm_scale), float(softcap), int(window), int(stride)
        key = (device, dtype, shape_q, Sk, sm_scale, score_kind, softcap, mask_kind, window, stride, backend, user_score)
        image = Problem._images.get(key)
        if image is None:
            p = FlexAttnParams()
            p.batch, p.heads, p.seq_q, p.seq_k, p.head_dim = B, H, Sq, Sk, D
            p.dtype = DTYPE_BF16 if dtype == torch.bfloat16 else DTYPE_F32
            p.sm_scale = sm_scale
            p.score_kind, p.softcap = int(score_kind), softcap
            p.mask_kind, p.window, p.stride = int(mask_kind), window, stride
            p.backend = int(backend)
            p.user_score = int(user_score)
            p.workspace_bytes = lib.flexattn_workspace_bytes(ctypes.byref(p))
            self._bwd_scratch = lib.flexattn_bwd_scratch_bytes(ctypes.byref(p))
            if p.workspace_bytes:
                if len(Problem._images) >= 256:
                    Problem._images.clear()
                Problem._images[key] = bytes(p), self._bwd_scratch
        else:
            p, self._bwd_scratch = FlexAttnParams.from_buffer_copy(image[0]), image[1]
        # Tensors of the problem itself whose pointers sit in `p`, by field name.  The tensors of a call are not among them:
        # autograd keeps the problem with the graph of the output, so a problem that held its output would hold itself.
        self._keep = {}
        if mask_kind == MASK_DOCUMENT:
            if doc_ids is None:
                raise ValueError("document mask needs segment/doc ids")
            doc_ids = torch.as_tensor(doc_ids)
            if doc_ids.dim() == 1:
                doc_ids = doc_ids[None].expand(B, -1)
            doc_ids = doc_ids.to(device=device, dtype=torch.int32).contiguous()
            if doc_ids.shape != (B, max(Sq, Sk)):
                raise ValueError(f"doc ids must be [batch, {max(Sq, Sk)}], got {tuple(doc_ids.shape)}")
            p.doc_ids = doc_ids.data_ptr()
            self._keep["doc_ids"] = doc_ids
        self.doc_ids = doc_ids if mask_kind == MASK_DOCUMENT else None
        if score_kind == SCORE_ALIBI:
            slopes = self._device_slopes(alibi_slopes, H, stream, capturing)
            p.alibi_slopes = slopes.data_ptr()
            self._keep["alibi_slopes"] = slopes
        own_status = status is None
        if own_status:
            status = _mailbox(device)
        p.status = at = status.data_ptr()
        if own_status and ctypes.c_int32.from_address(at).value != 0:
            raise_if_failed(device)
        self._keep["status"] = status
        self.ab = None
        if ab is not None:
            # dense additive bias [B,H,Sq,Sk], float32
            if not (isinstance(ab, torch.Tensor) and ab.is_cuda):
                raise ValueError("ab must be a CUDA tensor")
            if tuple(ab.shape) != (B, H, Sq, Sk):
                raise ValueError(f"Attention bias shape mismatch: expected {(B, H, Sq, Sk)}, got {tuple(ab.shape)}")
            self.ab = ab.to(torch.float32).contiguous()
            p.ab = self.ab.data_ptr()
            self._keep["ab"] = self.ab
        self.p = p
        self._bind_workspace(stream, capturing, (device.index, mask_kind, window, stride, B, Sq, Sk))

    _slope_cache: "OrderedDict[tuple, torch.Tensor]" = OrderedDict()
    _SLOPE_CACHE_ENTRIES = 64

    def _device_slopes(self, alibi_slopes, H, stream, capturing):
        """[H] float32 slopes on the device.  Host values are uploaded once and cached: a pageable
        host-to-device copy waits for the stream, which would serialise every call behind the last.
        A copy belongs to its stream like a mask map does (`_bind_workspace`)."""
        if isinstance(alibi_slopes, torch.Tensor) and alibi_slopes.is_cuda:
            slopes = alibi_slopes.to(torch.float32).flatten()
            if slopes.numel() == 1:
                slopes = slopes.expand(H)
            if slopes.numel() != H:
                raise ValueError(f"need one ALiBi slope per head ({H}), got {slopes.numel()}")
            return slopes.contiguous()
        cache = Problem._slope_cache
        find = Problem._hold_for_graph if capturing else OrderedDict.get
        if type(alibi_slopes) is tuple:   # the host values of a score spec: known after its first call
            t = find(cache, (stream, self.device.index, alibi_slopes))
            if t is not None and t.numel() == H:
                return t
        vals = tuple(float(x) for x in torch.as_tensor(alibi_slopes, dtype=torch.float32).flatten().tolist())
        if len(vals) == 1:
            vals = vals * H
        if len(vals) != H:
            raise ValueError(f"need one ALiBi slope per head ({H}), got {len(vals)}")
        key = (stream, self.device.index, vals)
        t = find(cache, key)
        if t is None:
            t = cache[key] = torch.tensor(vals, dtype=torch.float32).to(self.device)
        if type(alibi_slopes) is tuple:
            cache[(stream, self.device.index, alibi_slopes)] = t
        while len(cache) > Problem._SLOPE_CACHE_ENTRIES:
            cache.popitem(last=False)
        return t

    # ------------------------------------------------------------------ mask map
    def _bind_workspace(self, stream, capturing, sizes):
        """The workspace with the mask map, which depends on `sizes` and, for documents, on the ids."""
        p = self.p
        nbytes = p.workspace_bytes
        if nbytes == 0:
            raise FlexAttnError(2, "flexattn_workspace_bytes")
        doc_key = None
        if self.doc_ids is not None:
            doc_key = (self.doc_ids.data_ptr(), self.doc_ids._version)
        # A map belongs to the stream it was built on: there it is complete before any kernel reads it, and an evicted buffer
        # goes back to the pool of that stream, behind the kernels that still read it.  Another stream builds its own.
        key = (stream, *sizes, doc_key)
        cache = Problem._map_cache
        # Under capture a map of document ids is part of the graph: a replay reads the ids it finds.  So is a map that has not
        # been built before, and no later call may take it for a finished one.
        if capturing:
            entry = None if doc_key is not None else self._hold_for_graph(cache, key)
        else:
            entry = cache.get(key)
            if entry is not None:
                try:
                    cache.move_to_end(key)
                except KeyError:   # another thread has just evicted it
                    pass
        fresh = entry is None
        if fresh:
            # the entry keeps the doc-id tensor alive, so its (pointer, version) key cannot be recycled
            entry = (torch.empty(nbytes, dtype=torch.uint8, device=self.device), self.doc_ids)
        self.workspace = entry[0]
        p.workspace = self.workspace.data_ptr()
        if fresh:
            check(lib.flexattn_build_mask_map(stream, ctypes.byref(p)), "flexattn_build_mask_map")
            if not capturing:
                cache[key] = entry
                while len(cache) > Problem._MAP_CACHE_ENTRIES:
                    cache.popitem(last=False)

    @staticmethod
    def _hold_for_graph(cache, key):
        """The entry under `key` that a call outside the capture has made, on whatever stream (work enqueued before the
        capture comes before the replays), or None.  It outlives the cache from here on."""
        held, what = Problem._graph_held, (cache is Problem._map_cache, *key[1:])
        entry = held.get(what)
        if entry is None and (not what[0] or len(held) < Problem._GRAPH_HELD_ENTRIES):
            entry = next((e for k, e in list(cache.items()) if k[1:] == key[1:]), None)
            if entry is not None:
                held[what] = entry
        return entry

    def read_map(self, which: int, b: int, index: int):
        out = (ctypes.c_int32 * 4)()
        check(lib.flexattn_read_mask_map(_stream_ptr(self.device), ctypes.byref(self.p), which, b, index, out),
              "flexattn_read_mask_map")
        return tuple(out)

    # ------------------------------------------------------------------ tensors
    def _bind(self, **tensors):
        p, dtype, index = self.p, self.dtype, self.device.index
        for name, t in tensors.items():
            if t is None:
                continue
            if t.get_device() != index:
                raise ValueError(f"{name} must be on {self.device}")
            if not t.is_contiguous():
                raise ValueError(f"{name} must be contiguous")
            want = torch.float32 if name in ("l", "m", "delta") else dtype
            if t.dtype != want:
                raise ValueError(f"{name} must be {want}, got {t.dtype}")
            setattr(p, name, t.data_ptr())

    def _new(self, shape, dtype=None):
        if POISON_OUTPUTS:
            return torch.full(shape, float("nan"), dtype=dtype or self.dtype, device=self.device)
        return torch.empty(shape, dtype=dtype or self.dtype, device=self.device)

    def forward(self, q, k, v):
        B, H, Sq, D = self.shape_q
        o, l, m = self._new(self.shape_q), self._new((B, H, Sq), torch.float32), self._new((B, H, Sq), torch.float32)
        self._bind(q=q, k=k, v=v)
        self.p.o, self.p.l, self.p.m = o.data_ptr(), l.data_ptr(), m.data_ptr()
        check_user(lib.flexattn_fwd(_stream_ptr(self.device), ctypes.byref(self.p)), "flexattn_fwd", self.p.user_score)
        return o, l, m

    def preprocess(self, o, do):
        B, H, Sq, _ = self.shape_q
        delta = self._new((B, H, Sq), torch.float32)
        self._bind(o=o, d_o=do, delta=delta)
        check(lib.flexattn_bwd_preprocess(_stream_ptr(self.device), ctypes.byref(self.p)), "flexattn_bwd_preprocess")
        return delta

    def bwd_dq(self, q, k, v, do, l, m, delta, want_dab=False):
        """dq, or (dq, dab) with ``want_dab`` (dab: float32 [B,H,Sq,Sk], the gradient of the dense bias)."""
        dq = self._new(self.shape_q)
        self._bind(q=q, k=k, v=v, d_o=do, l=l, m=m, delta=delta, dq=dq)
        dab = None
        if want_dab:
            if self.ab is None:
                raise ValueError("dab was requested but the problem has no bias `ab`")
            dab = self._new(self.ab.shape, torch.float32)
            self.p.dab = dab.data_ptr()
        try:
            check_user(lib.flexattn_bwd_dq(_stream_ptr(self.device), ctypes.byref(self.p)), "flexattn_bwd_dq", self.p.user_score)
        finally:
            self.p.dab = None
        return (dq, dab) if want_dab else dq

    def bwd_dkv(self, q, k, v, do, l, m, delta):
        dk, dv = self._new(self.shape_k), self._new(self.shape_k)
        self._bind(q=q, k=k, v=v, d_o=do, l=l, m=m, delta=delta, dk=dk, dv=dv)
        check_user(lib.flexattn_bwd_dkv(_stream_ptr(self.device), ctypes.byref(self.p)), "flexattn_bwd_dkv", self.p.user_score)
        return dk, dv

    def backward(self, q, k, v, o, do, l, m, need_dq=True, need_dkv=True, want_dab=False, two_streams=None):
        """delta, dQ, dK and dV.  Where the library asks for scratch (`flexattn_bwd_scratch_bytes`) and there is room for it, one
        kernel computes all of them in one pass over the tile pairs, on the current stream.  Otherwise, and with a dense bias,
        dQ and dK/dV have a kernel each; they only share inputs, so dK/dV is launched on a side stream: both kernels fill
        every SM on their own, but the tail of one then overlaps the head of the other.  Everything is ordered after the
        current stream's work and the current stream waits for both.  ``two_streams=False`` launches those two on the current
        stream (the host-buffer pipeline does: there the extra stream only adds synchronisation between the copy and compute
        streams)."""
        if not (need_dq or want_dab) or not need_dkv:
            delta = self.preprocess(o, do)
            dk, dv = self.bwd_dkv(q, k, v, do, l, m, delta) if need_dkv else (None, None)
            if want_dab:
                dq, dab = self.bwd_dq(q, k, v, do, l, m, delta, want_dab=True)
                return delta, dq, dk, dv, dab
            return delta, self.bwd_dq(q, k, v, do, l, m, delta) if need_dq else None, dk, dv
        if want_dab and self.ab is None:
            raise ValueError("dab was requested but the problem has no bias `ab`")
        if two_streams is None:
            two_streams = TWO_STREAM_BACKWARD
        B, H, Sq, _ = self.shape_q
        delta = self._new((B, H, Sq), torch.float32)                # everything is allocated on the current stream
        dq, dk, dv = self._new(self.shape_q), self._new(self.shape_k), self._new(self.shape_k)
        dab = self._new(self.ab.shape, torch.float32) if want_dab else None
        self._bind(q=q, k=k, v=v, o=o, d_o=do, l=l, m=m)
        p = self.p
        p.delta, p.dq, p.dk, p.dv = delta.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr()
        p.dab = dab.data_ptr() if want_dab else None
        stream = _stream_ptr(self.device)
        scratch = None
        if self._bwd_scratch and self.ab is None:
            try:
                scratch = torch.empty(self._bwd_scratch, dtype=torch.uint8, device=self.device)
            except torch.OutOfMemoryError:   # the separate kernels need none
                pass
        if scratch is not None:   # one kernel for all three gradients, on one stream
            code = lib.flexattn_bwd_fused(stream, ctypes.byref(p), scratch.data_ptr(), self._bwd_scratch)
            if code not in (10, 13):   # those: not built for this call, and nothing launched
                check(code, "flexattn_bwd_fused")
                return delta, dq, dk, dv
        side = _side_stream(self.device).cuda_stream if two_streams else stream
        try:
            check_user(lib.flexattn_bwd(stream, side, ctypes.byref(p)), "flexattn_bwd", p.user_score)
        finally:
            p.dab = None
        return (delta, dq, dk, dv, dab) if want_dab else (delta, dq, dk, dv)


_SIDE_STREAMS = {}
# dK/dV on a side stream next to dQ (see Problem.backward); False launches the two kernels one after the other
TWO_STREAM_BACKWARD = os.environ.get("FLEXATTN_TWO_STREAM", "1") != "0"


def _side_stream(device):
    """One long-lived side stream per device for `Problem.backward` (created on first use)."""
    key = _device_index(device)
    st = _SIDE_STREAMS.get(key)
    if st is None:
        st = _SIDE_STREAMS[key] = torch.cuda.Stream(device)
    return st


def selftest_umma(variant: int, a: torch.Tensor, b: torch.Tensor, status=None) -> torch.Tensor:
    """Single-tile tensor-core self check (see flexattn_selftest_umma in the header)."""
    kdim = a.shape[1]
    d = torch.empty(128, 128, dtype=torch.float32, device=a.device)
    check(lib.flexattn_selftest_umma(_stream_ptr(a.device), int(variant), _ptr(a), _ptr(b), _ptr(d), int(kdim),
                                     _ptr(status)), "flexattn_selftest_umma")
    return d


def selftest_timeout(limit_ms: int, status=None, device=None):
    """Launches the time-out self check (see flexattn_selftest_timeout in the header): a wait that runs out
    after `limit_ms` and reports like an attention kernel would.  With ``status=None`` the report goes to the
    binding's own status words."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if status is None:
        status = _mailbox(device)
    check(lib.flexattn_selftest_timeout(_stream_ptr(device), int(limit_ms), _ptr(status)), "flexattn_selftest_timeout")
