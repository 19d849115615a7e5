"""Autograd functions and functional entry points of the operator set.

Host-side mirror of the reference's ``*_Func`` autograd classes and ``*_fn``
entries (same names, argument order, defaults and error behaviour), with every
Triton launch replaced by one call into librgd_b200.so through the C ABI:

===========================  =======================================================
entry point here             reference entry it replaces
===========================  =======================================================
``triton_norm_func_fn``      normalization/l2normalize_cached.py:435-436
``triton_fused_norm_func_fn``  normalization/fused_l2normalize_cached.py:506-507
``triton_fused_ln_func_fn``  normalization/head_layernorm_cached.py:455-456
``triton_rms_func_fn``       normalization/rmsnorm_cached.py:628-629
``triton_fused_rms_func_fn``  normalization/fused_rmsnorm_cached.py:801-802
``triton_rope_fn``           rope/head_rope_cached.py:326-327
``triton_fused_ln_rope_fn``  rope/fused_ln_rope_cached.py:695-696
``flash_attn_func``          flash_attn/flash_attn_triton_cached.py:1131-1133
===========================  =======================================================

Differences from the reference, all deliberate:

* the entry points run on the native host path (``csrc/host/torch_host.cpp``: checks, allocation,
  launch and the autograd node in C++); what it does not cover comes back as None and is handled
  here, by the ``*_Func`` classes: arguments that are wrong (the exceptions are raised here), tensor
  subclasses, channel strides other than 1, empty tensors, bias gradients, in-place rotation, calls
  under a tracer, a dispatch mode or a functorch transform.
* ``kernel_cache`` slots hold a validated launch key (shapes, strides, dtypes)
  instead of a compiled-kernel handle.  A call whose key differs re-validates
  and replaces the slot, so one module can be reused across shapes and dtypes
  (the reference silently mis-launches in that case).
* Row statistics are recomputed in the backward kernels, so nothing but the
  inputs is saved for backward (attention still saves O and LSE).
* ``triton_rope_fn`` is out of place unless ``in_place=True`` is passed by
  keyword; the reference's positional slip made the cached module path
  overwrite its inputs (rope/head_rope_cached.py:326-327 vs :279).
* RMSNorm's dweight is summed over batches in fp32 and rounded once.

Argument checks raise ``AssertionError`` explicitly (not ``assert``), so they
survive ``python -O``.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import threading
import weakref

import torch

from . import _lib
from ._lib import Bias, Heads, Rows

_FLOATS = (torch.float16, torch.bfloat16, torch.float32)


def _require(cond: bool, msg: str = "") -> None:
    if not cond:
        raise AssertionError(msg)


def _last_contig(t: torch.Tensor) -> torch.Tensor:
    """The kernels need a unit channel stride; anything else is copied, as in
    the reference.  Empty and single-channel tensors may report any stride."""
    if t.stride(-1) == 1:
        return t
    t = t.contiguous()
    if t.stride(-1) != 1:              # numel == 0 or a size-1 last dimension
        t = t.new_empty(t.shape).copy_(t)
    return t


def _i64(*vals) -> C.Array:
    return (C.c_int64 * len(vals))(*vals)


def _key(*tensors, extra=()) -> tuple:
    return tuple((tuple(t.shape), t.stride(), t.dtype, t.device.index) for t in tensors if t is not None) + tuple(extra)


def _plan(cache, slot: str, key, validate):
    """Launch plan of `slot` for this key.

    With a module cache: when the slot already holds `key` (same shapes,
    strides, dtypes, device as the last validated call) the stored plan is
    returned and host-side validation is skipped; otherwise `validate()` runs,
    the slot takes the new key and a fresh, empty plan.  The plan is a dict in
    which the launch helpers keep their marshalled ctypes arguments, so a
    repeated call only refreshes the data pointers.  A plan belongs to the thread
    that made it: another one, which could refresh the same pointers between this
    thread's refresh and its launch, makes its own.  Without a cache every call
    validates and marshals from scratch (returns None)."""
    if cache is None:
        validate()
        return None
    store, thread = cache.__dict__, threading.get_ident()
    ent = store.get("_plan_" + slot)
    if ent is not None and ent[0] == key and ent[2] == thread:
        return ent[1]
    validate()
    setattr(cache, slot, key)
    plan = {}
    store["_plan_" + slot] = (key, plan, thread)
    return plan


def _native_cache(cache):
    """The library's launch-plan cache behind a module cache (None without one)."""
    native = getattr(cache, "native", None)
    return native() if native is not None else None


def _tracing() -> bool:
    """True while torch.compile is tracing: the entry points then call the registered custom
    operators (rgd_triton_b200.library) instead of the eager path, which a tracer cannot follow
    into ctypes."""
    if torch.compiler.is_compiling():
        from . import library  # noqa: F401  (registers torch.ops.rgd_b200.*)
        return True
    return False


_HOST = None


def _bind_host(t):
    """The native host path, loaded on the first CUDA tensor.  None for anything else: the Python path
    then raises (there is no CPU path)."""
    global _HOST
    if _HOST is None and isinstance(t, torch.Tensor) and t.is_cuda:
        host = _lib.host()
        host.set_single_pass(_ATTN_BWD_MODE == "single_pass")
        _HOST = host
    return _HOST


def _needs_grad(*tensors) -> bool:
    """Whether autograd has to record this call.  When it does not, the entry
    points run the forward directly instead of through autograd.Function, whose
    bookkeeping costs more host time than a small operator's whole launch."""
    if not torch.is_grad_enabled():
        return False
    for t in tensors:
        if t is not None and t.requires_grad:
            return True
    return False


def _rows_arr(plan, tag: str, tensors):
    """ctypes array of rgd_rows for `tensors`; kept in the plan, pointers refreshed."""
    arr = plan.get(tag) if plan is not None else None
    if arr is None:
        arr = (Rows * len(tensors))(*[_lib.rows(t) for t in tensors])
        if plan is not None:
            plan[tag] = arr
    else:
        for a, t in zip(arr, tensors):
            a.ptr = t.data_ptr()
    return arr


def _heads_refs(plan, tag: str, tensors, layout):
    """byref()s of rgd_heads structs for `tensors` (None stays None); `layout` maps a tensor
    to its struct.  The structs are kept in the plan, pointers refreshed."""
    hs = plan.get(tag) if plan is not None else None
    if hs is None:
        hs = [None if t is None else layout(t) for t in tensors]
        if plan is not None:
            plan[tag] = hs
    else:
        for h, t in zip(hs, tensors):
            if h is not None:
                h.ptr = t.data_ptr()
    return [None if h is None else C.byref(h) for h in hs]


def _const(plan, tag: str, make):
    """A value that depends only on the launch key (sizes, dtype codes), made once per plan."""
    if plan is None:
        return make()
    v = plan.get(tag)
    if v is None:
        v = plan[tag] = make()
    return v


# --------------------------------------------------------------------------
# Row L2 normalise
# --------------------------------------------------------------------------
def _check_rows(xs, what: str) -> None:
    for x in xs:
        _require(x.ndim == 3, f"{what}: expected [B, N, C] tensors, got {tuple(x.shape)}")
        _require(x.dtype in _FLOATS, "Only support fp16, bf16, and fp32")
        _require(x.stride(-1) == 1 or x.numel() == 0 or x.shape[-1] == 1,
                 f"{what}: last dimension must be contiguous")
        _lib.require_device(x)
    _require(all(x.dtype == xs[0].dtype for x in xs), "All tensors must have the same type")
    _require(all(x.shape[0] == xs[0].shape[0] for x in xs), f"{what}: batch sizes differ")


def _row_sizes(plan, xs):
    return _const(plan, "sizes", lambda: (_i64(*[t.shape[1] for t in xs]), _i64(*[t.shape[2] for t in xs]),
                                          xs[0].shape[0], _lib.dtype_code(xs[0].dtype)))


def _l2_launch(plan, xs, dys, outs, eps: float, bwd: bool) -> None:
    lib = _lib.load()
    n = len(xs)
    N, Cc, B, dt = _row_sizes(plan, xs)
    xa, oa = _rows_arr(plan, "x", xs), _rows_arr(plan, "out", outs)
    with _lib.device_guard(xs[0]):
        if bwd:
            code = lib.rgd_l2norm_bwd(n, xa, _rows_arr(plan, "dy", dys), oa, N, Cc, B, float(eps), dt, _lib.stream_ptr())
        else:
            code = lib.rgd_l2norm_fwd(n, xa, oa, N, Cc, B, float(eps), dt, _lib.stream_ptr())
    if code:
        _lib.check(code, "l2norm_bwd" if bwd else "l2norm_fwd")


def _l2_forward(xs, eps, cache, tag):
    xs = [_last_contig(x) for x in xs]
    plan = _plan(cache, "fwd", _key(*xs, extra=("l2", tag)), lambda: _check_rows(xs, tag))
    ys = [torch.empty_like(x) for x in xs]
    _l2_launch(plan, xs, None, ys, eps, bwd=False)
    return xs, ys


def _l2_backward(xs, dys, eps, cache, tag):
    dys = [_last_contig(d) for d in dys]

    def validate():
        _check_rows([*xs, *dys], tag + " backward")
        _require(all(d.shape == x.shape for d, x in zip(dys, xs)), "gradient shape mismatch")
    plan = _plan(cache, "bwd", _key(*xs, *dys, extra=("l2", tag)), validate)
    dxs = [torch.empty_like(x) for x in xs]
    _l2_launch(plan, xs, dys, dxs, eps, bwd=True)
    return dxs


class Norm_Func(torch.autograd.Function):
    """y = x / max(||x||_2, eps) over the last dim of [B, N, C] (l2normalize_cached.py:402-433)."""

    @staticmethod
    def forward(ctx, x, norm_eps=1e-6, use_ptx=False, kernel_cache=None):
        (x,), (y,) = _l2_forward([x], norm_eps, kernel_cache, "L2Normalize")
        ctx.save_for_backward(x)
        ctx.norm_eps = norm_eps
        ctx.kernel_cache = kernel_cache
        return y

    @staticmethod
    def backward(ctx, dy):
        (dx,) = _l2_backward(list(ctx.saved_tensors), [dy], ctx.norm_eps, ctx.kernel_cache, "L2Normalize")
        return dx, None, None, None


def triton_norm_func_fn(x, norm_eps=1e-6, use_ptx=False, kernel_cache=None):
    """L2-normalise the rows of x.  ``use_ptx`` is accepted and ignored."""
    if _tracing():
        return torch.ops.rgd_b200.l2norm([x], float(norm_eps))[0]
    host = _HOST or _bind_host(x)
    if host is not None:
        out = host.rows(kernel_cache, norm_eps, False, x)
        if out is not None:
            return out
    if not _needs_grad(x):
        return _l2_forward([x], norm_eps, kernel_cache, "L2Normalize")[1][0]
    return Norm_Func.apply(x, norm_eps, use_ptx, kernel_cache)


class Fused_Norm_Func(torch.autograd.Function):
    """Two L2 normalisations in one launch (fused_l2normalize_cached.py:464-503)."""

    @staticmethod
    def forward(ctx, x1, x2, norm_eps=1e-6, kernel_cache=None):
        xs, ys = _l2_forward([x1, x2], norm_eps, kernel_cache, "FusedL2Normalize2")
        ctx.save_for_backward(*xs)
        ctx.norm_eps = norm_eps
        ctx.kernel_cache = kernel_cache
        return ys[0], ys[1]

    @staticmethod
    def backward(ctx, dy1, dy2):
        dx1, dx2 = _l2_backward(list(ctx.saved_tensors), [dy1, dy2], ctx.norm_eps, ctx.kernel_cache,
                                "FusedL2Normalize2")
        return dx1, dx2, None, None


def triton_fused_norm_func_fn(x1, x2, norm_eps=1e-6, kernel_cache=None):
    if _tracing():
        y1, y2 = torch.ops.rgd_b200.l2norm([x1, x2], float(norm_eps))
        return y1, y2
    host = _HOST or _bind_host(x1)
    if host is not None:
        out = host.rows(kernel_cache, norm_eps, False, x1, x2)
        if out is not None:
            return out
    if not _needs_grad(x1, x2):
        ys = _l2_forward([x1, x2], norm_eps, kernel_cache, "FusedL2Normalize2")[1]
        return ys[0], ys[1]
    return Fused_Norm_Func.apply(x1, x2, norm_eps, kernel_cache)


# --------------------------------------------------------------------------
# Row RMS norm with affine weight
# --------------------------------------------------------------------------
def _prep_weight(w: torch.Tensor, x: torch.Tensor):
    """Return (weight tensor, batch stride, per_batch) for the accepted weight
    forms [C], [1,1,C] (shared) and [B,1,C] (per batch) — rmsnorm_cached.py:582-589."""
    w = _last_contig(w)
    B, _, Cx = x.shape
    if w.ndim == 1:
        _require(w.shape[0] == Cx, f"weight has {w.shape[0]} channels, x has {Cx}")
        return w, 0, False
    _require(w.ndim == 3, f"weight must be [C] or [B|1, 1, C], got {tuple(w.shape)}")
    _require(w.shape[1] == 1, "sequence-dependent weights are not supported")
    _require(w.shape[2] == Cx, f"weight has {w.shape[2]} channels, x has {Cx}")
    if w.shape[0] == 1:
        return w, 0, False
    _require(w.shape[0] == B, "weight batch must be 1 or match x")
    return w, w.stride(0), True


def _check_weights(preps, xs) -> None:
    _require(all(p[0].dtype == preps[0][0].dtype for p in preps), "weights must share one dtype")
    for p in preps:
        _require(p[0].dtype in _FLOATS, "Only support fp16, bf16, and fp32")
        _require(p[0].device == xs[0].device, "weight and input are on different devices")


def _weight_ptrs(plan, ws):
    wp = plan.get("w") if plan is not None else None
    if wp is None:
        wp = (C.c_void_p * len(ws))(*[w.data_ptr() for w in ws])
        if plan is not None:
            plan["w"] = wp
    else:
        for i, w in enumerate(ws):
            wp[i] = w.data_ptr()
    return wp


def _rms_forward(xs, ws, eps, cache, tag):
    xs = [_last_contig(x) for x in xs]
    preps = None

    def validate():
        _check_rows(xs, tag)
        _check_weights([_prep_weight(w, x) for w, x in zip(ws, xs)], xs)
    plan = _plan(cache, "fwd", _key(*xs, *ws, extra=("rms", tag)), validate)
    meta = _const(plan, "wmeta", lambda: [_prep_weight(w, x)[1:] for w, x in zip(ws, xs)])   # (batch stride, per batch)
    wk = [_last_contig(w) for w in ws]
    lib = _lib.load()
    n = len(xs)
    N, Cc, B, dt = _row_sizes(plan, xs)
    wsb, wdt = _const(plan, "wconst", lambda: (_i64(*[m[0] for m in meta]), _lib.dtype_code(wk[0].dtype)))
    ys = [torch.empty_like(x) for x in xs]
    with _lib.device_guard(xs[0]):
        code = lib.rgd_rmsnorm_fwd(n, _rows_arr(plan, "x", xs), _weight_ptrs(plan, wk), wsb, _rows_arr(plan, "out", ys),
                                   N, Cc, B, float(eps), dt, wdt, _lib.stream_ptr())
    if code:
        _lib.check(code, "rmsnorm_fwd")
    return xs, wk, ys


def _rms_backward(xs, ws, dys, eps, cache, tag):
    dys = [_last_contig(d) for d in dys]

    def validate():
        _check_rows([*xs, *dys], tag + " backward")
        _check_weights([_prep_weight(w, x) for w, x in zip(ws, xs)], xs)
    plan = _plan(cache, "bwd", _key(*xs, *ws, *dys, extra=("rms", tag)), validate)
    if cache is not None:
        cache.bwd_dw = cache.bwd
    meta = _const(plan, "wmeta", lambda: [_prep_weight(w, x)[1:] for w, x in zip(ws, xs)])
    lib = _lib.load()
    n = len(xs)
    N, Cc, B, dt = _row_sizes(plan, xs)
    wsb, wdt, per, nbytes = _const(plan, "wconst", lambda: (
        _i64(*[m[0] for m in meta]), _lib.dtype_code(ws[0].dtype), (C.c_int * n)(*[1 if m[1] else 0 for m in meta]),
        int(lib.rgd_rmsnorm_bwd_workspace_bytes(n, N, Cc, B))))
    _require(nbytes >= 0, "rmsnorm_bwd: bad sizes")
    dxs = [torch.empty_like(x) for x in xs]
    dws = [torch.empty((B, x.shape[2]) if m[1] else (x.shape[2],), dtype=w.dtype, device=w.device)
           for m, x, w in zip(meta, xs, ws)]
    work = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=xs[0].device)
    dwp = (C.c_void_p * n)(*[t.data_ptr() for t in dws])
    with _lib.device_guard(xs[0]):
        code = lib.rgd_rmsnorm_bwd(n, _rows_arr(plan, "x", xs), _weight_ptrs(plan, ws), wsb, _rows_arr(plan, "dy", dys),
                                   _rows_arr(plan, "out", dxs), dwp, per, N, Cc, B, float(eps), dt, wdt,
                                   work.data_ptr(), work.numel(), _lib.stream_ptr())
    if code:
        _lib.check(code, "rmsnorm_bwd")
    return dxs, dws


class RMS_Func(torch.autograd.Function):
    """y = x * rsqrt(mean(x^2) + eps) * w  (rmsnorm_cached.py:572-625)."""

    @staticmethod
    def forward(ctx, x, w, norm_eps=1e-6, kernel_cache=None):
        (x,), (wk,), (y,) = _rms_forward([x], [w], norm_eps, kernel_cache, "FusedRMSNorm")
        ctx.save_for_backward(x, wk)
        ctx.wshape = w.shape
        ctx.norm_eps = norm_eps
        ctx.kernel_cache = kernel_cache
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        (dx,), (dw,) = _rms_backward([x], [w], [dy], ctx.norm_eps, ctx.kernel_cache, "FusedRMSNorm")
        return dx, dw.view(ctx.wshape), None, None


def triton_rms_func_fn(x, w, norm_eps=1e-6, kernel_cache=None):
    if _tracing():
        return torch.ops.rgd_b200.rmsnorm([x], [w], float(norm_eps))[0]
    host = _HOST or _bind_host(x)
    if host is not None:
        out = host.rows(kernel_cache, norm_eps, True, x, w)
        if out is not None:
            return out
    if not _needs_grad(x, w):
        return _rms_forward([x], [w], norm_eps, kernel_cache, "FusedRMSNorm")[2][0]
    return RMS_Func.apply(x, w, norm_eps, kernel_cache)


class Fused_RMS_Func(torch.autograd.Function):
    """Two RMS norms with separate weights in one launch (fused_rmsnorm_cached.py:725-798)."""

    @staticmethod
    def forward(ctx, x1, x2, w1, w2, norm_eps=1e-6, kernel_cache=None):
        xs, wk, ys = _rms_forward([x1, x2], [w1, w2], norm_eps, kernel_cache, "FusedRMSNorm2")
        ctx.save_for_backward(*xs, *wk)
        ctx.w1shape, ctx.w2shape = w1.shape, w2.shape
        ctx.norm_eps = norm_eps
        ctx.kernel_cache = kernel_cache
        return ys[0], ys[1]

    @staticmethod
    def backward(ctx, dy1, dy2):
        x1, x2, w1, w2 = ctx.saved_tensors
        (dx1, dx2), (dw1, dw2) = _rms_backward([x1, x2], [w1, w2], [dy1, dy2], ctx.norm_eps, ctx.kernel_cache,
                                               "FusedRMSNorm2")
        return dx1, dx2, dw1.view(ctx.w1shape), dw2.view(ctx.w2shape), None, None


def triton_fused_rms_func_fn(x1, x2, w1, w2, norm_eps=1e-6, kernel_cache=None):
    if _tracing():
        y1, y2 = torch.ops.rgd_b200.rmsnorm([x1, x2], [w1, w2], float(norm_eps))
        return y1, y2
    host = _HOST or _bind_host(x1)
    if host is not None:
        out = host.rows(kernel_cache, norm_eps, True, x1, x2, w1, w2)
        if out is not None:
            return out
    if not _needs_grad(x1, x2, w1, w2):
        ys = _rms_forward([x1, x2], [w1, w2], norm_eps, kernel_cache, "FusedRMSNorm2")[2]
        return ys[0], ys[1]
    return Fused_RMS_Func.apply(x1, x2, w1, w2, norm_eps, kernel_cache)


# --------------------------------------------------------------------------
# Head operators: LayerNorm, RoPE, LayerNorm -> RoPE
# --------------------------------------------------------------------------
def _head_dims(q, k, heads_second: bool):
    if heads_second:
        bq, hq, nq, dq = q.shape
        bk, hk, nk, dk = k.shape
    else:
        bq, nq, hq, dq = q.shape
        bk, nk, hk, dk = k.shape
    _require((bq, hq, dq) == (bk, hk, dk), f"q and k must share (batch, heads, head_dim): {q.shape} vs {k.shape}")
    return bq, hq, nq, nk, dq


def _check_heads(ts, what: str, dmax: int) -> None:
    for t in ts:
        _require(t.ndim == 4, f"{what}: expected 4-D tensors, got {tuple(t.shape)}")
        _require(t.dtype in _FLOATS, "Only support fp16, bf16, and fp32")
        _require(t.stride(-1) == 1 or t.numel() == 0 or t.shape[-1] == 1,
                 f"{what}: last dimension must be contiguous")
        _lib.require_device(t)
    _require(all(t.dtype == ts[0].dtype for t in ts), "All tensors must have the same type")
    _require(ts[0].shape[-1] <= dmax, f"Only supports head dimensions up to {dmax}")


def _cutoffs(seq_cutoff, nq: int, nk: int):
    """seq_cutoff: None, an int, or a (q, k) pair (head_rope_cached.py:193-201)."""
    if seq_cutoff is None:
        return nq, nk
    if isinstance(seq_cutoff, (tuple, list)):
        return int(seq_cutoff[0]), int(seq_cutoff[1])
    return int(seq_cutoff), int(seq_cutoff)


def _prep_pos(pos_emb: torch.Tensor, x: torch.Tensor, nq: int, nk: int) -> torch.Tensor:
    _require(pos_emb.ndim == 3, f"pos_emb must be [2, P, R], got {tuple(pos_emb.shape)}")
    _require(pos_emb.shape[0] == 2, "pos_emb[0] is sin and pos_emb[1] is cos")
    _require(pos_emb.is_cuda and pos_emb.device == x.device, "pos_emb must be on the tensors' device")
    _require(pos_emb.dtype in _FLOATS, "Only support fp16, bf16, and fp32")
    _require(nq < pos_emb.shape[1] and nk < pos_emb.shape[1],
             "pos_emb must hold more positions than the longest sequence")
    pos_emb = _last_contig(pos_emb)
    # Arithmetic runs in the promoted type of x and the table: a table that is
    # neither x's type nor fp32 promotes to fp32 anyway.
    if pos_emb.dtype != x.dtype and pos_emb.dtype != torch.float32:
        pos_emb = pos_emb.float()
    return pos_emb


def _ln_launch(plan, q, k, dqo, dko, qo, ko, heads_second, eps, bwd):
    lib = _lib.load()
    dims = _const(plan, "dims", lambda: (*_head_dims(q, k, heads_second), _lib.dtype_code(q.dtype)))
    B, H, nq, nk, d, dt = dims
    lay = lambda t: _lib.heads(t, heads_second)
    with _lib.device_guard(q):
        if bwd:
            h = _heads_refs(plan, "h", (q, k, dqo, dko, qo, ko), lay)
            code = lib.rgd_headln_bwd(*h, B, H, nq, nk, d, float(eps), dt, _lib.stream_ptr())
        else:
            h = _heads_refs(plan, "h", (q, k, qo, ko), lay)
            code = lib.rgd_headln_fwd(*h, B, H, nq, nk, d, float(eps), dt, _lib.stream_ptr())
    if code:
        _lib.check(code, "headln_bwd" if bwd else "headln_fwd")


def _ln_forward(q, k, heads_second, eps, cache):
    q, k = _last_contig(q), _last_contig(k)

    def validate():
        _check_heads([q, k], "FusedHeadLayerNorm", 256)
        _head_dims(q, k, heads_second)
    plan = _plan(cache, "fwd", _key(q, k, extra=("ln", bool(heads_second))), validate)
    qo, ko = torch.empty_like(q), torch.empty_like(k)
    _ln_launch(plan, q, k, None, None, qo, ko, heads_second, eps, bwd=False)
    return q, k, qo, ko


class Fused_LNQK_Func(torch.autograd.Function):
    """Non-affine LayerNorm over head_dim of Q and K in one launch
    (head_layernorm_cached.py:416-453)."""

    @staticmethod
    def forward(ctx, q, k, heads_second=True, norm_eps=1e-6, kernel_cache=None):
        q, k, qo, ko = _ln_forward(q, k, heads_second, norm_eps, kernel_cache)
        ctx.save_for_backward(q, k)
        ctx.heads_second, ctx.norm_eps, ctx.kernel_cache = heads_second, norm_eps, kernel_cache
        return qo, ko

    @staticmethod
    def backward(ctx, dqo, dko):
        q, k = ctx.saved_tensors
        dqo, dko = _last_contig(dqo), _last_contig(dko)

        def validate():
            _check_heads([q, k, dqo, dko], "FusedHeadLayerNorm backward", 256)
            _require(dqo.shape == q.shape and dko.shape == k.shape, "gradient shape mismatch")
        plan = _plan(ctx.kernel_cache, "bwd", _key(q, k, dqo, dko, extra=("ln", bool(ctx.heads_second))), validate)
        dq, dk = torch.empty_like(dqo), torch.empty_like(dko)
        _ln_launch(plan, q, k, dqo, dko, dq, dk, ctx.heads_second, ctx.norm_eps, bwd=True)
        return dq, dk, None, None, None


def triton_fused_ln_func_fn(query, key, heads_second=True, norm_eps=1e-6, kernel_cache=None):
    if _tracing():
        return torch.ops.rgd_b200.headln(query, key, bool(heads_second), float(norm_eps))
    host = _HOST or _bind_host(query)
    if host is not None:
        out = host.headln(kernel_cache, norm_eps, heads_second, query, key)
        if out is not None:
            return out
    if not _needs_grad(query, key):
        return _ln_forward(query, key, heads_second, norm_eps, kernel_cache)[2:]
    return Fused_LNQK_Func.apply(query, key, heads_second, norm_eps, kernel_cache)


def _rope_consts(plan, q, k, pos, cuts, heads_second):
    return _const(plan, "dims", lambda: (*_head_dims(q, k, heads_second), pos.shape[1], pos.shape[2], cuts[0], cuts[1],
                                         _lib.dtype_code(q.dtype), _lib.dtype_code(pos.dtype), pos.stride(0),
                                         pos.stride(1)))


def _rope_launch(plan, q, k, pos, qo, ko, cuts, heads_second, transposed):
    lib = _lib.load()
    B, H, nq, nk, d, P, R, cq, ck, dt, pdt, ps0, ps1 = _rope_consts(plan, q, k, pos, cuts, heads_second)
    qh, kh, qoh, koh = _heads_refs(plan, "h", (q, k, qo, ko), lambda t: _lib.heads(t, heads_second))
    with _lib.device_guard(q):
        code = lib.rgd_rope(qh, kh, pos.data_ptr(), ps0, ps1, qoh, koh, B, H, nq, nk, d, P, R, cq, ck,
                            1 if transposed else 0, dt, pdt, _lib.stream_ptr())
    if code:
        _lib.check(code, "rope")


def _rope_forward(q, k, pos_emb, seq_cutoff, heads_second, in_place, cache):
    q, k = _last_contig(q), _last_contig(k)
    plan = _plan(cache, "fwd", _key(q, k, pos_emb, extra=("rope", bool(heads_second), _cut_key(seq_cutoff))),
                 lambda: _check_heads([q, k], "RoPE", 128))
    if plan is not None and "pos_ok" in plan and pos_emb.dtype in (q.dtype, torch.float32) and pos_emb.stride(-1) == 1:
        pos, cuts = pos_emb, plan["cuts"]          # validated for this key before; no conversion needed
    else:
        B, H, nq, nk, d = _head_dims(q, k, heads_second)
        pos = _prep_pos(pos_emb, q, nq, nk)
        cuts = _cutoffs(seq_cutoff, nq, nk)
        if plan is not None:
            plan["pos_ok"], plan["cuts"] = True, cuts
    if in_place:
        qo, ko = q, k
    else:
        qo, ko = torch.empty_like(q), torch.empty_like(k)
    _rope_launch(plan, q, k, pos, qo, ko, cuts, heads_second, transposed=False)
    return q, k, pos, cuts, qo, ko


def _cut_key(seq_cutoff):
    return tuple(seq_cutoff) if isinstance(seq_cutoff, (tuple, list)) else seq_cutoff


class CombinedRoPEFunc(torch.autograd.Function):
    """Interleaved-pair rotary embedding on the first R channels of the first
    `cutoff` tokens of Q and K, one launch (head_rope_cached.py:277-323).  The
    backward is the same kernel with the rotation inverted, applied to the
    upstream gradients."""

    @staticmethod
    def forward(ctx, q, k, pos_emb, seq_cutoff=None, heads_second=True, in_place=False, kernel_cache=None):
        q, k, pos, cuts, qo, ko = _rope_forward(q, k, pos_emb, seq_cutoff, heads_second, in_place, kernel_cache)
        if in_place:
            ctx.mark_dirty(q, k)
        ctx.save_for_backward(pos)
        ctx.cuts, ctx.heads_second, ctx.kernel_cache = cuts, heads_second, kernel_cache
        return qo, ko

    @staticmethod
    def backward(ctx, dqo, dko):
        (pos,) = ctx.saved_tensors
        _require(not ctx.needs_input_grad[2], "CombinedRoPE does not support gradients in position embeddings")
        dqo, dko = _last_contig(dqo), _last_contig(dko)
        plan = _plan(ctx.kernel_cache, "bwd", _key(dqo, dko, pos, extra=("rope", bool(ctx.heads_second), ctx.cuts)),
                     lambda: _check_heads([dqo, dko], "RoPE backward", 128))
        dq, dk = torch.empty_like(dqo), torch.empty_like(dko)
        _rope_launch(plan, dqo, dko, pos, dq, dk, ctx.cuts, ctx.heads_second, transposed=True)
        return dq, dk, None, None, None, None, None


def triton_rope_fn(query, key, pos_emb, seq_cutoff=None, heads_second=True, fused_ln=False, kernel_cache=None,
                   in_place=False):
    """Rotary embedding on (query, key).  ``fused_ln`` is accepted for
    signature parity and ignored, as in the reference."""
    if _tracing() and not in_place:
        nq, nk = (query.shape[2], key.shape[2]) if heads_second else (query.shape[1], key.shape[1])
        cq, ck = _cutoffs(seq_cutoff, nq, nk)
        return torch.ops.rgd_b200.rope(query, key, pos_emb, cq, ck, bool(heads_second), False)
    host = _HOST or _bind_host(query)
    if host is not None and not in_place:
        out = host.rotary(kernel_cache, None, heads_second, query, key, pos_emb, seq_cutoff)
        if out is not None:
            return out
    if not _needs_grad(query, key, pos_emb):
        return _rope_forward(query, key, pos_emb, seq_cutoff, heads_second, in_place, kernel_cache)[4:]
    return CombinedRoPEFunc.apply(query, key, pos_emb, seq_cutoff, heads_second, in_place, kernel_cache)


def _lnrope_launch(plan, q, k, dqo, dko, pos, qo, ko, cuts, heads_second, eps, bwd):
    lib = _lib.load()
    B, H, nq, nk, d, P, R, cq, ck, dt, pdt, ps0, ps1 = _rope_consts(plan, q, k, pos, cuts, heads_second)
    lay = lambda t: _lib.heads(t, heads_second)
    tail = (B, H, nq, nk, d, P, R, cq, ck, float(eps), dt, pdt, _lib.stream_ptr())
    with _lib.device_guard(q):
        if bwd:
            qh, kh, dqh, dkh, qoh, koh = _heads_refs(plan, "h", (q, k, dqo, dko, qo, ko), lay)
            code = lib.rgd_lnrope_bwd(qh, kh, dqh, dkh, pos.data_ptr(), ps0, ps1, qoh, koh, *tail)
        else:
            qh, kh, qoh, koh = _heads_refs(plan, "h", (q, k, qo, ko), lay)
            code = lib.rgd_lnrope_fwd(qh, kh, pos.data_ptr(), ps0, ps1, qoh, koh, *tail)
    if code:
        _lib.check(code, "lnrope_bwd" if bwd else "lnrope_fwd")


def _lnrope_forward(q, k, pos_emb, seq_cutoff, heads_second, eps, cache):
    q, k = _last_contig(q), _last_contig(k)
    plan = _plan(cache, "fwd", _key(q, k, pos_emb, extra=("lnrope", bool(heads_second), _cut_key(seq_cutoff))),
                 lambda: _check_heads([q, k], "FusedLNRoPE", 128))
    if plan is not None and "pos_ok" in plan and pos_emb.dtype in (q.dtype, torch.float32) and pos_emb.stride(-1) == 1:
        pos, cuts = pos_emb, plan["cuts"]
    else:
        B, H, nq, nk, d = _head_dims(q, k, heads_second)
        pos = _prep_pos(pos_emb, q, nq, nk)
        cuts = _cutoffs(seq_cutoff, nq, nk)
        if plan is not None:
            plan["pos_ok"], plan["cuts"] = True, cuts
    qo, ko = torch.empty_like(q), torch.empty_like(k)
    _lnrope_launch(plan, q, k, None, None, pos, qo, ko, cuts, heads_second, eps, bwd=False)
    return q, k, pos, cuts, qo, ko


class FusedRoPEFunc(torch.autograd.Function):
    """Head LayerNorm followed by rotary embedding in one launch; backward is
    inverse rotation then LayerNorm backward (fused_ln_rope_cached.py:649-692)."""

    @staticmethod
    def forward(ctx, q, k, pos_emb, seq_cutoff=None, heads_second=True, norm_eps=1e-6, kernel_cache=None):
        q, k, pos, cuts, qo, ko = _lnrope_forward(q, k, pos_emb, seq_cutoff, heads_second, norm_eps, kernel_cache)
        ctx.save_for_backward(q, k, pos)
        ctx.cuts, ctx.heads_second, ctx.norm_eps, ctx.kernel_cache = cuts, heads_second, norm_eps, kernel_cache
        return qo, ko

    @staticmethod
    def backward(ctx, dqo, dko):
        q, k, pos = ctx.saved_tensors
        _require(not ctx.needs_input_grad[2], "CombinedRoPE does not support gradients in position embeddings")
        dqo, dko = _last_contig(dqo), _last_contig(dko)
        plan = _plan(ctx.kernel_cache, "bwd",
                     _key(q, k, dqo, dko, pos, extra=("lnrope", bool(ctx.heads_second), ctx.cuts)),
                     lambda: _check_heads([q, k, dqo, dko], "FusedLNRoPE backward", 128))
        dq, dk = torch.empty_like(dqo), torch.empty_like(dko)
        _lnrope_launch(plan, q, k, dqo, dko, pos, dq, dk, ctx.cuts, ctx.heads_second, ctx.norm_eps, bwd=True)
        return dq, dk, None, None, None, None, None


def triton_fused_ln_rope_fn(query, key, pos_emb, seq_cutoff=None, heads_second=True, norm_eps=1e-6,
                            kernel_cache=None):
    if _tracing():
        nq, nk = (query.shape[2], key.shape[2]) if heads_second else (query.shape[1], key.shape[1])
        cq, ck = _cutoffs(seq_cutoff, nq, nk)
        return torch.ops.rgd_b200.lnrope(query, key, pos_emb, cq, ck, bool(heads_second), float(norm_eps))
    host = _HOST or _bind_host(query)
    if host is not None:
        out = host.rotary(kernel_cache, norm_eps, heads_second, query, key, pos_emb, seq_cutoff)
        if out is not None:
            return out
    if not _needs_grad(query, key, pos_emb):
        return _lnrope_forward(query, key, pos_emb, seq_cutoff, heads_second, norm_eps, kernel_cache)[4:]
    return FusedRoPEFunc.apply(query, key, pos_emb, seq_cutoff, heads_second, norm_eps, kernel_cache)


# --------------------------------------------------------------------------
# FlashAttention
# --------------------------------------------------------------------------
def _attn_heads(t: torch.Tensor) -> Heads:
    # attention tensors are (batch, seqlen, nheads, headdim)
    return Heads(t.data_ptr(), t.stride(0), t.stride(2), t.stride(1))


def _prep_bias(bias, q, seqlen_q: int, seqlen_k: int):
    """Validate the bias and return (last-dim-contiguous bias, rgd_bias struct).
    Same rules as flash_attn_triton_cached.py:771-788."""
    if bias is None:
        return None, Bias(None, 0, 0, 0, _lib.RGD_BIAS_NONE, _lib.RGD_F32, None)
    batch, _, nheads, _ = q.shape
    _require(bias.dtype in (q.dtype, torch.float32), "bias must have q's dtype or float32")
    _require(bias.is_cuda and bias.device == q.device, "bias must be on q's device")
    _require(bias.dim() == 4, "bias must be 4-D")
    if bias.stride(-1) != 1:
        bias = bias.contiguous()
    if tuple(bias.shape[2:]) == (1, seqlen_k):
        kind = _lib.RGD_BIAS_VECTOR
    elif tuple(bias.shape[2:]) == (seqlen_q, seqlen_k):
        kind = _lib.RGD_BIAS_MATRIX
    else:
        raise RuntimeError("Last 2 dimensions of bias must be (1, seqlen_k) or (seqlen_q, seqlen_k)")
    full = bias.expand(batch, nheads, seqlen_q, seqlen_k)   # broadcast dims get stride 0
    sq = full.stride(2) if kind == _lib.RGD_BIAS_MATRIX else 0
    return bias, Bias(full.data_ptr(), full.stride(0), full.stride(1), sq, kind, _lib.dtype_code(full.dtype), None)


def _check_attn(q, k, v) -> None:
    _require(q.ndim == 4 and k.ndim == 4 and v.ndim == 4, "q, k, v must be (batch, seqlen, nheads, headdim)")
    batch, seqlen_q, nheads, d = q.shape
    seqlen_k = k.shape[1]
    _require(tuple(k.shape) == (batch, seqlen_k, nheads, d), f"k shape {tuple(k.shape)} does not match q")
    _require(tuple(v.shape) == (batch, seqlen_k, nheads, d), f"v shape {tuple(v.shape)} does not match k")
    _require(d <= 128, "FlashAttention only support head dimensions up to 128")
    _require(q.dtype == k.dtype == v.dtype, f"All tensors must have the same type {q.dtype=}, {k.dtype=}, {v.dtype=}")
    _require(q.dtype in (torch.float16, torch.bfloat16), "Only support fp16 and bf16")
    for t in (q, k, v):
        _lib.require_device(t)


# Block-sparse skip of masked bias tiles.  A matrix bias that a module's cache sees for the second
# time (the same tensor object, unchanged: identity through a weak reference plus the tensor's
# version counter) is scanned once for 128 x 128 tiles whose every element is <= -1e4 (-9984, which is
# what bf16 makes of -1e4); the
# tensor-memory kernels then skip those tiles (their probabilities are exactly zero, so results are
# bit-identical as long as |score * scale| stays far below 5e3; a query block containing a row with
# no unmasked key keeps all its tiles).  One-shot biases are never scanned: the scan reads the
# whole bias once, which only pays when the result is reused; and the lists are used only when they
# leave out at least a fifth of the tiles.
_SKIP_MASKED_TILES = True
_SKIP_THRESHOLD = -9984.0   # -1e4 as bf16 stores it (fp16 and fp32 hold -1e4 itself): masked means <= this
_SKIP_MIN_TILES = 64        # score tiles per (batch, head) below which the lists are not worth making
_SKIP_MIN_FRACTION = 0.2    # the list-following kernel instantiations run about 7 % slower per visited tile
                            # (dK/dV 17 %, forward 2 %, dQ 0 %): lists are used when at least this share is skipped


def set_skip_masked_tiles(enable: bool) -> bool:
    """Turn the block-sparse skip of masked bias tiles on or off; returns the previous setting."""
    global _SKIP_MASKED_TILES
    prev, _SKIP_MASKED_TILES = _SKIP_MASKED_TILES, bool(enable)
    return prev


def _bias_tiles(cache, bias, bias_t, bias_s, q, seqlen_q, seqlen_k, causal):
    """The tile-list buffer for this bias, or None (see above)."""
    if (cache is None or bias is None or causal or not _SKIP_MASKED_TILES or bias_s.kind != _lib.RGD_BIAS_MATRIX
            or bias_t.dtype == torch.float32 or bias.requires_grad or _tracing()
            or ((seqlen_q + 127) // 128) * ((seqlen_k + 127) // 128) < _SKIP_MIN_TILES):
        return None
    ent = getattr(cache, "_tiles", None)
    ver = bias._version
    if ent is not None and ent[0]() is bias and ent[1] == ver:
        if ent[2] is None:          # seen before, unchanged: scan it now
            lib = _lib.load()
            batch, _, nheads, _ = q.shape
            nbytes = int(lib.rgd_attn_bias_tiles_bytes(batch, nheads, seqlen_q, seqlen_k))
            buf = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=q.device)
            with _lib.device_guard(q):
                code = lib.rgd_attn_bias_tiles_build(C.byref(bias_s), batch, nheads, seqlen_q, seqlen_k,
                                                     _SKIP_THRESHOLD, buf.data_ptr(), buf.numel(), _lib.stream_ptr())
            if code == 0:
                # one read-back per bias tensor: how many tiles the lists leave out
                nqb, nkb = (seqlen_q + 127) // 128, (seqlen_k + 127) // 128
                slices = (1 if bias_s.stride_b == 0 else batch) * (1 if bias_s.stride_h == 0 else nheads)
                counts = buf[:2 * slices * nqb].view(torch.int16).to(torch.int32) & 0xFFFF      # qcnt comes first
                skipped = 1.0 - float(counts.sum().item()) / float(slices * nqb * nkb)
                ent[2] = buf if skipped >= _SKIP_MIN_FRACTION else False
                ent.append(skipped)
            else:
                ent[2] = False
        return ent[2] if torch.is_tensor(ent[2]) else None
    cache._tiles = [weakref.ref(bias), ver, None]
    return None


def _broadcast(bias, q):
    """Over which of (batch, heads) the bias is broadcast: stride 0 there."""
    return None if bias is None else tuple(s == 0 for s in bias.expand(q.shape[0], q.shape[2], -1, -1).stride()[:2])


def _native_tiles(cache, bias, q, k, causal):
    """_bias_tiles for the native host path: the same policy, with the cheap refusals first so that an
    ordinary call does not describe its bias twice."""
    if (cache is None or causal or not _SKIP_MASKED_TILES or bias.ndim != 4 or q.ndim != 4 or k.ndim != 4
            or bias.shape[2] == 1 or bias.dtype == torch.float32 or bias.requires_grad or bias.stride(-1) != 1
            or not bias.is_cuda or tuple(bias.shape[2:]) != (q.shape[1], k.shape[1])
            or ((q.shape[1] + 127) // 128) * ((k.shape[1] + 127) // 128) < _SKIP_MIN_TILES):
        return None
    ent = getattr(cache, "_tiles", None)
    if ent is not None and ent[2] is not None and ent[0]() is bias and ent[1] == bias._version:
        return ent[2] if torch.is_tensor(ent[2]) else None
    _check_attn(q, k, k)
    bias_t, bias_s = _prep_bias(bias, q, q.shape[1], k.shape[1])
    return _bias_tiles(cache, bias, bias_t, bias_s, q, q.shape[1], k.shape[1], causal)


def _attn_forward(q, k, v, bias, causal, softmax_scale, cache):
    q, k, v = _last_contig(q), _last_contig(k), _last_contig(v)
    plan = _plan(cache, "fwd", _key(q, k, v, bias, extra=("attn", bool(causal))), lambda: _check_attn(q, k, v))
    lib = _lib.load()
    batch, seqlen_q, nheads, d = q.shape
    seqlen_k = k.shape[1]
    softmax_scale = softmax_scale or 1.0 / math.sqrt(d)
    bias_t, bias_s = _prep_bias(bias, q, seqlen_q, seqlen_k)
    tiles = _bias_tiles(cache, bias, bias_t, bias_s, q, seqlen_q, seqlen_k, causal)
    if tiles is not None:
        bias_s.tiles = tiles.data_ptr()
    o = torch.empty_like(q)
    lse_rows, dt = _const(plan, "c", lambda: (int(lib.rgd_attn_lse_rows(seqlen_q)), _lib.dtype_code(q.dtype)))
    lse = torch.empty((batch, nheads, lse_rows), device=q.device, dtype=torch.float32)
    qh, kh, vh, oh = _heads_refs(plan, "h", (q, k, v, o), _attn_heads)
    with _lib.device_guard(q):
        code = lib.rgd_attn_fwd(qh, kh, vh, C.byref(bias_s), oh, lse.data_ptr(), batch, nheads, seqlen_q, seqlen_k, d,
                                float(softmax_scale), 1 if causal else 0, dt, _native_cache(cache), _lib.stream_ptr())
    if code:
        _lib.check(code, "attn_fwd")
    return q, k, v, o, lse, bias_t, softmax_scale, tiles


class FlashAttnFunc(torch.autograd.Function):
    """softmax(Q K^T * scale + bias) V with O(T) memory
    (flash_attn_triton_cached.py:1079-1129).  Returns (o, lse)."""

    @staticmethod
    def forward(ctx, q, k, v, bias=None, causal=False, softmax_scale=None, kernel_cache=None):
        q, k, v, o, lse, bias_t, softmax_scale, tiles = _attn_forward(q, k, v, bias, causal, softmax_scale, kernel_cache)
        ctx.save_for_backward(q, k, v, o, lse, bias_t)
        ctx.causal, ctx.softmax_scale, ctx.kernel_cache = causal, softmax_scale, kernel_cache
        # the backward of this call skips the same tiles, if the bias is still broadcast over the dimensions by
        # which their lists are indexed (saved-tensor hooks may have materialised it)
        ctx.tiles, ctx.tiles_bcast = tiles, _broadcast(bias_t, q)
        ctx.mark_non_differentiable(lse)
        return o, lse

    @staticmethod
    def backward(ctx, do, dlse):
        q, k, v, o, lse, bias = ctx.saved_tensors
        cache = ctx.kernel_cache
        want_dbias = bias is not None and ctx.needs_input_grad[3]
        tiles = ctx.tiles if ctx.tiles_bcast == _broadcast(bias, q) else None
        dq, dk, dv, dbias = _attn_backward(q, k, v, bias, o, lse, do, ctx.causal, ctx.softmax_scale, cache, want_dbias, tiles)
        if cache is not None:
            cache.bwd_odot = cache.bwd
        return dq, dk, dv, dbias, None, None, None


# How the attention backward forms dQ where the library offers a choice (on the tensor-memory kernels:
# head_dim 64, and smaller ones from 2^24 scores on):
#   "single_pass"  S, dP and the exponentials are evaluated once per tile pair and the dQ partial tiles
#                  are added into an fp32 accumulator (B * H * Tq * 64 * 4 bytes of scratch per call) with
#                  vector reductions, like the reference's atomic adds into dq
#                  (flash_attn_triton_cached.py:556-561): dK, dV bit-reproducible, dQ to its last bits only;
#   "two_kernel"   a dK/dV kernel and a dQ kernel, every output bit-reproducible, no accumulator.
_ATTN_BWD_MODE = os.environ.get("RGD_B200_ATTN_BWD", "single_pass")


def set_attention_backward(mode: str) -> str:
    """Select "single_pass" (default) or "two_kernel"; returns the previous setting."""
    global _ATTN_BWD_MODE
    _require(mode in ("single_pass", "two_kernel"), "mode must be 'single_pass' or 'two_kernel'")
    prev, _ATTN_BWD_MODE = _ATTN_BWD_MODE, mode
    if _HOST is not None:
        _HOST.set_single_pass(mode == "single_pass")
    return prev


def _attn_bwd_bytes(lib, single, *dims) -> int:
    nbytes = int(lib.rgd_attn_bwd_workspace_bytes(*dims))
    if single and nbytes >= 0:
        nbytes = max(nbytes, int(lib.rgd_attn_bwd_single_pass_workspace_bytes(*dims)))
    return nbytes


def _attn_backward(q, k, v, bias, o, lse, do, causal, softmax_scale, cache, want_dbias=False, tiles=None):
    """dq, dk, dv and, when asked for, the gradient of the bias (the reference refuses it,
    flash_attn_triton_cached.py:1107): d bias = P * (dP - delta), summed over the dimensions along
    which the bias is broadcast; a vector bias's sum over the queries is formed inside the dK/dV
    kernel, a matrix bias's gradient is written by the dQ kernel."""
    do = _last_contig(do)
    if q.shape[-1] not in (64, 128) and q.shape[-1] % 8 == 0 and _pad_head_dim_pays(q, k) and not _addressable(do):
        do = _dense(do)         # as for the inputs (flash_attn_func): o.sum(1) hands over a gradient of stride 0
    plan = _plan(cache, "bwd", _key(q, k, v, o, do, bias, extra=("attn", bool(causal), bool(want_dbias))),
                 lambda: _require(do.shape == q.shape and do.dtype == q.dtype, "dO must match q"))
    lib = _lib.load()
    batch, seqlen_q, nheads, d = q.shape
    seqlen_k = k.shape[1]
    _, bias_s = _prep_bias(bias, q, seqlen_q, seqlen_k)
    if tiles is not None and not want_dbias:
        bias_s.tiles = tiles.data_ptr()
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    single = _ATTN_BWD_MODE == "single_pass" and d <= 64 and not want_dbias and tiles is None
    dt, nbytes = _const(plan, ("c", single), lambda: (_lib.dtype_code(q.dtype), _attn_bwd_bytes(
        lib, single, batch, nheads, seqlen_q, seqlen_k, d, _lib.dtype_code(q.dtype))))
    _require(nbytes >= 0, "attn_bwd: bad sizes")
    work = torch.empty(max(nbytes, 16), dtype=torch.uint8, device=q.device)
    qh, kh, vh, oh, doh, dqh, dkh, dvh = _heads_refs(plan, "h", (q, k, v, o, do, dq, dk, dv), _attn_heads)
    dbias_s, dbuf = None, None
    if want_dbias:
        if bias_s.kind == _lib.RGD_BIAS_VECTOR:
            dbuf = torch.empty((batch, nheads, 1, seqlen_k), dtype=torch.float32, device=q.device)   # zeroed by the call
            dbias_s = Bias(dbuf.data_ptr(), nheads * seqlen_k, seqlen_k, 0, bias_s.kind, _lib.RGD_F32, None)
        else:
            # key blocks above the diagonal are skipped, not written, under a causal mask
            make = torch.zeros if causal else torch.empty
            dbuf = make((batch, nheads, seqlen_q, seqlen_k), dtype=q.dtype, device=q.device)
            dbias_s = Bias(dbuf.data_ptr(), dbuf.stride(0), dbuf.stride(1), dbuf.stride(2), bias_s.kind,
                           _lib.dtype_code(q.dtype), None)
    with _lib.device_guard(q):
        code = lib.rgd_attn_bwd_dbias(qh, kh, vh, C.byref(bias_s), oh, lse.data_ptr(), doh, dqh, dkh, dvh,
                                      None if dbias_s is None else C.byref(dbias_s), batch, nheads,
                                      seqlen_q, seqlen_k, d, float(softmax_scale), 1 if causal else 0, dt,
                                      work.data_ptr(), work.numel(), _native_cache(cache), _lib.stream_ptr())
    if code:
        _lib.check(code, "attn_bwd")
    dbias = None
    if want_dbias:
        # sum over the dimensions along which the bias is broadcast, in fp32, one rounding
        dims = [i for i in range(3) if bias.shape[i] == 1 and dbuf.shape[i] != 1]
        dbias = (dbuf.sum(dim=dims, keepdim=True, dtype=torch.float32) if dims else dbuf).to(bias.dtype)
        dbias = dbias.reshape(bias.shape)
    return dq, dk, dv, dbias


def _pad_head_dim_pays(q, k) -> bool:
    """Padding head_dim costs four extra passes over q, k, v, o (and as many in the backward);
    it pays once the score matrix is large."""
    return q.is_cuda and q.dtype in (torch.float16, torch.bfloat16) and \
        q.shape[0] * q.shape[2] * q.shape[1] * k.shape[1] >= (1 << 24)


def _addressable(t, zero_strides=False) -> bool:
    """Whether the aligned attention kernels take this view as it is: 16-byte rows, and positive strides (what is
    expanded over batch or heads has stride 0; the few-query forward takes that too)."""
    return t.stride(-1) == 1 and t.data_ptr() % 16 == 0 and all(
        s % 8 == 0 and (s > 0 or n == 1 or zero_strides) for s, n in zip(t.stride()[:3], t.shape[:3]))


def _dense(t):
    return t.clone(memory_format=torch.contiguous_format)


def flash_attn_func(q, k, v, bias=None, causal=False, softmax_scale=None, return_lse=False, kernel_cache=None):
    """q: (batch, seqlen_q, nheads, headdim); k, v: (batch, seqlen_k, nheads,
    headdim); bias: optional, 4-D, last two dims (1, seqlen_k) or (seqlen_q,
    seqlen_k), leading dims broadcastable to (batch, nheads).

    The tensor-memory kernels bound every device-side wait; should one ever run
    out, the call still returns and the results of that launch are invalid.
    ``rgd_triton_b200._lib.load().rgd_device_status()`` reports (and clears) that
    condition; poll it at a point where a device synchronisation is acceptable."""
    if _tracing():
        scale = float(softmax_scale or 1.0 / math.sqrt(q.shape[-1]))
        o, lse = torch.ops.rgd_b200.attn(q, k, v, bias, bool(causal), scale)
        return (o, lse) if return_lse else o
    d = q.shape[-1] if q.ndim == 4 else 0
    if d % 8 != 0 and d < 128 and _pad_head_dim_pays(q, k):
        # The tensor-memory kernels take head dims that are multiples of 8 (16-byte rows): large
        # problems with others are zero-padded to the next one (zero channels add nothing to q k^T, and
        # the padded channels of v give output channels that are cut off again); the softmax scale
        # stays that of the true head_dim.  Small problems run on the general kernels, where the copies
        # would cost more than they save.
        dp = (d + 7) // 8 * 8
        pad = lambda t: torch.nn.functional.pad(t, (0, dp - d))
        res = flash_attn_func(pad(q), pad(k), pad(v), bias, causal, softmax_scale or 1.0 / math.sqrt(d), True,
                              kernel_cache)
        o = res[0][..., :d].contiguous()
        return (o, res[1]) if return_lse else o
    host = _HOST or _bind_host(q)
    if host is not None:
        tiles, seen = None, None
        if bias is not None:
            seen = getattr(kernel_cache, "_tiles", None)
            tiles = _native_tiles(kernel_cache, bias, q, k, causal)
        out = host.attn(kernel_cache, q, k, v, bias, tiles, causal, softmax_scale, return_lse)
        if out is not None:
            return out
        if bias is not None and kernel_cache is not None:
            kernel_cache._tiles = seen          # what follows counts this call's sight of the bias itself
    large = d not in (0, 64, 128) and d % 8 == 0 and d < 128 and _pad_head_dim_pays(q, k)
    if large:
        # Large problems of these head dims are worth a dense copy of what is not addressable (keys shared by the
        # heads, a slice at an odd offset; the native path hands them back): [2, 1100, 12, 96] with expanded keys
        # and values 114 us on the general kernels without the copy, 46 with it.  Head dims 64 and 128 keep to the
        # kernels that take the view as it is.
        few = q.shape[1] <= 16 and not causal and not _needs_grad(q, k, v, bias)
        dense = [t if _addressable(t, few) else _dense(t) for t in (q, k, v)]
        if any(a is not b for a, b in zip(dense, (q, k, v))):
            return flash_attn_func(*dense, bias, causal, softmax_scale, return_lse, kernel_cache)
    if not _needs_grad(q, k, v, bias):
        _, _, _, o, lse, _, _, _ = _attn_forward(q, k, v, bias, causal, softmax_scale, kernel_cache)
    else:
        o, lse = FlashAttnFunc.apply(q, k, v, bias, causal, softmax_scale, kernel_cache)
    if large:
        o = o.contiguous()      # as the native path and the padded head dims return it
    return (o, lse) if return_lse else o
