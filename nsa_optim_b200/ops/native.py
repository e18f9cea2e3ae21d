"""Autograd wrappers for the sm_100a kernels in ``ops/csrc``.

The shared library ``libnsa_b200.so`` lives beside this file (built by ``ops/build.py``) and
exports plain C entry points that take device pointers, sizes and a stream; output tensors
are allocated with PyTorch, by the extension module ``_nsa_host`` (``csrc/host_ops.cpp``) for most ops and here
for the others, whose entry points are called through ctypes.  Each differentiable op is one ``autograd.Function`` whose
forward and backward both call native kernels.  ``SUPPORTED`` lists the ops that have a
native implementation; ``ops/__init__.py`` consults :func:`supports`.

Kernel failures do not raise from the device: kernels record a status block in pinned host
memory (bounded waits, argument checks); :func:`check_status` turns it into an exception.
"""
from __future__ import annotations

import ctypes
import os
from typing import Optional, Tuple

import torch
from torch import Tensor
from torch.autograd import forward_ad

from . import quant, torch_impl
from .signatures import declare

_LIB_PATH = os.environ.get("NSA_B200_LIB") or os.path.join(os.path.dirname(os.path.abspath(__file__)), "libnsa_b200.so")
_lib: Optional[ctypes.CDLL] = None
_host = None
_SPLITK_MAX = int(os.environ.get("NSA_B200_SPLITK_MAX", "2"))

SUPPORTED = {
    "linear", "rms_norm", "gated_rms_norm", "swiglu", "l2_norm", "rope", "embedding",
    "causal_conv1d", "linear_cross_entropy", "adamw", "adamw_lowbit", "gated_delta_rule",
    "attention", "nsa_attention", "ssd_scan",
}

STATUS_NAMES = {
    101: "timeout waiting for a TMA stage (smem full barrier)",
    102: "timeout waiting for a free smem stage (smem empty barrier)",
    103: "timeout waiting for an accumulator (tmem full barrier)",
    104: "timeout waiting for a free accumulator (tmem empty barrier)",
    201: "timeout waiting for a flag written by a peer GPU",
    202: "timeout waiting for a flag written by another CTA",
    301: "bad argument",
    302: "an index read from a tensor was out of range (debug build)",
}


# Shapes a native kernel does not cover are computed by the PyTorch implementation of the same op.
# Every such call is counted per op, so that a benchmark or a test can show that none of its work
# took that route (``fallback_counts()``; ``NSA_B200_STRICT=1`` turns a fallback into an error).
_fallbacks: dict = {}
_STRICT = os.environ.get("NSA_B200_STRICT", "") not in ("", "0")


def _fallback(op: str, why: str = "") -> None:
    _fallbacks[op] = _fallbacks.get(op, 0) + 1
    if _STRICT:
        raise RuntimeError(f"native op '{op}' does not cover this call ({why}) and NSA_B200_STRICT is set")


def fallback_counts(reset: bool = False) -> dict:
    out = dict(_fallbacks)
    if reset:
        _fallbacks.clear()
    return out


def lib_path() -> str:
    return _LIB_PATH


def load() -> ctypes.CDLL:
    global _lib, _host
    if _lib is None:
        if not os.path.exists(_LIB_PATH):
            raise FileNotFoundError(f"{_LIB_PATH} is missing; run `python -m nsa_optim_b200.ops.build`")
        lib = ctypes.CDLL(_LIB_PATH)
        declare(lib)
        from . import _nsa_host
        _nsa_host.bind(_LIB_PATH, globals(), _SPLITK_MAX)
        _host, _lib = _nsa_host, lib
    return _lib


def _h():
    """The extension module that prepares, allocates and launches (``csrc/host_ops.cpp``)."""
    if _host is None:
        load()
    return _host


def supports(op: str, t: Tensor) -> bool:
    if op not in SUPPORTED or not t.is_cuda:
        return False
    return t.dtype == torch.bfloat16 or (t.dtype == torch.float32 and op in ("adamw", "adamw_lowbit"))


def _check(rc: int) -> None:
    if rc != 0:
        raise RuntimeError(f"nsa_optim_b200 native call failed ({rc}): {load().nsa_last_error().decode()}")


def _stream() -> int:
    # the raw handle of the current stream; torch.cuda.current_stream() builds a Stream object for it each time
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _p(t: Optional[Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


class _NoRecord:
    """Stands in for an autograd context where nothing will be differentiated."""
    needs_input_grad = (False,) * 32

    def save_for_backward(self, *tensors):
        pass

    mark_non_differentiable = save_for_backward


def _recorded(args) -> bool:
    """Whether autograd, a transform, a forward-mode derivative or a tracer has something to see in a call."""
    if torch.is_grad_enabled():
        for a in args:
            if isinstance(a, Tensor) and a.requires_grad:
                return True
    return (torch._C._are_functorch_transforms_active() or forward_ad._current_level >= 0 or torch._C._is_tracing()
            or torch.compiler.is_compiling())


def _run(fn, *args):
    """fn.apply(*args); where nothing is recorded, the forward alone (a third of the host time of a small op)."""
    return fn.apply(*args) if _recorded(args) else fn.forward(_NoRecord(), *args)


def launch_count() -> int:
    return load().nsa_launch_count()


def reset_launch_count() -> None:
    load().nsa_launch_count_reset()


def read_status(reset: bool = True) -> Tuple[int, int, int, int]:
    out = (ctypes.c_int * 4)()
    _check(load().nsa_status_read(out, 1 if reset else 0))
    return tuple(int(v) for v in out)


# --------------------------------------------------------------------------------------
# Output allocation.  With NSA_B200_DEBUG_CANARY=1 every tensor a wrapper allocates for a kernel
# sits between two 4 KB guard zones filled with a pattern; ``check_canaries()`` (also run by
# ``check_status()``) verifies them, which catches a kernel writing past either end of its
# output: the stand-in for a memory sanitizer on machines where none may be run.
# --------------------------------------------------------------------------------------
_CANARY = os.environ.get("NSA_B200_DEBUG_CANARY", "") not in ("", "0")
_GUARD = 4096
_GUARD_BYTE = 0xA5
_guards: list = []


def _shape_of(size) -> tuple:
    if len(size) == 1 and isinstance(size[0], (tuple, list, torch.Size)):
        return tuple(int(x) for x in size[0])
    return tuple(int(x) for x in size)


def _guarded(shape, dtype, device, zero: bool) -> Tensor:
    dtype = dtype or torch.get_default_dtype()
    n = 1
    for d in shape:
        n *= d
    nbytes = n * torch.empty((), dtype=dtype).element_size()
    pad = (-nbytes) % 256
    buf = torch.empty(_GUARD + nbytes + pad + _GUARD, dtype=torch.uint8, device=device)
    buf[:_GUARD].fill_(_GUARD_BYTE)
    buf[_GUARD + nbytes:].fill_(_GUARD_BYTE)
    _guards.append((buf, nbytes))
    out = buf[_GUARD:_GUARD + nbytes].view(dtype).view(shape)
    return out.zero_() if zero else out


def _empty(*size, dtype=None, device=None) -> Tensor:
    if _CANARY and device is not None and torch.device(device).type == "cuda":
        return _guarded(_shape_of(size), dtype, device, False)
    return torch.empty(*size, dtype=dtype, device=device)


def _zeros(*size, dtype=None, device=None) -> Tensor:
    if _CANARY and device is not None and torch.device(device).type == "cuda":
        return _guarded(_shape_of(size), dtype, device, True)
    return torch.zeros(*size, dtype=dtype, device=device)


def _empty_like(t: Tensor, dtype=None) -> Tensor:
    if _CANARY and t.is_cuda:
        return _guarded(tuple(t.shape), dtype or t.dtype, t.device, False)
    return torch.empty_like(t, dtype=dtype, memory_format=torch.contiguous_format)


def check_canaries() -> int:
    """Verify and release the guard zones recorded so far; returns how many buffers were checked."""
    torch.cuda.synchronize()
    n = len(_guards)
    for k, (buf, nbytes) in enumerate(_guards):
        head_ok = bool((buf[:_GUARD] == _GUARD_BYTE).all())
        tail_ok = bool((buf[_GUARD + nbytes:] == _GUARD_BYTE).all())
        if not (head_ok and tail_ok):
            _guards.clear()
            side = "before" if not head_ok else "after"
            raise RuntimeError(f"guard zone {side} kernel output #{k} ({nbytes} bytes) was overwritten")
    _guards.clear()
    return n


def check_status(sync: bool = True) -> None:
    """Raise if any kernel since the last check reported a failure."""
    if sync and torch.cuda.is_available():
        torch.cuda.synchronize()
    if _CANARY:
        check_canaries()
    code, block, info, count = read_status(reset=True)
    if code != 0:
        raise RuntimeError(f"native kernel reported status {code} ({STATUS_NAMES.get(code, 'unknown')}); "
                           f"block {block}, detail {info}, {count} report(s)")


# --------------------------------------------------------------------------------------
# GEMM
# --------------------------------------------------------------------------------------
def _as_2d(x: Tensor) -> Tensor:
    x2 = x if x.dim() == 2 else x.reshape(-1, x.shape[-1])
    pitch, step = x2.stride()
    if step != 1 or pitch % 8 or x2.data_ptr() % 16:
        x2 = x2.contiguous()
    return x2


def split_k_choice(M: int, N: int, K: int, clusters: int = 74) -> int:
    """Parts to cut the reduction of an M x N x K GEMM into.  The pair kernel gives each CTA pair
    256 x 256 tiles; with few tiles and a long reduction (weight gradients: K = tokens) the last wave
    is mostly empty, and splitting the reduction fills it.  Two parts added into a zeroed fp32 C
    give the same bits in either order, so the default limit of 2 keeps results reproducible;
    ``NSA_B200_SPLITK_MAX`` raises it."""
    return _h().split_k_choice(M, N, K, clusters)


def gemm(a: Tensor, b: Tensor, a_mn: bool, b_mn: bool, out: Optional[Tensor] = None,
         out_dtype: torch.dtype = torch.bfloat16, accumulate: bool = False, max_ctas: int = 0,
         split_k: Optional[int] = None) -> Tensor:
    """C = op(A) op(B): a_mn False -> A is (M, K), True -> A is (K, M); b_mn False -> B is (N, K),
    True -> B is (K, N).  Row pitches may exceed the logical width (sliced views).  ``split_k``
    (default: chosen by :func:`split_k_choice`) cuts the reduction into parts that run on different
    CTA pairs and meet in fp32 through TMA reduce-add stores."""
    parts = 0 if split_k is None else max(split_k, 1)        # 0: to be chosen
    return _h().matmul(a, b, a_mn, b_mn, out, out_dtype, accumulate, max_ctas, parts)


def gemm_select(which: str = "default") -> None:
    """Kernel used by plain GEMMs from now on: "pair" (two CTAs per 256 x 256 tile), "single"
    (one CTA per 128 x 256 tile) or "default" (pair unless NSA_B200_GEMM=single)."""
    load().nsa_gemm_select({"default": 0, "single": 1, "pair": 2}[which])
    _host.gemm_single(which == "single")


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x: Tensor, w: Tensor):
        y, x2 = _h().linear_fwd(x, w)
        ctx.save_for_backward(x2, w)
        return y

    @staticmethod
    def backward(ctx, dy: Tensor):
        x2, w = ctx.saved_tensors
        return _host.multi_linear_bwd(x2, (w,), (dy,), ctx.needs_input_grad[0], ctx.needs_input_grad[1:])


class _MultiLinear(torch.autograd.Function):
    """Several projections of one input, y_i = x W_i^T.  The forward is one GEMM per weight; the
    backward builds dx = sum_i dy_i W_i in place (the first GEMM stores, the others add through the
    epilogue's TMA reduce-add) instead of leaving len(ws) - 1 full-size additions to autograd."""

    @staticmethod
    def forward(ctx, x: Tensor, run_first, *ws: Tensor):
        if run_first is None:
            *ys, x2 = _h().multi_linear_fwd(x, ws)
        else:
            x2 = _as_2d(x)
            ys = [run_first(x2, ws[0]).view(*x.shape[:-1], ws[0].shape[0])]
            ys += _h().multi_linear_fwd(x, ws[1:])[:-1]
        ctx.save_for_backward(x2, *ws)
        return tuple(ys)

    @staticmethod
    def backward(ctx, *dys):
        x2, *ws = ctx.saved_tensors
        dx, *dws = _host.multi_linear_bwd(x2, tuple(ws), dys, ctx.needs_input_grad[0], ctx.needs_input_grad[2:])
        return (dx, None, *dws)


def multi_linear(x: Tensor, ws) -> tuple:
    """(x W_0^T, x W_1^T, ...) for weights that share the input (see :class:`_MultiLinear`)."""
    ws = list(ws)
    if (x.shape[-1] % 8) or any(w.shape[0] % 8 for w in ws) or x.shape[0] == 0:
        return tuple(linear(x, w) for w in ws)
    rows = x.numel() // x.shape[-1]
    if rows <= 128:                        # the single-CTA kernel has no adding epilogue
        return tuple(linear(x, w) for w in ws)
    run = None
    pg = _pending_gather
    if pg is not None:
        if pg[0] <= ws[0].data_ptr() < pg[1] and ws[0].is_contiguous():
            run = pg[2]
        else:
            flush_pending_gather()
    return _run(_MultiLinear, x, run, *ws)


# A sharded unit may defer its all-gather to the first matmul that touches one of its weights:
# (lo, hi) is the address range of the unit's gathered buffer, ``run(x, w)`` launches the GEMM
# whose kernel also assembles that buffer, ``fallback()`` gathers it without a matmul.
_pending_gather = None


def set_pending_gather(lo: int, hi: int, run, fallback) -> None:
    global _pending_gather
    flush_pending_gather()
    _pending_gather = (lo, hi, run, fallback)


def clear_pending_gather() -> None:
    global _pending_gather
    _pending_gather = None


def flush_pending_gather() -> None:
    global _pending_gather
    if _pending_gather is not None:
        fb = _pending_gather[3]
        _pending_gather = None
        fb()


class _LinearGather(torch.autograd.Function):
    """y = x W^T where the kernel that computes y also gathers W's sharded unit (see
    ``parallel/symm.py``); the backward is the ordinary one."""

    @staticmethod
    def forward(ctx, x, w, run):
        x2 = _as_2d(x)
        y = run(x2, w)
        ctx.save_for_backward(x2, w)
        return y.view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w = ctx.saved_tensors
        return (*_host.multi_linear_bwd(x2, (w,), (dy,), ctx.needs_input_grad[0], ctx.needs_input_grad[1:2]), None)


def linear(x: Tensor, w: Tensor) -> Tensor:
    if (x.shape[-1] % 8) or (w.shape[0] % 8):
        flush_pending_gather()
        _fallback("linear")
        return torch_impl.linear(x, w)
    pg = _pending_gather
    if pg is not None:
        if pg[0] <= w.data_ptr() < pg[1] and w.is_contiguous():
            return _run(_LinearGather, x, w, pg[2])
        flush_pending_gather()
    return _run(_Linear, x, w)


# --------------------------------------------------------------------------------------
# norms
# --------------------------------------------------------------------------------------
class _RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, eps):
        y, xc, wb, rstd = _h().rms_fwd(x, w, eps)
        ctx.save_for_backward(xc, wb, rstd)
        ctx.wdtype = w.dtype
        return y

    @staticmethod
    def backward(ctx, dy):
        xc, wb, rstd = ctx.saved_tensors
        return (*_host.rms_bwd(xc, wb, rstd, dy, None, ctx.wdtype), None)


def _norm_grads(ctx, dres, dy):
    """Gradients of a plain norm's input, which also receives `dres` by the residual route, and weight."""
    if dy is None:
        return dres, None
    h, wb, rstd = ctx.saved_tensors
    return _host.rms_bwd(h, wb, rstd, dy, dres, ctx.wdtype)


class _RMSNormSkip(torch.autograd.Function):
    """(y, x) with y = rmsnorm(x) * w.  The second output is the input itself, handed on to the
    residual stream; in backward its gradient and the norm's gradient meet in one kernel instead
    of two kernels and an add."""

    @staticmethod
    def forward(ctx, x, w, eps):
        y, xc, wb, rstd = _h().rms_fwd(x, w, eps)
        ctx.save_for_backward(xc, wb, rstd)
        ctx.wdtype = w.dtype
        return y, x.view_as(x)

    @staticmethod
    def backward(ctx, dy, dskip):
        return (*_norm_grads(ctx, dskip, dy), None)


class _AddRMSNorm(torch.autograd.Function):
    """(h, y) with h = x + r and y = rmsnorm(h) * w in one pass; backward adds the gradient that
    reaches h directly to the norm's gradient in the same kernel, and x and r share the result."""

    @staticmethod
    def forward(ctx, x, r, w, eps):
        h, y, wb, rstd = _h().add_rms_fwd(x, r, w, eps)
        ctx.save_for_backward(h, wb, rstd)
        ctx.wdtype = w.dtype
        return h, y

    @staticmethod
    def backward(ctx, dh, dy):
        dx, dw = _norm_grads(ctx, dh, dy)
        return dx, dx, dw, None


def rms_norm_skip(x, w, eps=1e-6):
    if x.shape[-1] % 8 or x.shape[-1] > 8192:
        _fallback("rms_norm_skip")
        return torch_impl.rms_norm_skip(x, w, eps)
    return _run(_RMSNormSkip, x, w, eps)


def add_rms_norm(x, r, w, eps=1e-6):
    if x.shape[-1] % 8 or x.shape[-1] > 8192 or x.shape != r.shape:
        _fallback("add_rms_norm")
        return torch_impl.add_rms_norm(x, r, w, eps)
    return _run(_AddRMSNorm, x, r, w, eps)


class _GatedRMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gate, w, eps, norm_before_gate):
        ctx.mode, ctx.wdtype, ctx.gshape = 1 if norm_before_gate else 2, w.dtype, gate.shape
        y, xc, g2, wb, rstd = _h().gated_rms_fwd(x, gate, w, eps, ctx.mode)
        ctx.save_for_backward(xc, g2, wb, rstd)
        return y

    @staticmethod
    def backward(ctx, dy):
        xc, g2, wb, rstd = ctx.saved_tensors
        dx, dg, dw = _host.gated_rms_bwd(xc, g2, wb, rstd, dy, ctx.mode, ctx.wdtype)
        return dx, dg.view(ctx.gshape), dw, None, None


def rms_norm(x, w, eps=1e-6):
    d = x.shape[-1]
    if d % 8 or d > 8192:
        _fallback("rms_norm")
        return torch_impl.rms_norm(x, w, eps)
    return _run(_RMSNorm, x, w, eps)


def gated_rms_norm(x, gate, w, eps=1e-6, norm_before_gate=True):
    d = x.shape[-1]
    if d % 8 or d > 8192:
        _fallback("gated_rms_norm")
        return torch_impl.gated_rms_norm(x, gate, w, eps, norm_before_gate)
    return _run(_GatedRMSNorm, x, gate, w, eps, norm_before_gate)


class _L2Norm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, eps):
        y, rinv = _h().l2_fwd(x, eps)
        ctx.save_for_backward(y, rinv)
        return y

    @staticmethod
    def backward(ctx, dy):
        return _host.l2_bwd(*ctx.saved_tensors, dy), None


def l2_norm(x, eps=1e-6):
    d = x.shape[-1]
    if d % 8 or d > 512:
        _fallback("l2_norm")
        return torch_impl.l2_norm(x, eps)
    return _run(_L2Norm, x, eps)


# --------------------------------------------------------------------------------------
# SwiGLU, RoPE
# --------------------------------------------------------------------------------------
class _SwiGLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate, up):
        y, g2, u2 = _h().swiglu_fwd(gate, up)
        ctx.save_for_backward(g2, u2)
        return y

    @staticmethod
    def backward(ctx, dy):
        return _host.swiglu_bwd(*ctx.saved_tensors, dy)


def swiglu(gate, up):
    if gate.shape[-1] % 8:
        _fallback("swiglu")
        return torch_impl.swiglu(gate, up)
    return _run(_SwiGLU, gate, up)


class _RoPE(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, cos, sin):
        cos = cos.float().contiguous()
        sin = sin.float().contiguous()
        ctx.save_for_backward(cos, sin)
        return _h().rope(x, cos, sin, False)

    @staticmethod
    def backward(ctx, dy):
        cos, sin = ctx.saved_tensors
        return _host.rope(dy, cos, sin, True), None, None


def rope(x, cos, sin):
    if x.shape[-1] % 16 or cos.shape[0] != x.shape[1]:
        _fallback("rope")
        return torch_impl.rope(x, cos, sin)
    return _run(_RoPE, x, cos, sin)


# --------------------------------------------------------------------------------------
# causal conv1d
# --------------------------------------------------------------------------------------
class _Conv1d(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, activation):
        y, xv, wb, bb = _h().conv_fwd(x, weight, bias, activation)
        ctx.save_for_backward(xv, wb, bb)
        ctx.activation, ctx.wdtype = activation, weight.dtype
        return y

    @staticmethod
    def backward(ctx, dy):
        xv, wb, bb = ctx.saved_tensors
        return (*_host.conv_bwd(xv, wb, bb, dy, ctx.activation, ctx.wdtype), None)


def causal_conv1d(x, weight, bias, activation=True):
    if x.shape[-1] % 8 or weight.shape[-1] != 4:
        _fallback("causal_conv1d")
        return torch_impl.causal_conv1d(x, weight, bias, activation)
    return _run(_Conv1d, x, weight, bias, activation)


# --------------------------------------------------------------------------------------
# embedding
# --------------------------------------------------------------------------------------
class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, weight):
        y, flat = _h().embedding_fwd(ids, weight)
        ctx.save_for_backward(flat)
        ctx.wshape, ctx.wdtype = weight.shape, weight.dtype
        return y

    @staticmethod
    def backward(ctx, dy):
        (flat,) = ctx.saved_tensors
        n, d = flat.numel(), ctx.wshape[1]
        sorted_ids, perm = torch.sort(flat, stable=True)
        dw = _zeros(ctx.wshape, dtype=torch.float32, device=dy.device)
        dy2 = dy.reshape(n, d).contiguous()
        _check(load().nsa_embedding_bwd(_p(sorted_ids), _p(perm), _p(dy2), _p(dw), n, d, _stream()))
        return None, dw.to(ctx.wdtype)


def embedding(ids, weight):
    if weight.shape[1] % 8 or ids.dtype != torch.long:
        _fallback("embedding")
        return torch_impl.embedding(ids, weight)
    return _run(_Embedding, ids, weight)


# --------------------------------------------------------------------------------------
# fused linear + cross entropy
# --------------------------------------------------------------------------------------
class _LinearCE(torch.autograd.Function):
    """Per token chunk: logits GEMM (tcgen05) -> softmax-CE kernel that overwrites the logits
    with their gradient -> two gradient GEMMs.  The (chunk, V) block is the largest temporary."""

    @staticmethod
    def forward(ctx, hidden, weight, labels, ignore_index, chunk):
        loss, dh, dw = _h().cross_entropy_fwd(hidden, weight, labels, ignore_index, chunk, *ctx.needs_input_grad[:2])
        ctx.save_for_backward(dh, dw)
        ctx.wdtype = weight.dtype
        return loss

    @staticmethod
    def backward(ctx, gout):
        dh, dw = ctx.saved_tensors
        return (None if dh is None else _scaled_by(dh, gout.to(dh.dtype), dh.dtype),
                None if dw is None else _scaled_by(dw, gout, ctx.wdtype), None, None, None)


def _scaled_by(t: Tensor, s: Tensor, dtype: torch.dtype) -> Tensor:
    """t * s rounded once to ``dtype``, s a one-element tensor: one pass for bf16 results.  Tensor arithmetic where the
    product is differentiated again with respect to s, or s stands for a batch of factors."""
    if (torch.is_grad_enabled() and s.requires_grad) or not torch._C._has_storage(s):     # a batch under vmap has none
        return (t * s).to(dtype)
    if dtype != torch.bfloat16 or t.dtype not in (torch.float32, torch.bfloat16) or not t.is_contiguous() or t.data_ptr() % 16:
        return (t * s).to(dtype)
    return _h().scale(t, s)


def linear_cross_entropy(hidden, weight, labels, ignore_index=-100, chunk=4096):
    if hidden.shape[-1] % 8 or weight.shape[0] % 8:
        _fallback("linear_cross_entropy")
        return torch_impl.linear_cross_entropy(hidden, weight, labels, ignore_index, chunk)
    return _run(_LinearCE, hidden, weight, labels, ignore_index, chunk)


# --------------------------------------------------------------------------------------
# optimizer steps
# --------------------------------------------------------------------------------------
def adamw_multi(items, step, lr, b1, b2, eps, wd, grad_scale) -> None:
    """AdamW over (p, g, exp_avg, exp_avg_sq, master or None, None) tuples that share a device, dtypes and step.  The kernels index
    every state tensor with the parameter's element count: a state restored from a checkpoint of another sharding is refused."""
    _h().adamw(items, grad_scale, step, lr, b1, b2, eps, wd)


def adamw8bit_multi(items, step, lr, b1, b2, eps, wd, grad_scale, block) -> None:
    """8-bit AdamW over (p, g, codes m, codes v, scales m, scales v) tuples that share a device, dtypes and step."""
    if block != 256:
        raise ValueError("the native 8-bit AdamW kernel uses 256-element blocks")
    dev = items[0][0].device
    _h().adamw8bit(items, quant.codebook(8, True, dev), quant.codebook(8, False, dev), grad_scale, step, lr, b1, b2, eps, wd, block)


def adamw_step(p, g, m, v, master, step, lr, b1, b2, eps, wd, grad_scale):
    adamw_multi([(p, g, m, v, master, None)], step, lr, b1, b2, eps, wd, grad_scale)


def adamw8bit_step(p, g, mq, mabs, vq, vabs, step, lr, b1, b2, eps, wd, grad_scale, block):
    adamw8bit_multi([(p, g, mq, vq, mabs, vabs)], step, lr, b1, b2, eps, wd, grad_scale, block)


# --------------------------------------------------------------------------------------
# gated delta rule (chunk 64, key width 128)
# --------------------------------------------------------------------------------------
class _GatedDelta(torch.autograd.Function):
    """Chunkwise gated delta rule, two kernels each way: per-chunk matrices and operands
    (``gdn_prep_kernel``), the state recurrence with the output (``csrc/gdn.cu``); backward the reverse recurrence,
    then every gradient of a chunk (``gdn_post_kernel``).  All tensors token-major, gates fp32."""

    @staticmethod
    def forward(ctx, q, k, v, g, beta, scale):
        train = any(ctx.needs_input_grad)
        o, *kept = _h().gdn_fwd(q, k, v, g, beta, scale, train)
        if train:
            ctx.save_for_backward(q, k, v, beta, *kept)
            ctx.scale = scale
        return o

    @staticmethod
    def backward(ctx, do):
        return (*_host.gdn_bwd(*ctx.saved_tensors, do, ctx.scale), None)


def _dense16(t: Tensor) -> Tensor:
    """Contiguous with a 16-byte aligned start, as the copy engine and 16-byte loads need."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone(memory_format=torch.contiguous_format)


def gated_delta_rule(q, k, v, g, beta, scale=None, chunk=64):
    """Chunkwise gated delta rule (:class:`_GatedDelta`).  Value columns are independent of one another given
    q, k and the gates, so values wider than one launch's shared memory go in slices."""
    B, T, H, K = q.shape
    V = v.shape[-1]
    if K != 128 or V % 64 or chunk != 64 or q.dtype != torch.bfloat16:
        _fallback("gated_delta_rule")
        return torch_impl.gated_delta_rule(q, k, v, g, beta, scale, chunk)
    scale = K ** -0.5 if scale is None else scale
    bf = torch.bfloat16
    args = [_dense16(q), _dense16(k.to(bf)), v.to(bf), g.float().contiguous(), beta.float().contiguous()]
    outs = [_run(_GatedDelta, args[0], args[1], _dense16(part), args[3], args[4], float(scale))
            for part in (args[2].split(512, -1) if V > 512 else (args[2],))]
    o = outs[0] if len(outs) == 1 else torch.cat(outs, -1)
    return o.to(v.dtype)


# --------------------------------------------------------------------------------------
# attention family (csrc/attention.cu)
# --------------------------------------------------------------------------------------
def _range_visits() -> int:
    """Query tiles per CTA of the dK / dV kernel over a contiguous key range, where a key block has more than 256.  The environment is
    read here, under the GIL: another thread's assignment to os.environ may move what a native getenv walks."""
    return int(os.environ.get("NSA_B200_KV_VISITS", "64"))


def _list_visits() -> int:
    """The same over a list of tokens."""
    return int(os.environ.get("NSA_B200_KV_VISITS_SEL", "64"))


def _bwd_is_split(D: int, G: int, selected: bool) -> bool:
    return os.environ.get("NSA_B200_ATTN_BWD", "split") == "split" and (not selected or (D == 128 and G >= 8))


class _Attn(torch.autograd.Function):
    """Softmax attention on (B, T, H, D) tensors through the tcgen05 kernels.  ``tiles`` is
    ``None`` (contiguous key range bounded by causality / window) or the per-query-tile block
    lists from :func:`union_blocks` (selected-block attention).  Key positions are
    ``index * kp_stride + kp_off``.  Returns (output, L) with L the log2-sum-exp per row."""

    @staticmethod
    def forward(ctx, q, k, v, causal, window, scale, kp_stride, kp_off, tiles):
        o, L, q, k, v = _h().attn_fwd(q, k, v, causal, window, scale, kp_stride, kp_off, tiles)
        ctx.save_for_backward(q, k, v, o, L)
        ctx.cfg = (causal, window, scale, kp_stride, kp_off)
        ctx.tiles = tiles
        ctx.mark_non_differentiable(L)
        return o, L

    @staticmethod
    def backward(ctx, do, _dL):
        q, k, v, o, L = ctx.saved_tensors
        (causal, window, _, kp_stride, _), tiles, lists, walks = ctx.cfg, ctx.tiles, None, 0
        visits = _range_visits() if tiles is None else _list_visits()
        B, T, Hq, D = q.shape
        S, Hkv = k.shape[1], k.shape[2]
        split = _bwd_is_split(D, Hq // Hkv, tiles is not None)
        if split and tiles is None:
            walks_of = load().nsa_attn_bwd_walks if D == 128 else load().nsa_attn_bwd_walks_d64
            walks = walks_of(B, T, S, Hq, Hkv, int(causal), window, kp_stride)
        elif split:
            lists = _inverse_of(tiles, Hq // Hkv, visits)
        return (*_host.attn_bwd(q, k, v, o, do, L, *ctx.cfg, tiles, lists, visits, walks, split), None, None, None, None, None, None)


def _attn_ok(q, k) -> bool:
    Hq, Hkv, D = q.shape[2], k.shape[2], q.shape[3]
    G = Hq // max(Hkv, 1)
    return D in (64, 128) and Hkv > 0 and Hq % Hkv == 0 and G <= 128 and (G & (G - 1)) == 0


def attention(q, k, v, causal=True, window=0, scale=None):
    if not _attn_ok(q, k) or q.shape[1] != k.shape[1]:
        _fallback("attention")
        return torch_impl.attention(q, k, v, causal, window, scale)
    scale = q.shape[-1] ** -0.5 if scale is None else scale
    return _run(_Attn, q, k, v, causal, int(window), float(scale), 1, 0, None)[0]


def union_blocks(idx: Tensor, G: int, nS: int):
    """idx (B, Hkv, T, top_n) int32 selection-block ids (-1 = none) -> per query tile
    (128 // G tokens) ascending union list, token bit masks and counts."""
    tb, tm, tc = _h().union_blocks(idx, G, nS)
    return tb, tm, tc, tb.shape[-1]


def inverse_blocks(idx: Tensor, nS: int, R: int, visits_per_cta: int):
    """Inverse of the selection map (count, scan, fill kernels of ``csrc/attention.cu``; no sort, the
    same lists on every run).  Same results as :func:`_inverse_blocks_torch`."""
    B, Hkv, T, n = idx.shape
    if not idx.is_cuda or nS > 12288 or n > 32:
        return _inverse_blocks_torch(idx, nS, R, visits_per_cta)
    tok, list_start, item_start = _h().inverse_blocks(idx, nS, R, visits_per_cta)
    bound = (B * Hkv * T * n) // (R * visits_per_cta) + B * Hkv * nS
    return tok, list_start, item_start, nS, bound


def _inverse_of(tiles, G: int, visits: int):
    """Inverse lists of a selection's tiles for a dK / dV kernel of ``visits`` query tiles per CTA."""
    return inverse_blocks(tiles[4], tiles[5], 128 // G, visits)


def _inverse_blocks_torch(idx: Tensor, nS: int, R: int, visits_per_cta: int):
    """Inverse of the selection map.  idx (B, Hkv, T, top_n) -> (tok_list, list_start, item_start,
    nS, item_bound): for every (b, h, block) the ascending tokens that selected the block, laid out
    back to back; ``list_start`` / ``item_start`` are the exclusive prefixes of the list lengths and
    of the CTAs per list (a CTA covers ``visits_per_cta`` groups of R tokens); ``item_bound`` is a
    host-side upper bound of the CTA count, so nothing here waits for the device.  Entries that are
    negative, out of range or repeated inside a token's list are dropped."""
    B, Hkv, T, n = idx.shape
    dev = idx.device
    lists = B * Hkv * nS
    s, _ = idx.sort(dim=-1)
    ok = (s >= 0) & (s < nS)
    ok[..., 1:] &= s[..., 1:] != s[..., :-1]
    bh = torch.arange(B * Hkv, device=dev, dtype=torch.int64).view(B, Hkv, 1, 1)
    key = torch.where(ok, bh * nS + s.to(torch.int64), torch.full((), lists, device=dev, dtype=torch.int64)).reshape(-1)
    skey, order = key.sort(stable=True)                       # (b, h, t) order survives inside a list
    tok = ((order // n) % T).to(torch.int32)
    list_start = torch.searchsorted(skey, torch.arange(lists + 1, device=dev, dtype=torch.int64)).to(torch.int32)
    cnt = list_start[1:] - list_start[:-1]
    items = (-(-cnt // R) + visits_per_cta - 1) // visits_per_cta
    item_start = _zeros(lists + 1, dtype=torch.int32, device=dev)
    item_start[1:] = items.cumsum(0)
    bound = (B * Hkv * T * n) // (R * visits_per_cta) + lists
    return tok, list_start, item_start, nS, bound


def selected_attention(q, k, v, idx, scale=None):
    """Causal attention of each query token over its own list of 64-key blocks ``idx``
    (B, Hkv, T, top_n)."""
    scale = q.shape[-1] ** -0.5 if scale is None else scale
    G = q.shape[2] // k.shape[2]
    nS = -(-k.shape[1] // 64)
    idx = idx.to(torch.int32).contiguous()
    tiles = union_blocks(idx, G, nS) + (idx, nS)
    return _run(_Attn, q, k, v, True, 0, float(scale), 1, 0, tiles)[0]


def nsa_attention_indexed(q, k, v, idx, g_slc, g_swa, sel_block=64, window=512, scale=None):
    """Selected-block attention over caller-given block lists ``idx`` (B, Hkv, T, n) plus the sliding
    window, gated: both branches on the tcgen05 attention kernels."""
    B, T, Hq, D = q.shape
    G = Hq // k.shape[2]
    if not _attn_ok(q, k) or sel_block != 64 or G < 2 or G > 32:
        _fallback("nsa_attention_indexed")
        return torch_impl.nsa_attention_indexed(q, k, v, idx, g_slc, g_swa, sel_block, window, scale)
    scale = D ** -0.5 if scale is None else scale
    o_slc = selected_attention(q, k, v, idx, scale)
    o_swa = _run(_Attn, q, k, v, True, int(window), float(scale), 1, 0, None)[0]
    return g_slc.unsqueeze(-1) * o_slc + g_swa.unsqueeze(-1) * o_swa


def nsa_importance(q, k_cmp, L_cmp, nS, stride, block, scale):
    return _h().importance(q, k_cmp, L_cmp, nS, stride, block, scale)


def nsa_select(imp: Tensor, sel_block: int, top_n: int) -> Tensor:
    """imp (B, Hkv, T, nS) -> int32 (B, Hkv, T, top_n): block 0, the query's own block and the one
    before it always, then the most important causal blocks (ties: lower index); -1 where fewer
    are visible.  One warp per row (``nsa_select_kernel``); more than 2048 blocks use torch.topk."""
    B, H, T, nS = imp.shape
    if imp.is_cuda and nS <= 2048 and imp.dtype == torch.float32:
        return _h().select(imp, sel_block, top_n)
    return _nsa_select_torch(imp, sel_block, top_n)


def _nsa_select_torch(imp: Tensor, sel_block: int, top_n: int) -> Tensor:
    B, H, T, nS = imp.shape
    own = (torch.arange(T, device=imp.device) // sel_block)[:, None]
    j = torch.arange(nS, device=imp.device)[None, :]
    forced = (j == 0) | (j == own) | (j == own - 1)
    score = imp.masked_fill(forced, float("inf")).masked_fill_(j > own, float("-inf"))
    n = min(top_n, nS)
    val, idx = torch.topk(score, n, dim=-1)
    idx = idx.masked_fill(val == float("-inf"), -1).to(torch.int32)
    if n < top_n:
        idx = torch.nn.functional.pad(idx, (0, top_n - n), value=-1)
    return idx.contiguous()


class _GateCombine(torch.autograd.Function):
    """o = g1 o1 + g2 o2 + g3 o3 with one gate per (token, head): the sigmoid-gated combine of the
    three sparse-attention branches in one pass each way (``csrc/elementwise.cu``)."""

    @staticmethod
    def forward(ctx, o1, o2, o3, g1, g2, g3):
        o1, o2, o3 = o1.contiguous(), o2.contiguous(), o3.contiguous()
        g1, g2, g3 = (g.to(torch.bfloat16).contiguous() for g in (g1, g2, g3))
        D = o1.shape[-1]
        rows = o1.numel() // D
        o = _empty_like(o1)
        _check(load().nsa_gate_combine_fwd(_p(o1), _p(o2), _p(o3), _p(g1), _p(g2), _p(g3), _p(o), rows, D,
                                           _stream()))
        ctx.save_for_backward(o1, o2, o3, g1, g2, g3)
        return o

    @staticmethod
    def backward(ctx, do):
        o1, o2, o3, g1, g2, g3 = ctx.saved_tensors
        do = do.contiguous()
        D = o1.shape[-1]
        rows = o1.numel() // D
        d1, d2, d3 = _empty_like(o1), _empty_like(o1), _empty_like(o1)
        e1, e2, e3 = _empty_like(g1), _empty_like(g1), _empty_like(g1)
        _check(load().nsa_gate_combine_bwd(_p(o1), _p(o2), _p(o3), _p(g1), _p(g2), _p(g3), _p(do), _p(d1), _p(d2), _p(d3),
                                           _p(e1), _p(e2), _p(e3), rows, D, _stream()))
        return d1, d2, d3, e1, e2, e3


def _gate_logits_forward(o1, o2, o3, gates):
    """(combined output, bf16 logits) with the three gates as logits straight from the gate projection: ``gates`` is
    (B, T, 3*Hq) (or wider; columns [0, Hq) compressed, [Hq, 2Hq) selected, [2Hq, 3Hq) window)."""
    return _h().gates_fwd(o1, o2, o3, gates)


def _gate_logits_backward(o1, o2, o3, gl, do, sums=(None, None, None)):
    """(do1, do2, do3, d logits); ``sums``, three fp32 tensors of one value per row, receive rowsum(do_i * o_i)."""
    return _h().gates_bwd(o1, o2, o3, gl, do, *sums)


class _GateCombineLogits(torch.autograd.Function):
    """The same combine with the gates given as logits.  The sigmoid runs inside the combine kernel and its
    derivative inside the backward kernel, which writes d(logits) in the projection's own layout."""

    @staticmethod
    def forward(ctx, o1, o2, o3, gates):
        o1, o2, o3 = o1.contiguous(), o2.contiguous(), o3.contiguous()
        o, gl = _gate_logits_forward(o1, o2, o3, gates)
        ctx.save_for_backward(o1, o2, o3, gl)
        ctx.gdtype = gates.dtype
        return o

    @staticmethod
    def backward(ctx, do):
        d1, d2, d3, dgl = _gate_logits_backward(*ctx.saved_tensors, do)
        return d1, d2, d3, dgl.to(ctx.gdtype)


def _nsa_select_tiles(q, kc, L_cmp, nS, stride, block, sel_block, top_n, scale):
    """Importance of the selection blocks, the top_n of each token, and the per-tile lists of :class:`_Attn`."""
    idx = nsa_select(nsa_importance(q, kc, L_cmp, nS, stride, block, scale), sel_block, top_n)
    return union_blocks(idx, q.shape[2] // kc.shape[2], nS) + (idx, nS)


class _NSA(torch.autograd.Function):
    """The three branches and their gated combine as one node.  With separate nodes the backward read every do_i and
    o_i again for rowsum(do_i * o_i) and added the branches' dq, dk and dv in passes of their own (16384 tokens x 32
    heads: 280 of 6810 us; 6400 in all now); here the combine's backward leaves the sums, and each branch adds to the gradients of the one
    before it: dq in the kernel's epilogue, dk and dv of the selected and window branches in one fp32 buffer."""

    @staticmethod
    def forward(ctx, q, k, v, kc, vc, gates, stride, block, sel_block, top_n, window, scale):
        h = _h()
        o1, L1, q, kc, vc = h.attn_fwd(q, kc, vc, True, 0, scale, stride, block - 1, None)
        tiles = _nsa_select_tiles(q, kc, L1, -(-q.shape[1] // sel_block), stride, block, sel_block, top_n, scale)
        o2, L2, _, k, v = h.attn_fwd(q, k, v, True, 0, scale, 1, 0, tiles)
        o3, L3, *_ = h.attn_fwd(q, k, v, True, window, scale, 1, 0, None)
        o, gl = _gate_logits_forward(o1, o2, o3, gates)
        ctx.save_for_backward(q, k, v, kc, vc, gl, o1, o2, o3, L1, L2, L3)
        ctx.cfg, ctx.tiles, ctx.gdtype = (stride, block, window, scale), tiles, gates.dtype
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, kc, vc, gl, o1, o2, o3, L1, L2, L3 = ctx.saved_tensors
        e1, e2, e3 = (_empty_like(L1) for _ in range(3))
        d1, d2, d3, dgl = _gate_logits_backward(o1, o2, o3, gl, do, (e1, e2, e3))
        visits = _list_visits()
        lists = _inverse_of(ctx.tiles, q.shape[2] // k.shape[2], visits)
        grads = _host.nsa_bwd(q, k, v, kc, vc, o1, d1, L1, e1, o2, d2, L2, e2, o3, d3, L3, e3, ctx.tiles, lists,
                              _range_visits(), visits, *ctx.cfg)
        return (*grads, dgl.to(ctx.gdtype), None, None, None, None, None, None)


class _Pool(torch.autograd.Function):
    """Mean pooling of (B, T, H, D) keys / values over windows [i*stride, i*stride + block) ->
    (B, nC, H, D), forward and backward in ``csrc/elementwise.cu`` (fla's ``mean_pooling`` in the
    reference's NSA stack)."""

    @staticmethod
    def forward(ctx, x, block, stride):
        ctx.cfg = x.shape[1], block, stride
        return _h().pool_fwd(x, block, stride)

    @staticmethod
    def backward(ctx, dy):
        return _host.pool_bwd(dy, *ctx.cfg), None, None


def nsa_compress(x, block, stride):
    if x.dtype != torch.bfloat16 or (x.shape[2] * x.shape[3]) % 8 or x.shape[1] < block:
        _fallback("nsa_compress")
        return torch_impl.nsa_compress(x, block, stride)
    return _run(_Pool, x, int(block), int(stride))


def nsa_attention(q, k, v, g_cmp, g_slc, g_swa, cmp_block=32, cmp_stride=16, sel_block=64, top_n=16,
                  window=512, scale=None, gate_logits=None):
    """``gate_logits`` (B, T, 3*Hq), when given, replaces the three gate tensors: the sigmoid is taken
    inside the combine kernel."""
    B, T, Hq, D = q.shape
    Hkv = k.shape[2]
    G = Hq // Hkv
    if (not _attn_ok(q, k) or sel_block != 64 or sel_block != 4 * cmp_stride or cmp_block != 2 * cmp_stride
            or G < 2 or G > 32 or T < cmp_block):
        _fallback("nsa_attention")
        if gate_logits is not None:
            g_cmp, g_slc, g_swa = torch.sigmoid(gate_logits.float()).to(q.dtype)[..., :3 * Hq].split(Hq, dim=-1)
        return torch_impl.nsa_attention(q, k, v, g_cmp, g_slc, g_swa, cmp_block, cmp_stride, sel_block, top_n,
                                        window, scale)
    scale = D ** -0.5 if scale is None else scale
    kc = nsa_compress(k, cmp_block, cmp_stride)
    vc = nsa_compress(v, cmp_block, cmp_stride)
    if gate_logits is not None and window > 0 and q.dtype == torch.bfloat16 and _bwd_is_split(D, G, True):
        return _run(_NSA, q, k, v, kc, vc, gate_logits, cmp_stride, cmp_block, sel_block, top_n, int(window), float(scale))
    o_cmp, L_cmp = _run(_Attn, q, kc, vc, True, 0, float(scale), cmp_stride, cmp_block - 1, None)
    with torch.no_grad():
        tiles = _nsa_select_tiles(q, kc, L_cmp, -(-T // sel_block), cmp_stride, cmp_block, sel_block, top_n, float(scale))
    o_slc = _run(_Attn, q, k, v, True, 0, float(scale), 1, 0, tiles)[0]
    o_swa = _run(_Attn, q, k, v, True, int(window), float(scale), 1, 0, None)[0]
    if gate_logits is not None:
        if q.dtype == torch.bfloat16 and D in (64, 128, 256):
            return _run(_GateCombineLogits, o_cmp, o_slc, o_swa, gate_logits)
        g_cmp, g_slc, g_swa = torch.sigmoid(gate_logits.float()).to(q.dtype)[..., :3 * Hq].split(Hq, dim=-1)
    if q.dtype == torch.bfloat16 and D in (64, 128, 256):
        return _run(_GateCombine, o_cmp, o_slc, o_swa, g_cmp, g_slc, g_swa)
    return g_cmp.unsqueeze(-1) * o_cmp + g_slc.unsqueeze(-1) * o_slc + g_swa.unsqueeze(-1) * o_swa


# --------------------------------------------------------------------------------------
# Mamba-2 SSD
# --------------------------------------------------------------------------------------
class _SSDStatePass(torch.autograd.Function):
    """Hprev[c+1] = gamma[c] * Hprev[c] + S[c] over chunks (``csrc/ssd.cu``).
    S (B, nc, H, P, N) fp32, gamma (B, nc, H) fp32 -> Hprev, same shape as S."""

    @staticmethod
    def forward(ctx, S, gamma):
        S, gamma = S.contiguous(), gamma.contiguous()
        B, nc, H = gamma.shape
        E = S[0, 0, 0].numel()
        Hprev = _empty_like(S)
        _check(load().nsa_ssd_state_fwd(_p(S), _p(gamma), _p(Hprev), None, None, B, nc,
                                        H, E, _stream()))
        ctx.save_for_backward(gamma, Hprev)
        return Hprev

    @staticmethod
    def backward(ctx, dHprev):
        gamma, Hprev = ctx.saved_tensors
        B, nc, H = gamma.shape
        E = Hprev[0, 0, 0].numel()
        dHprev = dHprev.contiguous().float()
        dS = _empty_like(Hprev)
        _check(load().nsa_ssd_state_bwd(_p(dHprev), _p(gamma), _p(dS), None, B, nc, H, E,
                                        _stream()))
        dgamma = (Hprev * dS).sum((-1, -2))
        return dS, dgamma


class _SSD(torch.autograd.Function):
    """Mamba-2 SSD through the tcgen05 chunk kernels of ``csrc/ssd.cu`` (chunk 128, d_state 128,
    headdim 64, one B/C group)."""

    @staticmethod
    def forward(ctx, x, dt, A, Bm, Cm, D):
        y, *kept = _h().ssd_fwd(x, dt, A, Bm, Cm, D)
        ctx.save_for_backward(*kept)
        ctx.has_D = D is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        return _host.ssd_bwd(*ctx.saved_tensors, dy, ctx.has_D)


def _gates(a, b, dt_bias, A_log):
    """The two results of one launch (``csrc/gates.cu``), or None where autograd records, the layout is another or a tensor
    is elsewhere, which PyTorch's expressions refuse or take as they do."""
    f32, bf, shape, at = torch.float32, torch.bfloat16, a.shape, a.get_device()
    row = shape[-1:]
    if (a.dtype != bf or len(shape) < 2 or a.numel() == 0 or dt_bias.dtype not in (f32, bf) or A_log.dtype not in (f32, bf)
            or dt_bias.shape != row or A_log.shape != row or dt_bias.get_device() != at or A_log.get_device() != at
            or (b is not None and (b.dtype != bf or b.shape != shape or b.get_device() != at)) or _recorded((a, b, dt_bias, A_log))):
        return None
    return _h().gates(a, b, dt_bias, A_log)


def step_sizes(dt, dt_bias, A_log):
    return _gates(dt, None, dt_bias, A_log)


def delta_gates(a, b, dt_bias, A_log):
    return _gates(a, b, dt_bias, A_log)


def copy_columns(dst: Tensor, src: Tensor) -> bool:
    """dst[...] = src for two tensors that are column slices of row-major matrices (last dimension
    contiguous, one uniform row pitch): a pitched device copy instead of a generic strided kernel.
    Returns False (nothing done) when the layouts do not qualify."""
    if dst.shape != src.shape or dst.dtype != src.dtype or not (dst.is_cuda and src.is_cuda) or dst.dim() < 2:
        return False
    def pitch(t):
        if t.stride(-1) != 1:
            return None
        p = t.stride(-2)
        if p < t.shape[-1]:
            return None
        exp = p
        for d in range(t.dim() - 2, -1, -1):           # leading dims must fold into rows of pitch p
            if t.shape[d] != 1 and t.stride(d) != exp:
                return None
            exp *= t.shape[d]
        return p
    dp, sp = pitch(dst), pitch(src)
    if dp is None or sp is None:
        return False
    es = dst.element_size()
    rows = dst.numel() // dst.shape[-1]
    _check(load().nsa_copy2d(_p(dst), dp * es, _p(src), sp * es, dst.shape[-1] * es, rows,
                             _stream()))
    return True


def sumsq(tensors) -> Tensor:
    """Sum of squares over a list of bf16 / fp32 CUDA tensors -> fp32 device scalar (no host sync)."""
    lib = load()
    dev = tensors[0].device
    out = _zeros((), dtype=torch.float32, device=dev)
    partial = _empty(int(lib.nsa_sumsq_parts()), dtype=torch.float32, device=dev)
    for g in tensors:
        if g.dtype not in (torch.bfloat16, torch.float32) or not g.is_contiguous():
            g = g.float().contiguous()
        _check(lib.nsa_sumsq(_p(g), g.numel(), int(g.dtype == torch.float32), _p(partial), _p(out), 1,
                             _stream()))
    return out


def affine_quantize(t: Tensor, bits: int, q_block: int):
    """CUDA form of :func:`nsa_optim_b200.ops.quant.affine_quantize` for fp32 matrices."""
    rows, cols = t.shape
    nblk = -(-cols // q_block)
    t = t.float().contiguous()
    q = _empty(rows, nblk * q_block, dtype=torch.uint8, device=t.device)
    scale = _empty(rows, nblk, dtype=torch.float32, device=t.device)
    zero = _empty(rows, nblk, dtype=torch.float32, device=t.device)
    _check(load().nsa_affine_quant(_p(t), _p(q), _p(scale), _p(zero), rows, cols, q_block, bits,
                                   _stream()))
    return q, scale, zero, cols


def affine_dequantize(q: Tensor, scale: Tensor, zero: Tensor, orig_cols: int) -> Tensor:
    rows = q.shape[0]
    q_block = q.shape[1] // scale.shape[1]
    out = _empty(rows, orig_cols, dtype=torch.float32, device=q.device)
    _check(load().nsa_affine_dequant(_p(q.contiguous()), _p(scale.contiguous()), _p(zero.contiguous()), _p(out), rows,
                                     orig_cols, q_block, _stream()))
    return out


def mamba3_gate(u: Tensor, dt: Tensor, A: Tensor, Bc: Tensor, Cc: Tensor, D: Tensor) -> Tensor:
    """Forward-only sequential scan of the complex-state SSM (``csrc/mamba3.cu``).
    u, dt (B, L, H) ; A (H, N, 2) ; Bc, Cc (B, L, H, N, 2) ; D (H)  ->  gate (B, L, H) fp32 with
    gate_t = Re<C_t, h_t> + D; the block output is x_t * gate_t."""
    B, L, H = u.shape
    N = A.shape[1]
    f = lambda t: t.detach().float().contiguous()
    u, dt, A, Bc, Cc, D = f(u), f(dt), f(A), f(Bc), f(Cc), f(D)
    gate = _empty(B, L, H, dtype=torch.float32, device=u.device)
    _check(load().nsa_mamba3_scan(_p(u), _p(dt), _p(A), _p(Bc), _p(Cc), _p(D), _p(gate), B, L, H,
                                  N, _stream()))
    return gate


def ssd_scan(x, dt, A, Bm, Cm, D=None, chunk=256):
    """Mamba-2 SSD.  The shapes of the hybrid models (d_state 128, headdim 64, one group) run on
    the fused tcgen05 chunk kernels; other shapes use batched matmuls plus the native
    inter-chunk state pass."""
    if (x.shape[-1] == 64 and Bm.shape[-1] == 128 and Bm.shape[2] == 1 and x.dtype == torch.bfloat16
            and Bm.dtype == torch.bfloat16 and Cm.dtype == torch.bfloat16):
        return _run(_SSD, x, dt, A, Bm, Cm, D)
    return _ssd_scan_batched(x, dt, A, Bm, Cm, D, chunk)


def _ssd_scan_batched(x, dt, A, Bm, Cm, D=None, chunk=256):
    """Chunked SSD: the per-chunk terms are batched tensor-core matmuls over all chunks at once,
    the inter-chunk recurrence is one native kernel (forward) and one (backward)."""
    F = torch.nn.functional
    Bsz, T, H, P = x.shape
    G, N = Bm.shape[2], Bm.shape[3]
    L = min(chunk, 128, T)
    pad = (-T) % L
    if pad:
        x = F.pad(x, (0, 0, 0, 0, 0, pad))
        dt = F.pad(dt, (0, 0, 0, pad))
        Bm = F.pad(Bm, (0, 0, 0, 0, 0, pad))
        Cm = F.pad(Cm, (0, 0, 0, 0, 0, pad))
    Tp = T + pad
    nc = Tp // L
    rep = H // G
    cdt = x.dtype
    xr = x.reshape(Bsz, nc, L, H, P)
    dtr = dt.float().reshape(Bsz, nc, L, H)
    Br = Bm.reshape(Bsz, nc, L, G, N)
    Cr = Cm.reshape(Bsz, nc, L, G, N)
    a = dtr * A.float()[None, None, None, :]
    cum = torch.cumsum(a, dim=2)
    total = cum[:, :, -1]
    xdt = (xr.float() * dtr[..., None]).to(cdt)
    CB = torch.einsum("bclgn,bcsgn->bcgls", Cr, Br)                      # (B,nc,G,L,L) in the compute dtype
    seg = cum.permute(0, 1, 3, 2)                                        # (B,nc,H,L)
    tri = torch.ones(L, L, dtype=torch.bool, device=x.device).tril()
    dec = torch.exp((seg[..., :, None] - seg[..., None, :]).masked_fill(~tri, float("-inf"))).to(cdt)
    M = CB.repeat_interleave(rep, dim=2) * dec if rep > 1 else CB * dec  # (B,nc,H,L,L)
    y = torch.einsum("bchls,bcshp->bclhp", M, xdt)
    w_end = torch.exp(total[:, :, None, :] - cum)
    Bh = Br.repeat_interleave(rep, dim=3) if rep > 1 else Br
    S_loc = torch.einsum("bclhp,bclhn->bchpn", (xdt.float() * w_end[..., None]).to(cdt), Bh).float()
    Hprev = _run(_SSDStatePass, S_loc, torch.exp(total))                 # (B,nc,H,P,N) fp32
    Ch = Cr.repeat_interleave(rep, dim=3) if rep > 1 else Cr
    y_inter = torch.einsum("bclhn,bchpn->bclhp", (Ch.float() * torch.exp(cum)[..., None]).to(cdt), Hprev.to(cdt))
    y = (y + y_inter).reshape(Bsz, Tp, H, P)[:, :T]
    if D is not None:
        y = y + (x[:, :T].float() * D.float()[None, None, :, None]).to(cdt)
    return y.to(cdt)
