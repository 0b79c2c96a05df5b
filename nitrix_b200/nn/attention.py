"""Scaled-dot-product / flash attention on B200, PyTorch-hosted.

Drop-in for the reference's public entry
``nitrix.nn.attention.scaled_dot_product_attention``
(reference ``src/nitrix/nn/attention/__init__.py:126-230``): same positional
and keyword surface ``(q, k, v, *, bias, mask, scale, causal, qk_norm,
backend)``, same validation errors (``:40-60``), same differentiation contract
as its ``custom_vjp`` (reference ``src/nitrix/_kernels/cuda/attention.py:661-700``):
residuals ``(q, k, v, bias, mask, out, lse)``, cotangents
``(dq, dk, dv, dbias-or-None, None)`` with ``scale`` and ``causal`` static.

Differences, all on purpose:

* tensors are ``torch`` CUDA tensors (device memory, streams); the arithmetic
  is done by the CUDA library behind ``include/nitrix_b200_attention.h``, the
  differentiation rule is a C++ autograd function over it
  (``csrc/host/torch_ops.cpp``);
* bias and mask are passed by stride, never broadcast-materialised, and q/k/v
  stay in ``(..., h, s, d)`` layout (the reference transposes and materialises,
  ``attention.py:507-514,560-569``);
* ``dbias`` is produced only when ``bias.requires_grad`` (the reference always
  produces it when a bias is present, ``attention.py:408,437``);
* there is no host fallback: a problem the fused kernels decline runs on the
  CUDA-core family of the same library, with the reference's warn-once
  contract.
"""
from __future__ import annotations

import ctypes as C
import math
from typing import Optional, Tuple

import torch

from .. import _cabi
from ..backend import fallback, resolve_backend

__all__ = ["scaled_dot_product_attention", "default_scale", "qk_rms_norm", "sdpa_forward", "sdpa_backward"]

_QK_RMS_EPS = 1e-6  # reference _reference.py:32

_DTYPES = {torch.float32: _cabi.F32, torch.bfloat16: _cabi.BF16, torch.float16: _cabi.F16}
_KERNELS = {"cuda-sm100": _cabi.KERNEL_AUTO, "cuda-simt": _cabi.KERNEL_SIMT}


def default_scale(head_dim: int) -> float:
    """``1/sqrt(d)`` (reference ``_reference.py:35-49``)."""
    return 1.0 / math.sqrt(float(head_dim))


def qk_rms_norm(z: torch.Tensor) -> torch.Tensor:
    """RMS-normalise over the head dim, no learnable scale (reference ``_reference.py:52-77``).

    Runs outside the fused kernels' differentiation rule, as in the reference
    (``nn/attention/__init__.py:193-197``), so autograd chains its gradient.
    """
    acc = torch.promote_types(z.dtype, torch.float32)
    zf = z.to(acc)
    return (zf * torch.rsqrt(zf.square().mean(-1, keepdim=True) + _QK_RMS_EPS)).to(z.dtype)


def _qk_norm_fusable(q: torch.Tensor, k: torch.Tensor) -> bool:
    """Both on one CUDA device, same supported dtype and head dim, rows the kernel can read with 16-byte loads."""
    return _cabi.torch_ops().qk_norm_fits(q, k)


def qk_rms_norm_pair(q: torch.Tensor, k: torch.Tensor):
    """``qk_rms_norm`` of q and k: one kernel launch each way (``nb200_qk_rms_norm`` / ``nb200_qk_rms_norm_grad``) where
    that pre-op's layout rules hold, else the element-wise form.  Same place in the call sequence as the reference's
    (``nn/attention/__init__.py:193-197``): outside the attention kernels' own differentiation rule."""
    if _qk_norm_fusable(q, k):
        return _cabi.torch_ops().qk_norm(q, k)
    return qk_rms_norm(q), qk_rms_norm(k)


def _validate(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> None:
    # reference nn/attention/__init__.py:40-60
    if q.ndim < 3 or k.ndim < 3 or v.ndim < 3:
        raise ValueError(
            "scaled_dot_product_attention: q, k, v must have at least 3 dims (..., h, s, d); "
            f"got ndim {q.ndim}, {k.ndim}, {v.ndim}."
        )
    if q.shape[-1] != k.shape[-1]:
        raise ValueError(
            f"scaled_dot_product_attention: q/k head-dim mismatch (q d={q.shape[-1]}, k d={k.shape[-1]})."
        )
    if k.shape[-2] != v.shape[-2]:
        raise ValueError(
            f"scaled_dot_product_attention: k/v key-length mismatch (k t={k.shape[-2]}, v t={v.shape[-2]})."
        )


# ---------------------------------------------------------------------------
# shape canonicalisation: everything becomes 4-D (B, H, rows, cols)
# ---------------------------------------------------------------------------

def _to_bhxd(x: torch.Tensor, lead: Tuple[int, ...], h: int) -> torch.Tensor:
    """(..., h, n, d) -> (B, h, n, d) with the leading dims broadcast to ``lead``."""
    n, d = x.shape[-2], x.shape[-1]
    x = x.expand(*lead, h, n, d) if tuple(x.shape[:-3]) != lead or x.shape[-3] != h else x
    x = x.reshape(-1, h, n, d) if x.ndim != 4 else x
    if x.stride(-1) != 1 or _has_expanded_axis(x):
        # the tensor-core kernels address q, k, v by absolute (batch, head): an expanded view is materialised
        x = x.contiguous()
    return x


def _has_expanded_axis(x: torch.Tensor) -> bool:
    return 0 in x.stride() and any(st == 0 and n > 1 for st, n in zip(x.stride(), x.shape))


def _to_own_extent(x: torch.Tensor, lead: Tuple[int, ...], h: int, s: int, t: int) -> torch.Tensor:
    """bias / mask broadcastable to (*lead, h, s, t) -> 4-D (Bb, Hb, Sb, Tb), each extent 1 or full.

    Only differentiable view/expand ops are used, so a bias gradient of this
    4-D shape flows back to the caller's bias shape through autograd.  Leading
    dims are merged without copying whenever they are all broadcast or all
    present; a partially broadcast multi-dim batch is expanded over the batch.
    """
    full = (*lead, h, s, t)
    if x.ndim == 4 and len(full) == 4 and all(have == 1 or have == want for have, want in zip(x.shape, full)):
        return x   # already there (a view of a view would only be two more nodes for autograd to walk)
    if x.ndim > len(full):
        raise ValueError(f"bias/mask of shape {tuple(x.shape)} has more dims than (..., h, s, t) = {full}")
    x = x.reshape((1,) * (len(full) - x.ndim) + tuple(x.shape))
    for have, want in zip(x.shape, full):
        if have != 1 and have != want:
            raise ValueError(f"bias/mask of shape {tuple(x.shape)} does not broadcast to {full}")
    nl = len(lead)
    lead_have = tuple(x.shape[:nl])
    if all(a == 1 for a in lead_have):
        x = x.reshape(1, *x.shape[nl:])
    elif lead_have == lead:
        x = x.reshape(-1, *x.shape[nl:])
    else:
        x = x.expand(*lead, *x.shape[nl:]).reshape(-1, *x.shape[nl:])
    return x


def _strides4(x: Optional[torch.Tensor], full: Tuple[int, int, int, int]):
    """Element strides with 0 on every broadcast (extent-1) axis."""
    arr = (C.c_int64 * 4)()
    if x is not None:
        for a in range(4):
            arr[a] = 0 if (x.shape[a] == 1 and full[a] != 1) else x.stride(a)
    return arr


class PackedMask:
    """A boolean mask bit-packed once by ``nb200_mask_pack`` for one problem shape and reused by the forward, the
    backward and later calls.  ``level`` 1: packed without the key-major copy; 2: with it (what the backward of a
    mask with a query axis reads).  ``like`` is the 4-D byte mask it was packed from (strides tell the library
    which axes the mask broadcasts over)."""

    def __init__(self, blob: torch.Tensor, level: int, like: torch.Tensor):
        self.blob, self.level, self.like = blob, int(level), like


def _fill_common(p, q, k, v, out, lse, bias, mask, scale, causal, kernel, bh_range):
    B, H, S, D = q.shape
    T, Dv = k.shape[2], v.shape[3]
    p.dtype = _DTYPES[q.dtype]
    p.B, p.H, p.S, p.T, p.D, p.Dv = B, H, S, T, D, Dv
    p.q, p.k, p.v, p.out, p.lse = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr()
    full = (B, H, S, T)
    for name, ten in (("q_stride", q), ("k_stride", k), ("v_stride", v), ("out_stride", out)):
        getattr(p, name)[:] = list(ten.stride())
    if bias is not None:
        p.bias = bias.data_ptr()
        p.bias_dtype = _DTYPES[bias.dtype]
        p.bias_stride = _strides4(bias, full)
    if isinstance(mask, PackedMask):
        p.mask = mask.blob.data_ptr()
        p.mask_stride = _strides4(mask.like, full)
        p.mask_is_bitpacked = mask.level
    elif mask is not None:
        p.mask = mask.data_ptr()
        p.mask_stride = _strides4(mask, full)
    p.scale = float(scale)
    p.causal = int(bool(causal))
    p.kernel = int(kernel)
    lo, hi = (0, B * H) if bh_range is None else bh_range
    p.bh_begin, p.bh_end = int(lo), int(hi)


def _check(rc: int, what: str) -> None:
    if rc != _cabi.OK:
        raise RuntimeError(f"{what} failed (status {rc}): {_cabi.last_error()}")


def _launch(fn, p, device, what: str) -> None:
    """Call a library entry point on `device`'s current stream (the device is switched only when it is not current)."""
    _check(_cabi.enqueue(fn, p, device), what)


def _mask_bytes(mask):
    if mask is None or isinstance(mask, PackedMask):
        return mask
    if mask.dtype == torch.bool:
        return mask.view(torch.uint8)
    if mask.dtype == torch.uint8:
        return mask
    return (mask != 0).view(torch.uint8)


_plan_cache: dict = {}


def planned_kernel(q, k, v, bias=None, mask=None, *, scale=1.0, causal=False, which=_cabi.PASS_FWD,
                   kernel=_cabi.KERNEL_AUTO, want_dbias=False) -> int:
    """Kernel family the library would run for these 4-D operands (no launch; remembered by their layout)."""
    key = (_meta(q), _meta(k), _meta(v), _meta(bias), _mask_meta(mask), float(scale), bool(causal), q.device.index, which,
           kernel, bool(want_dbias))
    if key in _plan_cache:
        return _plan_cache[key]
    p = _cabi.new_params()
    B, H, S, _ = q.shape
    out = q  # pointers are not dereferenced by the planner
    lse = q
    _fill_common(p, q, k, v, out, lse, bias, _mask_bytes(mask), scale, causal, kernel, None)
    p.dout = p.dq = p.dk = p.dv = q.data_ptr()
    p.dout_stride = p.dq_stride = p.out_stride
    p.dk_stride, p.dv_stride = p.k_stride, p.v_stride
    if want_dbias and bias is not None and which == _cabi.PASS_BWD:
        p.want_dbias = 1   # the planner needs no dbias buffer
        p.dbias_stride[:] = [bias.shape[1] * bias.shape[2] * bias.shape[3], bias.shape[2] * bias.shape[3], bias.shape[3], 1]
    chosen = C.c_int(0)
    _check(_cabi.lib().nb200_sdpa_plan(C.byref(p), which, C.byref(chosen)), "nb200_sdpa_plan")
    if len(_plan_cache) >= 512:
        _plan_cache.clear()
    _plan_cache[key] = chosen.value
    return chosen.value


def pack_mask(q, k, v, mask, *, with_transpose: bool = True) -> PackedMask:
    """Bit-pack a 4-D boolean / byte mask for these operands' shape (enqueued on the current stream)."""
    mask_b = _mask_bytes(mask)
    p = _cabi.new_params()
    _fill_common(p, q, k, v, q, q, None, mask_b, 1.0, False, _cabi.KERNEL_AUTO, None)
    need = C.c_size_t(0)
    _check(_cabi.lib().nb200_mask_pack_bytes(C.byref(p), int(with_transpose), C.byref(need)), "nb200_mask_pack_bytes")
    blob = torch.empty(max(int(need.value), 1), dtype=torch.uint8, device=q.device)
    _check(_cabi.enqueue(lambda a, stream: _cabi.lib().nb200_mask_pack(a, int(with_transpose), blob.data_ptr(),
                                                                      blob.numel(), stream), p, q.device),
           "nb200_mask_pack")
    return PackedMask(blob, 2 if with_transpose else 1, mask_b)


def _meta(x: Optional[torch.Tensor]):
    # everything the planner looks at: dtype, extents, strides and the 16-byte alignment of the base address
    return None if x is None else (x.dtype, x.shape, x.stride(), x.data_ptr() & 15)


_POINTERS = ("q", "k", "v", "out", "lse", "bias", "mask", "dout", "dq", "dk", "dv", "dbias", "workspace")
_call_cache: dict = {}


def _call_params(key, fill):
    """A parameter block for operands of the layout that ``key`` describes, and the bytes of workspace the call needs.
    ``fill()`` returns ``(block, bytes)``; all of the block but its pointers is remembered by the key, which holds
    everything the library's answer depends on (the scale itself: families and scratch differ with its sign, with zero and
    with whether 1 / scale is a number of the storage type) (filling its 70 fields and asking the library took 25 us of a 60 us call), and every caller gets a copy of its own."""
    hit = _call_cache.get(key)
    if hit is None:
        p, need = fill()
        proto = _cabi.SdpaParams.from_buffer_copy(p)
        for name in _POINTERS:
            setattr(proto, name, None)
        if len(_call_cache) >= 512:
            _call_cache.clear()
        _call_cache[key] = (bytes(proto), need)
        return p, need
    return _cabi.SdpaParams.from_buffer_copy(hit[0]), hit[1]


def _workspace_need(p, which: int, query: str = "nb200_sdpa_workspace_bytes") -> int:
    need = C.c_size_t(0)
    _check(getattr(_cabi.lib(), query)(C.byref(p), which, C.byref(need)), query)
    return need.value


def _least_workspace(p, which: int, need: int, device) -> Optional[torch.Tensor]:
    """For a device without room for all of a call's ``need`` bytes of scratch: the least with which the call runs (the
    planes of fp32 operands take up to 1 GiB that the other kernels do without)."""
    least = _workspace_need(p, which, "nb200_sdpa_workspace_least_bytes")
    if least >= need:
        raise torch.OutOfMemoryError(f"no room for {need} bytes of workspace")
    return torch.empty(least, dtype=torch.uint8, device=device) if least else None


def _mask_meta(mask):
    # (a packed mask by the address of its bits, the layout it was packed from and its level)
    if isinstance(mask, PackedMask):
        return (_meta(mask.like), mask.level, mask.blob.data_ptr() & 15)
    return _meta(mask)


def sdpa_forward(q, k, v, bias=None, mask=None, *, scale: float, causal: bool = False,
                 kernel: int = _cabi.KERNEL_AUTO, bh_range=None, out=None, lse=None, out_peers=()):
    """Enqueue the forward on the current stream; 4-D operands.  Returns ``(out, lse)``.

    ``q`` (B,H,S,D), ``k`` (B,H,T,D), ``v`` (B,H,T,Dv); ``bias`` / ``mask`` 4-D
    with each extent 1 (broadcast) or full.  ``lse`` is fp32 (B,H,S), base 2.
    ``out_peers``: device addresses (ints) of further buffers with ``out``'s shape and strides that receive every
    output row as well (the fused all-gather of :mod:`nitrix_b200.parallel`).
    """
    B, H, S, _ = q.shape
    Dv = v.shape[3]
    if out is None:
        out = torch.empty((B, H, S, Dv), dtype=q.dtype, device=q.device)
    if lse is None:
        lse = torch.empty((B, H, S), dtype=torch.float32, device=q.device)
    mask_b = _mask_bytes(mask)
    bh_range = None if bh_range is None else tuple(map(int, bh_range))

    def fill():
        p = _cabi.new_params()
        _fill_common(p, q, k, v, out, lse, bias, mask_b, scale, causal, kernel, bh_range)
        p.n_out_peers = len(out_peers)
        for i, ptr in enumerate(out_peers):
            p.out_peers[i] = int(ptr)
        return p, _workspace_need(p, _cabi.PASS_FWD)

    if out_peers:
        p, need = fill()
    else:
        p, need = _call_params((_cabi.PASS_FWD, _meta(q), _meta(k), _meta(v), _meta(bias), _mask_meta(mask_b), _meta(out),
                                float(scale), bool(causal), kernel, bh_range, q.device.index), fill)
    p.scale = float(scale)
    p.q, p.k, p.v, p.out, p.lse = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr()
    if bias is not None:
        p.bias = bias.data_ptr()
    if mask_b is not None:
        p.mask = (mask_b.blob if isinstance(mask_b, PackedMask) else mask_b).data_ptr()
    ws = None
    if need:
        try:
            ws = torch.empty(need, dtype=torch.uint8, device=q.device)
        except torch.OutOfMemoryError:
            ws = _least_workspace(p, _cabi.PASS_FWD, need, q.device)
        if ws is not None:
            p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    _launch(_cabi.lib().nb200_sdpa_fwd, p, q.device, "nb200_sdpa_fwd")
    del ws  # same-stream reuse is ordered by the caching allocator
    return out, lse


def sdpa_backward(q, k, v, bias, mask, out, lse, dout, *, scale: float, causal: bool = False,
                  want_dbias: bool = False, kernel: int = _cabi.KERNEL_AUTO, bh_range=None, grads=None):
    """Enqueue the backward on the current stream; returns ``(dq, dk, dv, dbias_or_None)``.

    ``dbias`` has the bias' own 4-D extent (broadcast axes already reduced) and dtype.  ``grads`` = existing
    ``(dq, dk, dv, dbias_or_None)`` buffers to write into (several ``bh_range`` calls filling one set of buffers).
    """
    if dout.stride(-1) != 1 or _has_expanded_axis(dout):
        dout = dout.contiguous()   # e.g. the cotangent of out.sum() or out.mean(0) arrives as an expanded view
    if grads is not None:
        dq, dk, dv, dbias_buf = grads
    else:
        dq = torch.empty_like(q, memory_format=torch.contiguous_format)
        dk = torch.empty_like(k, memory_format=torch.contiguous_format)
        dv = torch.empty_like(v, memory_format=torch.contiguous_format)
        dbias_buf = None
    dbias = None
    if want_dbias:
        if bias is None:
            raise ValueError("want_dbias without a bias")
        if _has_expanded_axis(bias):   # (a stride of 0 is a broadcast axis to the library, which has one gradient for it)
            bias = bias.contiguous()
        dbias = dbias_buf if dbias_buf is not None else torch.empty(bias.shape, dtype=bias.dtype, device=bias.device)
    mask_b = _mask_bytes(mask)
    bh_range = None if bh_range is None else tuple(map(int, bh_range))

    def fill():
        p = _cabi.new_params()
        _fill_common(p, q, k, v, out, lse, bias, mask_b, scale, causal, kernel, bh_range)
        p.dout, p.dq, p.dk, p.dv = dout.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr()
        p.dout_stride[:] = list(dout.stride())
        p.dq_stride[:] = list(dq.stride())
        p.dk_stride[:] = list(dk.stride())
        p.dv_stride[:] = list(dv.stride())
        if dbias is not None:
            p.dbias = dbias.data_ptr()
            p.dbias_stride[:] = list(dbias.stride())
        return p, _workspace_need(p, _cabi.PASS_BWD)

    p, need = _call_params((_cabi.PASS_BWD, _meta(q), _meta(k), _meta(v), _meta(bias), _mask_meta(mask_b), _meta(out),
                            _meta(dout), _meta(dq), _meta(dk), _meta(dv), _meta(dbias), lse.data_ptr() & 15, float(scale), bool(causal),
                            kernel, bh_range, q.device.index), fill)
    p.scale = float(scale)
    p.q, p.k, p.v, p.out, p.lse = q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr()
    p.dout, p.dq, p.dk, p.dv = dout.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr()
    if bias is not None:
        p.bias = bias.data_ptr()
    if mask_b is not None:
        p.mask = (mask_b.blob if isinstance(mask_b, PackedMask) else mask_b).data_ptr()
    if dbias is not None:
        p.dbias = dbias.data_ptr()
    ws = None
    if need:
        try:
            ws = torch.empty(need, dtype=torch.uint8, device=q.device)
        except torch.OutOfMemoryError:
            ws = _least_workspace(p, _cabi.PASS_BWD, need, q.device)
        if ws is not None:
            p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
    _launch(_cabi.lib().nb200_sdpa_bwd, p, q.device, "nb200_sdpa_bwd")
    del ws  # same-stream reuse is ordered by the caching allocator
    return dq, dk, dv, dbias


def scaled_dot_product_attention(
    q: torch.Tensor,
    k: torch.Tensor,
    v: torch.Tensor,
    *,
    bias: Optional[torch.Tensor] = None,
    mask: Optional[torch.Tensor] = None,
    scale: Optional[float] = None,
    causal: bool = False,
    qk_norm: bool = False,
    backend: str = "auto",
    return_lse: bool = False,
):
    """``softmax(scale * q k^T + bias [masked]) v`` over the key axis, differentiable.

    Parameters follow the reference entry point: ``q`` ``(..., h, s, d)``, ``k``
    ``(..., h, t, d)``, ``v`` ``(..., h, t, d_v)``; ``bias`` (additive, applied
    after scaling) and ``mask`` (boolean, ``True`` keeps) broadcast to
    ``(..., h, s, t)``; ``causal`` keeps keys ``j <= i`` with indices aligned at
    zero and is AND-ed with ``mask``; ``scale`` defaults to ``1/sqrt(d)``;
    ``qk_norm`` RMS-normalises q and k first.  The result has shape
    ``(..., h, s, d_v)`` and the common dtype of q, k, v.  Computation is fp32
    (accumulators, softmax) whatever the storage dtype.  A query row with no
    kept key yields NaN, like the reference's ``jnp`` path.

    ``backend``: ``'auto'`` | ``'cuda-sm100'`` (alias ``'pallas-cuda'``) |
    ``'cuda-simt'``; see :mod:`nitrix_b200.backend`.
    """
    _validate(q, k, v)
    resolved_scale = default_scale(q.shape[-1]) if scale is None else float(scale)
    resolved = resolve_backend(backend)
    if not (q.is_cuda and k.is_cuda and v.is_cuda):
        raise ValueError("scaled_dot_product_attention: q, k, v must be CUDA tensors (no host path exists)")
    out_dtype = q.dtype
    if k.dtype != out_dtype or v.dtype != out_dtype:
        out_dtype = torch.promote_types(torch.promote_types(q.dtype, k.dtype), v.dtype)
    if out_dtype not in _DTYPES:
        raise ValueError(f"scaled_dot_product_attention: dtype {out_dtype} is not supported (fp32, bf16, fp16)")
    q, k, v = q.to(out_dtype), k.to(out_dtype), v.to(out_dtype)
    if qk_norm:
        q, k = qk_rms_norm_pair(q, k)

    kernel = _KERNELS[resolved]
    attention = _cabi.torch_ops().attention
    operands = (q, k, v, bias, mask)
    lead, (h, s) = tuple(q.shape[:-3]), q.shape[-3:-1]
    dv = v.shape[-1]
    out4, lse4, fit = attention(*operands, resolved_scale, bool(causal), kernel, False)
    if not fit:
        t, lk, lv = k.shape[-2], tuple(k.shape[:-3]), tuple(v.shape[:-3])
        lead = lead if (lead == lk and lead == lv) else tuple(torch.broadcast_shapes(lead, lk, lv))
        if k.shape[-3] != h or v.shape[-3] != h:
            raise ValueError(f"scaled_dot_product_attention: head-count mismatch (q {h}, k {k.shape[-3]}, v {v.shape[-3]})")
        if bias is not None:
            bias = _to_own_extent(bias if bias.dtype in _DTYPES else bias.to(torch.float32), lead, h, s, t)
        if mask is not None:
            mask = _mask_bytes(_to_own_extent(mask, lead, h, s, t))
        operands = (_to_bhxd(q, lead, h), _to_bhxd(k, lead, h), _to_bhxd(v, lead, h), bias, mask)
        out4, lse4, fit = attention(*operands, resolved_scale, bool(causal), kernel, False)
        if not fit:
            raise ValueError("scaled_dot_product_attention: q, k, v, bias and mask must be on one CUDA device")
    if out4 is None:
        # fp32 operands on the tensor-core kernels are a fused path too (fp32 is the one dtype the reference's fused
        # kernels accept, attention.py:736-744): only a problem that leaves the tensor paths altogether warns
        fallback(
            function="scaled_dot_product_attention",
            requested="cuda-sm100",
            resolved="cuda-simt",
            reason=(
                "the fused tcgen05 kernels take bf16/fp16 with d == d_v in {64, 128} (any query/key lengths); "
                "the fp32 tensor-core kernels take d, d_v in {32, 64, 128}"
            ),
            shapes=(tuple(q.shape), tuple(k.shape), tuple(v.shape)),
            dtype=out_dtype,
        )
        out4, lse4, _ = attention(*operands, resolved_scale, bool(causal), kernel, True)
    out = out4 if len(lead) == 1 else out4.reshape(*lead, h, s, dv)
    if return_lse:
        return out, lse4 if len(lead) == 1 else lse4.reshape(*lead, h, s)
    return out
