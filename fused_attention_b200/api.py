"""Host-side mirror of the reference operator, on top of the C ABI.

``attention_forward`` has the signature, argument meaning and error behaviour of the reference's
torch binding (``src/fused_attn_extention.cu:15-117``): fp16 CUDA contiguous rank-3 tensors
``[B, L, F]``, ``RuntimeError`` on any violated precondition, a freshly allocated fp16 output.
Differences, all relaxations: ``L`` need not be a multiple of ``chunk_size`` (ragged tails are
masked inside the kernel), the output is allocated on ``queries.device`` (the reference uses the
current device, ``:67-70``), the launch goes to the caller's current stream, and the mask is
applied to every key tile (the reference applies it to the first chunk only,
``include/fused_attn.cuh:732-742``).
"""
from __future__ import annotations

import ctypes
import importlib.util
import os
import warnings
from typing import Optional

import torch

from . import _lib


def _raw_stream(device: int) -> int:
    """The current stream of a device as the integer that the C ABI takes."""
    return torch.cuda.current_stream(device).cuda_stream


# (torch's own lookup of the same handle, without the Stream object around it: 0.07 us against 2.3)
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", _raw_stream)


def _require(cond: bool, what: str) -> None:
    if not cond:
        raise RuntimeError(f"attention_forward: {what}")


def _check_tensor(t: torch.Tensor, name: str) -> None:
    # src/fused_attn_extention.cu:24-43
    _require(isinstance(t, torch.Tensor), f"{name} must be a tensor")
    _require(t.dtype == torch.float16, f"{name} must be float16")
    _require(t.device.type == "cuda", f"{name} must be a CUDA tensor")
    _require(t.is_contiguous(), f"{name} must be contiguous")
    _require(t.dim() == 3, f"{name} must have 3 dimensions")


# The (head_dim, chunk_size) pairs of src/fused_attn_extention.cu:45-47.
_SIZES = frozenset((h, c) for h in (16, 32, 64, 128) for c in (16, 32, 64, 128) if c <= 2 * h and (h, c) != (128, 16))


def _check_call(head_dim: int, chunk_size: int, queries: torch.Tensor, keys: torch.Tensor, values: torch.Tensor,
                mask: Optional[torch.Tensor]) -> None:
    """Every precondition by itself, with the message of the one that is violated."""
    _check_tensor(queries, "queries")
    _check_tensor(keys, "keys")
    _check_tensor(values, "values")
    if mask is not None:
        _check_tensor(mask, "mask")
    head_dim, chunk_size = int(head_dim), int(chunk_size)
    # src/fused_attn_extention.cu:45-47
    _require(head_dim > 0 and not (head_dim & (head_dim - 1)) and 16 <= head_dim <= 128,
             "head_dim must be a power of two in [16, 128]")
    _require(chunk_size > 0 and not (chunk_size & (chunk_size - 1)) and 16 <= chunk_size <= 128
             and chunk_size <= 2 * head_dim, "chunk_size must be a power of two in [16, 128] and <= 2*head_dim")
    _require(not (chunk_size == 16 and head_dim == 128), "chunk_size 16 with head_dim 128 is not supported")
    B, L, F = queries.shape
    # :55-64 (the L % chunk_size requirement is lifted)
    _require(tuple(keys.shape) == (B, L, F), "keys must have the shape of queries")
    _require(tuple(values.shape) == (B, L, F), "values must have the shape of queries")
    _require(F % head_dim == 0, "the feature size must be divisible by head_dim")
    _require(B > 0 and L > 0 and F > 0, "empty tensors are not supported")
    _require(keys.device == queries.device and values.device == queries.device,
             "queries, keys and values must be on one device")
    if mask is not None:
        _require(tuple(mask.shape) == (B, L, L), "mask must have shape [B, L, L]")
        _require(mask.device == queries.device, "mask must be on the device of queries")


def _is_fp16_cuda(t, device: int) -> bool:
    return isinstance(t, torch.Tensor) and t.dtype is torch.float16 and t.is_cuda and t.get_device() == device and t.is_contiguous()


def _load_native():
    """The call in native code, from the extension module where it has been built: checks, allocation and launch without
    ctypes (B=1 R=4 L=256 H=64: 5.7 us a call, 8.4 through ctypes).  A function that always answers None where there is none,
    or, with a warning, one that cannot be loaded (built for another torch, or from older sources)."""
    from .build import ext_path
    path = os.path.abspath(ext_path())
    if not os.path.exists(path):
        return lambda *args: None
    try:
        spec = importlib.util.spec_from_file_location("fused_attn", path)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        return module._forward_through
    except (ImportError, AttributeError, OSError) as e:
        warnings.warn(f"{path} cannot be used, so calls go through ctypes, which takes some 3 us more each: {e}; rebuild it with "
                      "python -m fused_attention_b200.build --ext", RuntimeWarning, stacklevel=3)
        return lambda *args: None


_native = None


def attention_forward(head_dim: int, chunk_size: int, queries: torch.Tensor, keys: torch.Tensor,
                      values: torch.Tensor, mask: Optional[torch.Tensor] = None, *,
                      flags: int = _lib.FLAG_DEFAULT) -> torch.Tensor:
    """Fused multi-head attention forward ``softmax(Q K^T / sqrt(head_dim)) V`` on the GPU."""
    global _native
    lib = _lib.load()  # raises when the CUDA library is missing: no fallback
    if _native is None:
        _native = _load_native()
    out = _native(lib.forward_entry, head_dim, chunk_size, queries, keys, values, mask, flags)
    if out is not None:
        if out.__class__ is int:
            _lib.check(out)
        return out
    # All preconditions in one expression, nothing formatted and no device object built while they hold; what does not
    # pass goes through the checks one by one (measured on B=1 R=4 L=256 without the native call: 8.3 us a call, 13.8 with the checks in a row
    # and their messages formatted on every call).
    if not (isinstance(queries, torch.Tensor) and queries.is_cuda):
        _check_call(head_dim, chunk_size, queries, keys, values, mask)
    dev = queries.get_device()
    shape = queries.shape
    if not ((head_dim, chunk_size) in _SIZES and _is_fp16_cuda(queries, dev) and _is_fp16_cuda(keys, dev)
            and _is_fp16_cuda(values, dev) and len(shape) == 3 and keys.shape == shape and values.shape == shape
            and shape[2] % head_dim == 0 and 0 not in shape
            and (mask is None or (_is_fp16_cuda(mask, dev) and mask.shape == (shape[0], shape[1], shape[1])))):
        _check_call(head_dim, chunk_size, queries, keys, values, mask)
    out = torch.empty_like(queries)
    rc = lib.fa_b200_attention_forward(
        queries.data_ptr(), keys.data_ptr(), values.data_ptr(), None if mask is None else mask.data_ptr(),
        out.data_ptr(), shape[0], shape[1], shape[2], int(head_dim), int(chunk_size), dev, _raw_stream(dev), int(flags))
    if rc != _lib.OK:
        _lib.check(rc)
    return out


def bind_forward(head_dim: int, chunk_size: int, queries: torch.Tensor, keys: torch.Tensor, values: torch.Tensor,
                 mask: Optional[torch.Tensor] = None, *, out: Optional[torch.Tensor] = None,
                 flags: int = _lib.FLAG_DEFAULT):
    """The same call with its arguments checked and converted once: returns ``(launch, out)`` where ``launch()``
    does nothing but call ``fa_b200_attention_forward`` on the current stream of the tensors' device, writing
    into ``out``.  For loops over fixed tensors (benchmarks, CUDA-graph capture), where the checks and the
    allocation of ``attention_forward`` would cost more than a small problem's kernel."""
    lib = _lib.load()
    probe = attention_forward   # the checks live there; run them once on these tensors
    y = probe(head_dim, chunk_size, queries, keys, values, mask, flags=flags)
    if out is None:
        out = y
    else:
        _check_tensor(out, "out")
        _require(tuple(out.shape) == tuple(queries.shape) and out.device == queries.device, "out must match queries")
    B, L, F = queries.shape
    dev = queries.device.index if queries.device.index is not None else torch.cuda.current_device()
    ptrs = (queries.data_ptr(), keys.data_ptr(), values.data_ptr(), mask.data_ptr() if mask is not None else None,
            out.data_ptr())
    fn, H, C, fl = lib.fa_b200_attention_forward, int(head_dim), int(chunk_size), int(flags)
    keep = (queries, keys, values, mask, out)   # the tensors live as long as the closure

    def launch() -> None:
        rc = fn(ptrs[0], ptrs[1], ptrs[2], ptrs[3], ptrs[4], B, L, F, H, C, dev, _raw_stream(dev), fl)
        if rc != 0:
            _lib.check(rc)
    launch.tensors = keep
    return launch, out


def attention_forward_host(head_dim: int, chunk_size: int, queries: torch.Tensor, keys: torch.Tensor,
                           values: torch.Tensor, mask: Optional[torch.Tensor] = None, *, device: int = 0,
                           out: Optional[torch.Tensor] = None, flags: int = _lib.FLAG_DEFAULT) -> torch.Tensor:
    """Same operator for HOST tensors: copies in, runs on ``device``, copies out, returns when done.

    Goes through ``fa_b200_attention_forward_host``; pinned tensors make the copies asynchronous
    with respect to the host and reach full PCIe speed.
    """
    lib = _lib.load()
    for t, name in ((queries, "queries"), (keys, "keys"), (values, "values")) + (
            ((mask, "mask"),) if mask is not None else ()):
        _require(t.dtype == torch.float16 and t.device.type == "cpu" and t.is_contiguous() and t.dim() == 3,
                 f"{name} must be a contiguous float16 CPU tensor of rank 3")
    B, L, F = queries.shape
    _require(tuple(keys.shape) == (B, L, F) and tuple(values.shape) == (B, L, F), "shape mismatch")
    if mask is not None:
        _require(tuple(mask.shape) == (B, L, L), "mask must have shape [B, L, L]")
    if out is None:
        out = torch.empty_like(queries)
    else:
        _require(out.dtype == torch.float16 and out.device.type == "cpu" and out.is_contiguous()
                 and tuple(out.shape) == (B, L, F), "out must match queries")
    rc = lib.fa_b200_attention_forward_host(
        queries.data_ptr(), keys.data_ptr(), values.data_ptr(),
        mask.data_ptr() if mask is not None else None, out.data_ptr(),
        B, L, F, int(head_dim), int(chunk_size), int(device), int(flags))
    _lib.check(rc)
    return out


def read_status(device: int = 0) -> tuple[int, int]:
    """(first failure code, reporting CTA count) of the device status word; clears it."""
    w = (ctypes.c_uint32 * 2)()
    _lib.check(_lib.load().fa_b200_read_status(int(device), w))
    return int(w[0]), int(w[1])


def query(device: int = 0) -> dict:
    o = (ctypes.c_int32 * 4)()
    _lib.check(_lib.load().fa_b200_query(int(device), o))
    return {"cc_major": o[0], "cc_minor": o[1], "sm_count": o[2], "smem_optin": o[3]}


def describe_call(B: int, L: int, F: int, head_dim: int, mask_alignment: int = 0, flags: int = 0, sm_count: int = 148) -> dict:
    """What a call launches (``fa_b200_describe_call``): ``kernel``, whether it is ``planned`` on a stream that has scratch,
    and the number of ``launches`` then.  ``mask_alignment``: 0 without a mask, else what its address is a multiple of."""
    o = (ctypes.c_uint32 * 3)()
    _lib.check(_lib.load().fa_b200_describe_call(B, L, F, head_dim, int(mask_alignment), int(flags), int(sm_count), o))
    return {"kernel": ("short sequences", "simple", "pipelined", "pipelined on pairs of CTAs")[o[0]], "planned": bool(o[1]),
            "launches": int(o[2])}


def stream_has_scratch(stream: int = 0, device: int = 0) -> bool:
    """Whether a call on a stream (its handle) would find scratch for a divided or planned call."""
    o = (ctypes.c_uint32 * 1)()
    _lib.check(_lib.load().fa_b200_stream_has_scratch(int(device), int(stream), o))
    return bool(o[0])


def plan_taken(stream: int = 0, device: int = 0) -> Optional[bool]:
    """Whether the planned kernel had the last planned call on a stream (its handle), or the kernel behind it; None where
    that is not known (``fa_b200_plan_taken``).  Synchronises the stream."""
    o = (ctypes.c_uint32 * 2)()
    _lib.check(_lib.load().fa_b200_plan_taken(int(device), int(stream), o))
    return bool(o[1]) if o[0] else None


def select_kernel(B: int, L: int, F: int, head_dim: int, has_mask: bool = False, flags: int = 0) -> str:
    rc = _lib.load().fa_b200_select_kernel(B, L, F, head_dim, int(has_mask), flags)
    if rc < 0:
        _lib.check(rc)
    return {1: "simple", 2: "pipelined", 3: "pipelined on pairs of CTAs"}[rc]


def describe_schedule(B: int, L: int, F: int, head_dim: int, flags: int = 0, sm_count: int = 148) -> dict:
    """How the warp-specialised kernel spreads a call over its CTAs (``fa_b200_describe_schedule``)."""
    o = (ctypes.c_uint32 * 7)()
    _lib.check(_lib.load().fa_b200_describe_schedule(B, L, F, head_dim, int(flags), int(sm_count), o))
    return {"kernel": {1: "simple", 2: "pipelined", 3: "pipelined on pairs of CTAs"}[o[0]], "grid": o[1], "full_rounds": o[2],
            "tail_items": o[3], "tail_steps": o[4], "key_steps": o[5], "tail_grid": o[6]}


def cta_segments(sched: dict, n_items: int, cta: int) -> list[tuple[int, int, int]]:
    """The (work item, first key step, key steps) runs that CTA ``cta`` works through under ``sched``, in
    the kernel's order and with its arithmetic: whole items round-robin, then its share of a divided
    round (at most two runs)."""
    grid, n, T = sched["grid"], sched["key_steps"], sched["tail_steps"]
    if T == 0:
        return [(item, 0, n) for item in range(cta, n_items, grid)]
    segs = [(cta + k * grid, 0, n) for k in range(sched["full_rounds"])]
    tg = sched["tail_grid"]
    a, b = (cta * T // tg, (cta + 1) * T // tg) if cta < tg else (0, 0)
    base = sched["full_rounds"] * grid
    if b > a:
        t0, j0 = divmod(a, n)
        len0 = min(n - j0, b - a)
        segs.append((base + t0, j0, len0))
        if b - a > len0:
            segs.append((base + t0 + 1, 0, b - a - len0))
    return segs
