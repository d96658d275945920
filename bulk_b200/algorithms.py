"""Device-wide algorithms over torch CUDA tensors, calling the C-ABI.

These mirror the reference's device-wide drivers (their names, argument
meaning and in-place behaviour) so tests and benchmarks read like the
reference's own drivers:

=====================  ======================================================
this module            reference (jaredhoberock/bulk)
=====================  ======================================================
``reduce``             ``my_reduce(first, last, init, op)``  reduce.cu:58-97
``inclusive_scan``     ``::inclusive_scan(first, last, result, init, op)``
                       scan.cu:87-148
``merge``              ``my_merge(first1, last1, first2, last2, result, comp)``
                       merge.cu:127-162 (+ by-key block merge merge.hpp:507-607)
``stable_sort_by_key`` ``stable_merge_sort_by_key(keys_first, keys_last,
                       values_first, comp)`` merge_sort_by_key.cu:150-209
``reduce_by_key``      ``my_reduce_by_key(keys_first, keys_last, values_first,
                       keys_result, values_result, pred, op)``
                       reduce_by_key.cu:176-272
=====================  ======================================================

torch provides device memory and streams only; every computation runs in
libbulkb200.so.  Errors raise :class:`bulk_b200.BulkError`.
"""
from __future__ import annotations

import threading
from functools import lru_cache

import torch

from . import _lib
from ._lib import check, lib

_TORCH_TO_TAG = {
    torch.int32: "i32",
    torch.int64: "i64",
    torch.float32: "f32",
    torch.float64: "f64",
}
for _name, _tag in (("uint32", "u32"), ("uint64", "u64")):
    if hasattr(torch, _name):
        _TORCH_TO_TAG[getattr(torch, _name)] = _tag


def dtype_tag(t: torch.dtype) -> str:
    try:
        return _TORCH_TO_TAG[t]
    except KeyError:
        raise TypeError(f"unsupported dtype {t}") from None


def _stream_obj(stream: torch.cuda.Stream | None, device: torch.device) -> torch.cuda.Stream:
    return stream if stream is not None else torch.cuda.current_stream(device)


# the current stream's raw handle without a Stream object around it, where torch has it
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_handle(stream: torch.cuda.Stream | None, device: torch.device) -> int:
    if stream is None and _raw_stream is not None and device.index is not None:
        return _raw_stream(device.index)
    return _stream_obj(stream, device).cuda_stream


def _require_cuda(*ts: torch.Tensor) -> torch.device:
    first = None
    for t in ts:
        if t is None:
            continue
        if not t.is_cuda:
            raise ValueError("bulk_b200 operates on CUDA tensors (device memory)")
        if not t.is_contiguous():
            raise ValueError("bulk_b200 needs contiguous tensors")
        if first is None:
            first, index = t, t.get_device()
        elif t.get_device() != index:
            raise ValueError("all tensors must be on the same device")
    return None if first is None else first.device


class _WorkspacePool:
    """One zero-initialised device workspace per (device, stream), grown on demand.

    The library leaves every workspace's counters zeroed after each call, so a
    workspace is reused across calls on the same stream without re-clearing.
    A workspace is allocated and zero-filled on the stream that uses it, so the
    fill is ordered before the library's kernels there; when it grows, the old
    buffer goes back to torch's caching allocator as a block of that stream,
    which hands it out again only in that stream's order, after the kernels
    already queued on it.
    """

    def __init__(self):
        self._lock = threading.Lock()
        self._ws: dict[tuple[int, int], tuple[torch.Tensor, int, int]] = {}  # the buffer, its address and size

    def get(self, nbytes: int, device: torch.device, stream: torch.cuda.Stream | None,
            handle: int | None = None) -> tuple[int, int]:
        """(pointer, bytes) of the workspace of ``stream`` (``handle``: its
        raw handle, when the caller has it; None: the current stream)."""
        if handle is None:
            handle = _stream_handle(stream, device)
        key = (device.index if device.index is not None else torch.cuda.current_device(), handle)
        with self._lock:
            have = self._ws.get(key)
            if have is None or have[2] < nbytes:
                size = max(nbytes, 1 << 16, 0 if have is None else 2 * have[2])
                with torch.cuda.stream(_stream_obj(stream, device)):
                    t = torch.zeros(size, dtype=torch.uint8, device=device)
                have = self._ws[key] = (t, t.data_ptr(), size)
            return have[1], have[2]

    def status(self, device: torch.device | None = None, stream: torch.cuda.Stream | None = None) -> int:
        device = device or torch.device("cuda", torch.cuda.current_device())
        s = _stream_handle(stream, device)
        key = (device.index if device.index is not None else torch.cuda.current_device(), s)
        have = self._ws.get(key)
        if have is None:
            return _lib.BK_OK
        return lib.bk_workspace_status(have[1], have[2], s)

    def clear(self):
        with self._lock:
            self._ws.clear()


workspaces = _WorkspacePool()


def workspace_bytes(algo: str, key: str, value: str | None, n: int) -> int:
    return lib.bk_workspace_bytes(_lib.ALGO[algo], _lib.DTYPE[key], _lib.DTYPE[value], n)


def workspace_status(device=None, stream=None) -> int:
    """Synchronize and return (and clear) the device-side status of this stream's workspace."""
    return workspaces.status(device, stream)


def debug_set_fault(skip_publish_tile: int = -1, spin_limit_ns: int = 0) -> None:
    check(lib.bk_debug_set_fault(skip_publish_tile, spin_limit_ns), "bk_debug_set_fault")


@lru_cache(maxsize=4096)
def _need_bytes(device: int, algo: str, key: str, value: str | None, n: int) -> int:
    """The workspace a call on ``device`` needs.  It depends on types, length
    and device (the reduce's partials: on its SMs) alone: kept for the lengths
    in use, so that a repeated call asks the library once."""
    if device == torch.cuda.current_device():
        return workspace_bytes(algo, key, value, n)
    with torch.cuda.device(device):
        return workspace_bytes(algo, key, value, n)


@lru_cache(maxsize=None)
def _entry(*name: str):
    """The library's entry point bk_<name parts joined>."""
    return getattr(lib, "bk_" + "_".join(name))


def _call(fn, dev: torch.device, stream: torch.cuda.Stream | None, need: int, *args) -> None:
    """``fn(*args, workspace, its bytes, stream)`` with ``dev`` current; no workspace where ``need`` is 0."""
    if dev.index != torch.cuda.current_device():
        with torch.cuda.device(dev):
            return _call(fn, dev, stream, need, *args)
    s = _stream_handle(stream, dev)
    ws, wsb = workspaces.get(need, dev, stream, s) if need else (None, 0)
    status = fn(*args, ws, wsb, s)
    if status != _lib.BK_OK:
        check(status, fn.__name__)


def _need(dev: torch.device, algo: str, key: str, value: str | None, n: int) -> int:
    need = _need_bytes(dev.index, algo, key, value, n)
    return max(need, 256) if need or algo == "reduce" else 0


# ---------------------------------------------------------------------------
def reduce(x: torch.Tensor, init=0, op: str = "sum", out: torch.Tensor | None = None,
           stream: torch.cuda.Stream | None = None) -> torch.Tensor:
    """Return a 1-element device tensor holding init (+) x[0] (+) ... (+) x[n-1]."""
    dev = _require_cuda(x, out)
    tag = dtype_tag(x.dtype)
    if out is None:
        out = torch.empty(1, dtype=x.dtype, device=dev)
    n = x.numel()
    need = _need(dev, "reduce", tag, None, n)
    _call(_entry("reduce", op, tag), dev, stream, need, x.data_ptr(), n, init, out.data_ptr())
    return out


def inclusive_scan(x: torch.Tensor, init=0, op: str = "sum", out: torch.Tensor | None = None,
                   stream: torch.cuda.Stream | None = None) -> torch.Tensor:
    """out[i] = init (+) x[0] (+) ... (+) x[i]; ``out`` may be ``x`` (in place).

    ``init`` may be a device tensor of x's dtype (one element, or a view of
    one, e.g. the last output of a previous scan): it is then read on the
    device when the scan runs, with no copy to the host."""
    dev = _require_cuda(x, out)
    tag = dtype_tag(x.dtype)
    if out is None:
        out = torch.empty_like(x)
    dinit = isinstance(init, torch.Tensor)
    if dinit:
        if not init.is_cuda or init.device != dev or init.dtype != x.dtype or init.numel() != 1:
            raise ValueError("a tensor init must be one element of x's dtype on x's device")
    n = x.numel()
    need = _need(dev, "inclusive_scan", tag, None, n)
    if dinit:
        _call(_entry("inclusive_scan", op, tag, "dinit"), dev, stream, need, x.data_ptr(), n, init.data_ptr(),
              out.data_ptr())
    else:
        _call(_entry("inclusive_scan", op, tag), dev, stream, need, x.data_ptr(), n, init, out.data_ptr())
    return out


def _payload_tag(t: torch.Tensor | None) -> str | None:
    if t is None:
        return None
    if t.element_size() == 4:
        return "u32"
    if t.element_size() == 8:
        return "u64"
    raise TypeError("payloads must be 4- or 8-byte elements")


def merge(a: torch.Tensor, b: torch.Tensor, a_vals: torch.Tensor | None = None, b_vals: torch.Tensor | None = None,
          out: torch.Tensor | None = None, out_vals: torch.Tensor | None = None,
          stream: torch.cuda.Stream | None = None):
    """Stable merge of sorted a and b (ties: a first).  Returns keys, or (keys, vals) with payloads."""
    dev = _require_cuda(a, b, a_vals, b_vals, out, out_vals)
    if a.dtype != b.dtype:
        raise TypeError("a and b must have the same dtype")
    tag = dtype_tag(a.dtype)
    n = a.numel() + b.numel()
    if out is None:
        out = torch.empty(n, dtype=a.dtype, device=dev)
    if a_vals is not None and (b_vals is None or a_vals.element_size() != b_vals.element_size()):
        raise TypeError("a_vals and b_vals must both be given, with the same element size")
    if a_vals is not None and out_vals is None:
        out_vals = torch.empty(n, dtype=a_vals.dtype, device=dev)
    vt = _payload_tag(a_vals)
    need = _need(dev, "merge", tag, vt, n)
    if a_vals is None:
        _call(_entry("merge", tag), dev, stream, need, a.data_ptr(), a.numel(), b.data_ptr(), b.numel(), out.data_ptr())
        return out
    _call(_entry("merge_by_key", tag, vt), dev, stream, need, a.data_ptr(), a_vals.data_ptr(), a.numel(), b.data_ptr(),
          b_vals.data_ptr(), b.numel(), out.data_ptr(), out_vals.data_ptr())
    return out, out_vals


def stable_sort_by_key(keys: torch.Tensor, vals: torch.Tensor | None = None,
                       stream: torch.cuda.Stream | None = None):
    """In-place stable sort of keys (and vals with them).  Returns keys, or (keys, vals)."""
    dev = _require_cuda(keys, vals)
    tag = dtype_tag(keys.dtype)
    n = keys.numel()
    if vals is not None and vals.numel() != n:
        raise ValueError("keys and vals must have the same length")
    vt = _payload_tag(vals)
    need = _need(dev, "sort_by_key", tag, vt, n)
    if vals is None:
        _call(_entry("sort_keys", tag), dev, stream, need, keys.data_ptr(), n)
        return keys
    _call(_entry("sort_by_key", tag, vt), dev, stream, need, keys.data_ptr(), vals.data_ptr(), n)
    return keys, vals


def reduce_by_key(keys: torch.Tensor, vals: torch.Tensor, out_keys: torch.Tensor | None = None,
                  out_vals: torch.Tensor | None = None, num_out: torch.Tensor | None = None,
                  stream: torch.cuda.Stream | None = None, sync: bool = True):
    """One (key, sum) pair per run of equal consecutive keys.

    Returns (out_keys, out_vals, count).  With ``sync=True`` (the reference's
    behaviour, reduce_by_key.cu:269) count is a Python int and the outputs are
    trimmed to it; with ``sync=False`` count stays a 1-element device tensor
    and the outputs are the full-length buffers.
    """
    dev = _require_cuda(keys, vals, out_keys, out_vals, num_out)
    n = keys.numel()
    if vals.numel() != n:
        raise ValueError("keys and vals must have the same length")
    kt, vt = dtype_tag(keys.dtype), dtype_tag(vals.dtype)
    if out_keys is None:
        out_keys = torch.empty(max(n, 1), dtype=keys.dtype, device=dev)
    if out_vals is None:
        out_vals = torch.empty(max(n, 1), dtype=vals.dtype, device=dev)
    if num_out is None:
        num_out = torch.empty(1, dtype=torch.int64, device=dev)
    _call(_entry("reduce_by_key", kt, vt), dev, stream, _need(dev, "reduce_by_key", kt, vt, n), keys.data_ptr(),
          vals.data_ptr(), n, out_keys.data_ptr(), out_vals.data_ptr(), num_out.data_ptr())
    if not sync:
        return out_keys, out_vals, num_out
    c = int(num_out.item())
    return out_keys[:c], out_vals[:c], c
