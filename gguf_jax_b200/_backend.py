"""Device plumbing shared by the host-side modules: torch tensors, streams, scratch.

PyTorch is used for device memory, streams and process groups only; every computation on
quantized data goes through the C ABI in include/ggq.h.
"""
from __future__ import annotations

import numpy as np
import torch

from . import _lib

_DTYPE_CODE = {torch.float32: _lib.GGQ_F32, torch.bfloat16: _lib.GGQ_BF16, torch.float16: _lib.GGQ_F16}


def canon_dtype(dtype) -> torch.dtype:
    """Accept torch dtypes, numpy dtypes and names ('bfloat16', 'float32', ...)."""
    if isinstance(dtype, torch.dtype):
        return dtype
    name = getattr(dtype, "name", None) or getattr(dtype, "__name__", None) or str(dtype)
    name = str(name).replace("torch.", "")
    try:
        return getattr(torch, np.dtype(name).name)
    except TypeError:
        pass
    out = getattr(torch, name, None)
    if not isinstance(out, torch.dtype):
        raise TypeError(f"unsupported dtype {dtype!r}")
    return out


def dtype_code(dtype: torch.dtype) -> int:
    try:
        return _DTYPE_CODE[dtype]
    except KeyError:
        raise TypeError(f"the kernels write float32, bfloat16 or float16, not {dtype}") from None


def default_device() -> torch.device:
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


def as_tensor(data, device=None) -> torch.Tensor:
    """numpy / torch / buffer -> torch tensor on ``device`` (default: the current CUDA
    device when there is one), mirroring ``jnp.asarray`` in the reference."""
    if isinstance(data, torch.Tensor):
        return data if device is None else data.to(device)
    t = torch.as_tensor(np.ascontiguousarray(data))
    return t.to(default_device() if device is None else device)


def require_cuda(t: torch.Tensor, what: str) -> int:
    if not t.is_cuda:
        raise RuntimeError(
            f"{what}: the data lives on {t.device}; this library computes on a CUDA device only "
            "(there is no CPU fallback). Move the array to a B200 first.")
    return t.device.index if t.device.index is not None else torch.cuda.current_device()


def stream_ptr(device_index: int) -> int:
    return torch.cuda.current_stream(device_index).cuda_stream


def _capture_id(stream: int) -> int:
    """Identity of the CUDA graph capture that the stream takes part in, 0 outside any."""
    return _lib.native().capture_id(stream)


class _Buffers:
    """One device buffer per (device, stream), grown on demand: the calls of a stream are ordered, so one serves them all.

    CUDA graphs keep the addresses they were captured with.  So a buffer that a capture has been given stays allocated when a
    larger one takes its place (which is then at least twice as large: those kept never add up to more than the current
    one).  And a buffer that is first allocated under capture belongs to that capture alone: it is the graph's memory and
    its zero fill runs on replay, so no other graph and no call outside may take it for a cleared one.
    Graphs captured on a stream that had its buffer share it: their replays must not overlap each other or the stream's calls."""

    def __init__(self, smallest: int, zeroed: bool, publish: bool):
        self.smallest, self.zeroed, self.publish = smallest, zeroed, publish
        self.current: dict[tuple[int, int], torch.Tensor] = {}
        self.in_graphs: set[tuple[int, int]] = set()               # keys whose current buffer a capture was given
        self.kept: dict[tuple[int, int], list[torch.Tensor]] = {}
        self.of_capture: dict[tuple[int, int], tuple[int, torch.Tensor]] = {}

    def _new(self, device_index: int, nbytes: int) -> torch.Tensor:
        make = torch.zeros if self.zeroed else torch.empty
        return make(max(nbytes, self.smallest), dtype=torch.uint8, device=torch.device("cuda", device_index))

    def get(self, device_index: int, nbytes: int, stream: int, least: int | None = None) -> torch.Tensor | None:
        """At least ``nbytes``; under capture, where none is that large yet, ``least`` will do."""
        key = (device_index, stream)
        buf = self.current.get(key)
        capture = _capture_id(stream)
        if capture:
            own = self.of_capture.get(key)
            if own is not None and own[0] == capture and own[1].numel() >= nbytes:
                return own[1]
            if least is not None and least < nbytes and (buf is None or buf.numel() < nbytes):
                return self.get(device_index, least, stream)
            if buf is not None and buf.numel() >= nbytes > 0:
                self.in_graphs.add(key)
                return buf
            if nbytes > 0:
                buf = self._new(device_index, nbytes)
                self.of_capture[key] = (capture, buf)
                return buf
        if nbytes == 0:
            return None
        if buf is None or buf.numel() < nbytes:
            if key in self.in_graphs:
                self.in_graphs.discard(key)
                self.kept.setdefault(key, []).append(buf)
                nbytes = max(nbytes, 2 * buf.numel())
            buf = self.current[key] = self._new(device_index, nbytes)
            if self.publish:
                _lib.native().set_scratch(key[0], key[1], buf)
        return buf


_workspaces = _Buffers(1 << 20, zeroed=True, publish=True)
_stagings = _Buffers(1 << 16, zeroed=False, publish=False)


def staging(device_index: int, nbytes: int, stream: int | None = None) -> torch.Tensor:
    """Device buffer that receives host-resident activations.  ``stream``: the current stream's handle if the caller already
    has it."""
    return _stagings.get(device_index, nbytes, stream_ptr(device_index) if stream is None else stream)


def workspace(device_index: int, nbytes: int, stream: int | None = None, least: int | None = None) -> torch.Tensor | None:
    """Zero-filled scratch for the fused kernels.  The kernels leave it zeroed, so it is cleared only when (re)allocated.
    ``stream``: the current stream's handle if the caller already has it.  ``least``: what the call cannot do without; a
    capturing stream gets no more than that newly allocated."""
    return _workspaces.get(device_index, nbytes, stream_ptr(device_index) if stream is None else stream, least)
