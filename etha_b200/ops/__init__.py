"""Native ops: sm_100a copy/convert/reduce kernels, flag kernels, table packer, IPC helpers."""

from __future__ import annotations

from ctypes import byref as _byref

import torch

from . import lib as _L
from .lib import STATUS_BAD_OP, STATUS_OK, STATUS_TIMEOUT, cuda_lib
from .table import LAUNCH_COUNT, CopyTable, SliceRef, dtype_code, make_spec

FLAG_LAUNCH_COUNT = [0]  # set_flags / wait_flags kernels launched in this process

__all__ = [
    "CopyTable",
    "SliceRef",
    "dtype_code",
    "cuda_lib",
    "local_copy",
    "set_flags",
    "wait_flags",
    "device_info",
    "STATUS_OK",
    "STATUS_TIMEOUT",
    "STATUS_BAD_OP",
]


def _handle(stream: torch.cuda.Stream | None, index: int) -> int:
    return torch._C._cuda_getCurrentRawStream(index) if stream is None else stream.cuda_stream


def _reachable(src: torch.Tensor, device: torch.device) -> None:
    """Raise unless kernels on `device` can read `src`, which is not there: its address goes into the launch as it is."""
    if src.is_cuda:
        with torch.cuda.device(device):
            if cuda_lib().etha_enable_peer_access(src.device.index):
                raise ValueError(f"{device} cannot read the memory of {src.device}: {_L.last_error()}")
    elif not src.is_pinned():
        raise ValueError(f"the source must be on a CUDA device or in pinned host memory, not on {src.device}")


def _after_current(stream: torch.cuda.Stream, index: int) -> int:
    """Handle of `stream`, made to wait for the current stream of device `index`, which may still be writing the source."""
    current = torch.cuda.current_stream(index)
    with torch.cuda.stream(stream):
        capturing = torch.cuda.is_current_stream_capturing()
    if capturing:
        with torch.cuda.stream(current):
            if not torch.cuda.is_current_stream_capturing():
                return stream.cuda_stream  # a graph cannot wait for work outside of it
    stream.wait_stream(current)
    return stream.cuda_stream


def local_copy(src: torch.Tensor, dst: torch.Tensor, stream: torch.cuda.Stream | None = None) -> None:
    """`dst[...] = src` (any strides, fp32/bf16/fp16 conversion) through the copy kernels.  `dst` is on a CUDA device, `src`
    on the same one, on a peer of it or in pinned host memory.  A copy on another `stream` than the device's current one
    comes after what the current stream holds at the call; whoever uses `dst` elsewhere, or frees either tensor, waits for it."""
    shape = tuple(src.shape)
    if shape != tuple(dst.shape):
        raise ValueError(f"shape mismatch {shape} vs {tuple(dst.shape)}")
    if len(shape) > 8:
        raise ValueError("at most 8 dims")
    if not dst.is_cuda:
        raise ValueError(f"the destination must be on a CUDA device, not on {dst.device}")
    # one op, launched with the op in the kernel's arguments: no table is built or uploaded
    spec = make_spec(shape, [SliceRef.of(src)], [SliceRef.of(dst)], (), (), 0, 0)
    if not src.numel():
        return
    index = dst.get_device()
    if src.get_device() != index:
        _reachable(src, dst.device)
    s = torch._C._cuda_getCurrentRawStream(index)
    if stream is not None and stream.cuda_stream != s:
        s = _after_current(stream, index)
    rc = cuda_lib().etha_run_spec(_byref(spec), index, s)
    if -100 < rc < 0:  # refused by the packer
        raise ValueError(f"cannot pack op ({rc}): {_L.last_error()}")
    _L.check(rc, "local copy")
    LAUNCH_COUNT[0] += 1


def set_flags(addresses: torch.Tensor, epoch: int, stream: torch.cuda.Stream | None = None) -> None:
    """Store `epoch` (release, system scope) to every uint32 flag whose address is in `addresses` (int64, device)."""
    index = addresses.get_device()
    rc = cuda_lib().etha_set_flags(addresses.data_ptr(), addresses.numel(), epoch & 0xFFFFFFFF, index, _handle(stream, index))
    _L.check(rc, "set_flags")
    FLAG_LAUNCH_COUNT[0] += 1


def wait_flags(
    flags: torch.Tensor,
    which: torch.Tensor,
    epoch: int,
    status: torch.Tensor,
    timeout_s: float = 2.0,
    stream: torch.cuda.Stream | None = None,
) -> None:
    """Enqueue a bounded wait until `flags[which[i]] >= epoch` for all i.

    `status` (int32[2], device or pinned-mapped) receives `[STATUS_OK | STATUS_TIMEOUT, index of the
    first missing flag]`.  The wait gives up after `timeout_s`; the context stays usable.
    """
    index = flags.get_device()
    rc = cuda_lib().etha_wait_flags(flags.data_ptr(), which.data_ptr(), which.numel(), epoch & 0xFFFFFFFF, int(timeout_s * 1e9),
                                    status.data_ptr(), index, _handle(stream, index))
    if rc:
        _L.check(rc, "wait_flags")
    FLAG_LAUNCH_COUNT[0] += 1


def device_info() -> dict:
    import ctypes as C

    sm, maj, mnr, mc = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    _L.check(cuda_lib().etha_device_info(C.byref(sm), C.byref(maj), C.byref(mnr), C.byref(mc)), "device_info")
    return {"sm_count": sm.value, "cc": (maj.value, mnr.value), "multicast": bool(mc.value)}
