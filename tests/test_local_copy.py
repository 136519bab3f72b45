"""`local_copy`: what it refuses and where it launches."""

import pytest
import torch

from etha_b200 import ops


class _Cuda:
    """A host tensor that says it is on a CUDA device."""

    def __init__(self, t, index=0):
        self._t, self.device, self.is_cuda = t, torch.device("cuda", index), True

    def __getattr__(self, name):
        return getattr(self._t, name)


class _Stream:
    cuda_stream = 77


class _Lib:
    """Stands in for the native library: records the calls, launches nothing."""

    def __init__(self, peers=True):
        self.calls, self.peers = [], peers

    def etha_run_spec(self, spec, stream):
        self.calls.append(("run", stream))
        return 0

    def etha_enable_peer_access(self, index):
        self.calls.append(("peer", index))
        return 0 if self.peers else -1

    def etha_last_error(self):
        return b"no peer access"


class _Guard:
    """`torch.cuda.device` / `current_device` without a GPU; device 0 is current."""

    now = 0

    def __init__(self, device):
        self.index = device if isinstance(device, int) else device.index

    def __enter__(self):
        self.before, _Guard.now = _Guard.now, self.index

    def __exit__(self, *exc):
        _Guard.now = self.before


@pytest.fixture
def lib(monkeypatch):
    fake = _Lib()
    monkeypatch.setattr(ops, "cuda_lib", lambda: fake)
    monkeypatch.setattr(ops._L, "cuda_lib", lambda: fake)
    monkeypatch.setattr(torch.cuda, "device", _Guard)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: _Guard.now)
    return fake


def test_a_pageable_host_source_is_refused(lib):
    src = torch.zeros(4, 8)
    with pytest.raises(ValueError, match="pinned"):
        ops.local_copy(src, _Cuda(torch.zeros(4, 8)), _Stream())
    assert not lib.calls
    ops.local_copy(torch.zeros(0, 8), _Cuda(torch.zeros(0, 8)), _Stream())  # nothing to read
    assert not lib.calls


def test_a_host_destination_is_refused(lib):
    with pytest.raises(ValueError, match="destination"):
        ops.local_copy(_Cuda(torch.zeros(8)), torch.zeros(8), _Stream())
    assert not lib.calls


def test_a_source_on_another_gpu_needs_peer_access(lib):
    src, dst = _Cuda(torch.zeros(8), 1), _Cuda(torch.zeros(8), 0)
    ops.local_copy(src, dst, _Stream())
    assert lib.calls == [("peer", 1), ("run", 77)]
    lib.calls, lib.peers = [], False
    with pytest.raises(ValueError, match="cuda:0 cannot read the memory of cuda:1"):
        ops.local_copy(src, dst, _Stream())
    assert lib.calls == [("peer", 1)]


@pytest.mark.gpu
def test_host_sources_on_the_gpu():
    dst = torch.zeros(33, 65, device="cuda:0")
    src = torch.randn(33, 65)
    with pytest.raises(ValueError, match="pinned"):
        ops.local_copy(src, dst)
    pinned = src.pin_memory()
    ops.local_copy(pinned, dst)
    assert torch.equal(dst.cpu(), src)
