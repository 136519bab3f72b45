"""`local_copy`: what it refuses, which device the launches go to, what they come after; every kernel class through it."""

from contextlib import nullcontext
from types import SimpleNamespace

import pytest
import torch

from etha_b200 import ops
from etha_b200.ops.table import _Blob


class _Cuda:
    """A host tensor that says it is on a CUDA device."""

    def __init__(self, t, index=0):
        self._t, self.device, self.is_cuda = t, torch.device("cuda", index), True

    def get_device(self):
        return self.device.index

    def __getattr__(self, name):
        return getattr(self._t, name)


class _Stream:
    cuda_stream = 77


class _Lib:
    """Stands in for the native library: records the calls, launches nothing."""

    def __init__(self, peers=True):
        self.calls, self.peers = [], peers

    def etha_run_spec(self, spec, device, stream):
        self.calls.append(("run", stream, device))
        return 0

    def etha_set_flags(self, addresses, n, epoch, device, stream):
        self.calls.append(("set", stream, device))
        return 0

    def etha_wait_flags(self, flags, which, n, epoch, timeout, status, device, stream):
        self.calls.append(("wait", stream, device))
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
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 77)
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
    assert lib.calls == [("peer", 1), ("run", 77, 0)]
    lib.calls, lib.peers = [], False
    with pytest.raises(ValueError, match="cuda:0 cannot read the memory of cuda:1"):
        ops.local_copy(src, dst, _Stream())
    assert lib.calls == [("peer", 1)]


@pytest.mark.parametrize("index", [0, 1])
def test_launches_go_to_the_device_of_their_memory(lib, index):
    """Whatever device is current: a default stream has the same handle on all of them."""
    x = _Cuda(torch.zeros(8), index)
    ops.local_copy(x, _Cuda(torch.zeros(8), index), _Stream())
    ops.set_flags(x, 1, _Stream())
    ops.wait_flags(x, x, 1, x, 1.0, _Stream())
    assert lib.calls == [(name, 77, index) for name in ("run", "set", "wait")]


@pytest.mark.parametrize("device,index", [("cuda:0", 0), ("cuda:1", 1), ("cuda", -1)])
def test_a_table_names_its_device_in_every_launch(device, index):
    t = ops.CopyTable(torch.device("cpu"))  # packed and laid out on the host
    t.device = torch.device(device)
    for n, dtype in [(64, torch.float32), (16, torch.bfloat16), (7, torch.float32)]:
        t.add((n,), [ops.SliceRef(1 << 30, (1,), torch.float32)], [ops.SliceRef(1 << 32, (1,), dtype)])
    ks = t._lay_out(t._packed, _Blob())
    assert len(ks.ldst) == 3 and len(ks.bulk) == 3
    assert {one.device for one in ks.ldst + ks.bulk} == {index}


@pytest.mark.gpu
def test_an_unknown_device_is_an_error_and_the_current_one_stays():
    x = torch.zeros(8, dtype=torch.int64, device="cuda:0")
    lib, before = ops.cuda_lib(), torch.cuda.current_device()
    assert lib.etha_set_flags(x.data_ptr(), 0, 1, torch.cuda.device_count(), 0) < 0
    assert torch.cuda.current_device() == before
    assert lib.etha_set_flags(x.data_ptr(), 0, 1, before, 0) == 0 and lib.etha_set_flags(x.data_ptr(), 0, 1, -1, 0) == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("handle", [77, 78])
def test_a_copy_on_another_stream_is_ordered(lib, monkeypatch, handle):
    current, waits = object(), []
    stream = SimpleNamespace(cuda_stream=handle, wait_stream=lambda other: waits.append((other, len(lib.calls))))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda index: current)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: nullcontext())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    ops.local_copy(_Cuda(torch.zeros(8)), _Cuda(torch.zeros(8)), stream)
    assert waits == ([] if handle == 77 else [(current, 0)])  # before the launch
    assert lib.calls == [("run", handle, 0)]


@pytest.mark.gpu
def test_another_stream_waits_for_the_current_one():
    """The source is still being written on the current stream when the copy is put on a side stream."""
    src = torch.zeros(1 << 20, dtype=torch.int32, device="cuda:0")
    dst = torch.zeros_like(src)
    side = torch.cuda.Stream("cuda:0")
    torch.cuda.synchronize()
    for k in range(1, 4):
        torch.cuda._sleep(20_000_000)  # about 10 ms
        src.fill_(k)
        ops.local_copy(src, dst, side)
        side.synchronize()
        assert bool((dst == k).all())
    torch.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("forked", [False, True])
def test_other_streams_under_capture(forked):
    """Into a capturing stream that is not current, and from a capture into a stream forked off it."""
    src = torch.arange(1000, dtype=torch.float32, device="cuda:0")
    dst = torch.zeros_like(src)
    one, two = torch.cuda.Stream("cuda:0"), torch.cuda.Stream("cuda:0")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(one):
        graph.capture_begin()
        if forked:
            ops.local_copy(src, dst, two)
            one.wait_stream(two)
        else:
            with torch.cuda.stream(two):
                ops.local_copy(src, dst, one)
        graph.capture_end()
    assert not dst.any()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(dst, src)


VIEWS = {  # kernel class -> (source, destination) shaped views of one buffer each
    "fast run": lambda x, y: (x[:64].view(-1), y[:64].view(-1)),
    "fast rows": lambda x, y: (x[:, 8:264], y[:, 16:272]),
    "one element": lambda x, y: (x[3, 3:4], y[5, 7:8]),
    "no element": lambda x, y: (x[:0], y[:0]),
    "no dimension": lambda x, y: (x[2, 2], y[3, 3]),
    "ragged": lambda x, y: (x[:, 1:258], y[:, 3:260]),
    "ragged, two strided dims": lambda x, y: (x.view(16, 8, 272)[:, 1:7:2, 5:133], y.view(16, 8, 272)[:, ::3, 3:131]),
    "transposing": lambda x, y: (x[:, :128], y[:, :128].t()),
    "transposing, unaligned": lambda x, y: (x[1:100, 3:80], y[2:79, 5:104].t()),
    "short rows": lambda x, y: (x[:, 1:4], y[:, 2:5]),
    "element by element": lambda x, y: (x[:, ::2], y[:, 1::2]),
    "broadcast source": lambda x, y: (x[:1].expand(128, 272), y),
}


@pytest.mark.gpu
@pytest.mark.parametrize("view", VIEWS)
@pytest.mark.parametrize("sdt,ddt", [(torch.bfloat16,) * 2, (torch.float32,) * 2, (torch.uint8,) * 2, (torch.float32, torch.bfloat16),
                                     (torch.bfloat16, torch.float32), (torch.float16, torch.bfloat16)])
def test_every_class_launched_alone(view, sdt, ddt):
    x = torch.randint(-99, 99, (128, 272), device="cuda:0").to(sdt)
    y = torch.randint(0, 9, (128, 272), device="cuda:0").to(ddt)
    want = y.clone()
    src, dst = VIEWS[view](x, y)
    VIEWS[view](x, want)[1].copy_(src)
    ops.local_copy(src, dst)
    assert torch.equal(y, want)  # the rest of the destination included


@pytest.mark.gpu
def test_host_sources_on_the_gpu():
    dst = torch.zeros(33, 65, device="cuda:0")
    src = torch.randn(33, 65)
    with pytest.raises(ValueError, match="pinned"):
        ops.local_copy(src, dst)
    pinned = src.pin_memory()
    ops.local_copy(pinned, dst)
    assert torch.equal(dst.cpu(), src)
