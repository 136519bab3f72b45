"""Tile layout of a launch and the dynamic walk over it: every unit of every op is copied exactly where it belongs."""

import numpy as np
import pytest
import torch

from etha_b200.ops import lib as L
from etha_b200.ops.table import CopyTable, SliceRef

from test_table_pack import OpView

UNITS = [1, 31, 255, 256, 257, 511, 512, 1023, 1024, 1025, 2047, 2049, 40000]  # edges of tiles and trips, in 16-byte units


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("scale", [1, 7, 500])
def test_layout_covers_every_unit(kernel, scale):
    t = CopyTable(torch.device("cpu"))
    for i, n in enumerate(UNITS):
        t.add((n * scale * 16,), [SliceRef((i + 1) << 40, (1,), torch.uint8)], [SliceRef((i + 101) << 40, (1,), torch.uint8)])
    ops = np.frombuffer(b"".join(e[2] for e in t._packed), dtype=np.uint8).copy()
    before = [OpView.from_buffer_copy(e[2]) for e in t._packed]
    starts = np.zeros(len(before) + 1, dtype=np.uint32)
    lib = L.cuda_lib()
    total = lib.etha_layout_tiles(ops.ctypes.data, len(before), kernel, starts.ctypes.data)
    size = lib.etha_sizeof_op()
    assert starts[0] == 0 and starts[-1] == total
    for i, b in enumerate(before):
        op = OpView.from_buffer_copy(ops[i * size : (i + 1) * size].tobytes())
        tiles = int(starts[i + 1] - starts[i])
        assert 256 <= op.tile_units <= b.tile_units and op.total_units == b.total_units
        assert (tiles - 1) * op.tile_units < op.total_units <= tiles * op.tile_units


@pytest.mark.gpu
@pytest.mark.parametrize("bulk", [False, True])
@pytest.mark.parametrize("repeat", [1, 24])
def test_every_class_walks_all_tiles(bulk, repeat):
    """One table with all kernel classes, ops of every edge size; launched twice, with a flag that has to come last."""
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(3)
    t, pairs = CopyTable(dev), []
    for _ in range(repeat):
        for n in UNITS:
            raw = torch.randint(0, 255, (n * 16,), generator=g, device=dev, dtype=torch.uint8)
            f32 = torch.randn(n * 8, generator=g, device=dev)
            rows = torch.randn(n, 1024, generator=g, device=dev).to(torch.bfloat16) if n <= 1024 else None
            for src, dst in [(raw, torch.zeros_like(raw)), (f32, torch.zeros(n * 8, dtype=torch.bfloat16, device=dev)),
                             (f32[: n * 8 - 1], torch.zeros(n * 8 - 1, device=dev))]:
                pairs.append((src, dst))
            if rows is not None:
                pairs.append((rows[:, 256:640], torch.zeros(n, 384, dtype=torch.bfloat16, device=dev)))
    for src, dst in pairs:
        t.add_copy(src, dst)
    t.finalize()
    flags = torch.zeros(1, dtype=torch.int32, device=dev)
    addrs = torch.tensor([flags.data_ptr()], dtype=torch.int64, device=dev)
    for epoch in (1, 2):
        for _, dst in pairs:
            dst.zero_()
        t.launch(signals=addrs, epoch=epoch, bulk=bulk)
        torch.cuda.synchronize()
        assert t.error_word() == 0 and flags.item() == epoch
        assert all(torch.equal(dst, src.to(dst.dtype)) for src, dst in pairs)


@pytest.mark.gpu
def test_two_streams_share_a_table():
    """Launches of one table, without signals, that overlap on the GPU take their tiles from queues of their own."""
    dev = torch.device("cuda", 0)
    src = torch.arange(64 << 20, device=dev, dtype=torch.int32)
    dst = torch.zeros_like(src)
    t = CopyTable(dev)
    t.add_copy(src, dst)
    t.finalize()
    streams = [torch.cuda.Stream(dev) for _ in range(2)]
    marks = []
    torch.cuda.synchronize()
    for s in streams:
        t.launch(s)
        with torch.cuda.stream(s):
            marks.append((dst == src).all())  # what this stream sees after its own launch
    torch.cuda.synchronize()
    assert all(bool(m) for m in marks)


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n", [8, 100_003, 4_000_000])
def test_chained_launches_see_each_other(graph, n):
    """A kernel that is resident before its predecessor ends still reads what that one, and the ones before it, wrote."""
    dev = torch.device("cuda", 0)
    bufs = [torch.zeros(n + 1, dtype=torch.int32, device=dev)[i % 2 :][:n] for i in range(12)]  # aligned and not
    tables = []
    for src, dst in zip(bufs, bufs[1:]):
        t = CopyTable(dev)
        t.add_copy(src, dst)
        tables.append(t.finalize())
    stream = torch.cuda.Stream(dev)
    start = torch.zeros(1, dtype=torch.int32, device=dev)

    def chain():
        start.add_(1)
        bufs[0].copy_(start.expand(n))
        for t in tables:
            t.launch(stream)
        return bufs[-1] + 0  # what the next kernel in the stream sees

    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        out = chain()
        if graph:
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream):
                out = chain()
        for k in range(2, 12):
            if graph:
                g.replay()
            else:
                out = chain()
            stream.synchronize()
            assert bool((out == k).all()), k
