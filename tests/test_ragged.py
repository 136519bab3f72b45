"""Ragged class: rows of any alignment, against the general kernel and plain PyTorch; chunk arithmetic on the CPU."""

import random

import pytest
import torch

from etha_b200.ops import CopyTable, SliceRef

from test_table_emulation import _fast_div
from test_table_pack import OpView

DEV = "cuda:0"


def _view(rows, cols, lead, dtype, seed):
    """[rows, cols] view whose rows start `lead` elements into wider rows of odd width."""
    g = torch.Generator().manual_seed(seed)
    width = cols + lead + 3 + (cols + lead) % 2
    bits = torch.randn(rows, width, generator=g) * 3
    return bits.to(dtype).to(DEV)[:, lead : lead + cols]


def _table(shape, srcs, dsts, sizes=(), ops=(), streaming=True):
    t = CopyTable(DEV)
    t.stream_typed = streaming
    t.add(shape, [SliceRef.of(s) for s in srcs], [SliceRef.of(d) for d in dsts], sizes, ops)
    return t


def _run(t):
    t.finalize().launch()
    torch.cuda.synchronize()
    assert t.error_word() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16, torch.bfloat16, torch.float32, torch.int64])
@pytest.mark.parametrize("rows,cols", [(1, 97), (3, 101), (37, 257), (513, 801)])
def test_bit_copies_at_every_offset(dtype, rows, cols):
    for lead_s in range(0, 17, 3):
        for lead_d in (0, 1, 2, 5, 7, 16):
            src = _view(rows, cols, lead_s, dtype, lead_s)
            dst = _view(rows, cols, lead_d, dtype, 100)
            whole = torch.as_strided(dst, (rows, dst.stride(0)), dst.stride(), dst.storage_offset() - lead_d)
            want = whole.clone()
            want[:, lead_d : lead_d + cols] = src
            t = _table((rows, cols), [src], [dst])
            assert t._packed[0][0] == 0 or t._packed[0][4] == 0x1000 or cols * src.element_size() < 48
            _run(t)
            assert torch.equal(whole, want), (lead_s, lead_d)  # neighbours of the rows included


@pytest.mark.gpu
@pytest.mark.parametrize("sdt,ddt", [(a, b) for a in (torch.float32, torch.bfloat16, torch.float16) for b in (torch.float32, torch.bfloat16, torch.float16)])
@pytest.mark.parametrize("sizes,opnames", [((), ()), ((2,), ("sum",)), ((3,), ("avg",)), ((8,), ("max",)), ((2, 3), ("sum", "max")), ((2, 2), ("avg", "avg"))])
def test_typed_rows_equal_the_general_kernel(sdt, ddt, sizes, opnames):
    if not sizes and sdt == ddt:
        pytest.skip("a same-dtype copy is a bit copy")
    n = 1
    for s in sizes:
        n *= s
    for rows, cols, lead_s, lead_d in [(1, 24, 0, 1), (5, 27, 1, 0), (67, 333, 3, 2), (40, 1024, 7, 5)]:
        srcs = [_view(rows, cols, lead_s, sdt, 10 + i) for i in range(n)]
        if not all(s.storage_offset() == srcs[0].storage_offset() for s in srcs):
            raise AssertionError
        outs = []
        for streaming in (True, False):
            dsts = [torch.full((rows, cols + lead_d + 4), 7.0, dtype=ddt, device=DEV) for _ in range(2)]
            t = _table((rows, cols), srcs, [d[:, lead_d : lead_d + cols] for d in dsts], sizes, opnames, streaming)
            assert (t._packed[0][4] >> 12 == 1) == streaming
            _run(t)
            assert torch.equal(dsts[0], dsts[1])
            outs.append(dsts[0])
        assert torch.equal(outs[0].view(torch.uint8), outs[1].view(torch.uint8))
        assert bool((outs[0][:, :lead_d] == 7).all()) and bool((outs[0][:, lead_d + cols :] == 7).all())


@pytest.mark.gpu
def test_strided_dims_and_fan_out():
    src = torch.randn(6, 9, 10, 56, device=DEV)[:, 1:8, ::2, 3:51]
    dst = torch.zeros(6, 11, 10, 61, device=DEV)
    dsts = [dst[:, 2:9, 1::2, 5:53], torch.zeros(6, 11, 10, 61, device=DEV)[:, 2:9, 1::2, 5:53]]
    t = _table(tuple(src.shape), [src], dsts)
    assert t._packed[0][4] == 0x1000
    _run(t)
    assert torch.equal(dsts[0], src) and torch.equal(dsts[1], src)
    mask = torch.zeros_like(dst, dtype=torch.bool)
    mask[:, 2:9, 1::2, 5:53] = True
    assert not dst[~mask].any()


@pytest.mark.gpu
def test_special_values_pass_unchanged():
    vals = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), 65504.0, -65504.0, 1e-8, 3e38], device=DEV).repeat(13)[:97]
    for ddt in (torch.bfloat16, torch.float16):
        src = vals.repeat(5, 1)[:, 1:90]
        dst = torch.zeros(5, 91, dtype=ddt, device=DEV)
        _run(_table((5, 89), [src], [dst[:, 2:]]))
        assert torch.equal(dst[:, 2:], src.to(ddt))
    a, b = vals.repeat(5, 1)[:, 1:90], torch.full((5, 97), float("-inf"), device=DEV)[:, 1:90]
    dst = torch.zeros(5, 91, device=DEV)
    _run(_table((5, 89), [a, b], [dst[:, 1:90]], (2,), ("max",)))
    assert torch.equal(dst[:, 1:90], torch.maximum(a, b))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("sizes,opnames", [((2,), ("sum",)), ((3,), ("avg",)), ((2,), ("max",)), ((3,), ("min",)), ((2,), ("product",)), ((2, 2), ("max", "sum"))])
def test_nan_and_infinity_through_collapses(dtype, sizes, opnames):
    """Every pair of special values meets in some column; NaN wins over everything, as in torch."""
    special = torch.tensor([float("nan"), float("inf"), float("-inf"), 0.0, -0.0, 1.5, torch.finfo(dtype).min, torch.finfo(dtype).max], device=DEV)
    n, cols = 1, 8 * 8 + 25
    for s in sizes:
        n *= s
    srcs = []
    for i in range(n):
        row = torch.full((cols,), 2.0, device=DEV)
        row[:64] = special.repeat_interleave(8) if i % 2 else special.repeat(8)
        srcs.append(row.to(dtype).repeat(3, 1 + 8 // n)[:, 1 : cols - 3])  # odd rows, not on a 16-byte boundary
    steps = {"sum": torch.add, "avg": torch.add, "max": torch.maximum, "min": torch.minimum, "product": torch.mul}

    def fold(values, name):
        acc = values[0]
        for v in values[1:]:
            acc = steps[name](acc, v)
        return acc / len(values) if name == "avg" else acc

    want = [s.float() for s in srcs]
    for size, name in zip(sizes, opnames):
        want = [fold(want[k : k + size], name) for k in range(0, len(want), size)]
    outs = []
    for streaming in (True, False):
        dst = torch.zeros(3, cols, dtype=dtype, device=DEV)
        t = _table(tuple(srcs[0].shape), srcs, [dst[:, 3 : cols - 1]], sizes, opnames, streaming)
        assert (t._packed[0][4] >> 12 == 1) == streaming
        _run(t)
        assert torch.equal(dst[:, 3 : cols - 1].isnan(), want[0].isnan())
        torch.testing.assert_close(dst[:, 3 : cols - 1], want[0].to(dtype), rtol=0, atol=0, equal_nan=True)
        outs.append(dst.view(torch.uint8))
    assert torch.equal(*outs)


@pytest.mark.parametrize("seed", range(40))
def test_chunks_cover_every_row_once(seed):
    """The packer's chunk description of randomly strided boxes, walked like the kernel: every element of every row lies in
    exactly one chunk, and whole chunks start on 16-byte boundaries of the destination."""
    rng = random.Random(seed)
    sdt, ddt = rng.choice([(torch.uint8,) * 2, (torch.bfloat16,) * 2, (torch.float32,) * 2, (torch.int64,) * 2,
                           (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float16, torch.bfloat16)])
    es, ed = sdt.itemsize, ddt.itemsize
    shape = [rng.randint(1, 5) for _ in range(rng.randint(0, 3))] + [rng.randint(48 // min(es, ed), 300)]
    strides = []
    for _ in range(2):  # nested, with gaps; some aligned, some reversed
        step, out = 1, []
        for n in reversed(shape):
            out.insert(0, step)
            step = step * n + rng.choice([0, 1, 3, 16])
            step = (step + 15) // 16 * 16 if rng.random() < 0.4 else step
        strides.append(tuple(-s if i < len(shape) - 1 and rng.random() < 0.1 else s for i, s in enumerate(out)))
    sptr, dptr = (1 << 30) + es * rng.randint(0, 16), (1 << 32) + ed * rng.randint(0, 16)
    t = CopyTable(torch.device("cpu"))
    t.add(shape, [SliceRef(sptr, strides[0], sdt)], [SliceRef(dptr, strides[1], ddt)])
    op = OpView.from_buffer_copy(t._packed[0][2])
    chunks, per_row, mul, shr, _ = op.pad
    if not chunks:
        assert op.ndim <= 1 and (op.unit_bytes_src == 16 if op.mode == 0 else op.unit_elems == 8)
        return
    raw = op.mode == 0
    size = op.unit_bytes_dst if raw else ed  # bytes of what is counted
    step, unit = (32, 1) if raw else (8, ed)
    length = op.inner_units * (op.unit_bytes_dst if raw else op.unit_elems)
    rows = op.total_units // op.inner_units
    assert chunks == rows * per_row and size >= 1
    seen = [0] * rows
    for chunk in range(chunks):
        row = _fast_div(chunk, mul, shr)
        assert row == chunk // per_row
        off, r = 0, row
        for d in reversed(range(op.ndim)):
            q = 0 if d == 0 else _fast_div(r, op.div_mul[d], op.div_shr[d])
            off += (r - q * op.extent[d]) * op.dst_stride[d]
            r = q
        head = (-(op.dst[0] + off) % 16) // ed
        lead = (op.dst[0] + off) % 16 if raw else (8 - head if head else 0)
        e0 = (chunk % per_row) * step - lead
        assert (op.dst[0] + off + e0 * unit) % 16 == 0
        lo, hi = max(e0, 0), min(e0 + step, length)
        if lo < hi:
            assert lo == seen[row], "chunks of a row follow each other"
            seen[row] = hi
    assert seen == [length] * rows
