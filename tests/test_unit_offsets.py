"""Byte offsets of an op's units, by the kernels' own arithmetic: boxes whose rows pass 4 GiB as well as small ones."""

import ctypes as C

import pytest
import torch

from etha_b200.ops import lib as L
from etha_b200.ops import local_copy
from etha_b200.ops.table import CopyTable, SliceRef

BIG = 2**31 + 8  # bf16 elements of a row: 4 GiB + 16 bytes


def _packed(shape, sstr, dstr, dtype):
    t = CopyTable(torch.device("cpu"))
    t.add(shape, [SliceRef(1 << 44, sstr, dtype)], [SliceRef(1 << 45, dstr, dtype)])
    return t._packed[0]


@pytest.mark.parametrize("shape,sstr,dstr,dtype,klass", [
    ((2, BIG), (BIG + 8, 1), (BIG, 1), torch.bfloat16, 0),  # rows of the fast kernel
    ((2, BIG // 2), (BIG // 2 + 4, 1), (BIG // 2 + 8, 1), torch.float32, 0),
    ((1, BIG), (BIG, 1), (BIG, 1), torch.bfloat16, 0),  # one run
    ((3, 2**28 + 8), (2**28 + 16, 1), (2**28 + 8, 1), torch.bfloat16, 0),
    ((2, 2, 2**28 + 8), (2**31, 2**29, 1), (2**31, 2**29 + 16, 1), torch.float32, 1),  # rows of the general kernel
    ((5, 64), (80, 1), (64, 1), torch.bfloat16, 0),
    ((2, 3, 64), (1000, 72, 1), (256, 64, 1), torch.float32, 1),
])
def test_units_lie_where_the_strides_say(shape, sstr, dstr, dtype, klass):
    cls, _, raw, *_ = _packed(shape, sstr, dstr, dtype)
    assert cls == klass
    numel = 1
    for n in shape:
        numel *= n
    per = 16 // dtype.itemsize  # elements of a unit
    row = shape[-1] // per
    units = {u for r in range(numel // shape[-1]) for k in (0, 1, 2**28 - 1, 2**28, 2**28 + 1, row // 2, row - 2, row - 1)
             if 0 <= k < row for u in [r * row + k]}
    so, do = C.c_int64(), C.c_int64()
    for unit in sorted(units):
        L.cuda_lib().etha_op_unit_offsets(raw, unit, C.byref(so), C.byref(do))
        e, src, dst = unit * per, 0, 0
        for n, s, d in zip(reversed(shape), reversed(sstr), reversed(dstr)):
            e, i = divmod(e, n)
            src, dst = src + i * s, dst + i * d
        assert (so.value, do.value) == (src * dtype.itemsize, dst * dtype.itemsize), unit


@pytest.mark.gpu
def test_rows_longer_than_4_gib_are_copied_whole():
    """13 GB on the device: one padded source row of 4 GiB + 64 bytes, read by both rows of the destination."""
    n = 2**32 + 64
    row = torch.empty(n, dtype=torch.uint8, device="cuda:0")
    row.view(torch.int32).copy_(torch.arange(n // 4, dtype=torch.int32, device="cuda:0"))
    dst = torch.zeros(2, n, dtype=torch.uint8, device="cuda:0")
    local_copy(row.expand(2, n), dst)
    torch.cuda.synchronize()
    for k in range(2):
        assert torch.equal(dst[k].view(torch.int64), row.view(torch.int64))
