"""Transposing class: which boxes it takes (CPU) and what it writes, against plain PyTorch and the general kernel."""

import pytest
import torch

from etha_b200.ops import CopyTable, SliceRef

from test_table_pack import OpView

DEV = "cuda:0"


def _key(t):
    return t._packed[0][4] >> 12


@pytest.mark.parametrize("shape,sstr,dstr,taken", [
    ((96, 160), (1, 96), (160, 1), True),
    ((8, 8), (1, 8), (8, 1), True),
    ((7, 160), (1, 7), (160, 1), False),  # too narrow
    ((96, 160), (2, 192), (160, 1), False),  # no unit stride in the source
    ((96, 160), (160, 1), (160, 1), False),  # one run
    ((3, 96, 160), (96 * 160, 1, 96), (160, 480, 1), True),
    ((96, 3, 160), (1, 96 * 160, 96), (480, 160, 1), True),
])
def test_rule(shape, sstr, dstr, taken):
    for sdt, ddt in [(torch.bfloat16,) * 2, (torch.float32,) * 2, (torch.float32, torch.float16), (torch.int8,) * 2]:
        t = CopyTable(torch.device("cpu"))
        t.add(shape, [SliceRef(1 << 20, sstr, sdt)], [SliceRef(1 << 30, dstr, ddt)])
        assert (_key(t) == 3) == (taken and sdt != torch.int8)
        if _key(t) == 3:
            op = OpView.from_buffer_copy(t._packed[0][2])
            blocks = op.pad[0]
            flags, a, b = op.pad[4] & 0xFF, op.pad[4] >> 8 & 0xFF, op.pad[4] >> 16 & 0xFF
            assert flags & 1 and op.dst_stride[a] == ddt.itemsize and op.src_stride[b] == sdt.itemsize and a != b
            kb = 256 // sdt.itemsize
            want = -(-op.extent[a] // 64) * -(-op.extent[b] // kb)
            for d in range(op.ndim):
                want *= 1 if d in (a, b) else op.extent[d]
            assert blocks == want


def _run(src, dsts, streaming=True):
    t = CopyTable(DEV)
    t.stream_typed = streaming
    t.add(tuple(src.shape), [SliceRef.of(src)], [SliceRef.of(d) for d in dsts])
    assert (_key(t) == 3) == streaming
    t.finalize().launch()
    torch.cuda.synchronize()
    assert t.error_word() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("sdt,ddt", [(torch.bfloat16,) * 2, (torch.int32,) * 2, (torch.float32, torch.bfloat16), (torch.float32, torch.float16),
                                     (torch.bfloat16, torch.float32), (torch.float16, torch.bfloat16), (torch.float16, torch.float32)])
@pytest.mark.parametrize("m,n", [(8, 8), (64, 128), (65, 129), (63, 127), (200, 72), (333, 257)])
@pytest.mark.parametrize("lead_s,lead_d", [(0, 0), (8, 0), (0, 1), (3, 8), (5, 7)])
def test_transposed_matrix(sdt, ddt, m, n, lead_s, lead_d):
    g = torch.Generator().manual_seed(m * n)
    pad = 16 if (lead_s % 8 == 0 and lead_d % 8 == 0) else 1  # widths that keep or break the alignment of the rows
    wide = (torch.randn(m, (n + 7) // 8 * 8 + lead_s + pad, generator=g) * 100).to(sdt).to(DEV)
    src = wide[:, lead_s : lead_s + n].t()  # [n, m], unit stride along n
    back = torch.full((n, (m + 7) // 8 * 8 + lead_d + pad), 3, dtype=ddt, device=DEV)
    want = back.clone()
    want[:, lead_d : lead_d + m] = src.to(ddt)
    other = back.clone()
    _run(src, [back[:, lead_d : lead_d + m], other[:, lead_d : lead_d + m]])
    assert torch.equal(back, want) and torch.equal(other, want)
    slow = torch.full_like(back, 3)
    _run(src, [slow[:, lead_d : lead_d + m]], streaming=False)
    assert torch.equal(slow.view(torch.uint8), back.view(torch.uint8))


@pytest.mark.gpu
def test_batched_and_permuted():
    x = torch.randn(5, 72, 3, 136, device=DEV)
    for perm in [(3, 1, 0, 2), (0, 3, 2, 1), (3, 0, 2, 1), (1, 2, 3, 0)]:
        src = x.permute(perm)
        dst = torch.zeros(src.shape, device=DEV)
        t = CopyTable(DEV)
        t.add_copy(src, dst)
        t.finalize().launch()
        torch.cuda.synchronize()
        assert t.error_word() == 0 and torch.equal(dst, src)
