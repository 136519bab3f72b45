"""Collapse instances (3 and 5 to 8 sources, two levels, mixed 16-bit types) give the general kernel's bits."""

import pytest
import torch

from etha_b200.ops import CopyTable, SliceRef

DEV = "cuda:0"
FLOATS = (torch.float32, torch.bfloat16, torch.float16)


@pytest.mark.gpu
@pytest.mark.parametrize("sdt,ddt", [(a, b) for a in FLOATS for b in FLOATS])
@pytest.mark.parametrize("sizes,opnames", [((2,), ("sum",)), ((3,), ("sum",)), ((4,), ("avg",)), ((5,), ("max",)), ((6,), ("product",)),
                                          ((7,), ("avg",)), ((8,), ("min",)), ((2, 2), ("sum", "avg")), ((2, 3), ("avg", "sum")),
                                          ((4, 2), ("sum", "max")), ((1, 3), ("sum", "sum")), ((2, 4), ("min", "avg"))])
def test_equal_to_the_general_kernel(sdt, ddt, sizes, opnames):
    n = 1
    for s in sizes:
        n *= s
    # one run shorter than a CTA's trip, a run with a remainder, rows of a matrix
    for rows, cols, width in [(1, 8, 8), (3, 1000, 1000), (129, 512, 520)]:
        wide = [torch.randn(rows, width, generator=torch.Generator().manual_seed(i)).to(sdt).to(DEV) * 1.7 for i in range(n)]
        wide[0].view(-1)[:4] = torch.tensor([float("nan"), float("inf"), float("-inf"), 0.0], device=DEV).to(sdt)
        srcs = [w[:, :cols] for w in wide]
        outs = []
        for streaming in (True, False):
            dsts = [torch.zeros(rows, cols, dtype=ddt, device=DEV) for _ in range(2)]
            t = CopyTable(DEV)
            t.stream_typed = streaming
            t.add((rows, cols), [SliceRef.of(s) for s in srcs], [SliceRef.of(d) for d in dsts], sizes, opnames)
            t.finalize().launch()
            torch.cuda.synchronize()
            assert t.error_word() == 0 and torch.equal(dsts[0].view(torch.uint8), dsts[1].view(torch.uint8))
            outs.append(dsts[0])
        assert torch.equal(outs[0].view(torch.uint8), outs[1].view(torch.uint8))
