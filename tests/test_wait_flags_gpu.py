"""Waits for more flags than the warp has lanes: one deadline for all, the first missing flag is named."""

import pytest
import torch

from etha_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,missing", [(70, (3, 35)), (70, (35, 67)), (300, (299,)), (300, (31, 63, 95, 127, 159, 191, 223, 255, 287))])
def test_missing_flags_share_a_deadline(n, missing):
    flags = torch.full((n,), 5, dtype=torch.int32, device=DEV)
    which = torch.arange(n, dtype=torch.int32, device=DEV)
    status = torch.zeros(2, dtype=torch.int32, device=DEV)
    ops.wait_flags(flags, which, 5, status, timeout_s=0.1)  # all set
    torch.cuda.synchronize()
    assert status.tolist() == [ops.STATUS_OK, -1]
    for i in missing:
        flags[i] = 4
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    begin.record()
    ops.wait_flags(flags, which, 5, status, timeout_s=0.2)
    end.record()
    torch.cuda.synchronize()
    assert status.tolist() == [ops.STATUS_TIMEOUT, missing[0]]
    assert 190 < begin.elapsed_time(end) < 300


@pytest.mark.parametrize("n", [0, 1, 32, 33, 257])
def test_flags_that_are_set_end_the_wait(n):
    flags = torch.full((n + 1,), -(2**31), dtype=torch.int32, device=DEV)  # one epoch after 2^31 - 1
    which = torch.arange(n, 0, -1, dtype=torch.int32, device=DEV)
    status = torch.full((2,), 7, dtype=torch.int32, device=DEV)
    ops.wait_flags(flags, which, 2**31 - 1, status, timeout_s=0.5)
    torch.cuda.synchronize()
    assert status.tolist() == [ops.STATUS_OK, -1]
