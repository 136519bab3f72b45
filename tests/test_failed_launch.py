"""A launch that reports a failure, or runs on a table that has reported one, publishes nothing and leaves its counter closed."""

import pytest
import torch

from etha_b200.ops import STATUS_BAD_OP, STATUS_TIMEOUT, CopyTable
from etha_b200.ops import lib as L

from test_table_pack import OpView

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _flag():
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    return flag, torch.tensor([flag.data_ptr()], dtype=torch.int64, device=DEV)


def _launch(t, addrs, epoch, **kw):
    t.launch(signals=addrs, epoch=epoch, **kw)
    torch.cuda.synchronize()


def _of_class(kernel):
    """(source, destination) views that one kernel class runs."""
    x = torch.randn(300, 515, device=DEV)
    y = torch.zeros(300, 515, device=DEV)
    if kernel == "fast" or kernel == "bulk":
        return x[:, :512].contiguous(), y[:, :512].contiguous()
    if kernel == "typed":
        return x[:, :512].contiguous(), y[:, :512].to(torch.bfloat16)
    if kernel == "ragged":
        return x, torch.zeros(300, 516, device=DEV)[:, 1:]
    if kernel == "transposing":
        return x, torch.zeros(515, 300, device=DEV).t()
    return x[:, ::2], y[:, ::2]


@pytest.mark.parametrize("kernel", ["fast", "bulk", "typed", "ragged", "transposing", "general"])
def test_a_table_with_a_failure_publishes_nothing(kernel):
    src, dst = _of_class(kernel)
    t = CopyTable(DEV)
    t.add_copy(src, dst)
    t.finalize()
    flag, addrs = _flag()
    _launch(t, addrs, 1, bulk=kernel == "bulk")
    assert flag.item() == 1 and t._sync.tolist() == [0, 0, 0, 0]
    for left in (0, 1):  # tiles that an abandoned launch left in the counter
        t._sync[0], t._sync[1] = left, STATUS_TIMEOUT
        dst.zero_()
        _launch(t, addrs, 2, bulk=kernel == "bulk")
        assert flag.item() == 1 and t.error_word() == STATUS_TIMEOUT
        assert torch.equal(dst, src.to(dst.dtype))
    t._sync.zero_()
    for epoch in (3, 4):
        _launch(t, addrs, epoch, bulk=kernel == "bulk")
        assert flag.item() == epoch and t._sync[0].item() == 0


def test_a_refused_op_keeps_the_flag_back():
    """An op whose dtype is not the instance's is reported and not run; the rest of the table is delivered."""
    pairs = [(torch.randn(n, device=DEV), torch.zeros(n, dtype=torch.bfloat16, device=DEV)) for n in (8 * 40000, 8 * 333)]
    t = CopyTable(DEV)
    for src, dst in pairs:
        t.add_copy(src, dst)
    t.finalize()
    (launches, _, n) = t._all.ldst
    assert n == 1 and launches[0].n_ops == 2 and launches[0].key < L.KEY_RAGGED
    at = launches[0].ops - t._buffer.data_ptr() + OpView.src_dtype.offset
    flag, addrs = _flag()
    _launch(t, addrs, 1)
    assert flag.item() == 1
    for _, dst in pairs:
        dst.zero_()
    t._buffer[at] = L.DT_F16
    _launch(t, addrs, 2)
    assert flag.item() == 1 and t.error_word() == STATUS_BAD_OP and t._sync[0].item() == 0
    assert not pairs[0][1].any() and torch.equal(pairs[1][1], pairs[1][0].to(torch.bfloat16))
