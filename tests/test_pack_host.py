"""Which blocks the one-launch pack takes; the others go through one copy per block."""
import pytest
import torch

from dpnegf_b200 import rgf_plan

CPU = torch.device("cpu")


def _at(offset, rows, cols):
    """A complex128 [rows, cols] tensor whose data starts ``offset`` bytes behind a 16-byte boundary."""
    raw = bytearray(16 * rows * cols + 32)
    base = torch.frombuffer(raw, dtype=torch.uint8).data_ptr()
    t = torch.frombuffer(raw, dtype=torch.complex128, count=rows * cols, offset=(-base) % 16 + offset)
    assert t.data_ptr() % 16 == offset
    return t.view(rows, cols)


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 5), (32, 32)])
def test_only_aligned_blocks_are_packed(rows, cols):
    good, bad = _at(0, rows, cols), _at(8, rows, cols)
    assert rgf_plan._packable([(0, good), (rows * cols, good.mT)], CPU)
    assert not rgf_plan._packable([(0, good), (rows * cols, bad)], CPU)
    assert not rgf_plan._packable([(0, bad.mT)], CPU)


def test_other_blocks_are_not_packed():
    t = _at(0, 4, 4)
    assert not rgf_plan._packable([], CPU)
    assert not rgf_plan._packable([(0, t.to(torch.complex64))], CPU)
    assert not rgf_plan._packable([(0, t.expand(2, 4, 4))], CPU)
    assert not rgf_plan._packable([(0, t[:0])], CPU)
    assert not rgf_plan._packable([(0, torch._neg_view(t))], CPU)
    assert not rgf_plan._packable([(0, t)], torch.device("meta"))


def test_tensors_of_a_function_transform_are_not_packed():
    """Inside torch.func.grad and jvp a tensor has no address; the copy path takes it."""
    seen = []

    def f(x):
        seen.append(rgf_plan._packable([(0, x)], CPU))
        return x.abs().sum()

    t = torch.ones(2, 2, dtype=torch.complex128)
    torch.func.grad(f)(t)
    torch.func.jvp(f, (t,), (t,))
    assert seen == [False, False]
