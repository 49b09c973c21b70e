"""What the attention bindings hand to the kernels: rows on 16 bytes, copied only where they are not."""
import pytest
import torch

from flextrain_b200.ops.attention_cuda import _rows, _strided_ok


def _at(shift, *shape):
    """A contiguous bf16 tensor that starts ``shift`` elements past a 16-byte boundary."""
    n = torch.Size(shape).numel()
    buf = torch.arange(n + 16, dtype=torch.float32).to(torch.bfloat16)
    lead = (-buf.data_ptr() // 2) % 8
    return buf[lead + shift:lead + shift + n].view(shape)


@pytest.mark.parametrize("shift", [1, 2, 4, 7])
@pytest.mark.parametrize("T", [1, 5])
def test_a_contiguous_tensor_off_the_grid_is_copied(shift, T):
    t = _at(shift, T, 2, 64)
    assert t.is_contiguous() and not _strided_ok(t)
    r = _rows(t)
    assert _strided_ok(r) and torch.equal(r, t)


def test_tensors_on_the_grid_are_passed_on():
    t = _at(0, 5, 2, 64)
    assert _rows(t) is t
    view = _at(0, 5, 4, 64)[:, 1:3]                 # heads of a wider projection
    assert _rows(view) is view


def test_strides_over_one_row_do_not_count():
    t = torch.as_strided(_at(0, 2, 64).view(-1), (1, 2, 64), (3, 64, 1))
    assert t.is_contiguous() and not _strided_ok(t)
    assert _strided_ok(_rows(t)) and torch.equal(_rows(t), t)


def test_transposed_heads_become_rows():
    t = _at(0, 2, 5, 64).transpose(0, 1)
    assert _strided_ok(_rows(t)) and torch.equal(_rows(t), t)
