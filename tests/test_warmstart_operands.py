"""Which operands the weight gradient's product takes as they lie, and the transposed
copies of the others -- host only."""

import pytest
import torch

torch_bf16 = torch.bfloat16


def matrix(rows, cols, stride, start=0):
    flat = torch.arange(start + rows * stride + 64, dtype=torch.float32).to(torch_bf16)
    base = (-flat.data_ptr() // 2) % 8 + start  # elements from a 16-byte boundary
    return flat.as_strided((rows, cols), (stride, 1), base)


@pytest.mark.parametrize("rows,cols,stride,start,taken", [
    (16, 24, 24, 0, True), (16, 24, 32, 0, True), (16, 24, 32, 8, True), (16, 20, 24, 0, True),
    (16, 24, 24, 3, False),   # off 16 bytes
    (16, 9, 9, 0, False),     # rows off 16 bytes
    (16, 1, 1, 0, False),     # a column
    (1, 24, 8, 0, False),     # one row, whose stride says nothing
    (1, 24, 0, 0, False)])
def test_operands_as_they_lie(rows, cols, stride, start, taken):
    from dgc_b200.warmstart import _as_tensor_maps_take

    assert _as_tensor_maps_take(matrix(rows, cols, stride, start)) == taken


@pytest.mark.parametrize("rows,cols", [(16, 1), (1, 16), (5, 3), (8, 8)])
def test_transposed_copies_are_rows(rows, cols):
    from dgc_b200.warmstart import _padded_t, _round8

    x = matrix(rows, cols, cols)
    for wide in {_round8(rows), rows}:
        t = _padded_t(x, wide)
        assert t.shape == (cols, wide) and t.stride() == (wide, 1)
        assert t.data_ptr() != x.data_ptr()
        assert torch.equal(t[:, :rows], x.t()) and not t[:, rows:].any()
