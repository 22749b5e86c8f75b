"""One row has no row stride: whatever its tensor says, gemm_sm100 passes the row's own length."""

import pytest
import torch

from machete_b200.kernels.gemm.gemm_sm100 import _rows

K = 256


@pytest.mark.parametrize("make", [
    lambda: torch.zeros(K, 1).t(),                            # stride 1
    lambda: torch.zeros(K).as_strided((1, K), (0, 1)),        # stride 0
    lambda: torch.zeros(5, K + 3)[2:3, :K],                   # a stride that is no multiple of 8
    lambda: torch.zeros(1, K),
    lambda: torch.zeros(1, 1, K),
    lambda: torch.zeros(4, 3, K + 3)[1:2, 1:2, :K],
    lambda: torch.zeros(K),
])
def test_one_row(make):
    t = make()
    assert _rows(t, K) == (1, K) == (t.view(-1, K).shape[0], t.view(-1, K).stride(0))


def test_several_rows_keep_their_stride():
    assert _rows(torch.zeros(5, K + 8)[:, :K], K) == (5, K + 8)
    assert _rows(torch.zeros(2, 3, K), K) == (6, K)
    with pytest.raises(RuntimeError):
        _rows(torch.zeros(2, 3, K + 8)[:, :2, :K], K)         # rows that are not equally spaced
