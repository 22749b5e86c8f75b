"""Products at the edges of the row tiles: whole pairs of 64-value tiles, a single one behind them, pages that end in either."""

import pytest
import torch

from machete_b200.kernels.decode_matvec import MatvecSm100Op
from machete_b200.megakernel import Megakernel
from tests.util import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 8, 9, 16, 17, 24, 25, 32])
@pytest.mark.parametrize("k", [64, 128, 192, 1024, 1088, 1152])
def test_rows_and_tile_counts(dtype, rows, k):
    g = torch.Generator().manual_seed(rows * k)
    x = torch.randn(1, rows, k, generator=g).to(dtype)
    w = (torch.randn(200, k, generator=g) * 0.02).to(dtype)
    y = torch.full((1, rows, 200), float("nan"), dtype=dtype, device="cuda")
    Megakernel(MatvecSm100Op.schedule(a=x.cuda(), weight=w.cuda(), y=y)).compile().run()
    assert_parity(y[0], x[0].float() @ w.float().t(), f"{rows} x {k}")
