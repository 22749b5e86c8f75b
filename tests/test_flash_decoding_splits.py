"""The split counts of split-KV attention at head dim 64."""

import math

import pytest

from machete_b200.kernels.attention.flash_decoding import default_num_splits, splits_by_cost


@pytest.mark.parametrize("batch", [1, 2, 3, 7, 8, 37, 200])
@pytest.mark.parametrize("kv", [1, 63, 64, 300, 1931, 32768, 131072])
def test_splits_stay_in_range_and_never_cost_more_waves_of_tokens(batch, kv):
    s, old = splits_by_cost(batch, 8, 1, kv, 148), default_num_splits(batch, 8, 1, kv, 148)
    assert 1 <= s <= max(1, min(64, kv // 64))

    def cost(n):
        return math.ceil(batch * 8 * n / 148) * (200 + -(-kv // n))

    assert cost(s) <= cost(old)
