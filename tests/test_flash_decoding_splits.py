"""The split counts of split-KV attention: which rule a call takes, and what the rules answer."""

import pytest
import torch

from machete_b200.kernels.attention import flash_decoding_schedule
from machete_b200.kernels.attention.flash_decoding import default_num_splits, layer_num_splits, splits_by_cost

BF = torch.bfloat16


@pytest.mark.parametrize("batch", [1, 2, 3, 7, 8, 37, 200])
@pytest.mark.parametrize("kv", [1, 63, 64, 300, 1931, 32768, 131072])
def test_splits_stay_in_range(batch, kv):
    assert 1 <= splits_by_cost(batch, 8, 1, kv, 148) <= max(1, min(64, kv // 64))


@pytest.mark.parametrize("batch,kv,by_cost,by_waves", [(8, 1931, 2, 9), (4, 1931, 4, 9), (8, 4096, 2, 9), (8, 32768, 9, 9)])
def test_the_measured_choices(batch, kv, by_cost, by_waves):
    assert splits_by_cost(batch, 8, 1, kv, 148) == by_cost
    assert default_num_splits(batch, 8, 1, kv, 148) == by_waves


def _splits(B, H, Hkv, D, kv, M=1, **kw):
    q, k = torch.empty(B, M, H, D, dtype=BF), torch.empty(B, kv, Hkv, D, dtype=BF)
    ops, _ = flash_decoding_schedule(q, k, k, torch.empty_like(q), kv_group_size=H // Hkv, **kw)
    return ops[0].static_dims["num_splits"]


def test_which_rule_a_call_takes():
    assert _splits(8, 32, 8, 64, 1931) == 2                            # head dim 64, a static length: by cost
    assert _splits(8, 32, 8, 64, 1931, dynamic_len=True) == 9          # the length follows the position
    assert _splits(8, 32, 8, 128, 1931) == 9
    assert _splits(8, 32, 8, 64, 1931, num_splits=5) == 5
    q, k = torch.empty(8, 1, 32, 64, dtype=BF), torch.empty(8, 1931, 8, 64, dtype=BF)
    assert layer_num_splits(q, k) == 9                                 # the layers of a model keep theirs


@pytest.mark.parametrize("H,Hkv,D,most", [(32, 4, 64, 32), (8, 2, 64, 32), (4, 2, 64, 64), (2, 2, 64, 64), (32, 2, 128, 64)])
def test_defaults_stay_within_one_trip_of_the_combine(H, Hkv, D, most):
    """128 lse values at a time: four rows of 32 splits at head dim 64, two of 64 at 128."""
    rows = min(H // Hkv, 256 // D)
    for kv in (3889, 12729, 32768):
        q, k = torch.empty(1, 1, H, D, dtype=BF), torch.empty(1, kv, Hkv, D, dtype=BF)
        for splits in (_splits(1, H, Hkv, D, kv), _splits(1, H, Hkv, D, kv, dynamic_len=True), layer_num_splits(q, k)):
            assert splits <= most and rows * splits <= 128
    assert _splits(1, H, Hkv, D, 32768, num_splits=100) == 100         # what the caller asks for stands
