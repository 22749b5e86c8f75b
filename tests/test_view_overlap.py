"""Which views of one storage share values (CPU): against the sets of addresses, whatever the order of their axes."""

import random

import pytest
import torch

from machete_b200.megakernel import tensor_meta_overlaps
from machete_b200.megakernel.lowering import meta_of


def values(t):
    """Storage indices of a view's values."""
    return set(torch.arange(t.untyped_storage().nbytes() // 2).as_strided(t.shape, t.stride(), t.storage_offset()).reshape(-1).tolist())


def cut(rng, t):
    for axis in range(t.ndim):
        lo = rng.randrange(t.shape[axis])
        t = t.narrow(axis, lo, rng.randint(1, t.shape[axis] - lo))
    return t


@pytest.mark.parametrize("seed", range(8))
def test_slices_of_a_buffer_in_any_order_of_axes(seed):
    rng = random.Random(seed)
    for _ in range(60):
        shape = [rng.randint(1, 4) for _ in range(rng.randint(1, 4))]
        order = rng.sample(range(len(shape)), len(shape))
        whole = torch.zeros(shape, dtype=torch.bfloat16).permute(order)
        a, b = cut(rng, whole), cut(rng, whole)
        assert tensor_meta_overlaps(meta_of(a), meta_of(b)) == bool(values(a) & values(b)), (whole.shape, whole.stride(), a.shape, b.shape)


@pytest.mark.parametrize("seed", range(8))
def test_nothing_shared_is_missed_in_windows_that_overlap(seed):
    rng = random.Random(seed)
    for _ in range(60):
        ndim = rng.randint(1, 3)
        strides = tuple(rng.randint(1, 9) for _ in range(ndim))
        flat = torch.zeros(200, dtype=torch.bfloat16)
        a, b = (flat.as_strided([rng.randint(1, 4) for _ in range(ndim)], strides, rng.randint(0, 40)) for _ in range(2))
        if values(a) & values(b):
            assert tensor_meta_overlaps(meta_of(a), meta_of(b)), (a.shape, b.shape, strides, a.storage_offset(), b.storage_offset())


def test_heads_of_a_head_major_cache():
    cache = torch.zeros(3, 4, 128, 64, dtype=torch.bfloat16).transpose(1, 2)          # (B, T, H, D)
    window, heads = cache[:, :101], cache[:, :, 2:]
    assert tensor_meta_overlaps(meta_of(window), meta_of(heads))
    assert not tensor_meta_overlaps(meta_of(cache[:, :, :2]), meta_of(heads))
    assert not tensor_meta_overlaps(meta_of(cache[:, :100]), meta_of(cache[:, 100:]))
