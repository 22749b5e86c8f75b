"""Prompt attention with the heads of a KV head packed into a tile's rows: groups that divide 128, groups of which only
a power of two does, and query counts at the edges of what a tile then holds; and both forms of the head-dim-64 kernel."""

import pytest
import torch

from machete_b200.kernels.attention import flash_prefill
from tests.test_gpu_prefill_attention import _reference
from tests.util import assert_parity

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("layout", ["bhmd", "bmhd"])
@pytest.mark.parametrize("H,Hkv,M,N", [(3, 1, 127, 300), (6, 1, 65, 65), (12, 2, 31, 1000), (16, 1, 8, 129), (16, 1, 9, 640),
                                       (32, 1, 5, 64), (64, 1, 3, 77), (128, 1, 2, 130), (8, 8, 129, 200), (256, 1, 2, 70)])
def test_packed_heads(D, layout, H, Hkv, M, N):
    g = torch.Generator(device="cuda").manual_seed(H + M)
    q = torch.randn(2, H, M, D, generator=g, device="cuda").to(BF)
    k, v = (torch.randn(2, Hkv, N, D, generator=g, device="cuda").to(BF) for _ in range(2))
    mem = (lambda t: t) if layout == "bhmd" else (lambda t: t.transpose(1, 2).contiguous())
    o = torch.full_like(mem(q), 7.0)
    lse = torch.zeros(2, H, M, device="cuda")
    flash_prefill(mem(q), mem(k), mem(v), o, causal=True, layout=layout, lse=lse, check_status=True)
    want, want_lse = _reference(q, k, v, True)
    assert_parity(o if layout == "bhmd" else o.transpose(1, 2), want, f"H={H}/{Hkv} M={M} N={N} D={D}")
    assert float((lse.double() - want_lse).abs().max()) < 2e-3


# 148 SMs: 296 tiles of 32 queries x 4 heads are two each, 444 three; which form a count takes goes by its KV tiles
@pytest.mark.parametrize("batch,M,N", [(1, 1184, 1184), (1, 1185, 1200), (2, 700, 1000), (2, 864, 900), (2, 897, 900)])
def test_tile_counts_at_the_edges_of_the_two_forms(batch, M, N):
    g = torch.Generator(device="cuda").manual_seed(M)
    q = torch.randn(batch, 32, M, 64, generator=g, device="cuda").to(BF)
    k, v = (torch.randn(batch, 8, N, 64, generator=g, device="cuda").to(BF) for _ in range(2))
    o = torch.zeros_like(q)
    flash_prefill(q, k, v, o, causal=True, check_status=True)
    assert_parity(o, _reference(q, k, v, True)[0], f"B={batch} M={M} N={N}")


@pytest.mark.parametrize("D,M", [(64, 70), (64, 1400), (128, 70)])
def test_row_maxima_that_keep_growing(D, M):
    # every tile raises the exponent reference of every row: the rescaling of O in its turn
    g = torch.Generator(device="cuda").manual_seed(D)
    q = torch.ones(1, 32, M, D, device="cuda").to(BF)
    k = (torch.arange(M + 600, device="cuda")[None, None, :, None] / 16 + torch.rand(1, 8, M + 600, D, generator=g, device="cuda")).to(BF)
    v = torch.randn(1, 8, M + 600, D, generator=g, device="cuda").to(BF)
    o = torch.zeros_like(q)
    flash_prefill(q, k, v, o, causal=True, check_status=True)
    assert_parity(o, _reference(q, k, v, True)[0], f"growing maxima D={D}")


# two tiles' boundaries at the edges of a 32-query block, prefixes that are multiples of 32 and not; the last of 400 tiles
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("batch,H,Hkv,M,N", [(1, 8, 2, 100, 100), (1, 8, 2, 97, 360), (2, 32, 8, 777, 1000), (1, 6, 1, 65, 80),
                                             (1, 64, 1, 40, 99), (1, 16, 2, 33, 1055)])
def test_the_grouping_of_heads_leaves_the_bits(D, batch, H, Hkv, M, N):
    g = torch.Generator(device="cuda").manual_seed(M * N)
    q = torch.randn(batch, H, M, D, generator=g, device="cuda").to(BF)
    k, v = (torch.randn(batch, Hkv, N, D, generator=g, device="cuda").to(BF) for _ in range(2))
    packed, single = torch.zeros_like(q), torch.zeros_like(q)
    flash_prefill(q, k, v, packed, causal=True, check_status=True)
    each = (t.repeat_interleave(H // Hkv, dim=1).contiguous() for t in (k, v))      # a KV head of its own for every head
    flash_prefill(q, *each, single, causal=True, check_status=True)
    assert torch.equal(packed, single)
