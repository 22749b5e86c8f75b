"""Prompt attention with three tiles a CTA (head dim 64): last CTAs of one, two and three tiles, tiles of one CTA that see
different numbers of KV tiles, one KV tile and less, and both forms' results bit for bit.

Tolerance: that of the suite (`assert_parity`: a few bf16 roundings of values of size one against an fp64 attention)."""

import ctypes as C

import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.attention import flash_prefill
from tests import test_gpu_launch_overlap as overlap
from tests.test_gpu_prefill_attention import _reference
from tests.util import assert_parity

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _form(B, H, Hkv, M, Nk, causal, sms=148):
    out = (C.c_int32 * 4)()
    assert N.lib().mk_flash_prefill_plan(B, H, Hkv, M, Nk, 64, int(causal), sms, out) == 0
    return list(out)


def _inputs(B, H, Hkv, M, Nk):
    g = torch.Generator(device="cuda").manual_seed(M + Nk)
    q = torch.randn(B, H, M, 64, generator=g, device="cuda").to(BF)
    k, v = (torch.randn(B, Hkv, Nk, 64, generator=g, device="cuda").to(BF) for _ in range(2))
    return q, k, v


# (row tiles mod 3: 0, 1, 2; without packed heads the tiles of a CTA are 128 queries, two KV tiles, apart)
@pytest.mark.parametrize("B,H,Hkv,M,Nk,causal", [(5, 8, 8, 1100, 3100, True), (5, 8, 8, 1153, 3153, True), (4, 10, 10, 1281, 3300, True),
                                                 (2, 32, 8, 777, 2000, True), (1, 32, 8, 1400, 1, False), (1, 32, 8, 1300, 64, False),
                                                 (1, 32, 8, 1200, 65, False), (1, 32, 8, 2600, 2900, True)])
def test_three_tiles_a_cta(B, H, Hkv, M, Nk, causal):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _form(B, H, Hkv, M, Nk, causal)[0] == 3
    q, k, v = _inputs(B, H, Hkv, M, Nk)
    o, lse = torch.full_like(q, 7.0), torch.zeros(B, H, M, device="cuda")
    flash_prefill(q, k, v, o, causal=causal, lse=lse, check_status=True)
    for b in range(B):
        want, want_lse = _reference(q[b:b + 1], k[b:b + 1], v[b:b + 1], causal)
        assert_parity(o[b:b + 1], want, f"sequence {b} of B={B} H={H}/{Hkv} M={M} N={Nk}")
        assert float((lse[b:b + 1].double() - want_lse).abs().max()) < 2e-3


def test_the_form_leaves_the_bits():
    # two sequences together take three tiles a CTA, each by itself one
    q, k, v = _inputs(2, 32, 8, 777, 3000)
    both, each = torch.zeros_like(q), torch.zeros_like(q)
    for _ in range(3):                       # (the warps of a tile run at their own pace)
        flash_prefill(q, k, v, both, causal=True, check_status=True)
        for b in range(2):
            flash_prefill(q[b:b + 1], k[b:b + 1], v[b:b + 1], each[b:b + 1], causal=True, check_status=True)
        assert torch.equal(both, each)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,M,Nk,causal", [(1, 200, 333, True), (1, 130, 77, False), (2, 777, 2000, True)])
@pytest.mark.parametrize("scale", [-0.125, 0.0, -0.0, 1e-40, -3.0])
def test_scales_of_either_sign_and_none(D, B, M, Nk, causal, scale):
    # masked scores leave the softmax whatever the sign; no scale is the mean over the visible tokens
    g = torch.Generator(device="cuda").manual_seed(M + D)
    q = torch.randn(B, 32, M, D, generator=g, device="cuda").to(BF)
    k, v = (torch.randn(B, 8, Nk, D, generator=g, device="cuda").to(BF) for _ in range(2))
    o, lse = torch.full_like(q, 7.0), torch.zeros(B, 32, M, device="cuda")
    flash_prefill(q, k, v, o, causal=causal, scale=scale, lse=lse, check_status=True)
    want, want_lse = _reference(q.double() * (scale * D ** 0.5), k, v, causal)
    assert_parity(o, want, f"scale {scale}")
    # (fp32 products of D terms of size 1, scaled: a few 2^-24 of the largest score, some 40 * 3)
    assert float((lse.double() - want_lse).abs().max()) < 2e-3


@pytest.mark.parametrize("B,M,Nk", [(2, 777, 2000), (5, 1100, 3100)])
@pytest.mark.parametrize("falling", [False, True])
def test_row_maxima_that_keep_growing_in_three_tiles(B, M, Nk, falling):
    # every KV tile raises the exponent reference of every row (or of every other query's, beside rows that keep theirs): O is
    # rescaled while the other tiles' products run.  Tolerance: as for the same values in the form of one tile
    H, Hkv = (32, 8) if B == 2 else (8, 8)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _form(B, H, Hkv, M, Nk, True)[0] == 3
    g = torch.Generator(device="cuda").manual_seed(M + falling)
    q = torch.ones(B, H, M, 64, device="cuda").to(BF)
    if falling:
        q[:, :, 1::2] = -1
    k = (torch.arange(Nk, device="cuda")[None, None, :, None] / 16 + torch.rand(B, Hkv, Nk, 64, generator=g, device="cuda")).to(BF)
    v = torch.randn(B, Hkv, Nk, 64, generator=g, device="cuda").to(BF)
    o = torch.full_like(q, 7.0)
    for _ in range(3):
        flash_prefill(q, k, v, o, causal=True, check_status=True)
        for b in range(B):
            assert_parity(o[b:b + 1], _reference(q[b:b + 1], k[b:b + 1], v[b:b + 1], True)[0], f"growing maxima, sequence {b}")


def test_three_tiles_a_cta_between_other_kernels():
    # all of an SM's tensor memory is taken and given back between kernels that start early
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert _form(1, overlap.HEADS, overlap.KV_HEADS, 8100, 8100, True)[0] == 3
    overlap.test_a_chain_of_kernels_sees_what_the_one_before_it_wrote(8100, 64)
