"""How prompt attention is cut (CPU): three tiles a CTA only where the busiest SM then has less to do."""

import ctypes as C

import pytest

from machete_b200 import _native as N


def plan(B, M, Nk, D=64, causal=True, H=32, Hkv=8, sms=148):
    out = (C.c_int32 * 4)()
    assert N.lib().mk_flash_prefill_plan(B, H, Hkv, M, Nk, D, int(causal), sms, out) == 0
    return list(out)


@pytest.mark.parametrize("B,M,Nk", [(1, 1185, 1185), (1, 1408, 1408), (1, 1760, 1760), (2, 593, 593), (2, 864, 864), (1, 1400, 2000),
                                    (1, 1400, 3000), (1, 1200, 3800), (2, 777, 1000)])
def test_short_tiles_fill_the_second_round(B, M, Nk):
    ctas, pack, rows, tiles = plan(B, M, Nk)
    assert 296 < tiles <= 444 and ctas == 2 and pack == 4 and rows == -(-M // 32)


@pytest.mark.parametrize("B,M,Nk,causal", [(2, 777, 3000, True), (2, 777, 2000, True), (1, 1400, 4000, True), (1, 1700, 4300, True),
                                           (1, 1300, 1300, False), (1, 1760, 4096, False), (1, 1400, 500, False)])
def test_long_tiles_all_at_once(B, M, Nk, causal):
    assert plan(B, M, Nk, causal=causal)[0] == 3


def test_edges_of_the_window():
    # 8 tiles a row of tiles: 37 rows fill two CTAs an SM, 55 are the last below three
    for M, ctas in ((1184, 2), (1185, 3), (1760, 3), (1761, 2)):
        assert plan(1, M, 4096, causal=False)[0] == ctas, M
    assert plan(1, 1300, 1300, D=128, causal=False)[0] == 2      # one form only
    assert plan(1, 1, 1)[0] == 2 and plan(65535, 1, 1)[3] == 65535 * 8
    assert plan(1, 1300, 1300, causal=False, H=8, Hkv=8)[1:] == [1, 11, 88]


@pytest.mark.parametrize("B,M,Nk,causal,form", [(1, 2048, 2048, True, 2), (1, 2600, 2600, True, 2), (1, 4096, 4096, True, 3), (1, 1900, 1900, False, 2),
                                                (1, 3000, 3000, False, 3), (2, 4096, 4096, True, 3)])
def test_several_rounds(B, M, Nk, causal, form):
    assert plan(B, M, Nk, causal=causal)[0] == form and plan(B, M, Nk, causal=causal)[3] > 444


def test_sequences_together_and_by_themselves():
    # what tests/test_gpu_prefill_forms.py compares bit for bit
    assert plan(2, 777, 3000)[0] == 3 and plan(1, 777, 3000)[0] == 2


def _busiest(B, M, Nk, causal, group, slots):
    """KV tiles of the busiest of five slots, every CTA dealt out there and back, the longest first."""
    rows, per_row = -(-M // 32), 8 * B
    n = per_row * -(-rows // group)

    def kv(rank):
        end = (rows - rank // per_row * group) * 32
        return -(-(min(Nk, Nk - M + end) if causal else Nk) // 64)

    def slot_sum(slot):
        ranks = (r * slots + (slots - 1 - slot if r & 1 else slot) for r in range(-(-n // slots)))
        return sum(kv(x) for x in ranks if x < n)
    return max(slot_sum(q * (slots - 1) // 4) for q in range(5))


# 60 to 4000 rounds; short prompts of which each has one CTA of three tiles or two, filled or not
@pytest.mark.parametrize("B,M,Nk,causal", [(b, m, n, c) for c in (True, False) for b, m, n in (
    (17, 4096, 4096), (19, 4096, 4096), (24, 4096, 4096), (32, 4096, 4096), (100, 4096, 4096), (1, 131072, 131072), (5000, 32, 900),
    (60000, 64, 100), (9000, 96, 96), (9000, 128, 128), (30000, 170, 400), (3000, 333, 1000))])
def test_many_rounds_are_looked_at_in_full(B, M, Nk, causal):
    one, three = _busiest(B, M, Nk, causal, 1, 296), _busiest(B, M, Nk, causal, 3, 148)
    assert plan(B, M, Nk, causal=causal)[0] == (3 if 5 * three < 4 * one else 2), (one, three)


def test_bad_sizes_are_refused():
    out = (C.c_int32 * 4)()
    for args in ((1, 32, 8, 10, 9, 64, 1, 148), (1, 32, 7, 9, 9, 64, 1, 148), (1, 32, 8, 9, 9, 96, 1, 148), (1, 32, 8, 9, 9, 64, 1, 0)):
        assert N.lib().mk_flash_prefill_plan(*args, out) != 0
