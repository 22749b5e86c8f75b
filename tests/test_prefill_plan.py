"""How prompt attention is cut (CPU): three CTAs an SM only where the second round of two an SM would be the longer way."""

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


def test_bad_sizes_are_refused():
    out = (C.c_int32 * 4)()
    for args in ((1, 32, 8, 10, 9, 64, 1, 148), (1, 32, 7, 9, 9, 64, 1, 148), (1, 32, 8, 9, 9, 96, 1, 148), (1, 32, 8, 9, 9, 64, 1, 0)):
        assert N.lib().mk_flash_prefill_plan(*args, out) != 0
