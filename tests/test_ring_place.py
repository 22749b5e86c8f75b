"""Where a chain's matvec launch keeps a CTA's pages (CPU): slot and lap of every page, as the kernels' consumers work them out, are
those of a loader that steps from slot to slot, also for weights of many more pages than a ring has slots."""

import ctypes as C

import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.gemm import GemmOp
from machete_b200.megakernel import Megakernel, MegakernelConfig


def place(stages, page):
    out = (C.c_int32 * 2)()
    assert N.lib().mk_ring_place(stages, page, out) == 0
    return out[0], out[1]


@pytest.mark.parametrize("stages", range(1, 13))
def test_slot_and_lap(stages):
    # (a 32-bit product with a shift of 22 ends at 1024 pages a slot)
    pages = {0, 1, stages - 1, stages, stages + 1, (1 << 26) - 1}
    for k in (1, 512, 1023, 1024, 1025, 2048, 4096, 1 << 20, (1 << 26) // stages - 1):
        pages |= {k * stages + d for d in (-1, 0, 1)}
    for page in sorted(p for p in pages if 0 <= p < 1 << 26):
        assert place(stages, page) == (page % stages, page // stages), page


def test_every_page_of_a_large_weight():
    # 3.8 GB of weights that nothing touches; pages of 64 values are the shortest, 224 of them a unit of 16 rows
    out, k, rows = 132000, 14336, 5
    w = torch.empty(out, k, dtype=torch.bfloat16)
    a, c = torch.empty(rows, k, dtype=torch.bfloat16)[:, None], torch.empty(rows, 1, out, dtype=torch.bfloat16)
    mk = Megakernel(GemmOp.schedule(a=a, b=w, c=c), config=MegakernelConfig(native_kc=64))
    plan = mk.launch_plan()
    assert len(plan) == 1 and plan[0]["kind"] == N.LAUNCH_MATVEC
    stages, units = plan[0]["stages"], -(-out // 16)
    pages = -(-units // plan[0]["grid"]) * (k // 64)
    assert pages > 1024 * stages
    slot = lap = 0
    for page in range(pages):
        assert place(stages, page) == (slot, lap), page
        slot += 1
        if slot == stages:
            slot, lap = 0, lap + 1


def test_bad_arguments_are_refused():
    out = (C.c_int32 * 2)()
    for stages, page in ((0, 0), (13, 0), (4, -1), (4, 1 << 26)):
        assert N.lib().mk_ring_place(stages, page, out) != 0
    assert N.lib().mk_ring_place(4, 0, None) != 0
