"""K blocks side by side (CPU): who waits for whom, where the units go, and which chains stay chains."""

import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.allreduce import AllReduceSm100Op
from machete_b200.kernels.decode_matvec import MatvecResidualSm100Op, MatvecSm100Op
from machete_b200.megakernel import Megakernel, MegakernelConfig, OverlapTileScheduler
from machete_b200.megakernel.fusion import in_place_of
from machete_b200.megakernel.peer import PeerBuffers
from machete_b200.megakernel.scheduling import share_out, simulate

BF = torch.bfloat16


def chain(a, w, y, blocks):
    k = a.shape[-1] // blocks
    ops = MatvecSm100Op.schedule(a=a[..., :k], weight=w[:, :k], y=y)
    for b in range(1, blocks):
        s = slice(b * k, (b + 1) * k)
        ops += MatvecResidualSm100Op.schedule(a=a[..., s], weight=w[:, s], residual_in=y, residual_out=y)
    return ops


def test_blocks_wait_for_the_input_and_the_next_op_for_all_of_them():
    x, h = torch.zeros(16, 1, 256, dtype=BF), torch.zeros(16, 1, 4096, dtype=BF)
    y, z = torch.zeros(16, 1, 256, dtype=BF), torch.zeros(16, 1, 256, dtype=BF)
    w = torch.zeros(256, 4096, dtype=BF)
    ops = MatvecSm100Op.schedule(a=x, weight=torch.zeros(4096, 256, dtype=BF), y=h)
    ops += chain(h, w, y, 4)
    ops += MatvecSm100Op.schedule(a=y, weight=torch.zeros(256, 256, dtype=BF), y=z)
    ops += chain(h, w, y, 4)                                    # again into y: behind its reader
    for sched in (None, OverlapTileScheduler()):
        mk = Megakernel(ops, config=MegakernelConfig(num_sms=16), scheduler=sched)
        assert [op.i[N.MV_EPI] for op in mk.native_ops] == [N.EPI_STORE] + [N.EPI_KSUM] * 4 + [N.EPI_STORE] + [N.EPI_KSUM] * 4
        deps = [d.coarse for d in mk.program.deps]
        assert deps == [[]] + [[0]] * 4 + [[1, 2, 3, 4]] + [[5]] * 4
        # every block on CTAs of its own: 16 units on 4 CTAs
        where = [set(int(c) for c in mk.program.placement[j]) for j in (1, 2, 3, 4)]
        assert all(len(s) == 4 for s in where) and len(set().union(*where)) == 16
        final = simulate(mk.program)
        assert (final == mk.program.counter_expected[:len(final)]).all()


def test_chains_that_read_their_own_output_stay_chains():
    a, w = torch.zeros(16, 1, 4096, dtype=BF), torch.zeros(1024, 4096, dtype=BF)
    inside = chain(a, w, a[..., 1024:2048], 4)                  # the second block reads what the first one writes
    other = torch.zeros(16, 1, 1024, dtype=BF)
    broken = chain(a, w, torch.zeros(16, 1, 1024, dtype=BF), 2)[:1]
    broken += MatvecResidualSm100Op.schedule(a=a[..., 2048:], weight=w[:, 2048:], residual_in=other, residual_out=other)
    for ops in (inside, broken):
        mk = Megakernel(ops, config=MegakernelConfig(num_sms=16))
        assert all(op.commutes is None for op in mk.native_ops)
        assert mk.program.deps[1].coarse == ([0] if ops is inside else [])


def test_programs_with_an_all_reduce_keep_their_chains():
    # (no kernel has both but the generic one)
    x, y = torch.zeros(16, 1, 4096, dtype=BF), torch.zeros(16, 1, 256, dtype=BF)
    part, total = torch.zeros(16, 1, 256), torch.zeros(16, 1, 256, dtype=BF)
    ops = chain(x, torch.zeros(256, 4096, dtype=BF), y, 4)
    ops += MatvecSm100Op.schedule(a=y, weight=torch.zeros(256, 256, dtype=BF), y=part)
    reduced = AllReduceSm100Op.schedule(peers=PeerBuffers(1 << 20, rank=0, world_size=2), x=part, y=total)
    for with_reduce in (False, True):
        mk = Megakernel(ops + (reduced if with_reduce else []), config=MegakernelConfig(num_sms=16))
        assert [op.commutes is not None for op in mk.native_ops[:4]] == [not with_reduce] * 4


def test_a_replaced_block_keeps_its_place_in_the_group():
    a, w, y = torch.zeros(16, 1, 4096, dtype=BF), torch.zeros(256, 4096, dtype=BF), torch.zeros(16, 1, 256, dtype=BF)
    cfg = MegakernelConfig(num_sms=16)
    mine = Megakernel(chain(a, w, y, 4), config=cfg).native_ops
    w2 = torch.zeros(256, 4096, dtype=BF)
    fresh = Megakernel(chain(a, w2, y, 4), config=cfg).native_ops                   # blocks of another program
    plain = Megakernel(chain(a, w2, y, 4), config=MegakernelConfig(num_sms=16, fuse=False)).native_ops
    for b in range(4):
        for new in (fresh[b], plain[b]):
            got = in_place_of(mine[b], new)
            for slot in (N.MV_P_KPART, N.MV_P_KARRIVE):
                assert got.p[slot] == mine[b].p[slot]
            assert got.p[N.MV_P_W0] == w2[:, b * 1024:].data_ptr() and got.i[N.MV_EPI] == N.EPI_KSUM
            assert (got.i[N.MV_KBLOCK], got.i[N.MV_KBLOCKS], got.commutes) == (b, 4, mine[0].commutes)
            assert got.zero_on_reset == mine[b].zero_on_reset
            assert in_place_of(got, got).record(1) == got.record(1)
        # a block in a program of single ops is what the chain has
        assert in_place_of(plain[b], fresh[b]).record(1) == plain[b].record(1)
    # what is no block of the product is refused: another epilogue, another residual, more rows than the buffer holds
    with pytest.raises(ValueError, match="block 0 of 4"):
        in_place_of(mine[0], plain[1])
    other = MatvecResidualSm100Op.schedule(a=a[..., :1024], weight=w[:, :1024], residual_in=torch.zeros_like(y), residual_out=y)
    with pytest.raises(ValueError, match="block 1 of 4"):
        in_place_of(mine[1], Megakernel(other, config=cfg).native_ops[0])
    wide, wide_y = torch.zeros(17, 1, 1024, dtype=BF), torch.zeros(17, 1, 256, dtype=BF)
    with pytest.raises(ValueError, match="17 rows do not fit"):
        in_place_of(mine[0], Megakernel(MatvecSm100Op.schedule(a=wide, weight=w[:, :1024], y=wide_y), config=cfg).native_ops[0])


def test_ctas_are_dealt_out_by_what_the_blocks_cost():
    assert share_out((7, 7, 7, 7), 14).tolist() == [c % 4 for c in range(14)]        # equal blocks: every n-th
    for costs, ctas in (((8192, 2048), 148), ((1, 1000), 148), ((3, 1, 4, 1, 5), 148), ((6144, 256, 6144), 7)):
        owner = share_out(costs, ctas)
        for i, cost in enumerate(costs):
            assert abs((owner == i).sum() - ctas * cost / sum(costs)) <= 1
        first = [owner.tolist().index(i) for i in range(len(costs)) if (owner == i).any()]
        assert max(first) - min(first) <= max(len(costs), sum(costs) // min(costs))  # spread out, not in runs


@pytest.mark.parametrize("edges", [(0, 3072, 4096), (0, 64, 4096), (0, 2048, 4096)])
@pytest.mark.parametrize("sched", [None, OverlapTileScheduler()])
def test_long_blocks_get_more_ctas(edges, sched):
    a, w, y = torch.zeros(16, 1, 4096, dtype=BF), torch.zeros(1024, 4096, dtype=BF), torch.zeros(16, 1, 1024, dtype=BF)
    ops = MatvecSm100Op.schedule(a=a[..., :edges[1]], weight=w[:, :edges[1]], y=y)
    ops += MatvecResidualSm100Op.schedule(a=a[..., edges[1]:], weight=w[:, edges[1]:], residual_in=y, residual_out=y)
    for ctas in (1, 2, 16):
        mk = Megakernel(ops, config=MegakernelConfig(num_sms=ctas), scheduler=sched)
        where = [set(int(c) for c in mk.program.placement[j]) for j in (0, 1)]
        if ctas == 1 or (ctas == 2 and edges[1] == 64):
            assert where[0] == where[1] == set(range(ctas))                          # no CTA left for the shorter one
        else:
            assert not where[0] & where[1] and len(where[0] | where[1]) == ctas
            assert abs(len(where[0]) - ctas * (edges[1] + 1280) / (4096 + 2 * 1280)) <= 1
        final = simulate(mk.program)
        assert (final == mk.program.counter_expected[:len(final)]).all()
