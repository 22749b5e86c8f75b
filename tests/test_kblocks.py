"""K blocks side by side (CPU): who waits for whom, where the units go, and which chains stay chains."""

import torch

from machete_b200 import _native as N
from machete_b200.kernels.allreduce import AllReduceSm100Op
from machete_b200.kernels.decode_matvec import MatvecResidualSm100Op, MatvecSm100Op
from machete_b200.megakernel import Megakernel, MegakernelConfig, OverlapTileScheduler
from machete_b200.megakernel.peer import PeerBuffers
from machete_b200.megakernel.scheduling import simulate

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
