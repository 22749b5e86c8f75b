"""The K blocks of one product as ops that run side by side, against the chain of stores and residual adds."""

import pytest
import torch

from machete_b200.kernels.decode_matvec import (MatvecNvfp4Sm120Op, MatvecResidualNvfp4Sm120Op, MatvecResidualSm100Op,
                                                MatvecSm100Op)
from machete_b200.megakernel import Megakernel, MegakernelConfig, OverlapTileScheduler
from machete_b200.quantization import quantize_nvfp4_weight

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# activations that no single op can stage; rows at the edges of the 8-row tiles, outputs at those of a unit's 16 rows
@pytest.mark.parametrize("rows,k,blocks,out", [(7, 2048, 4, 2048), (8, 3392, 2, 48), (9, 1536, 4, 1), (16, 2048, 4, 40),
                                               (16, 512, 8, 1000), (17, 1024, 4, 16), (32, 512, 4, 100)])
def test_bf16_blocks_equal_the_chain(rows, k, blocks, out):
    g = torch.Generator().manual_seed(rows * k)
    a = torch.randn(rows, 1, k * blocks, generator=g).to(BF).cuda()
    w = (0.05 * torch.randn(out, k * blocks, generator=g)).to(BF).cuda()
    w2 = (0.05 * torch.randn(64, 64, generator=g)).to(BF).cuda()

    def ops(y, h, z):
        chain = MatvecSm100Op.schedule(a=a[..., :k], weight=w[:, :k], y=y)
        for b in range(1, blocks):
            s = slice(b * k, (b + 1) * k)
            chain += MatvecResidualSm100Op.schedule(a=a[..., s], weight=w[:, s], residual_in=y, residual_out=y)
        return chain + (MatvecSm100Op.schedule(a=h, weight=w2, y=z) if h is not None else [])

    compare(ops, rows, out, blocks)


@pytest.mark.parametrize("rows,edges,out", [(1, (0, 2048, 3072), 64), (5, (0, 6144, 12288), 48), (8, (0, 4096, 8192), 1000),
                                            (9, (0, 256, 512, 768), 33), (32, (0, 1024, 2048), 16)])
def test_nvfp4_blocks_equal_the_chain(rows, edges, out):
    g = torch.Generator().manual_seed(rows)
    a = torch.randn(rows, 1, edges[-1], generator=g).to(BF).cuda()
    q = quantize_nvfp4_weight((0.02 * torch.randn(out, edges[-1], generator=g)).to(BF).cuda(), group_size=16)

    def ops(y, h, z):
        chain = []
        for lo, hi in zip(edges[:-1], edges[1:]):
            kw = dict(a=a[..., lo:hi], weight_packed=q.packed[:, lo // 2: hi // 2], weight_scales=q.scales[:, lo // 16: hi // 16],
                      group_size=16, global_scale=q.global_scale)
            chain += MatvecNvfp4Sm120Op.schedule(y=y, **kw) if lo == 0 else \
                MatvecResidualNvfp4Sm120Op.schedule(residual_in=y, residual_out=y, **kw)
        return chain

    compare(ops, rows, out, len(edges) - 1)


def compare(ops, rows, out, blocks):
    # (the sharing of a unit among warps, and with it the order of its sums, follows the number of CTAs)
    for sms, scheds in ((None, (None, OverlapTileScheduler())), (3, (None,))):
        want = result(ops, rows, out, blocks, MegakernelConfig(num_sms=sms, fuse=False), None)
        assert not want[0].isnan().any()
        for sched in scheds:
            got = result(ops, rows, out, blocks, MegakernelConfig(num_sms=sms), sched)
            # the same sums, in the same order, with the same roundings
            assert torch.equal(got[0], want[0]), (sms, sched)
            assert torch.equal(got[1], want[1]) or want[1].isnan().all()


def result(ops, rows, out, blocks, cfg, sched):
    y = torch.full((rows, 1, out), float("nan"), dtype=BF, device="cuda")
    h = y[..., :64] if out >= 64 and out % 8 == 0 and rows < 17 else None          # an op behind the product reads it
    z = torch.full((rows, 1, 64), float("nan"), dtype=BF, device="cuda")
    mk = Megakernel(ops(y, h, z), config=cfg, scheduler=sched)
    assert [op.commutes is not None for op in mk.native_ops[:blocks]] == [cfg.fuse] * blocks
    for _ in range(3):                                                             # the counters are left at zero
        y.fill_(float("nan"))
        mk.run()
    return y.clone(), z.clone()


@pytest.mark.parametrize("from_chain", [True, False])
def test_one_block_gets_other_weights(from_chain):
    g = torch.Generator().manual_seed(3)
    a = torch.randn(16, 1, 8192, generator=g).to(BF).cuda()
    w, w2 = ((0.05 * torch.randn(256, 8192, generator=g)).to(BF).cuda() for _ in range(2))

    def chain(weight, y):
        ops = MatvecSm100Op.schedule(a=a[..., :2048], weight=weight[:, :2048], y=y)
        for b in range(1, 4):
            s = slice(b * 2048, (b + 1) * 2048)
            ops += MatvecResidualSm100Op.schedule(a=a[..., s], weight=weight[:, s], residual_in=y, residual_out=y)
        return ops

    got = []
    for fuse in (True, False):
        cfg = MegakernelConfig(fuse=fuse)
        y = torch.full((16, 1, 256), float("nan"), dtype=BF, device="cuda")
        mk = Megakernel(chain(w, y), config=cfg)
        mk.run()
        fresh = Megakernel(chain(w2, y), config=MegakernelConfig(fuse=from_chain))
        for block in (2, 0):
            mk.update_op(block, fresh.native_ops[block])
            for _ in range(2):
                y.fill_(float("nan"))
                mk.run()
            got.append(y.clone())
    assert torch.equal(got[0], got[2]) and torch.equal(got[1], got[3]) and not torch.equal(got[0], got[1])
    assert not got[0].isnan().any()


@pytest.mark.parametrize("rows,edges,out", [(1, (0, 1024, 1088), 700), (8, (0, 6144, 6656, 8192), 64), (16, (0, 512, 3072), 2400)])
def test_blocks_of_different_lengths_equal_the_chain(rows, edges, out):
    g = torch.Generator().manual_seed(rows)
    a = torch.randn(rows, 1, edges[-1], generator=g).to(BF).cuda()
    w = (0.05 * torch.randn(out, edges[-1], generator=g)).to(BF).cuda()

    def ops(y, h, z):
        chain = MatvecSm100Op.schedule(a=a[..., :edges[1]], weight=w[:, :edges[1]], y=y)
        for lo, hi in zip(edges[1:-1], edges[2:]):
            chain += MatvecResidualSm100Op.schedule(a=a[..., lo:hi], weight=w[:, lo:hi], residual_in=y, residual_out=y)
        return chain

    compare(ops, rows, out, len(edges) - 1)
