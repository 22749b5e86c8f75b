"""The final residual add fused into the LM head that reads its sum, against the two separate ops."""

import pytest
import torch

from machete_b200.kernels.decode_matvec import MatvecSm100Op, schedule_final_sm100
from machete_b200.megakernel import Megakernel, MegakernelConfig

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("rows,hidden,vocab", [(1, 64, 17), (8, 2048, 400), (9, 2048, 401), (32, 1088, 64)])
def test_fused_final_add_equals_the_two_ops(rows, hidden, vocab):
    g = torch.Generator().manual_seed(rows)
    a, r = (torch.randn(rows, 1, hidden, generator=g).to(BF).cuda() for _ in range(2))
    w = (torch.randn(hidden, hidden, generator=g) / hidden ** 0.5).to(BF).cuda()
    x = torch.zeros_like(a)
    fn = (1 + 0.02 * torch.randn(hidden, generator=g)).to(BF).cuda()
    lm = (0.02 * torch.randn(vocab, hidden, generator=g)).to(BF).cuda()
    got = {}
    for fuse in (True, False):
        total = torch.full_like(x, float("nan"))
        logits = torch.full((rows, 1, vocab), float("nan"), dtype=BF, device="cuda")
        # a last projection and the head, as a step ends
        ops = MatvecSm100Op.schedule(a=a, weight=w, y=x) + schedule_final_sm100(
            x=x, residual_in=r, residual_out=total, final_norm=fn, lm_head=lm, logits=logits, seq_len=1)
        mk = Megakernel(ops, config=MegakernelConfig(fuse=fuse))
        assert len(mk.native_ops) == (2 if fuse else 3)
        mk.run()
        got[fuse] = (total, logits)
    # the same additions, roundings and dot products in the same order: equal bit for bit
    assert torch.equal(got[True][0], got[False][0]) and torch.equal(got[True][1], got[False][1])
    assert torch.equal(got[True][0], (x.float() + r.float()).to(BF))


def test_an_in_place_sum_keeps_the_two_ops():
    x, r = torch.zeros(1, 1, 256, dtype=BF, device="cuda"), torch.randn(1, 1, 256).to(BF).cuda()
    a, w = torch.randn(1, 1, 256).to(BF).cuda(), torch.eye(256).to(BF).cuda()
    want = (a.float() + r.float()).to(BF)
    logits = torch.zeros(1, 1, 16, dtype=BF, device="cuda")
    ops = MatvecSm100Op.schedule(a=a, weight=w, y=x) + schedule_final_sm100(
        x=x, residual_in=r, residual_out=r, final_norm=torch.ones(256, dtype=BF, device="cuda"),
        lm_head=torch.zeros(16, 256, dtype=BF, device="cuda"), logits=logits, seq_len=1)
    mk = Megakernel(ops)
    assert len(mk.native_ops) == 3
    mk.run()
    assert torch.equal(r, want)
