"""When the final residual add may run inside the LM head that reads its sum (lowering alone, no device)."""

import pytest
import torch

from machete_b200.kernels.decode_matvec import MatvecSm100Op, schedule_final_sm100
from machete_b200.megakernel import Megakernel, MegakernelConfig

BF = torch.bfloat16
HIDDEN, VOCAB = 256, 64


def _ops(x, residual_in, residual_out, logits, final_norm):
    a = torch.zeros(1, 1, HIDDEN, dtype=BF)
    ops = MatvecSm100Op.schedule(a=a, weight=torch.zeros(HIDDEN, HIDDEN, dtype=BF), y=x)
    ops += schedule_final_sm100(x=x, residual_in=residual_in, residual_out=residual_out, final_norm=final_norm,
                                lm_head=torch.zeros(VOCAB, HIDDEN, dtype=BF), logits=logits, seq_len=1)
    return len(Megakernel(ops, config=MegakernelConfig(num_sms=4)).native_ops)


def _row():
    return torch.zeros(1, 1, HIDDEN, dtype=BF)


@pytest.mark.parametrize("alias", ["none", "x", "residual_in"])
def test_logits_in_the_memory_of_an_addend_keep_the_two_ops(alias):
    """Two ops: the add has read its addends before the head stores a logit.  In one, some CTAs would store logits
    while others still read the addends."""
    x, r = _row(), _row()
    logits = {"none": torch.zeros(1, 1, VOCAB, dtype=BF), "x": x[..., :VOCAB], "residual_in": r[..., HIDDEN - VOCAB:]}[alias]
    assert _ops(x, r, _row(), logits, torch.ones(HIDDEN, dtype=BF)) == (2 if alias == "none" else 3)


def test_a_sum_in_the_memory_of_the_norm_weight_keeps_the_two_ops():
    total = _row()
    assert _ops(_row(), _row(), total, torch.zeros(1, 1, VOCAB, dtype=BF), total.view(-1)) == 3
