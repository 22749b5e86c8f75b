"""A projection behind attention has an event, whatever was staged before (CPU)."""

import torch

from machete_b200.kernels.attention import flash_decoding_schedule
from machete_b200.kernels.decode_matvec import MatvecSm100Op
from machete_b200.megakernel import Megakernel, MegakernelConfig, OverlapTileScheduler

BF = torch.bfloat16


def test_a_layer_whose_mlp_reads_the_input_of_its_attention():
    z = lambda *s: torch.zeros(*s, dtype=BF)                                       # noqa: E731
    x, q, o, h = z(4, 1, 256), z(4, 1, 256), z(4, 1, 256), z(4, 1, 512)
    ops = MatvecSm100Op.schedule(a=x, weight=z(256, 256), y=q)
    attn, cfg = flash_decoding_schedule(q.view(4, 1, 4, 64), z(4, 300, 2, 64), z(4, 300, 2, 64), o.view(4, 1, 4, 64), kv_group_size=2,
                                        num_splits=4)
    ops += attn + MatvecSm100Op.schedule(a=x, weight=z(512, 256), y=h) + MatvecSm100Op.schedule(a=o, weight=z(256, 256), y=z(4, 1, 256))
    for sched in (None, OverlapTileScheduler()):
        mk = Megakernel(ops, config=MegakernelConfig(num_sms=8), scheduler=sched)
        keys, events = mk.program.ops["act_key"], mk.program.events["op"].tolist()
        assert keys[0] == keys[2] != keys[3]
        # the MLP's projection too: the attention units beside it would use the staging buffer and the split-K slots
        assert [events.count(j) for j in range(4)] == [8, 8, 8, 8]
