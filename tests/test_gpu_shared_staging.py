"""Ops on one input that share what the first of them staged, with weights of different formats."""

import pytest
import torch

from machete_b200.kernels.decode_matvec import MatvecNvfp4Sm120Op, MatvecSm100Op
from machete_b200.megakernel import Megakernel, MegakernelConfig
from machete_b200.quantization import dequantize_nvfp4_weight, quantize_nvfp4_weight
from tests.util import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,group", [(1, 512, 16), (4, 1024, 16), (5, 2048, 32), (8, 4096, 16), (16, 2048, 32), (32, 1536, 16)])
@pytest.mark.parametrize("packed_first", [False, True])
def test_fp16_and_packed_weights_on_one_input(rows, k, group, packed_first):
    g = torch.Generator().manual_seed(rows + k)
    x = torch.randn(rows, 1, k, generator=g).half().cuda()
    w = (torch.randn(80, k, generator=g) * 0.02).half().cuda()
    q = quantize_nvfp4_weight((torch.randn(80, k, generator=g) * 0.02).half().cuda(), group_size=group)
    y, z = (torch.full((rows, 1, 80), float("nan"), dtype=torch.float16, device="cuda") for _ in range(2))
    ops = [MatvecSm100Op.schedule(a=x, weight=w, y=y),
           MatvecNvfp4Sm120Op.schedule(a=x, weight_packed=q.packed, weight_scales=q.scales, y=z, group_size=group,
                                       global_scale=q.global_scale)]
    # fewer CTAs than units: every CTA holds units of both ops
    mk = Megakernel(sum(ops[::-1] if packed_first else ops, []), config=MegakernelConfig(num_sms=4)).compile()
    keys = mk.program.ops["act_key"]
    assert keys[0] == keys[1] != 0                      # the second op has nothing staged for it
    mk.run()
    assert_parity(y[:, 0], x[:, 0].float() @ w.float().t(), "fp16 weights")
    assert_parity(z[:, 0], x[:, 0].float() @ dequantize_nvfp4_weight(q).float().t(), "packed weights")
