"""Staging of the activation rows in the NVFP4 matvecs: conversion in place, residual add, RMSNorm, at the edges of
what a thread and a group of four rows take (224 chunks of 8 values; rows 1, 4, 5, 32)."""

import pytest
import torch

from machete_b200.kernels.decode_matvec import MatvecNvfp4Sm120Op, RmsMatvecNvfp4Sm120Op
from machete_b200.megakernel import Megakernel
from machete_b200.quantization import dequantize_nvfp4_weight, quantize_nvfp4_weight
from tests.util import assert_parity

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("rows,k", [(1, 256), (1, 4096), (2, 1792), (3, 2048), (4, 2048), (5, 4096), (8, 4096), (9, 2048), (32, 1536)])
def test_rows_converted_and_normalised_in_place(rows, k):
    g = torch.Generator().manual_seed(rows * k)
    x, r = (torch.randn(1, rows, k, generator=g).to(BF).cuda() for _ in range(2))
    norm = (1 + 0.02 * torch.randn(k, generator=g)).to(BF).cuda()
    q = quantize_nvfp4_weight((torch.randn(48, k, generator=g) * 0.02).to(BF).cuda(), group_size=16)
    w = dequantize_nvfp4_weight(q).float()
    y, z = (torch.full((1, rows, 48), float("nan"), dtype=BF, device="cuda") for _ in range(2))
    total = torch.full_like(x, float("nan"))
    packed = dict(weight_packed=q.packed, weight_scales=q.scales, group_size=16, global_scale=q.global_scale)
    ops = MatvecNvfp4Sm120Op.schedule(a=x, y=y, **packed)
    ops += RmsMatvecNvfp4Sm120Op.schedule(x=x, residual_in=r, residual_out=total, norm_weight=norm, y=z, eps=1e-6, **packed)
    Megakernel(ops).compile().run()
    want = (x.float() + r.float()).to(BF)
    assert torch.equal(total, want)                    # one rounding of an exact sum
    normed = want.float() * torch.rsqrt(want.float().pow(2).mean(-1, keepdim=True) + 1e-6) * norm.float()
    # the bar of the other matvec tests: f16 activations (2^-11 a value) and a bf16 result
    assert_parity(y[0], x[0].float() @ w.t(), f"converted {rows}x{k}")
    assert_parity(z[0], normed[0] @ w.t(), f"normalised {rows}x{k}")
