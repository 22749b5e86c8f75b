"""Steps of several rows or with NVFP4 weights: units found by one vote over windows of 32 records, a loader that issues
through an elected lane, partial attention states in the staging buffer."""

import pytest
import torch

from machete_b200.kernels.attention import flash_decoding_schedule
from machete_b200.kernels.decode_matvec import MatvecNvfp4Sm120Op
from machete_b200.megakernel import Megakernel, MegakernelConfig
from machete_b200.quantization import quantize_nvfp4_weight

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def step(batch, tokens, hidden=512, heads=4, kv_heads=2, head_dim=128, out=512, seed=0):
    """Q projection, attention, output projection, all with packed weights: ``(ops, outputs, keep)``."""
    g = torch.Generator().manual_seed(seed)

    def packed(n, k):
        return quantize_nvfp4_weight((torch.randn(n, k, generator=g) / k ** 0.5).to(BF).cuda(), group_size=16)

    def project(x, w, y):
        return MatvecNvfp4Sm120Op.schedule(a=x, weight_packed=w.packed, weight_scales=w.scales, y=y, group_size=16,
                                           global_scale=w.global_scale)

    x = torch.randn(batch, 1, hidden, generator=g).to(BF).cuda()
    k, v = (torch.randn(batch, tokens, kv_heads, head_dim, generator=g).to(BF).cuda() for _ in range(2))
    q, o = (torch.full((batch, 1, heads * head_dim), float("nan"), dtype=BF, device="cuda") for _ in range(2))
    y = torch.full((batch, 1, out), float("nan"), dtype=BF, device="cuda")
    wq, wo = packed(heads * head_dim, hidden), packed(out, heads * head_dim)
    attn, cfg = flash_decoding_schedule(q.view(batch, 1, heads, head_dim), k, v, o.view(batch, 1, heads, head_dim),
                                        kv_group_size=heads // kv_heads)
    ops = project(x, wq, q) + attn + project(o, wo, y)
    return ops, [q, o, y], (x, k, v, wq, wo, cfg)


@pytest.mark.parametrize("batch", [1, 3])
def test_the_trace_holds_every_page_that_was_issued(batch):
    ops, outs, keep = step(batch, 3000)
    mk = Megakernel(ops, config=MegakernelConfig(num_sms=24))
    mk.run()
    plain = [t.clone() for t in outs]
    mk.enable_trace(4096)
    mk.run()
    assert all(torch.equal(a, b) for a, b in zip(plain, outs)) and not any(t.isnan().any() for t in outs)
    issued = sum(int((rec["code"] == 2).sum()) for rec in mk.read_trace().values())
    assert issued == int(mk.program.instrs["n_pages"].sum()) > 0
