"""Rows that sixteen warps stage (9 to 16 rows, and up to 8 where a CTA has the multiprocessor): normalised with and without a
residual, K of less than a warp's chunks, of ragged parts and of several rounds, and residual rows that do not fit beside the
pages requested ahead.  The chain's results and residual output are the persistent kernel's, bit for bit."""

import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.decode_matvec import (FinalRmsLmHeadSm100Op, MatvecNvfp4Sm120Op, MatvecSm100Op, RmsGateUpSiluNvfp4Sm120Op,
                                                RmsMatvecNvfp4Sm120Op, RmsQMatvecRopeSm100Op)
from machete_b200.megakernel import Megakernel
from tests.test_gpu_chain import BF, Values, equal_forms

pytestmark = pytest.mark.gpu


def _warps(ops):
    return [p["warps"] for p in Megakernel(ops).launch_plan() if p["kind"] == N.LAUNCH_MATVEC]


@pytest.mark.parametrize("fmt,rows,k,out", [
    ("bf16", 9, 64, 64), ("bf16", 16, 2048, 3072), ("bf16", 16, 1856, 192), ("bf16", 10, 2112, 64), ("bf16", 16, 4096, 128),
    ("bf16", 13, 4096, 4992), ("bf16", 8, 2048, 4096), ("bf16", 2, 1024, 2368),
    ("nvfp4", 16, 256, 40), ("nvfp4", 9, 1792, 100), ("nvfp4", 16, 2048, 4000), ("nvfp4", 12, 4096, 64), ("nvfp4", 8, 4096, 6144),
    ("nvfp4-g32", 15, 1280, 48), ("nvfp4", 7, 8192, 2400), ("nvfp4", 16, 4096, 8000)])
@pytest.mark.parametrize("residual", [False, True])
def test_normalised_rows(fmt, rows, k, out, residual):
    v = Values(rows * k + out)
    # sequences of several tokens where the rows divide so, with strides of their own
    b, s = (rows // 2, 2) if rows % 2 == 0 else (rows, 1)
    x, n = v(b, s + 1, k + 8)[:, 1:, :k], 1 + v(k, std=0.02)
    res, res_out = v(b, s, k + 16)[..., :k], torch.zeros(b, s, k, dtype=BF, device="cuda")
    y, w = torch.zeros(b, s, out, dtype=BF, device="cuda"), v.weight(fmt, out, k)
    kw = dict(x=x, norm_weight=n, y=y, **(dict(residual_in=res, residual_out=res_out) if residual else {}))
    if fmt == "bf16" and residual:
        q = kw.pop("y")
        cos, sin = v(s, 32), v(s, 32)
        ops = RmsQMatvecRopeSm100Op.schedule(weight=w, q=q, cos=cos, sin=sin, **kw)
    elif fmt == "bf16":
        ops = FinalRmsLmHeadSm100Op.schedule(x=x, norm_weight=n, weight=w, logits=y)
    elif not residual:
        u = v.weight(fmt, out, k)
        ops = RmsGateUpSiluNvfp4Sm120Op.schedule(x=x, norm_weight=n, gate_packed=w.packed, gate_scales=w.scales, up_packed=u.packed,
                                                 up_scales=u.scales, group_size=w.group_size, global_scale=w.global_scale,
                                                 up_global_scale=u.global_scale, y=y)
    else:
        ops = RmsMatvecNvfp4Sm120Op.schedule(weight_packed=w.packed, weight_scales=w.scales, group_size=w.group_size,
                                             global_scale=w.global_scale, **kw)
    if rows > 8:
        assert _warps(ops) == [16]
    got = equal_forms(ops, [y, res_out], launches=1)
    assert got[0].float().abs().sum() > 0
    if residual:
        assert torch.equal(got[1], x + res)


@pytest.mark.parametrize("fmt,rows,k,out", [("nvfp4", 9, 256, 33), ("nvfp4", 16, 4096, 64), ("nvfp4", 11, 1536, 5000),
                                            ("nvfp4-g32", 16, 512, 17), ("bf16", 16, 4096, 64), ("fp16", 16, 4096, 64)])
def test_rows_as_they_come(fmt, rows, k, out):
    v = Values(rows * k + out)
    x = v(rows, 1, k + 8, dtype=torch.float16 if fmt == "fp16" else BF)[..., :k]
    y, w = torch.zeros(rows, 1, out, dtype=x.dtype, device="cuda"), v.weight(fmt, out, k)
    if fmt.startswith("nvfp4"):
        ops = MatvecNvfp4Sm120Op.schedule(a=x, weight_packed=w.packed, weight_scales=w.scales, y=y, group_size=w.group_size,
                                          global_scale=w.global_scale)
    else:
        ops = MatvecSm100Op.schedule(a=x, weight=w, y=y)
    assert equal_forms(ops, [y])[0].float().abs().sum() > 0
