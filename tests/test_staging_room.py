"""What lies where in the shared memory of a chain's matvec launch (CPU): partial sums, rows and ring do not meet, and the norm's weights
and residual rows that are copied to the ring lie behind the pages that are requested before the rows are staged."""

import ctypes as C

import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.decode_matvec import (FinalRmsLmHeadSm100Op, MatvecNvfp4Sm120Op, MatvecSm100Op, RmsGateUpSiluNvfp4Sm120Op,
                                                RmsMatvecNvfp4Sm120Op, RmsQMatvecRopeSm100Op)
from machete_b200.megakernel import Megakernel, MegakernelConfig

BF = torch.bfloat16
OPTIN = 232448            # bytes a CTA may have on an sm_100


def _e(*shape, dtype=BF):
    return torch.empty(*shape, dtype=dtype)


def _ops(fmt, rows, k, out, prologue):
    x, y, n, res = _e(1, rows, k), _e(1, rows, out), _e(k), dict(residual_in=_e(1, rows, k), residual_out=_e(1, rows, k))
    if fmt == "bf16":
        if prologue == "none":
            return MatvecSm100Op.schedule(a=x, weight=_e(out, k), y=y)
        if prologue == "norm":
            return FinalRmsLmHeadSm100Op.schedule(x=x, norm_weight=n, weight=_e(out, k), logits=y)
        return RmsQMatvecRopeSm100Op.schedule(x=x, norm_weight=n, weight=_e(out, k), q=y, cos=_e(rows, 32), sin=_e(rows, 32), **res)
    w = dict(weight_packed=_e(out, k // 2, dtype=torch.uint8), weight_scales=_e(out, k // 16, dtype=torch.float8_e4m3fn), group_size=16, global_scale=1.0)
    if prologue == "none":
        return MatvecNvfp4Sm120Op.schedule(a=x, y=y, **w)
    if prologue == "norm":
        two = dict(gate_packed=w["weight_packed"], gate_scales=w["weight_scales"], up_packed=_e(out, k // 2, dtype=torch.uint8),
                   up_scales=_e(out, k // 16, dtype=torch.float8_e4m3fn))
        return RmsGateUpSiluNvfp4Sm120Op.schedule(x=x, norm_weight=n, y=y, group_size=16, global_scale=1.0, up_global_scale=1.0, **two)
    return RmsMatvecNvfp4Sm120Op.schedule(x=x, norm_weight=n, y=y, **w, **res)


def _staging(mk, launch):
    prog, keep = mk._tables()
    out = (C.c_int32 * 8)()
    assert N.lib().mk_plan_staging(C.byref(prog), mk.num_sms, OPTIN, launch, out) == 0, N.lib().mk_last_error()
    return list(out)


@pytest.mark.parametrize("prologue", ["none", "norm", "add"])
@pytest.mark.parametrize("fmt", ["bf16", "nvfp4"])
@pytest.mark.parametrize("rows", [1, 2, 3, 8, 9, 13, 16, 17, 32])
def test_regions(fmt, rows, prologue):
    beside = set()
    for k in (256, 1024, 1792, 2048, 4096, 6144, 14336):
        for out in (64, 1024, 4096, 9024):
            for page_k in (0, 256):
                if rows * k > 70000 or (fmt == "nvfp4" and k > 2048 and k % 2048):
                    continue
                mk = Megakernel(_ops(fmt, rows, k, out, prologue), config=MegakernelConfig(native_kc=page_k) if page_k else None)
                plan = mk.launch_plan()
                if not plan:
                    continue                      # no room for a page beside the rows
                assert len(plan) == 1
                what, (slots, act, ring, page, stages, ahead, norm, res) = plan[0], _staging(mk, 0)
                where = (k, out, page_k, what)
                assert what["smem"] <= OPTIN and what["stages"] == stages >= 1 and ahead >= 1, where
                assert 4096 <= slots < act and act + rows * (2 * k + (16 if fmt == "bf16" else 0)) <= ring, where
                assert ring % 1024 == page % 1024 == 0 and ring + stages * page <= what["smem"], where
                room, held = what["smem"] - ring, min(ahead, stages) * page
                copied = what["warps"] == 16 and (rows > 8 or fmt == "nvfp4")
                if norm >= 0:
                    assert copied and prologue != "none" and norm >= held and norm % 16 == 0 and norm + 2 * k <= (res if res >= 0 else room), where
                elif copied and prologue != "none":
                    assert ring + held + 2 * k > OPTIN, where
                if res >= 0:
                    assert prologue == "add" and norm >= 0 and res % 16 == 0 and res + rows * 2 * k <= room, where
                elif copied and prologue == "add":
                    assert ring + held + 2 * k + rows * 2 * k > OPTIN, where
                if copied:
                    beside.add(res >= 0)
    if prologue == "add" and 8 < rows <= 16:
        assert beside == {True, False}            # both routes are among the sizes


def test_refusals():
    mk = Megakernel(_ops("bf16", 2, 256, 64, "none"))
    prog, keep = mk._tables()
    out = (C.c_int32 * 8)()
    for launch in (-1, 1):
        assert N.lib().mk_plan_staging(C.byref(prog), 148, OPTIN, launch, out) != 0
    assert N.lib().mk_plan_staging(C.byref(prog), 148, OPTIN, 0, None) != 0
    single = Megakernel(_ops("bf16", 2, 256, 64, "none"), config=MegakernelConfig(single_launch=True))
    prog, keep = single._tables()
    assert N.lib().mk_plan_staging(C.byref(prog), 148, OPTIN, 0, out) != 0
