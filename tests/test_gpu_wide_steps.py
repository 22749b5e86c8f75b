"""Steps of several rows or with NVFP4 weights: units found by one vote over windows of 32 records, a loader that issues
through an elected lane, partial attention states in the staging buffer."""

import ctypes as C

import numpy as np
import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.attention import flash_decoding_schedule
from machete_b200.kernels.decode_matvec import MatvecNvfp4Sm120Op
from machete_b200.megakernel import Megakernel, MegakernelConfig
from machete_b200.quantization import dequantize_nvfp4_weight, quantize_nvfp4_weight
from tests.util import assert_parity

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def packed(n, k, g):
    return quantize_nvfp4_weight((torch.randn(n, k, generator=g) / k ** 0.5).to(BF).cuda(), group_size=16)


def project(x, w, y):
    return MatvecNvfp4Sm120Op.schedule(a=x, weight_packed=w.packed, weight_scales=w.scales, y=y, group_size=16,
                                       global_scale=w.global_scale)


def placement(mk):
    out = (C.c_int32 * 3)()
    N.check(N.lib().mk_state_placement(mk._handle, out), "mk_state_placement")
    return list(out)


def step(batch, tokens, hidden=512, heads=4, kv_heads=2, head_dim=128, out=512, seed=0):
    """Q projection, attention, output projection, all with packed weights: ``(ops, outputs, keep)``."""
    g = torch.Generator().manual_seed(seed)

    x = torch.randn(batch, 1, hidden, generator=g).to(BF).cuda()
    k, v = (torch.randn(batch, tokens, kv_heads, head_dim, generator=g).to(BF).cuda() for _ in range(2))
    q, o = (torch.full((batch, 1, heads * head_dim), float("nan"), dtype=BF, device="cuda") for _ in range(2))
    y = torch.full((batch, 1, out), float("nan"), dtype=BF, device="cuda")
    wq, wo = packed(heads * head_dim, hidden, g), packed(out, heads * head_dim, g)
    attn, cfg = flash_decoding_schedule(q.view(batch, 1, heads, head_dim), k, v, o.view(batch, 1, heads, head_dim),
                                        kv_group_size=heads // kv_heads, num_splits=2)
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


@pytest.mark.parametrize("batch", [1, 4])
def test_every_place_of_the_states_gives_the_same_bits(batch):
    """Two participants a unit (17 KB of states): in the pages, and one, two and four units' in the staging buffer, whose
    size a projection beside the step sets."""
    got, seen = [], []
    for extra in (256, 17408 // 2, 2 * 17408 // 2, 4 * 17408 // 2):
        k = -(-extra // batch // 2048) * 2048 if extra > 256 else 256
        ops, outs, keep = step(batch, 500, heads=12, kv_heads=3)
        g = torch.Generator().manual_seed(1)
        x, y = torch.randn(batch, 1, k, generator=g).to(BF).cuda(), torch.full((batch, 1, 64), float("nan"), dtype=BF, device="cuda")
        w = packed(64, k, g)
        mk = Megakernel(ops + project(x, w, y), config=MegakernelConfig(num_sms=4, num_pages=4))
        mk.compile()
        size, sets, may = placement(mk)
        assert may == 1 and size in (0, 17408)
        seen.append(sets if size else 0)
        for _ in range(2):
            for t in outs:
                t.fill_(float("nan"))
            mk.run()
        got.append([t.clone() for t in outs])
        assert_parity(y[:, 0], x[:, 0].float() @ dequantize_nvfp4_weight(w).float().t(), "the projection beside it")
    assert seen == [0, 1, 2, 4]
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
    assert not any(t.isnan().any() for t in got[0])


def two_projections_of_one_input(fuse):
    """Projection of x, attention, another projection of x: the program, its op records without the second one's events."""
    ops, outs, keep = step(2, 500)
    g = torch.Generator().manual_seed(2)
    x = torch.randn(2, 1, 10240, generator=g).to(BF).cuda()
    ys = [torch.full((2, 1, 512), float("nan"), dtype=BF, device="cuda") for _ in range(2)]
    ws = [packed(512, 10240, g) for _ in range(2)]
    outs[0].copy_(torch.randn(2, 1, 512, generator=g))
    mk = Megakernel(project(x, ws[0], ys[0]) + ops[1:-1] + project(x, ws[1], ys[1]),
                    config=MegakernelConfig(num_sms=8, num_pages=4, fuse=fuse))
    want = [x[:, 0].float() @ dequantize_nvfp4_weight(w).float().t() for w in ws]
    return mk, ys, want, (outs, keep, x, ws)


def drop_events_of_the_last_op(mk):
    prog, last = mk.program, len(mk.native_ops) - 1
    assert prog.ops["act_key"][0] == prog.ops["act_key"][last] != 0
    drop = prog.events["op"] == last
    assert drop.any()
    prog.events["n_waits"][drop] = 0
    kept = np.concatenate([[0], np.cumsum(~drop)])
    prog.cta_event_begin[:] = kept[prog.cta_event_begin]
    prog.events = prog.events[~drop].copy()


def test_projections_of_one_input_around_attention():
    """The second projection must not start beside the attention units: their combine uses the slots of its partial sums."""
    mk, ys, want, keep = two_projections_of_one_input(fuse=True)
    first = None
    for _ in range(100):
        for y in ys:
            y.fill_(float("nan"))
        mk.run()
        first = first or [y.clone() for y in ys]
        assert all(torch.equal(a, b) for a, b in zip(first, ys))
    for y, ref in zip(ys, want):
        assert_parity(y[:, 0], ref, "projection")
    # tables that would let them run side by side are refused
    mk, ys, want, keep = two_projections_of_one_input(fuse=True)
    drop_events_of_the_last_op(mk)
    with pytest.raises(ValueError, match="no event between a fused combine"):
        mk.compile()


def test_rows_staged_before_attention_keep_the_buffer():
    """Hand-made tables in which the second projection relies on the rows that the first one staged (and no combine is fused):
    the states must not go there."""
    mk, ys, want, keep = two_projections_of_one_input(fuse=False)
    drop_events_of_the_last_op(mk)
    mk.compile()
    assert placement(mk) == [0, 4, 0]
    for _ in range(20):
        for y in ys:
            y.fill_(float("nan"))
        mk.run()
        for y, ref in zip(ys, want):
            assert_parity(y[:, 0], ref, "projection")


@pytest.mark.parametrize("units", [(31, 1, 32), (32, 33, 1), (1, 30, 1, 32, 64, 5), (63, 1, 64, 2, 31), (16, 16, 17, 15, 33)])
@pytest.mark.parametrize("rows,ctas", [(1, 1), (5, 1), (9, 2)])
def test_events_at_the_edges_of_the_record_windows(units, rows, ctas):
    """Projections of ``units`` x 16 outputs, each reading the one before, with attention among them: lists longer than 32
    records a CTA and events at every distance from a window's end."""
    g = torch.Generator().manual_seed(sum(units))
    ops, outs, keep = step(rows, 700, out=256)
    x = outs[2]                                        # the chain goes on from the step's output
    want = []
    for n in units:
        w = packed(16 * n * ctas, 256, g)
        y = torch.full((rows, 1, max(256, 16 * n * ctas)), float("nan"), dtype=BF, device="cuda")
        if n * ctas < 16:
            y[..., 16 * n * ctas:] = 0.5               # what the next projection reads besides
        ops = ops + project(x[..., :256], w, y[..., :16 * n * ctas])
        want.append((x, w, y))
        x = y
    mk = Megakernel(ops, config=MegakernelConfig(num_sms=ctas))
    for _ in range(2):
        mk.run()
    assert int(np.diff(mk.program.cta_instr_begin).max()) > 64
    for i, (a, w, y) in enumerate(want):
        ref = a[:, 0, :256].float() @ dequantize_nvfp4_weight(w).float().t()
        assert_parity(y[:, 0, :ref.shape[1]], ref, f"projection {i}")
