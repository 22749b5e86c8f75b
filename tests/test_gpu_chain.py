"""A program as a chain of kernels against the same program as one launch: the same sums in the same order, so the same bits."""

import threading

import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.attention import flash_decoding_schedule
from machete_b200.kernels.decode_matvec import (MatvecNvfp4Sm120Op, MatvecResidualNvfp4Sm120Op, MatvecResidualSm100Op,
                                                MatvecSm100Op, RmsGateUpSiluNvfp4Sm120Op, RmsGateUpSiluSm100Op,
                                                RmsKMatvecRopeCacheSm100Op, RmsQMatvecRopeSm100Op, RmsVMatvecCacheSm100Op,
                                                schedule_decode_layer_sm100)
from machete_b200.kernels.decode_matvec.nvfp4_model import schedule_decode_layer_nvfp4_sm100
from machete_b200.kernels.llama1b import schedule_decode_model_sm100
from machete_b200.megakernel import Megakernel, MegakernelConfig, OverlapTileScheduler
from machete_b200.quantization import quantize_nvfp4_weight

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


class Values:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, *shape, std=1.0, dtype=BF):
        return (torch.randn(*shape, generator=self.g, device="cuda") * std).to(dtype)

    def weight(self, fmt, o, k):
        w = self(o, k, std=0.02, dtype=torch.float16 if fmt == "fp16" else BF)
        return w if fmt in ("bf16", "fp16") else quantize_nvfp4_weight(w, group_size=16 if fmt == "nvfp4" else 32)


def equal_forms(ops, outs, launches=1, attention=None, **config):
    """Both forms, three launches each (the arrival counts and slots they leave behind included), from the same buffers.
    `launches`: at least so many kernels in the chain; `attention`: participants and CTAs a multiprocessor of its attention launch."""
    start, got = [t.clone() for t in outs], []
    for single in (True, False):
        for t, s in zip(outs, start):
            t.copy_(s)
        mk = Megakernel(ops, config=MegakernelConfig(single_launch=single, **config), scheduler=OverlapTileScheduler()).compile()
        for _ in range(3):
            mk.run()
        plan = mk.launch_plan()
        assert mk.launches_per_run == max(1, len(plan)) and (len(plan) == 0 if single else len(plan) >= launches)
        if attention and not single:
            assert [(p["warps"], p["per_sm"]) for p in plan if p["kind"] == N.LAUNCH_ATTENTION] == [attention]
        assert mk.launch_count() == 3 and not mk.read_counters().any()
        got.append([t.clone() for t in outs])
    for a, b in zip(*got):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    return got[1]


# rows at the edges of the kernels' row classes; outputs at those of a unit's 16 rows; K of one tile, of a ragged last page, of
# odd numbers of tiles, of as many pages as participants and of more
@pytest.mark.parametrize("fmt,rows,k,out", [
    ("bf16", 1, 64, 1), ("bf16", 1, 1088, 16), ("bf16", 1, 14336, 40), ("bf16", 2, 832, 4096), ("bf16", 8, 6144, 100),
    ("bf16", 9, 2880, 33), ("bf16", 16, 1024, 1024), ("bf16", 17, 1600, 15), ("bf16", 32, 1536, 5000),
    ("fp16", 1, 2048, 64), ("fp16", 5, 960, 200), ("fp16", 16, 1152, 17), ("fp16", 32, 512, 48),
    ("nvfp4", 1, 256, 1), ("nvfp4", 1, 14336, 1000), ("nvfp4", 4, 4096, 14336), ("nvfp4", 8, 1792, 24),
    ("nvfp4", 9, 2048, 520), ("nvfp4", 16, 768, 31), ("nvfp4", 25, 1280, 4096),
    ("nvfp4-g32", 1, 4096, 6144), ("nvfp4-g32", 3, 512, 16), ("nvfp4-g32", 12, 1024, 100), ("nvfp4-g32", 32, 256, 8)])
@pytest.mark.parametrize("residual", [False, True])
def test_products(fmt, rows, k, out, residual):
    v = Values(rows * k + out)
    dtype = torch.float16 if fmt == "fp16" else BF
    # sequences of several tokens where the rows divide so, with strides of their own
    b, s = (rows // 2, 2) if rows % 2 == 0 else (rows, 1)
    x, y = v(b, s, k + 8, dtype=dtype)[..., :k], torch.zeros(b, s + 1, out + 8, dtype=dtype, device="cuda")[:, 1:, :out]
    r, w = v(b, s, out, dtype=dtype), v.weight(fmt, out, k)
    if fmt.startswith("nvfp4"):
        kw = dict(a=x, weight_packed=w.packed, weight_scales=w.scales, group_size=w.group_size, global_scale=w.global_scale)
        ops = MatvecResidualNvfp4Sm120Op.schedule(residual_in=r, residual_out=y, **kw) if residual else \
            MatvecNvfp4Sm120Op.schedule(y=y, **kw)
    else:
        ops = MatvecResidualSm100Op.schedule(a=x, weight=w, residual_in=r, residual_out=y) if residual else \
            MatvecSm100Op.schedule(a=x, weight=w, y=y)
    assert equal_forms(ops, [y])[0].float().abs().sum() > 0


@pytest.mark.parametrize("fmt,rows,k,inter", [("bf16", 1, 2048, 8), ("bf16", 8, 4096, 104), ("bf16", 16, 1024, 2048), ("bf16", 32, 832, 24),
                                              ("nvfp4", 1, 4096, 12288), ("nvfp4", 7, 6144, 16), ("nvfp4-g32", 16, 2048, 1000),
                                              ("nvfp4", 32, 768, 2048)])
def test_normalised_rows_and_pairs(fmt, rows, k, inter):
    v = Values(rows + k)
    x, y, n = v(rows, 1, k), torch.zeros(rows, 1, inter, dtype=BF, device="cuda"), 1 + v(k, std=0.02)
    g, u = v.weight(fmt, inter, k), v.weight(fmt, inter, k)
    if fmt == "bf16":
        ops = RmsGateUpSiluSm100Op.schedule(x=x, norm_weight=n, gate_weight=g, up_weight=u, y=y)
    else:
        ops = RmsGateUpSiluNvfp4Sm120Op.schedule(x=x, norm_weight=n, gate_packed=g.packed, gate_scales=g.scales, up_packed=u.packed,
                                                 up_scales=u.scales, group_size=g.group_size, global_scale=g.global_scale,
                                                 up_global_scale=u.global_scale, y=y)
    assert equal_forms(ops, [y])[0].float().abs().sum() > 0


# (participants, CTAs a multiprocessor) of the launch on 148 multiprocessors
@pytest.mark.parametrize("batch,kv,heads,kv_heads,dim,splits,causal,m,form", [
    (1, 1, 8, 8, 64, 0, False, 1, (7, 2)), (1, 300, 32, 8, 64, 0, False, 1, (7, 2)), (2, 65, 16, 1, 128, 3, False, 1, (7, 2)),
    (3, 1930, 32, 4, 128, 0, False, 1, (7, 2)), (1, 2000, 8, 2, 64, 128, False, 1, (7, 2)), (1, 700, 8, 4, 128, 40, True, 16, (4, 3)),
    (2, 130, 4, 4, 64, 64, True, 5, (7, 2)), (8, 4096, 32, 8, 128, 0, False, 1, (7, 2)),
    # units of one to four pages in one, two and more waves of two, three and four CTAs a multiprocessor
    (13, 500, 8, 8, 64, 4, False, 1, (4, 3)), (11, 701, 32, 8, 64, 8, False, 1, (4, 3)), (16, 1931, 16, 8, 64, 8, False, 1, (4, 4)),
    (20, 250, 16, 8, 64, 2, True, 2, (4, 3)), (12, 380, 32, 8, 128, 4, False, 1, (4, 3)), (16, 129, 8, 8, 128, 4, False, 1, (7, 2))])
@pytest.mark.parametrize("fuse", [True, False])
def test_attention(batch, kv, heads, kv_heads, dim, splits, causal, m, form, fuse):
    v = Values(kv + dim)
    q, o = v(batch, m, heads, dim), torch.zeros(batch, m, heads, dim, dtype=BF, device="cuda")
    k, vv = v(batch, kv + 3, kv_heads, dim)[:, :kv], v(batch, kv, kv_heads, dim)
    ops, _ = flash_decoding_schedule(q, k, vv, o, num_splits=splits, causal=causal, kv_group_size=heads // kv_heads)
    lse = ops[1].tensor_refs["lse"]
    assert equal_forms(ops, [o, lse], attention=form, fuse=fuse)[0].float().abs().sum() > 0


# every kernel with the fused q/k norm; the new token in the first page, a middle one and the last
@pytest.mark.parametrize("batch,kv,heads,kv_heads,dim,splits,new,form", [
    (2, 300, 32, 8, 64, 0, 299, (7, 2)), (13, 500, 8, 8, 64, 4, 0, (4, 3)), (16, 1931, 16, 8, 64, 8, 1000, (4, 4)),
    (3, 1930, 32, 4, 128, 0, 1929, (7, 2)), (12, 380, 32, 8, 128, 4, 190, (4, 3))])
def test_attention_that_normalises(batch, kv, heads, kv_heads, dim, splits, new, form):
    v = Values(kv + dim)
    q, o = v(batch, 1, heads, dim), torch.zeros(batch, 1, heads, dim, dtype=BF, device="cuda")
    k, vv = v(batch, kv, kv_heads, dim), v(batch, kv, kv_heads, dim)
    norm = dict(q_weight=1 + v(dim, std=0.02), k_weight=1 + v(dim, std=0.02), cos=v(dim // 2), sin=v(dim // 2), new_token=new)
    ops, _ = flash_decoding_schedule(q, k, vv, o, num_splits=splits, kv_group_size=heads // kv_heads, qk_norm=norm)
    assert equal_forms(ops, [o, k], attention=form)[0].float().abs().sum() > 0


def layer_weights(v, fmt, hidden, inter, heads, kv_heads, dim, kv):
    w = {"cos": v(kv, dim // 2), "sin": v(kv, dim // 2), "layer.0.attn_norm": 1 + v(hidden, std=0.02), "layer.0.mlp_norm": 1 + v(hidden, std=0.02)}
    if fmt != "bf16":
        w["layer.0.q_norm"], w["layer.0.k_norm"] = 1 + v(dim, std=0.02), 1 + v(dim, std=0.02)
    for name, o, i in (("q", heads * dim, hidden), ("k", kv_heads * dim, hidden), ("v", kv_heads * dim, hidden), ("o", hidden, heads * dim),
                       ("gate", inter, hidden), ("up", inter, hidden), ("down", hidden, inter)):
        p = v.weight(fmt, o, i)
        if fmt == "bf16":
            w[f"layer.0.W_{name}"] = p
        else:
            w[f"layer.0.W_{name}.packed"], w[f"layer.0.W_{name}.scales"], w[f"layer.0.W_{name}.global_scale"] = p.packed, p.scales, float(p.global_scale)
    return w


# a whole layer: rows appended to the cache in the launch before the attention that reads them, whose other pages are
# fetched before that launch has finished; 16 rows: the down projection's K blocks side by side
@pytest.mark.parametrize("fmt,batch,seq,kv,pos", [("bf16", 1, 1, 700, 699), ("bf16", 3, 1, 130, 64), ("bf16", 2, 3, 70, 61), ("bf16", 16, 1, 300, 250),
                                                  ("nvfp4", 1, 1, 1000, 999), ("nvfp4", 8, 1, 66, 32), ("nvfp4", 2, 1, 40, 0)])
@pytest.mark.parametrize("moving", [False, True])
def test_layer(fmt, batch, seq, kv, pos, moving):
    if moving and seq > 1:
        pytest.skip("a moving position takes one token a sequence")
    hidden, inter, heads, kv_heads, dim = (2048, 8192, 16, 4, 64) if fmt == "bf16" else (2048, 6144, 8, 2, 128)
    v = Values(batch + kv)
    w = layer_weights(v, fmt, hidden, inter, heads, kv_heads, dim, kv)
    z = lambda n: torch.zeros(batch, seq, n, dtype=BF, device="cuda")      # noqa: E731
    kc, vc = v(batch, kv, kv_heads, dim), v(batch, kv, kv_heads, dim)
    x, r, xo, ro, q, at, h = v(batch, seq, hidden), v(batch, seq, hidden), z(hidden), z(hidden), z(heads * dim), z(heads * dim), z(inter)
    kw = dict(layer_idx=0, batch=batch, seq_len=seq, weights=w, k_cache=kc, v_cache=vc, x_in=x, residual_in=r, x_out=xo, residual_out=ro,
              q_buf=q, attn_out_buf=at, mlp_h_buf=h, eps=1e-5, num_q_heads=heads, num_kv_heads=kv_heads, head_dim=dim)
    config = {}
    if moving:
        config["position"] = torch.tensor([pos], dtype=torch.int32, device="cuda")
        kw.update(cache_pos=0, dynamic_position=True)
    else:
        kw["cache_pos"] = pos
    if fmt == "bf16":
        ops = schedule_decode_layer_sm100(hidden_size=hidden, intermediate_size=inter, **kw).ops
    else:
        ops = schedule_decode_layer_nvfp4_sm100(**kw).ops
    assert equal_forms(ops, [xo, ro, q, at, h, kc, vc], launches=5, **config)[0].float().abs().sum() > 0


# appends to one cache, to sequences one by one at positions of their own, to heads of a head-major cache: rows that lie somewhere
# else than token `position` of sequence 0 are waited for as well
@pytest.mark.parametrize("case", ["V alone", "K alone", "a later sequence", "sequences one by one", "later heads", "heads one by one"])
@pytest.mark.parametrize("heads_first", [False, True])
def test_appends_to_part_of_the_caches(case, heads_first):
    hidden, heads, kv_heads, dim, batch, kv, pos = 2048, 16, 4, 64, 3, 700, 699
    v = Values(len(case))
    caches = v(2, batch, kv_heads, kv, dim).transpose(2, 3) if heads_first else v(2, batch, kv, kv_heads, dim)
    k, vc = caches[0], caches[1]
    x, r, n = v(batch, 1, hidden), v(batch, 1, hidden), 1 + v(hidden, std=0.02)
    cos, sin, w = v(1, dim // 2), v(1, dim // 2), v(kv_heads * dim, hidden, std=0.05)
    q, o = torch.zeros(batch, 1, heads * dim, dtype=BF, device="cuda"), torch.zeros(batch, 1, heads, dim, dtype=BF, device="cuda")
    both = ((RmsKMatvecRopeCacheSm100Op, k), (RmsVMatvecCacheSm100Op, vc))
    append = {"V alone": [(*both[1], 0, pos)], "K alone": [(*both[0], 0, pos)],
              "a later sequence": [(c, t[1:2], 1, pos) for c, t in both],
              "sequences one by one": [(c, t[b:b + 1], b, p) for b, p in enumerate((pos, 40, 300)) for c, t in both],
              "later heads": [(c, t[:, :, 2:], 0, pos) for c, t in both],
              "heads one by one": [(c, t[:, :, h:h + 1], 0, pos) for h in range(kv_heads) for c, t in both]}[case]
    ops = RmsQMatvecRopeSm100Op.schedule(x=x, residual_in=r, residual_out=torch.zeros_like(x), norm_weight=n, q=q, cos=cos, sin=sin,
                                         weight=v(heads * dim, hidden, std=0.05))
    for cls, cache, first, at in append:
        rows = slice(first, first + cache.shape[0])
        ops += cls.schedule(x=x[rows], residual_in=r[rows], norm_weight=n, weight=w[:cache.shape[2] * dim], cos=cos, sin=sin, dst_cache=cache,
                            cache_pos=at)
    ops += flash_decoding_schedule(q.view(batch, 1, heads, dim), k, vc, o, kv_group_size=heads // kv_heads)[0]
    assert equal_forms(ops, [o, q, caches], launches=2)[0].float().abs().sum() > 0


def test_a_position_outside_the_cache_runs_nothing():
    v = Values(5)
    w = layer_weights(v, "bf16", 512, 1024, 8, 2, 64, 64)
    z = lambda n: torch.zeros(1, 1, n, dtype=BF, device="cuda")      # noqa: E731
    kc, vc, pos = v(1, 64, 2, 64), v(1, 64, 2, 64), torch.tensor([64], dtype=torch.int32, device="cuda")
    before, xo = kc.clone(), z(512)
    ops = schedule_decode_layer_sm100(layer_idx=0, batch=1, seq_len=1, cache_pos=0, dynamic_position=True, weights=w, k_cache=kc, v_cache=vc,
                                      x_in=v(1, 1, 512), residual_in=z(512), x_out=xo, residual_out=z(512), q_buf=z(512),
                                      attn_out_buf=z(512), mlp_h_buf=z(1024), eps=1e-5, hidden_size=512, intermediate_size=1024,
                                      num_q_heads=8, num_kv_heads=2, head_dim=64).ops
    mk = Megakernel(ops, config=MegakernelConfig(position=pos)).compile()
    with pytest.raises(RuntimeError, match="position"):
        mk.run()
    assert torch.equal(kc, before) and not xo.any()
    pos.fill_(3)
    mk.run()
    assert xo.any()


def test_replaced_records_change_the_chain():
    v = Values(9)
    x, w, w2 = v(3, 1, 1024), v(64, 1024, std=0.02), v(64, 1024, std=0.02)
    y = torch.zeros(3, 1, 64, dtype=BF, device="cuda")
    mk = Megakernel(MatvecSm100Op.schedule(a=x, weight=w, y=y)).compile()
    other = Megakernel(MatvecSm100Op.schedule(a=x, weight=w2, y=y)).compile()
    other.run()
    want = y.clone()
    mk.run()
    assert not torch.equal(y, want)
    mk.update_op(0, other.native_ops[0])
    mk.run()
    assert torch.equal(y, want)


def dependent_products(ws, first, last):
    """Projections, each on the rows of the one before it: as many launches, one graph from eight on."""
    ops, x = [], first
    for w in ws:
        y = last if w is ws[-1] else torch.zeros_like(first)
        ops += MatvecSm100Op.schedule(a=x, weight=w, y=y)
        x = y
    return ops


@pytest.mark.parametrize("n", [7, 8, 20])
def test_long_chains(n):
    v = Values(n)
    y = torch.zeros(2, 1, 256, dtype=BF, device="cuda")
    ops = dependent_products([v(256, 256, std=0.08) for _ in range(n)], v(2, 1, 256), y)
    assert equal_forms(ops, [y], launches=n)[0].float().abs().sum() > 0


@pytest.mark.parametrize("captured", [False, True])
def test_replaced_records_change_a_long_chain(captured):
    v = Values(11)
    x, x2, y = v(2, 1, 256), v(2, 1, 256), torch.zeros(2, 1, 256, dtype=BF, device="cuda")
    ws = [v(256, 256, std=0.08) for _ in range(9)]
    ops = dependent_products(ws, x, y)
    mk = Megakernel(ops).compile()
    mk.run()
    old = y.clone()
    first_y = ops[0].tensor_refs["y"]
    other = Megakernel(MatvecSm100Op.schedule(a=x2, weight=ws[0], y=first_y)).compile()
    mk.update_op(0, other.native_ops[0])
    if captured:      # planned again while the caller's stream is captured
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            mk.run(sync=False)
        graph.replay()
    else:
        mk.run()
    torch.cuda.synchronize()
    want = torch.zeros_like(y)
    Megakernel(dependent_products(ws, x2, want), config=MegakernelConfig(single_launch=True)).compile().run()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and not torch.equal(y, old)


# every row class and number of warps: two dependent projections are two kernels (one would be the persistent kernel)
@pytest.mark.parametrize("fmt", ["bf16", "fp16", "nvfp4"])
@pytest.mark.parametrize("rows,k,out", [(1, 1024, 1024), (2, 4096, 4096), (8, 2048, 256), (8, 6144, 2048), (9, 1024, 6144), (16, 2048, 2048),
                                        (16, 1792, 512), (17, 1024, 1024), (32, 1024, 256)])
def test_every_row_class_has_its_kernel(fmt, rows, k, out):
    v = Values(rows + k)
    dtype = torch.float16 if fmt == "fp16" else BF
    x, y, z = v(rows, 1, k, dtype=dtype), *(torch.zeros(rows, 1, n, dtype=dtype, device="cuda") for n in (out, 64))
    ops = []
    for a, b, o, i in ((x, y, out, k), (y, z, 64, out)):
        w = v.weight(fmt, o, i)
        if fmt == "nvfp4":
            ops += MatvecNvfp4Sm120Op.schedule(a=a, weight_packed=w.packed, weight_scales=w.scales, group_size=w.group_size,
                                               global_scale=w.global_scale, y=b)
        else:
            ops += MatvecSm100Op.schedule(a=a, weight=w, y=b)
    assert equal_forms(ops, [y, z], launches=2)[1].float().abs().sum() > 0


# every kernel with the sum of K blocks: the blocks of a product in one launch; (activation rows, consumer warps) of its kernel
@pytest.mark.parametrize("fmt,rows,k,out,form", [
    ("bf16", 4, 28672, 520, (8, 16)), ("bf16", 12, 8192, 520, (16, 16)), ("bf16", 20, 4096, 520, (32, 8)),
    ("fp16", 4, 28672, 520, (8, 16)), ("fp16", 12, 8192, 520, (16, 16)), ("fp16", 20, 4096, 520, (32, 8)),
    ("nvfp4", 1, 4096, 520, (8, 16)), ("nvfp4", 4, 4096, 2400, (8, 8)), ("nvfp4", 12, 4096, 520, (16, 16)), ("nvfp4", 20, 4096, 520, (32, 8))])
def test_k_blocks_side_by_side(fmt, rows, k, out, form):
    v = Values(rows + k)
    dtype = torch.float16 if fmt == "fp16" else BF
    a, y, ops, step = v(rows, 1, k, dtype=dtype), torch.zeros(rows, 1, out, dtype=dtype, device="cuda"), [], k // 4
    for b in range(4):
        part, sums = a[..., b * step:(b + 1) * step], dict(residual_in=y, residual_out=y) if b else dict(y=y)
        w = v.weight(fmt, out, step)
        if fmt == "nvfp4":
            cls = MatvecResidualNvfp4Sm120Op if b else MatvecNvfp4Sm120Op
            ops += cls.schedule(a=part, weight_packed=w.packed, weight_scales=w.scales, group_size=16, global_scale=w.global_scale, **sums)
        else:
            ops += (MatvecResidualSm100Op if b else MatvecSm100Op).schedule(a=part, weight=w, **sums)
    launch, = Megakernel(ops, scheduler=OverlapTileScheduler()).launch_plan()
    assert launch["n_ops"] == 4 and (launch["rows"], launch["warps"]) == form
    assert equal_forms(ops, [y])[0].float().abs().sum() > 0


def test_no_token_is_fed_back_after_a_failed_launch():
    """The status and the abort flag that a wait which ran out leaves, written by the host: the last op leaves position,
    token and input row alone, the error is raised, and the next step runs."""
    hidden, nq, nkv, hd, inter, vocab, T, start = 512, 8, 2, 64, 1024, 1024, 128, 40
    v = Values(21)
    w = layer_weights(v, "bf16", hidden, inter, nq, nkv, hd, T)
    z = lambda n: torch.zeros(1, 1, n, dtype=BF, device="cuda")      # noqa: E731
    x_in, position = v(1, 1, hidden), torch.tensor([start], dtype=torch.int32, device="cuda")
    tv, ti = torch.zeros(1, 1, device="cuda"), torch.full((1, 1), 7, dtype=torch.int32, device="cuda")
    ops, _keep = schedule_decode_model_sm100(
        batch=1, cache_pos=0, weights=w, k_cache=[v(1, T, nkv, hd)], v_cache=[v(1, T, nkv, hd)], x_buffers=[z(hidden), z(hidden)],
        residual_buffers=[z(hidden), z(hidden)], q_buf=z(nq * hd), attn_out_buf=z(nq * hd), mlp_h_buf=z(inter),
        final_norm=1 + v(hidden, std=0.02), lm_head=v(vocab, hidden, std=0.05), top_values=tv, top_indices=ti, num_layers=1, x_in=x_in,
        residual_in=z(hidden), position=position, hidden_size=hidden, intermediate_size=inter, num_q_heads=nq, num_kv_heads=nkv, head_dim=hd)
    mk = Megakernel(ops, config=MegakernelConfig(position=position), scheduler=OverlapTileScheduler()).compile()
    assert mk.launches_per_run > 1
    before, at = x_in.clone(), -mk._workspace.data_ptr() % 256
    state = mk._workspace[at:at + 128].view(torch.int32)      # status[16], abort flag, ...
    state[0] = state[16] = 1
    with pytest.raises(RuntimeError, match="aborted"):
        mk.run()
    assert int(position) == start and int(ti) == 7 and torch.equal(x_in, before)
    mk.run()
    assert int(position) == start + 1 and not torch.equal(x_in, before)


class MovingLayer:
    """One layer with a position in its records; V lies in front of K.  `at(pos)`: its ops at a position, on the same buffers."""

    def __init__(self, batch=2, length=600, seed=21):
        self.hidden, self.inter, self.heads, self.kv_heads, self.dim = 2048, 4096, 16, 4, 64
        self.batch, v = batch, Values(seed)
        self.w = layer_weights(v, "bf16", self.hidden, self.inter, self.heads, self.kv_heads, self.dim, length)
        z = lambda n: torch.zeros(batch, 1, n, dtype=BF, device="cuda")      # noqa: E731
        self.caches, self.x, self.r = v(2, batch, length, self.kv_heads, self.dim), v(batch, 1, self.hidden), v(batch, 1, self.hidden)
        self.xo, self.ro, self.q, self.a, self.h = z(self.hidden), z(self.hidden), z(self.heads * self.dim), z(self.heads * self.dim), z(self.inter)
        self.outs = [self.xo, self.ro, self.q, self.a, self.h, self.caches]
        self.start = [t.clone() for t in self.outs]

    def at(self, pos):
        return schedule_decode_layer_sm100(
            layer_idx=0, batch=self.batch, seq_len=1, cache_pos=pos, weights=self.w, k_cache=self.caches[1], v_cache=self.caches[0], x_in=self.x,
            residual_in=self.r, x_out=self.xo, residual_out=self.ro, q_buf=self.q, attn_out_buf=self.a, mlp_h_buf=self.h, eps=1e-5,
            hidden_size=self.hidden, intermediate_size=self.inter, num_q_heads=self.heads, num_kv_heads=self.kv_heads, head_dim=self.dim,
            fa_num_splits=4).ops

    def after(self, step):
        for t, s in zip(self.outs, self.start):
            t.copy_(s)
        step()
        torch.cuda.synchronize()
        return [t.clone() for t in self.outs]


def same_bytes(a, b):
    return all(torch.equal(p.view(torch.uint8), q.view(torch.uint8)) for p, q in zip(a, b))


def captured(mk):
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=stream):
        mk.run(sync=False, validate=False)
    return graph


# over a page's boundary and a split's, several at a time, and back: the rows that attention waits for move with the records
@pytest.mark.parametrize("single", [False, True])
def test_replaced_positions_move_a_captured_step(single):
    layer = MovingLayer()
    mk = Megakernel(layer.at(100), config=MegakernelConfig(single_launch=single), scheduler=OverlapTileScheduler()).compile()
    mk.run()
    graph = captured(mk)
    for pos in (101, 127, 128, 129, 300, 70, 511, 512, 599, 63):
        fresh = Megakernel(layer.at(pos), scheduler=OverlapTileScheduler()).compile()
        for i, record in enumerate(fresh.native_ops):
            mk.update_op(i, record)
        plan = mk.launch_plan()
        assert [(p["early"], p["wait_lo"], p["wait_hi"]) for p in plan if p["kind"] == 2] == ([] if single else [(1, pos, pos + 1)])
        want = layer.after(fresh.run)
        for step in (graph.replay, mk.run, graph.replay):
            assert same_bytes(layer.after(step), want), pos
        mk.wait()


# records that the captured launches cannot follow: K slices of another length; caches with the heads in front of the tokens
def test_replaced_sizes_and_strides_reach_a_captured_step():
    layer = MovingLayer()
    mk = Megakernel(layer.at(300), scheduler=OverlapTileScheduler()).compile()
    mk.run()
    graph = captured(mk)
    rows = layer.caches
    by_head = rows.new_zeros(2, layer.batch, layer.kv_heads, 600, layer.dim).transpose(2, 3)
    by_head.copy_(rows)
    other = MovingLayer(seed=22)
    for name in ("x", "r", "w", "xo", "ro", "q", "a", "h"):
        setattr(other, name, getattr(layer, name))
    other.caches = by_head
    layer.outs, layer.start = [*layer.outs, by_head], [*layer.start, by_head.clone()]
    counted = mk.launch_count()
    for at, config in ((layer.at, dict(native_kc=512)), (other.at, {}), (layer.at, {})):
        fresh = Megakernel(at(300), config=MegakernelConfig(single_launch=True, **config), scheduler=OverlapTileScheduler()).compile()
        for i, record in enumerate(fresh.native_ops):
            mk.update_op(i, record)
        want = layer.after(fresh.run)
        assert same_bytes(layer.after(graph.replay), want)
        assert same_bytes(layer.after(mk.run), want) and len(mk.launch_plan()) == 5
        again = captured(mk)
        assert same_bytes(layer.after(again.replay), want) and same_bytes(layer.after(graph.replay), want)
        mk.wait()
        counted += 4
        assert mk.launch_count() == counted


def test_two_threads_run_a_program_whose_record_was_replaced():
    v = Values(31)
    y = torch.zeros(2, 1, 256, dtype=BF, device="cuda")
    ops = dependent_products([v(256, 256, std=0.08) for _ in range(9)], v(2, 1, 256), y)
    mk = Megakernel(ops).compile()
    mk.run()
    want, rounds = y.clone(), 40
    records = [Megakernel(ops, config=MegakernelConfig(native_kc=kc)).native_ops for kc in (64, 1024)]   # (other launches each time)
    stream, errors = torch.cuda.Stream(), []

    def runs(gate):
        try:
            gate.wait(30)
            for _ in range(3):
                mk.run(stream=stream, sync=False, validate=False)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    for n in range(rounds):
        mk.update_op(n % 9, records[(n // 9) % 2][n % 9])
        y.zero_()
        torch.cuda.synchronize()
        gate = threading.Barrier(2)
        threads = [threading.Thread(target=runs, args=(gate,)) for _ in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join(60)
        mk.wait()
        assert not errors and (y.float() - want.float()).abs().max() <= 0.02 * want.float().abs().max()
    assert mk.launch_count() == 1 + 6 * rounds
