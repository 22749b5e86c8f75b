"""The launches of a chain as the library plans them (CPU): which cache pages an attention launch may load before the launch that
appends to the caches has finished."""

import numpy as np
import pytest
import torch

from machete_b200 import _native as N
from machete_b200.kernels.attention import flash_decoding_schedule
from machete_b200.kernels.decode_matvec import (MatvecSm100Op, RmsKMatvecRopeCacheSm100Op, RmsQMatvecRopeSm100Op, RmsVMatvecCacheSm100Op,
                                                schedule_decode_layer_sm100)
from machete_b200.megakernel import Megakernel, MegakernelConfig, OverlapTileScheduler

BF = torch.bfloat16
HIDDEN, D, HKV, HEADS = 256, 64, 4, 8


def z(*shape):
    return torch.zeros(*shape, dtype=BF)


class Layer:
    """Q, K and V projections and the attention behind them; `append`: (which cache, its slice that an op writes, at which token)."""

    def __init__(self, k, v, append, batch, tokens, seq=1, dynamic=False):
        x, r, n = z(batch, seq, HIDDEN), z(batch, seq, HIDDEN), z(HIDDEN)
        q, o = z(batch, seq, HEADS * D), z(batch, seq, HEADS, D)
        cos, sin = z(seq, D // 2), z(seq, D // 2)
        self.ops = RmsQMatvecRopeSm100Op.schedule(x=x, residual_in=r, residual_out=z(batch, seq, HIDDEN), norm_weight=n, q=q,
                                                  weight=z(HEADS * D, HIDDEN), cos=cos, sin=sin)
        for cls, cache, first, at in append:
            rows = slice(first, first + cache.shape[0])
            self.ops += cls.schedule(x=x[rows], residual_in=r[rows], norm_weight=n, weight=z(cache.shape[2] * D, HIDDEN), cos=cos, sin=sin,
                                     dst_cache=cache, cache_pos=0 if dynamic else at, dynamic_pos=dynamic)
        window = slice(None) if dynamic else slice(0, tokens)
        self.ops += flash_decoding_schedule(q.view(batch, seq, HEADS, D), k[:, window], v[:, window], o, kv_group_size=HEADS // HKV,
                                            num_splits=2, dynamic_len=dynamic)[0]
        config = MegakernelConfig(position=torch.zeros(1, dtype=torch.int32)) if dynamic else MegakernelConfig()
        self.mk = Megakernel(self.ops, config=config, scheduler=OverlapTileScheduler())
        plan = self.mk.launch_plan()
        assert [p["kind"] for p in plan][-1] == N.LAUNCH_ATTENTION and len(plan) >= 2
        self.attention = plan[-1]

    def tokens_written(self, pos):
        """From the records alone: tokens of K or V, as the attention op addresses them, of which some value is written before."""
        at = self.mk.native_ops[self.attention["first_op"]]
        here = np.arange(at.i[N.AT_D])
        written = []
        for op in self.mk.native_ops[:self.attention["first_op"]]:
            b, s = np.meshgrid(np.arange(op.i[N.MV_M] // op.i[N.MV_S]), np.arange(op.i[N.MV_S]), indexing="ij")
            token = s + op.i[N.MV_POS] + (pos if op.i.get(N.MV_DYNPOS, 0) & 2 else 0)
            rows = np.arange(op.i[N.MV_O])
            value = (rows // op.i[N.MV_HD]) * op.s[N.MV_S_O_H] + rows % op.i[N.MV_HD]
            row = b * op.s[N.MV_S_O_B] + token * op.s[N.MV_S_O_S]
            written.append(op.p[N.MV_P_OUT] + 2 * (row[..., None] + value).reshape(-1))
        written = np.concatenate(written)
        tokens = set()
        for base, s0 in ((N.AT_P_K, N.AT_S_K_B), (N.AT_P_V, N.AT_S_V_B)):
            for b in range(at.i[N.AT_B]):
                for n in range(at.i[N.AT_N]):
                    row = at.p[base] + 2 * (b * at.s[s0] + n * at.s[s0 + 1])
                    values = row + 2 * (np.arange(at.i[N.AT_HKV])[:, None] * at.s[s0 + 2] + here)
                    if np.isin(values, written).any():
                        tokens.add(n)
        return tokens

    def check(self, pos=0):
        """Every token that is written is waited for."""
        launch = self.attention
        if not launch["early"]:
            return
        add = pos if launch["wait_dyn"] else 0
        for n in self.tokens_written(pos):
            assert launch["wait_lo"] + add <= n < launch["wait_hi"] + add, (n, launch)


K, V = RmsKMatvecRopeCacheSm100Op, RmsVMatvecCacheSm100Op
T = 128
LAYOUTS = {
    "separate": lambda b: (z(b, T, HKV, D), z(b, T, HKV, D)),
    "one buffer": lambda b: tuple(z(2, b, T, HKV, D)),
    "V before K": lambda b: tuple(reversed(tuple(z(2, b, T, HKV, D)))),
    "K and V of a token together": lambda b: tuple(z(b, T, 2, HKV, D).unbind(2)),
    "heads of a token together": lambda b: tuple(z(b, T, HKV, 2, D).unbind(3)),
    "heads first": lambda b: tuple(t.transpose(1, 2) for t in z(2, b, HKV, T, D)),
    "tokens first": lambda b: tuple(t.transpose(0, 1) for t in z(2, T, b, HKV, D)),
    "padded rows": lambda b: tuple(t[:, :, :HKV] for t in z(2, b, T, HKV + 1, D)),
}


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("dynamic", [False, True])
def test_the_usual_layer_loads_early_but_for_the_new_rows(layout, dynamic):
    for batch, seq, pos in ((1, 1, 0), (1, 1, 77), (3, 1, 100), (2, 1, T - 1), (2, 3, 61)):
        if dynamic and seq > 1:
            continue
        k, v = LAYOUTS[layout](batch)
        layer = Layer(k, v, [(K, k, 0, pos), (V, v, 0, pos)], batch, pos + seq, seq, dynamic)
        want = dict(early=1, wait_dyn=1, wait_lo=0, wait_hi=1) if dynamic else dict(early=1, wait_dyn=0, wait_lo=pos, wait_hi=pos + seq)
        assert {name: layer.attention[name] for name in want} == want
        layer.check(pos)


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("dynamic", [False, True])
@pytest.mark.parametrize("case", ["V alone", "K alone", "a later sequence", "sequences one by one", "later heads", "heads one by one",
                                  "all but the first sequence", "K into V's rows"])
def test_rows_of_part_of_the_caches_are_waited_for(layout, dynamic, case):
    batch, pos = 3, 100
    k, v = LAYOUTS[layout](batch)
    at = {"V alone": [(V, v, 0, pos)], "K alone": [(K, k, 0, pos)],
          "a later sequence": [(K, k[1:2], 1, pos), (V, v[1:2], 1, pos)],
          "sequences one by one": [(c, t[b:b + 1], b, p) for b, p in enumerate((pos, 40, 63)) for c, t in ((K, k), (V, v))],
          "later heads": [(K, k[:, :, 2:], 0, pos), (V, v[:, :, 2:], 0, pos)],
          "heads one by one": [(c, t[:, :, h:h + 1], 0, pos) for h in range(HKV) for c, t in ((K, k), (V, v))],
          "all but the first sequence": [(K, k[1:], 1, pos), (V, v[1:], 1, pos)],
          "K into V's rows": [(K, v, 0, 17), (V, v, 0, pos)]}[case]
    layer = Layer(k, v, at, batch, pos + 1, 1, dynamic)
    assert layer.tokens_written(pos)
    layer.check(pos)
    if case in ("V alone", "K alone"):
        assert layer.attention["early"]      # (the gain stays)


def test_views_that_overlap_load_nothing_early():
    flat = z(4 * T * HKV * D)
    row = HKV * D
    same = z(2, T, HKV, D)
    sliding = flat.as_strided((2, T, HKV, D), (8 * row, row, D, 1))             # sequence 1 is sequence 0, 8 tokens on
    shifted = flat.as_strided((2, T, HKV, D), (T * row, row, D, 1), 4 * row)    # V is K, 4 tokens on
    plain = flat.as_strided((2, T, HKV, D), (T * row, row, D, 1))
    for k, v, early in ((same, same, 1), (sliding, z(2, T, HKV, D), 0), (plain, shifted, 0)):
        layer = Layer(k, v, [(K, k, 0, 50), (V, v, 0, 50)], 2, 51)
        assert layer.attention["early"] == early
        layer.check()


def test_the_layers_of_a_model_load_early():
    hidden, inter = 512, 1024
    w = {"cos": z(T, 32), "sin": z(T, 32), "layer.0.attn_norm": z(hidden), "layer.0.mlp_norm": z(hidden)}
    for name, o, i in (("q", 512, hidden), ("k", 128, hidden), ("v", 128, hidden), ("o", hidden, 512), ("gate", inter, hidden), ("up", inter, hidden),
                       ("down", hidden, inter)):
        w[f"layer.0.W_{name}"] = z(o, i)
    caches = z(2, 3, 2, T, 2, 64)       # K and V, layers
    ops = schedule_decode_layer_sm100(layer_idx=0, batch=2, seq_len=1, cache_pos=90, weights=w, k_cache=caches[0, 1], v_cache=caches[1, 1],
                                      x_in=z(2, 1, hidden), residual_in=z(2, 1, hidden), x_out=z(2, 1, hidden), residual_out=z(2, 1, hidden),
                                      q_buf=z(2, 1, 512), attn_out_buf=z(2, 1, 512), mlp_h_buf=z(2, 1, inter), eps=1e-5, hidden_size=hidden,
                                      intermediate_size=inter, num_q_heads=8, num_kv_heads=2, head_dim=64).ops
    plan = Megakernel(ops, scheduler=OverlapTileScheduler()).launch_plan()
    assert [p["kind"] for p in plan] == [N.LAUNCH_MATVEC, N.LAUNCH_ATTENTION] + 3 * [N.LAUNCH_MATVEC]
    assert [p["early"] for p in plan] == [0, 1, 1, 1, 1]
    assert (plan[1]["wait_lo"], plan[1]["wait_hi"], plan[1]["wait_dyn"]) == (90, 91, 0)


@pytest.mark.parametrize("seq", [1, 3])
def test_a_position_is_inside_only_if_every_token_of_the_step_is(seq):
    x, cache = z(2, seq, HIDDEN), z(2, T, HKV, D)
    ops = RmsVMatvecCacheSm100Op.schedule(x=x, residual_in=x.clone(), norm_weight=z(HIDDEN), weight=z(HKV * D, HIDDEN), cos=z(seq, D // 2),
                                          sin=z(seq, D // 2), dst_cache=cache, dynamic_pos=True)
    mk = Megakernel(ops, config=MegakernelConfig(position=torch.zeros(2, dtype=torch.int32)))
    assert mk._tables()[0].position_limit == T - seq + 1


# eight dense rows that leave a ring of at most four pages, and of more, by their length and by the length of a page
@pytest.mark.parametrize("rows,k,out,page_k,warps,ring", [(3, 14336, 4096, 1024, 8, 3), (8, 4608, 8192, 1024, 8, 4), (8, 3072, 8192, 1024, 16, 5),
                                                          (3, 14336, 4096, 512, 16, 7), (1, 4096, 14336, 1024, 8, 6), (16, 1024, 1024, 1024, 16, 1),
                                                          (17, 1024, 4096, 1024, 8, 2)])
def test_warps_follow_the_ring(rows, k, out, page_k, warps, ring):
    ops = MatvecSm100Op.schedule(a=z(1, rows, k), weight=z(out, k), y=z(1, rows, out))
    launch, = Megakernel(ops, config=MegakernelConfig(native_kc=page_k)).launch_plan()
    assert (launch["warps"], launch["stages"]) == (warps, ring)
