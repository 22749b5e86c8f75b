"""What a chain of kernels does where a run of it cannot do all: positions outside the caches, launches behind one that failed, ops behind
the one that moves the position; and records that only some of a launch's ops carry."""

import pytest
import torch

from machete_b200.kernels.attention import flash_decoding_schedule
from machete_b200.kernels.decode_matvec import (RmsKMatvecRopeCacheSm100Op, RmsQMatvecRopeSm100Op, RmsVMatvecCacheSm100Op,
                                                schedule_decode_layer_sm100)
from machete_b200.kernels.decode_matvec.top1 import schedule_final_top1_sm100
from machete_b200.megakernel import Megakernel, MegakernelConfig, OverlapTileScheduler

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def values(*shape, std=1.0, seed=3):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed + sum(shape))) * std).to(BF).cuda()


def positions(*at):
    return torch.tensor(at, dtype=torch.int32, device="cuda")


class Layer:
    """A layer that follows a device-resident position; every buffer that it writes holds 7 before a run."""

    def __init__(self, length=64, batch=2):
        hidden, inter, dim = 512, 1024, 64
        w = {"cos": values(length, 32), "sin": values(length, 32), "layer.0.attn_norm": values(hidden), "layer.0.mlp_norm": values(hidden)}
        for name, o, i in (("q", hidden, hidden), ("k", 128, hidden), ("v", 128, hidden), ("o", hidden, hidden), ("gate", inter, hidden),
                           ("up", inter, hidden), ("down", hidden, inter)):
            w[f"layer.0.W_{name}"] = values(o, i, std=0.02)
        z = lambda n: torch.empty(batch, 1, n, dtype=BF, device="cuda")      # noqa: E731
        self.caches, self.xo, self.ro, self.q, self.a, self.h = values(2, batch, length, 2, dim), z(hidden), z(hidden), z(hidden), z(hidden), z(inter)
        self.outs = [self.xo, self.ro, self.q, self.a, self.h]
        self.caches_before = self.caches.clone()
        self.ops = schedule_decode_layer_sm100(
            layer_idx=0, batch=batch, seq_len=1, cache_pos=0, dynamic_position=True, weights=w, k_cache=self.caches[0], v_cache=self.caches[1],
            x_in=values(batch, 1, hidden), residual_in=values(batch, 1, hidden, seed=5), x_out=self.xo, residual_out=self.ro, q_buf=self.q,
            attn_out_buf=self.a, mlp_h_buf=self.h, eps=1e-5, hidden_size=hidden, intermediate_size=inter, num_q_heads=8, num_kv_heads=2,
            head_dim=dim).ops

    def clear(self):
        for t in self.outs:
            t.fill_(7)
        self.caches.copy_(self.caches_before)

    def untouched(self):
        return all(bool((t == 7).all()) for t in self.outs) and torch.equal(self.caches, self.caches_before)


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("at", [(64,), (-1,), (3, 64)])
def test_a_position_outside_the_cache_writes_nothing_and_is_counted(at, single):
    layer, pos = Layer(), positions(*at)
    mk = Megakernel(layer.ops, config=MegakernelConfig(position=pos, single_launch=single)).compile()
    layer.clear()
    with pytest.raises(RuntimeError, match="position"):
        mk.run()
    assert layer.untouched() and mk.launch_count() == 1
    pos.fill_(3)
    mk.run()
    assert not any(bool((t == 7).all()) for t in layer.outs) and mk.launch_count() == 2


def test_attention_alone_counts_a_run_that_found_a_bad_position():
    q, o, k, pos = values(1, 1, 8, 64), torch.full((1, 1, 8, 64), 7, dtype=BF, device="cuda"), values(1, 64, 2, 64), positions(64)
    ops = flash_decoding_schedule(q, k, k.clone(), o, kv_group_size=4, dynamic_len=True)[0]
    mk = Megakernel(ops, config=MegakernelConfig(position=pos)).compile()
    with pytest.raises(RuntimeError, match="position"):
        mk.run()
    assert mk.launch_count() == 1 and bool((o == 7).all())


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("start", [5, 15])
def test_an_op_behind_the_feedback_sees_the_position_that_the_run_began_with(start, single):
    hidden, vocab, length, dim = 256, 512, 16, 64
    x, r, n, emb, pos = values(1, 1, hidden), values(1, 1, hidden, seed=4), values(hidden), values(vocab, hidden, std=0.05), positions(start)
    tv, ti = torch.zeros(1, 1, device="cuda"), torch.zeros(1, 1, dtype=torch.int32, device="cuda")
    ops = schedule_final_top1_sm100(x=x, residual_in=r, final_norm=n, lm_head=emb, top_values=tv, top_indices=ti, seq_len=1,
                                    feedback=dict(embedding=emb, x_in=x, position=pos))
    ops = list(ops[0] if isinstance(ops, tuple) else ops)
    cache = torch.full((1, length, 2, dim), 7, dtype=BF, device="cuda")
    ops += RmsVMatvecCacheSm100Op.schedule(x=x, residual_in=r, norm_weight=n, weight=values(2 * dim, hidden, std=0.05), cos=values(1, 32),
                                           sin=values(1, 32), dst_cache=cache, dynamic_pos=True)
    mk = Megakernel(ops, config=MegakernelConfig(position=pos, single_launch=single), scheduler=OverlapTileScheduler()).compile()
    mk.run()
    written = [t for t in range(length) if not bool((cache[0, t] == 7).all())]
    assert written == [start] and int(pos.item()) == start + 1


@pytest.mark.parametrize("single", [False, True])
def test_tokens_of_a_sequence_share_its_position(single):
    hidden, length, dim = 256, 32, 64
    x, r, n, pos = values(2, 3, hidden), values(2, 3, hidden, seed=4), values(hidden), positions(4, 20)
    cache = torch.full((2, length, 2, dim), 7, dtype=BF, device="cuda")
    ops = RmsVMatvecCacheSm100Op.schedule(x=x, residual_in=r, norm_weight=n, weight=values(2 * dim, hidden, std=0.05), cos=values(3, 32),
                                          sin=values(3, 32), dst_cache=cache, dynamic_pos=True)
    Megakernel(ops, config=MegakernelConfig(position=pos, single_launch=single)).run()
    written = [[t for t in range(length) if not bool((cache[b, t] == 7).all())] for b in range(2)]
    assert written == [[4, 5, 6], [20, 21, 22]]


@pytest.mark.parametrize("single", [False, True])
def test_every_op_of_a_group_leaves_its_residual(single):
    hidden, dim = 256, 64
    x, r, n, cos, sin = values(2, 1, hidden), values(2, 1, hidden, seed=4), values(hidden), values(1, 32), values(1, 32)
    sums, q = torch.full((2, 2, 1, hidden), 7, dtype=BF, device="cuda"), torch.zeros(2, 2, 1, 2 * dim, dtype=BF, device="cuda")
    cache = torch.zeros(2, 8, 2, dim, dtype=BF, device="cuda")
    common = dict(x=x, residual_in=r, norm_weight=n, cos=cos, sin=sin)
    ops = RmsVMatvecCacheSm100Op.schedule(weight=values(2 * dim, hidden), dst_cache=cache, cache_pos=3, **common)
    for i in range(2):
        ops += RmsQMatvecRopeSm100Op.schedule(weight=values(2 * dim, hidden), residual_out=sums[i], q=q[i], **common)
    Megakernel(ops, config=MegakernelConfig(single_launch=single), scheduler=OverlapTileScheduler()).run()
    want = (x.float() + r.float()).to(BF)
    assert torch.equal(sums[0], want) and torch.equal(sums[1], want)


def test_nothing_runs_behind_a_launch_that_failed():
    layer, pos = Layer(), positions(9)
    mk = Megakernel(layer.ops, config=MegakernelConfig(position=pos)).compile()
    layer.clear()
    # a wait that ran out, as its launch leaves it: the status code and the abort flag (word 16) of the workspace
    state = mk._workspace[(-mk._workspace.data_ptr()) % 256:][:256].view(torch.int32)
    state[0], state[16] = 2, 1
    with pytest.raises(RuntimeError, match="aborted"):
        mk.run()
    assert layer.untouched() and mk.launch_count() == 1
    mk.run()
    assert not any(bool((t == 7).all()) for t in layer.outs) and mk.launch_count() == 2
