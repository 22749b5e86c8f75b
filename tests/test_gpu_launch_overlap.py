"""Launches overlap their set-up with the kernel before them in the stream: every kernel must see all that the one
before it wrote, and must not write what that one still reads.  Decode programs, prompt attention, both GEMM kernels
and torch's own kernels run through each other's buffers, back to back and as a captured graph, against the same
chain with a synchronise after every step.  Everything here is deterministic, so the bits have to be equal."""

import pytest
import torch

from machete_b200.kernels.attention import flash_prefill
from machete_b200.kernels.decode_matvec import MatvecSm100Op
from machete_b200.kernels.gemm import gemm_sm100
from machete_b200.megakernel import Megakernel

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
HIDDEN, HEADS, KV_HEADS = 512, 16, 4


def _weight(g, rows, cols):
    return (torch.randn(rows, cols, generator=g, device="cuda") * cols ** -0.5).to(BF)


class _Chain:
    """x -> q, k, v -> attention -> projection + x -> first rows through two decode programs -> x of the next round.
    The two decode programs exchange two small buffers, so the second overwrites what the first reads."""

    def __init__(self, rows, head_dim, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.rows, self.d, self.g = rows, head_dim, g
        q_dim, kv_dim = HEADS * head_dim, KV_HEADS * head_dim
        self.wq, self.wk, self.wv = _weight(g, q_dim, HIDDEN), _weight(g, kv_dim, HIDDEN), _weight(g, kv_dim, HIDDEN)
        self.wo = _weight(g, HIDDEN, q_dim)
        self.x = torch.empty(1, rows, HIDDEN, dtype=BF, device="cuda")
        self.q, self.o = (torch.empty(1, rows, q_dim, dtype=BF, device="cuda") for _ in range(2))
        self.k, self.v = (torch.empty(1, rows, kv_dim, dtype=BF, device="cuda") for _ in range(2))
        self.y = torch.empty_like(self.x)
        self.a, self.b = (torch.empty(1, 8, HIDDEN, dtype=BF, device="cuda") for _ in range(2))
        w1, w2 = _weight(g, HIDDEN, HIDDEN), _weight(g, HIDDEN, HIDDEN)
        self.there = Megakernel(MatvecSm100Op.schedule(a=self.a, weight=w1, y=self.b)).compile()
        self.back = Megakernel(MatvecSm100Op.schedule(a=self.b, weight=w2, y=self.a)).compile()
        self.buffers = [self.q, self.k, self.v, self.o, self.y, self.a, self.b]

    def steps(self):
        n, d = self.rows, self.d

        def heads(t, h):
            return t.view(1, n, h, d)

        return [
            lambda: gemm_sm100(self.x, self.wq, self.q),
            lambda: gemm_sm100(self.x, self.wk, self.k),
            lambda: gemm_sm100(self.x, self.wv, self.v),
            lambda: flash_prefill(heads(self.q, HEADS), heads(self.k, KV_HEADS), heads(self.v, KV_HEADS),
                                  heads(self.o, HEADS), causal=True, layout="bmhd"),
            lambda: gemm_sm100(self.o, self.wo, self.y),
            lambda: self.y.add_(self.x),
            lambda: self.a.copy_(self.y[:, :8]),
            lambda: self.there.run(sync=False),
            lambda: self.back.run(sync=False),
            lambda: self.there.run(sync=False),
            lambda: self.y[:, :8].copy_(self.b),
            lambda: self.x.copy_(self.y).mul_(0.7),
            lambda: gemm_sm100(self.x, self.wo.view(-1, HIDDEN)[:HIDDEN], self.y),
        ]

    def start(self, seed):
        for t in self.buffers:
            t.fill_(float("nan"))
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.x.copy_(torch.randn(self.x.shape, generator=g, device="cuda").to(BF))
        torch.cuda.synchronize()

    def state(self):
        torch.cuda.synchronize()
        return [t.clone() for t in (self.x, *self.buffers)]


@pytest.mark.parametrize("rows,head_dim", [(96, 64), (320, 128), (1100, 64), (2100, 128)])
def test_a_chain_of_kernels_sees_what_the_one_before_it_wrote(rows, head_dim):
    c = _Chain(rows, head_dim, rows)
    want = {}
    for seed in range(3):
        c.start(seed)
        for _ in range(3):
            for step in c.steps():
                step()
                torch.cuda.synchronize()
        want[seed] = c.state()
        assert all(bool(torch.isfinite(t).all()) for t in want[seed])
    for seed in range(3):                                     # other inputs each time: nothing old is right by chance
        c.start(seed)
        for _ in range(3):
            for step in c.steps():
                step()
        assert all(torch.equal(p, q) for p, q in zip(c.state(), want[seed]))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(3):
            for step in c.steps():
                step()
    for seed in (2, 0, 1):
        c.start(seed)
        graph.replay()
        assert all(torch.equal(p, q) for p, q in zip(c.state(), want[seed]))
