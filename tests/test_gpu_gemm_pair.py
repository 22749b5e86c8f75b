"""Both tcgen05 GEMM kernels at the sizes where their cuts go wrong: one row, the edges of the 16-row granularity and
of a full tile, ragged columns and K, few tiles (K is split over a cluster) and many (persistent pairs that walk
several tiles each), odd column counts (no two-column stores), and every activation.

The bar of test_gpu_gemm_sm100.py: one bf16 rounding plus K * 2^-24 relative fp32 accumulation noise; silu adds a
relative 2^-9 for the exponential and the division."""

import ctypes

import pytest
import torch

from machete_b200 import _native as native
from machete_b200.kernels.gemm import gemm_pack_weight, gemm_sm100

pytestmark = pytest.mark.gpu
BF = torch.bfloat16

SHAPES = [(1, 256, 64), (15, 1000, 1000), (129, 257, 72), (160, 4096, 4096), (255, 512, 2048), (257, 300, 8192),
          (512, 4096, 512), (777, 1025, 1032), (1031, 5000, 328), (2049, 2304, 264), (96, 19000, 136),
          (1031, 14001, 328), (2049, 7000, 264)]


@pytest.mark.parametrize("M,N_out,K", SHAPES)
@pytest.mark.parametrize("activation", [None, "relu", "silu"])
def test_every_cut_against_fp64(M, N_out, K, activation):
    g = torch.Generator(device="cuda").manual_seed(M + N_out)
    a = torch.randn(M, K, generator=g, device="cuda").to(BF)
    b = (torch.randn(N_out, K, generator=g, device="cuda") * K ** -0.5).to(BF)
    want = a.double() @ b.double().t()
    noise = (a.double().abs() @ b.double().abs().t()) * K * 2.0 ** -24
    rounding = 2.0 ** -8
    if activation == "relu":
        want = want.clamp_min(0)
    elif activation == "silu":
        want, rounding = torch.nn.functional.silu(want), 2.0 ** -8 + 2.0 ** -9
        noise = noise * 1.1                                   # the slope of silu is below 1.1
    for weight in (b, gemm_pack_weight(b)) if K % 64 == 0 else (b,):
        c = torch.full((M, N_out), float("nan"), dtype=BF, device="cuda")
        gemm_sm100(a, weight, c, activation=activation, check_status=True)
        bad = ~((c.double() - want).abs() <= want.abs() * rounding + noise + 1e-30)
        assert not bool(bad.any()), f"{int(bad.sum())} of {bad.numel()} entries outside the bar"


def test_results_do_not_depend_on_the_launch_before():
    """Launches overlap their set-up with the kernel before them: a product that reads the one before it sees all of
    it.  Every chain starts from another x0 and from buffers of NaN, so that nothing an earlier chain left is right;
    long and short products alternate, so that a launch really is placed early."""
    g = torch.Generator(device="cuda").manual_seed(3)
    sizes = [512, 512, 4096, 512, 256, 8192, 512]
    w = [(torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).to(BF) for k, n in zip(sizes, sizes[1:])]
    x0 = [torch.randn(320, 512, generator=g, device="cuda").to(BF) for _ in range(4)]
    bufs = [torch.empty(320, n, dtype=BF, device="cuda") for n in sizes[1:]]

    def chain(x, wait):
        for t in bufs:
            t.fill_(float("nan"))
        torch.cuda.synchronize()
        for i in range(len(w)):
            x = gemm_sm100(x, w[i], bufs[i])
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return x.clone()

    want = [chain(x, True) for x in x0]
    assert all(bool(torch.isfinite(t).all()) for t in want) and not torch.equal(want[0], want[1])
    for _ in range(3):
        for x, y in zip(x0, want):
            assert torch.equal(chain(x, False), y)


def _plan(M, N_out, K, ldb=None):
    out = (ctypes.c_int32 * 4)()
    assert native.lib().mk_gemm_bf16_plan(M, N_out, K, ldb or K, out) == 0
    return tuple(out)                                         # pair kernel, split, rows per tile, tiles


def test_the_shapes_above_take_every_cut():
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    cuts = [_plan(*shape) for shape in SHAPES]
    assert {0, 1} <= {split > 1 for pair, split, _, _ in cuts if pair} and any(split > 1 for pair, split, _, _ in cuts if not pair)
    assert any(split == 1 for pair, split, _, _ in cuts if not pair)
    # a pair's two accumulators are waited for, and change their parity, from its third tile on
    assert sum(tiles > 3 * pairs for pair, split, _, tiles in cuts if pair and split == 1) >= 2


@pytest.mark.parametrize("M,N_out,K,split", [(320, 1000, 4096, True), (1031, 9001, 328, False)])
@pytest.mark.parametrize("pad", [1, 2, 4, 32])
def test_pair_kernel_on_strided_operands(M, N_out, K, split, pad):
    """Rows of C that allow four, two or no columns at once (an even, an odd and a 4-byte-aligned row stride), A and B
    cut from wider buffers; nothing beside C's columns is written."""
    pair, parts, _, _ = _plan(M, N_out, K, K + 8)
    assert pair and (parts > 1) == split
    g = torch.Generator(device="cuda").manual_seed(pad)
    a = torch.randn(M, K + 16, generator=g, device="cuda").to(BF)[:, :K]
    b = (torch.randn(N_out, K + 8, generator=g, device="cuda") * K ** -0.5).to(BF)[:, :K]
    whole = torch.full((M, N_out + pad), 7.0, dtype=BF, device="cuda")
    c = whole[:, :N_out]
    gemm_sm100(a, b, c, check_status=True)
    want = a.double() @ b.double().t()
    bar = want.abs() * 2.0 ** -8 + (a.double().abs() @ b.double().abs().t()) * K * 2.0 ** -24
    assert bool(((c.double() - want).abs() <= bar).all())
    assert bool((whole[:, N_out:] == 7.0).all())
    if pad == 32:                                             # leading dimensions over equally spaced rows
        lead = a[:M // 2 * 2].reshape(2, M // 2, K)
        out = torch.empty(2, M // 2, N_out, dtype=BF, device="cuda")
        gemm_sm100(lead, b, out, check_status=True)
        assert bool(((out.view(-1, N_out).double() - want[:M // 2 * 2]).abs() <= bar[:M // 2 * 2]).all())


@pytest.mark.parametrize("M,N_out,K", [(66, 8616, 5576), (48, 8160, 5352), (53, 8608, 9360), (76, 9240, 3256),
                                       (59, 5392, 10760), (91, 5128, 1544)])
def test_few_rows_use_the_device(M, N_out, K):
    """Where the weight's bytes are the bound, or nearly, a product must not settle for the fewest CTAs."""
    pair, split, _, tiles = _plan(M, N_out, K)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (2 if pair else 1) * split * tiles >= 0.6 * sms


@pytest.mark.parametrize("K,N_out", [(256, 264), (2048, 512)])
def test_one_row_of_any_stride(K, N_out):
    g = torch.Generator(device="cuda").manual_seed(K)
    b = (torch.randn(N_out, K, generator=g, device="cuda") * K ** -0.5).to(BF)
    x = torch.randn(K, generator=g, device="cuda").to(BF)
    odd = torch.zeros(5, K + 3, dtype=BF, device="cuda")
    odd[0, :K] = x
    want = x.double()[None] @ b.double().t()
    bar = want.abs() * 2.0 ** -8 + (x.double().abs()[None] @ b.double().abs().t()) * K * 2.0 ** -24
    for a in (x.view(K, 1).t(), x.as_strided((1, K), (0, 1)), odd[0:1, :K]):
        for c in (torch.zeros(1, N_out, dtype=BF, device="cuda"), torch.zeros(N_out, 1, dtype=BF, device="cuda").t()):
            gemm_sm100(a, b, c, check_status=True)
            assert bool(((c.double() - want).abs() <= bar).all())


@pytest.mark.parametrize("split_k", [0, 1, 2])
def test_a_wait_that_runs_out(split_k):
    """K is so long that its products take more than the millisecond a wait is given: the kernel gives up in the
    middle of its stream, with copies and products in flight, reports it, and the next call is right."""
    M, N_out, K = 300, 3840, 1 << 20
    if split_k == 0:
        pair, split, _, _ = _plan(M, N_out, K)
        assert pair and split > 1                             # 0 takes the pair kernel, the others the single one
    a = torch.zeros(M, K, dtype=BF, device="cuda")
    b = torch.zeros(N_out, K, dtype=BF, device="cuda")
    c = torch.zeros(M, N_out, dtype=BF, device="cuda")
    with pytest.raises(RuntimeError, match="aborted: wait"):
        gemm_sm100(a, b, c, split_k=split_k, timeout_ms=1, check_status=True)
    g = torch.Generator(device="cuda").manual_seed(split_k)
    a = torch.randn(M, 2048, generator=g, device="cuda").to(BF)
    b = (torch.randn(N_out, 2048, generator=g, device="cuda") * 2048 ** -0.5).to(BF)
    gemm_sm100(a, b, c, split_k=split_k, check_status=True)
    want = a.double() @ b.double().t()
    bar = want.abs() * 2.0 ** -8 + (a.double().abs() @ b.double().abs().t()) * 2048 * 2.0 ** -24
    assert bool(((c.double() - want).abs() <= bar).all())
