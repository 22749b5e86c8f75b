"""Timed cases: what a program built on this package has it do, through its public entry points.

Six kinds of work, each over the sizes that are met in use:

* ``decode_bf16``   one decode step of the 16-layer Llama-3.2-1B shape, bf16 weights, logits for sampling;
* ``decode_nvfp4``  one decode step of the 36-layer Qwen3-8B shape, block-scaled NVFP4 weights, q/k norm, logits;
* ``project``       one projection of a handful of rows as a program of its own (bf16 or NVFP4 weights);
* ``flash_decode``  split-KV attention of one new token per sequence against a long cache;
* ``prefill``       attention of a prompt, or of a chunk of one behind a cached prefix;
* ``gemm``          one projection of a prompt's rows.

A case is a dict of plain values; ``prepare`` builds what a program keeps between calls (weights, caches, buffers,
the compiled program), ``run`` is one pass, ``work`` what the pass cannot do without, ``tolerance`` how far another
correct implementation of the same precision may be.
"""

import math

import torch

from machete_b200.kernels.attention import flash_decoding_schedule, flash_prefill
from machete_b200.kernels.decode_matvec import MatvecNvfp4Sm120Op, RmsMatvecNvfp4Sm120Op
from machete_b200.kernels.decode_matvec.nvfp4_model import schedule_decode_layer_nvfp4_sm100
from machete_b200.kernels.gemm import GemmOp, gemm_sm100
from machete_b200.kernels.llama1b import schedule_decode_model_sm100
from machete_b200.megakernel import Megakernel, OverlapTileScheduler
from machete_b200.quantization import quantize_nvfp4_weight

BF = torch.bfloat16
DEV = "cuda"

LLAMA_1B = dict(layers=16, hidden=2048, inter=8192, heads=32, kv_heads=8, head_dim=64, vocab=128256, theta=500000.0,
                eps=1e-5)
QWEN3_8B = dict(layers=36, hidden=4096, inter=12288, heads=32, kv_heads=8, head_dim=128, vocab=151936, theta=1000000.0,
                eps=1e-6)


def listed():
    return [
        # One user's chat at 4096 tokens of context: the latency of a token.
        dict(name="decode-1b-b1-kv4096", kind="decode_bf16", batch=1, kv=4096),
        # A small server's batch, no length a round number.
        dict(name="decode-1b-b16-kv1931", kind="decode_bf16", batch=16, kv=1931),
        # The larger model with packed weights: one user with a long document, and a batch of eight.
        dict(name="decode-8b-nvfp4-b1-kv8192", kind="decode_nvfp4", batch=1, kv=8192),
        dict(name="decode-8b-nvfp4-b8-kv4096", kind="decode_nvfp4", batch=8, kv=4096),
        # Single layers called by themselves, as a program that mixes these ops with its own does: the widest
        # projection of an 8B layer for one token, the smallest call, and packed weights for four tokens.
        dict(name="project-bf16-1x4096x14336", kind="project", fmt="bf16", m=1, k=4096, n=14336),
        dict(name="project-bf16-16x1024x1024", kind="project", fmt="bf16", m=16, k=1024, n=1024),
        dict(name="project-nvfp4-4x4096x14336", kind="project", fmt="nvfp4", m=4, k=4096, n=14336),
        # Attention over long contexts, eight sequences.
        dict(name="flash-decode-b8-kv32768", kind="flash_decode", batch=8, kv=32768, heads=32, kv_heads=8, head_dim=128),
        # A whole prompt; and a chunk of a prompt behind a prefix that lies in the cache already, two sequences.
        dict(name="prefill-4096-d128", kind="prefill", batch=1, m=4096, n=4096, heads=32, kv_heads=8, head_dim=128,
             causal=True, layout="bhmd"),
        dict(name="prefill-chunk-777of3000-d64", kind="prefill", batch=2, m=777, n=3000, heads=32, kv_heads=8,
             head_dim=64, causal=True, layout="bmhd"),
        # Projections of a long prompt's rows and of a short, ragged one's.
        dict(name="gemm-2048x4096x14336", kind="gemm", m=2048, k=4096, n=14336, activation="silu"),
        dict(name="gemm-93x4096x4096", kind="gemm", m=93, k=4096, n=4096, activation=""),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode_bf16", "decode_nvfp4", "project", "project", "flash_decode", "prefill", "prefill", "gemm", "gemm"])
    if kind == "decode_bf16":
        return dict(kind=kind, batch=_log(rng, 1, 16), kv=_log(rng, 128, 4096))
    if kind == "decode_nvfp4":
        batch = _log(rng, 1, 8)
        return dict(kind=kind, batch=batch, kv=_log(rng, 256, min(8192, 32768 // batch)))
    if kind == "project":
        fmt = rng.choice(["bf16", "nvfp4", "nvfp4-g32"])
        m, n = _log(rng, 1, 32), _log(rng, 512, 14336)
        k = _log(rng, 512, min(14336, 50000 // m))
        if fmt == "bf16":
            k -= k % 64
        else:
            k -= k % 2048 if k > 2048 else k % 256     # what the packed layout takes
        return dict(kind=kind, fmt=fmt, m=m, k=k, n=n)
    if kind == "flash_decode":
        return dict(kind=kind, batch=_log(rng, 1, 8), kv=_log(rng, 256, 32768), heads=32, kv_heads=rng.choice([4, 8]),
                    head_dim=rng.choice([64, 128]))
    if kind == "prefill":
        m = _log(rng, 65, 4096)
        batch = rng.randint(1, 2) if m <= 2048 else 1
        n = m + rng.choice([0, rng.randint(0, 4096 - m)])
        return dict(kind=kind, batch=batch, m=m, n=n, heads=32, kv_heads=8, head_dim=rng.choice([64, 128]),
                    causal=n > m or rng.random() < 0.75, layout=rng.choice(["bhmd", "bmhd"]))
    m = _log(rng, 33, 2048)
    n, k = 8 * _log(rng, 128, 1792), 8 * _log(rng, 128, 1792)
    while m * n * k > 2048 * 4096 * 14336:
        n, k = 8 * _log(rng, 128, 1792), 8 * _log(rng, 128, 1792)
    return dict(kind=kind, m=m, k=k, n=n, activation=rng.choice(["", "", "silu", "relu"]))


class _Inputs:
    """Seeded values on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std=1.0):
        return torch.randn(*shape, generator=self.g, device=DEV, dtype=BF).mul_(std)

    def norm_weight(self, n):
        return 1.0 + self.normal(n, std=0.02)


def _zeros(*shape, dtype=BF):
    return torch.zeros(*shape, dtype=dtype, device=DEV)


def _rope(length, d2, theta):
    inv = 1.0 / (theta ** (torch.arange(0, d2, dtype=torch.float32, device=DEV) / d2))
    ang = torch.arange(length, dtype=torch.float32, device=DEV)[:, None] * inv[None, :]
    return torch.cos(ang).to(BF), torch.sin(ang).to(BF)


def _weights(cfg, kv, rnd, packed):
    h, i, d = cfg["hidden"], cfg["inter"], cfg["head_dim"]
    q, kvd = cfg["heads"] * d, cfg["kv_heads"] * d
    out = {}
    out["cos"], out["sin"] = _rope(kv, d // 2, cfg["theta"])

    def put(key, rows, cols):
        w = rnd.normal(rows, cols, std=0.02)
        if not packed:
            out[key] = w
            return
        p = quantize_nvfp4_weight(w, group_size=16)
        out[f"{key}.packed"], out[f"{key}.scales"], out[f"{key}.global_scale"] = p.packed, p.scales, float(p.global_scale)

    for layer in range(cfg["layers"]):
        p = f"layer.{layer}"
        out[f"{p}.attn_norm"], out[f"{p}.mlp_norm"] = rnd.norm_weight(h), rnd.norm_weight(h)
        if packed:
            out[f"{p}.q_norm"], out[f"{p}.k_norm"] = rnd.norm_weight(d), rnd.norm_weight(d)
        for name, rows, cols in (("W_q", q, h), ("W_k", kvd, h), ("W_v", kvd, h), ("W_o", h, q), ("W_gate", i, h),
                                 ("W_up", i, h), ("W_down", h, i)):
            put(f"{p}.{name}", rows, cols)
    out["final_norm"] = rnd.norm_weight(h)
    put("lm_head", cfg["vocab"], h)
    return out


def _decode_buffers(cfg, batch, kv, rnd):
    d, h = cfg["head_dim"], cfg["hidden"]
    q = cfg["heads"] * d
    return dict(
        k_cache=rnd.normal(cfg["layers"], batch, kv, cfg["kv_heads"], d),
        v_cache=rnd.normal(cfg["layers"], batch, kv, cfg["kv_heads"], d),
        x_in=rnd.normal(batch, 1, h), residual_in=_zeros(batch, 1, h),
        x=[_zeros(batch, 1, h) for _ in range(2)], residual=[_zeros(batch, 1, h) for _ in range(2)],
        q=_zeros(batch, 1, q), attn=_zeros(batch, 1, q), mlp=_zeros(batch, 1, cfg["inter"]),
        logits=_zeros(batch, 1, cfg["vocab"]))


def _prepare_decode_bf16(case, rnd):
    cfg, batch, kv = LLAMA_1B, case["batch"], case["kv"]
    w, b = _weights(cfg, kv, rnd, packed=False), _decode_buffers(cfg, batch, kv, rnd)
    ops, keep = schedule_decode_model_sm100(
        batch=batch, cache_pos=kv - 1, weights=w, k_cache=list(b["k_cache"]), v_cache=list(b["v_cache"]),
        x_buffers=b["x"], residual_buffers=b["residual"], q_buf=b["q"], attn_out_buf=b["attn"], mlp_h_buf=b["mlp"],
        final_norm=w["final_norm"], lm_head=w["lm_head"], logits=b["logits"], num_layers=cfg["layers"], eps=cfg["eps"],
        hidden_size=cfg["hidden"], intermediate_size=cfg["inter"], num_q_heads=cfg["heads"],
        num_kv_heads=cfg["kv_heads"], head_dim=cfg["head_dim"], x_in=b["x_in"], residual_in=b["residual_in"])
    mk = Megakernel(ops, scheduler=OverlapTileScheduler()).compile()
    return dict(mk=mk, keep=(w, b, keep), out=[b["logits"], *b["x"], *b["residual"], b["k_cache"], b["v_cache"]])


def _prepare_decode_nvfp4(case, rnd):
    cfg, batch, kv = QWEN3_8B, case["batch"], case["kv"]
    w, b = _weights(cfg, kv, rnd, packed=True), _decode_buffers(cfg, batch, kv, rnd)
    x, r, ops, keep = b["x_in"], b["residual_in"], [], []
    for i in range(cfg["layers"]):
        layer = schedule_decode_layer_nvfp4_sm100(
            layer_idx=i, batch=batch, seq_len=1, cache_pos=kv - 1, weights=w, k_cache=b["k_cache"][i],
            v_cache=b["v_cache"][i], x_in=x, residual_in=r, x_out=b["x"][i % 2], residual_out=b["residual"][i % 2],
            q_buf=b["q"], attn_out_buf=b["attn"], mlp_h_buf=b["mlp"], eps=cfg["eps"], num_q_heads=cfg["heads"],
            num_kv_heads=cfg["kv_heads"], head_dim=cfg["head_dim"])
        ops += layer.ops
        keep += layer.keep_alive
        x, r = b["x"][i % 2], b["residual"][i % 2]
    last = b["residual"][cfg["layers"] % 2]
    ops += RmsMatvecNvfp4Sm120Op.schedule(x=x, residual_in=r, residual_out=last, norm_weight=w["final_norm"],
                                          weight_packed=w["lm_head.packed"], weight_scales=w["lm_head.scales"],
                                          y=b["logits"], group_size=16, global_scale=w["lm_head.global_scale"],
                                          eps=cfg["eps"])
    mk = Megakernel(ops, scheduler=OverlapTileScheduler()).compile()
    return dict(mk=mk, keep=(w, b, keep), out=[b["logits"], *b["x"], *b["residual"], b["k_cache"], b["v_cache"]])


def _prepare_project(case, rnd):
    m, k, n = case["m"], case["k"], case["n"]
    x, y, w = rnd.normal(1, m, k), _zeros(1, m, n), rnd.normal(n, k, std=0.02)
    if case["fmt"] == "bf16":
        ops = GemmOp.schedule(a=x, b=w, c=y)
    else:
        group = 32 if case["fmt"] == "nvfp4-g32" else 16
        w = quantize_nvfp4_weight(w, group_size=group)
        ops = MatvecNvfp4Sm120Op.schedule(a=x, weight_packed=w.packed, weight_scales=w.scales, y=y, group_size=group,
                                          global_scale=w.global_scale)
    return dict(mk=Megakernel(ops).compile(), keep=(x, w), out=[y])


def _prepare_flash_decode(case, rnd):
    b, n, h, hkv, d = (case[k] for k in ("batch", "kv", "heads", "kv_heads", "head_dim"))
    q, k, v, o = rnd.normal(b, 1, h, d), rnd.normal(b, n, hkv, d), rnd.normal(b, n, hkv, d), _zeros(b, 1, h, d)
    ops, _ = flash_decoding_schedule(q, k, v, o, kv_group_size=h // hkv)
    return dict(mk=Megakernel(ops).compile(), keep=(q, k, v), out=[o])


def _prepare_prefill(case, rnd):
    b, m, n, h, hkv, d = (case[k] for k in ("batch", "m", "n", "heads", "kv_heads", "head_dim"))

    def rows(heads, length):
        return rnd.normal(*((b, heads, length, d) if case["layout"] == "bhmd" else (b, length, heads, d)))

    q, k, v = rows(h, m), rows(hkv, n), rows(hkv, n)
    return dict(q=q, k=k, v=v, o=torch.zeros_like(q), causal=case["causal"], layout=case["layout"])


def _prepare_gemm(case, rnd):
    m, k, n = case["m"], case["k"], case["n"]
    return dict(a=rnd.normal(1, m, k), b=rnd.normal(n, k, std=0.02), c=_zeros(1, m, n), activation=case["activation"] or None)


_PREPARE = dict(decode_bf16=_prepare_decode_bf16, decode_nvfp4=_prepare_decode_nvfp4, project=_prepare_project,
                flash_decode=_prepare_flash_decode, prefill=_prepare_prefill, gemm=_prepare_gemm)


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, _Inputs(seed)), kind=case["kind"])


def run(state):
    if state["kind"] == "prefill":
        return flash_prefill(state["q"], state["k"], state["v"], state["o"], causal=state["causal"], layout=state["layout"])
    if state["kind"] == "gemm":
        return gemm_sm100(state["a"], state["b"], state["c"], activation=state["activation"])
    state["mk"].run(sync=False)
    return state["out"]


def _decode_work(cfg, batch, kv, bytes_per_weight):
    h, i, q, kvd = cfg["hidden"], cfg["inter"], cfg["heads"] * cfg["head_dim"], cfg["kv_heads"] * cfg["head_dim"]
    weights = cfg["layers"] * (2 * q * h + 2 * kvd * h + 3 * i * h) + cfg["vocab"] * h
    cache = cfg["layers"] * batch * kv * kvd * 2
    return dict(bytes=weights * bytes_per_weight + cache * 2 + batch * cfg["vocab"] * 2,
                flops=2 * batch * weights + 2 * cache * cfg["heads"] // cfg["kv_heads"])


def work(case):
    kind = case["kind"]
    if kind == "decode_bf16":
        return _decode_work(LLAMA_1B, case["batch"], case["kv"], 2.0)
    if kind == "decode_nvfp4":
        return _decode_work(QWEN3_8B, case["batch"], case["kv"], 0.5625)
    if kind in ("project", "gemm"):
        m, k, n = case["m"], case["k"], case["n"]
        return dict(bytes=k * n * (0.5625 if "nvfp4" in case.get("fmt", "") else 2.0) + 2 * m * (k + n), flops=2 * m * k * n)
    b, h, hkv, d = (case[k] for k in ("batch", "heads", "kv_heads", "head_dim"))
    if kind == "flash_decode":
        return dict(bytes=4 * b * case["kv"] * hkv * d + 4 * b * h * d, flops=4 * b * case["kv"] * h * d)
    m, n = case["m"], case["n"]
    pairs = m * n - (m * (m - 1) // 2 if case["causal"] else 0)       # the last m of the n tokens are the queries
    return dict(bytes=4 * b * d * (m * h + n * hkv), flops=4 * b * h * d * pairs)


def tolerance(case):
    # bf16 results: one rounding is up to 2^-8 of a value.  A decode step stores its residual stream and its
    # intermediate rows in bf16 some five times a layer, and roundings that fall the other way add up over the layers.
    if case["kind"].startswith("decode"):
        return {"rel": 2e-2}
    # attention rounds its probabilities to bf16 as well as its result
    return {"rel": 1e-2 if case["kind"] in ("prefill", "flash_decode") else 5e-3}
