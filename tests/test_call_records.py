"""The records that carry the arguments of a prompt attention and of a GEMM to the library (CPU): sizes, order and refusals."""

import ctypes as C
import math

import pytest

from machete_b200 import _native as N


class _Prefill(C.Structure):
    _fields_ = ([(n, C.c_uint64) for n in ("q", "k", "v", "o", "lse", "workspace", "workspace_bytes", "cuda_stream")]
                + [(n, C.c_int64 * 3) for n in ("q_strides", "k_strides", "v_strides", "o_strides")]
                + [("timeout_ms", C.c_int64), ("scale", C.c_double)]
                + [(n, C.c_int32) for n in ("B", "H", "Hkv", "M", "N", "D", "causal", "reserved")])


class _Gemm(C.Structure):
    _fields_ = ([(n, C.c_uint64) for n in ("a", "b", "c", "workspace", "workspace_bytes", "cuda_stream")]
                + [(n, C.c_int64) for n in ("lda", "ldb", "ldc", "split_k", "timeout_ms")]
                + [(n, C.c_int32) for n in ("M", "N", "K", "activation", "packed", "reserved")])


@pytest.mark.parametrize("fmt,cls", [(N.PREFILL_CALL, _Prefill), (N.GEMM_CALL, _Gemm)])
def test_a_packed_record_is_the_c_structure(fmt, cls):
    assert fmt.size == C.sizeof(cls)
    values = list(range(1, len(fmt.unpack(bytes(fmt.size))) + 1))
    got = cls.from_buffer_copy(fmt.pack(*values))
    flat = []
    for name, _ in cls._fields_:
        v = getattr(got, name)
        flat += list(v) if hasattr(v, "__len__") else [v]
    assert flat == values


def _prefill(q=1 << 20, B=1, H=8, Hkv=2, M=4, Nk=4, D=64, causal=1, ws=1 << 20, ws_bytes=256, scale=0.125):
    strides = (H * M * D, M * D, D, Hkv * Nk * D, Nk * D, D, Hkv * Nk * D, Nk * D, D, H * M * D, M * D, D)
    return N.lib().mk_flash_prefill_call(N.PREFILL_CALL.pack(q, q, q, q, 0, ws, ws_bytes, 0, *strides, 1000, scale, B, H, Hkv, M, Nk, D, causal, 0))


def test_refusals_are_those_of_the_argument_form():
    lib = N.lib()
    assert lib.mk_flash_prefill_call(None) != 0 and lib.mk_gemm_bf16_call(None) != 0
    assert _prefill(q=0) == -1
    for bad in (dict(D=96), dict(Hkv=3), dict(M=5), dict(M=0), dict(ws_bytes=255), dict(ws=(1 << 20) + 128)):
        assert _prefill(**bad) == -2, bad
    for scale in (math.nan, math.inf, -math.inf, 1e39, 3e38):        # (3e38 * log2(e) is beyond fp32)
        assert _prefill(scale=scale) == -2, scale
        assert b"scale" in lib.mk_flash_prefill_last_error()
    one = 1 << 20

    def gemm(a=one, K=64, lda=64, packed=0, act=0):
        return lib.mk_gemm_bf16_call(N.GEMM_CALL.pack(a, one, one, one, 1 << 20, 0, lda, 64, 64, 0, 1000, 64, 64, K, act, packed, 0))
    assert gemm(a=0) == -1
    for bad in (dict(K=60), dict(K=0), dict(lda=32), dict(lda=65), dict(act=3), dict(K=72, lda=72, packed=1)):
        assert gemm(**bad) == -2, bad
