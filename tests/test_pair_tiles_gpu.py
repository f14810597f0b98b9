"""bf16 linears whose 256-row tiles are worked on by pairs of CTAs: a last tile that only the first CTA has rows of, remainders of
M, N and K, rings that wrap, several tiles to a pair, and every epilogue, against float64."""
import ctypes

import numpy as np
import pytest

from kandle_b200 import core, lib
from kandle_b200.core import Tensor
from kandle_b200.engine import interleave_gate_up
from oracle import vogozen

F = ctypes.c_float
KEEP = []


@pytest.fixture(autouse=True)
def _clear_keep():
    yield
    KEEP.clear()


def _r(t):
    if t is None:
        return None
    KEEP.append(t)
    return ctypes.byref(t._handle.c())


def _bf(shape, seed, sd=1.0):
    return lib.round_to_bf16((np.random.default_rng(seed).standard_normal(shape) * sd).astype(np.float32))


def _put(a):
    return Tensor(a, dtype="bfloat16")


def _pair(M, N, K, heads=0):
    p = ctypes.c_int(0)
    lib.call("kd_debug_linear_pair", M, N, K, heads, 148, ctypes.byref(p))
    return bool(p.value)


def _close(got, want, rel):
    """Within the rounding of the result (rel of its value) and of fp32 sums in any order (1e-5 of the largest)."""
    assert (np.abs(got - want) <= rel * np.abs(want) + 1e-5 * np.abs(want).max()).all()


# microseconds of one CTA and of a pair a tile, from measuring both
@pytest.mark.parametrize("M, N, K, one, two", [(700, 4096, 1024, 10.3, 11.5), (4096, 1024, 2048, 17.3, 19.4), (4096, 1024, 3072, 23.2, 25.0), (8192, 4096, 1024, 68.2, 61.5),
                                               (16384, 6144, 1024, 181, 147), (65536, 6144, 1024, 727, 588), (2103, 2560, 9728, 153, 143), (2103, 6144, 2560, 51.9, 47.9),
                                               (6000, 2048, 2048, 46.9, 44.1), (2103, 8448, 2048, 66.2, 68.6), (8192, 1024, 2048, 39.1, 39.8), (8192, 1024, 3072, 54.2, 53.3),
                                               (8192, 2304, 768, 29.7, 30.3), (12288, 768, 768, 18.0, 19.5), (96000, 768, 3072, 355, 317), (96000, 2304, 768, 311, 291),
                                               (32768, 1024, 3072, 170, 155), (65536, 768, 768, 90.1, 84.5)])
def test_pairs_where_they_are_the_faster_form(M, N, K, one, two):
    assert _pair(M, N, K) == (two < one)


@pytest.mark.gpu
@pytest.mark.parametrize("M, N, K", [(24577, 264, 72), (24800, 512, 200), (37900, 776, 64), (1409, 2312, 6152)])
def test_epilogues_of_pairs(backend, M, N, K):
    assert _pair(M, N, K)
    x, w = _bf((M, K), 1), _bf((N, K), 2, K ** -0.5)
    tx, tw = _put(x), _put(w)
    y = x.astype(np.float64) @ w.T.astype(np.float64)
    outs = [core.full((M, N), float("nan"), "float32") for _ in range(2)]
    for o in outs:
        lib.call("kd_linear_bf16", _r(tx), _r(tw), None, 0, _r(o))
    got = outs[0].dataAsync()
    _close(got, y, 0)
    assert np.array_equal(got, outs[1].dataAsync())
    r, b = _bf((M, N), 3), _bf((N,), 4, 0.5)
    res = core.full((M, N), float("nan"), "float32")
    lib.call("kd_linear_bf16", _r(tx), _r(tw), _r(Tensor(r)), 1, _r(res))
    _close(res.dataAsync(), y + r, 0)
    out = core.full((M, N), float("nan"), "bfloat16")
    lib.call("kd_linear_bf16_bias", _r(tx), _r(tw), _r(_put(b)), _r(_put(r)), 1, _r(out))
    _close(out.dataAsync(), vogozen.gelu_tanh(y + b) + r, 2.0 ** -8)
    n = N // 64 * 32
    head, tail = core.full((M, n), float("nan"), "bfloat16"), core.full((M, N - n), float("nan"), "float32")
    lib.call("kd_linear_ex", _r(tx), _r(tw), None, F(1.0), _r(head), _r(tail))
    _close(head.dataAsync(), y[:, :n], 2.0 ** -8)
    _close(tail.dataAsync(), y[:, n:], 0)


@pytest.mark.gpu
@pytest.mark.parametrize("epilogue", [2, 5])
def test_gated_epilogues_of_pairs(backend, epilogue):
    M, ff, K = 24800, 144, 200
    assert _pair(M, 2 * ff, K)
    x, g, u = _bf((M, K), 5), _bf((ff, K), 6, 2 * K ** -0.5), _bf((ff, K), 7, K ** -0.5)
    out = core.full((M, ff), float("nan"), "bfloat16")
    lib.call("kd_linear_glu", _r(_put(x)), _r(_put(interleave_gate_up(g, u))), epilogue, _r(out))
    xd = x.astype(np.float64)
    want = (vogozen.silu if epilogue == 2 else vogozen.gelu_tanh)(xd @ g.T) * (xd @ u.T)
    assert (np.abs(out.dataAsync() - want) <= 2.0 ** -8 * np.abs(want) + 2e-5 * np.abs(want).max()).all()


@pytest.mark.gpu
def test_heads_of_pairs(backend, oracle):
    """Query/key norm, rotation and cache rows: the fused epilogue against the linear and the kernel that does the same."""
    B, S, Hq, Hkv, K, d, max_s = 96, 257, 2, 1, 72, 128, 264
    n = (Hq + 2 * Hkv) * d
    assert _pair(B * S, n, K, 1)
    x, w = _bf((B * S, K), 8), _bf((n, K), 9, K ** -0.5)
    qw, kw = (_put(lib.round_to_bf16(1 + 0.1 * _bf((d,), s))) for s in (10, 11))
    cos_t, sin_t = core.empty((S, 64), "float32"), core.empty((S, 64), "float32")
    lib.call("kd_rope_table", _r(Tensor(oracle.rope_inv_freq(d, 1e6))), None, 0, S, _r(cos_t), _r(sin_t))
    caches = [core.zeros((B, Hkv, max_s, d), "bfloat16") for _ in range(4)]
    q = [core.full((B, S, Hq, d), float("nan"), "bfloat16") for _ in range(2)]
    lib.call("kd_qkv_linear_norm_rope_cachewrite", _r(_put(x)), _r(_put(w)), _r(qw), _r(kw), F(1e-6), _r(cos_t), _r(sin_t), _r(caches[0]), _r(caches[1]), 0, _r(q[0]))
    qkv = core.empty((1, B * S, n), "float32")               # (as one fp32 partial sum: unrounded, as in the epilogue)
    lib.call("kd_linear_bf16", _r(_put(x)), _r(_put(w)), None, 0, _r(qkv.view(B * S, n)))
    lib.call("kd_qkv_norm_rope_cachewrite", _r(qkv), _r(qw), _r(kw), F(1e-6), _r(cos_t), _r(sin_t), _r(caches[2]), _r(caches[3]), None, 0, _r(q[1]))
    for a, b in ((q[0], q[1]), (caches[0], caches[2]), (caches[1], caches[3])):
        a, b = a.dataAsync(), b.dataAsync()
        assert (np.abs(a - b) <= 2.0 ** -7 * np.abs(b) + 1e-5).all()
