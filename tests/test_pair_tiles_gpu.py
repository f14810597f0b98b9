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


# microseconds of one CTA and of a pair a tile, from measuring both with the epilogue that the size has in a model
@pytest.mark.parametrize("M, N, K, one, two", [(700, 6144, 1024, 10.8, 12.0), (700, 19456, 2560, 77.7, 64.1), (4096, 6144, 1024, 40.4, 36.2), (16384, 6144, 1024, 145, 128),
                                               (65536, 6144, 1024, 698, 604), (4096, 1024, 2048, 40.8, 41.5), (36000, 1024, 2048, 177, 168), (4096, 1024, 3072, 43.6, 45.3),
                                               (8192, 1024, 3072, 90.6, 85.3), (2103, 2560, 4096, 74.1, 67.8), (2103, 2560, 9728, 153, 135), (2103, 6144, 2560, 57.6, 52.9),
                                               (6000, 2048, 2048, 68.3, 67.1), (8192, 2304, 768, 37.7, 38.4), (36000, 768, 768, 38.3, 36.9), (96000, 768, 3072, 355, 319),
                                               (65536, 512, 512, 34.9, 37.8), (96000, 768, 240, 195, 205), (65536, 4096, 1024, 467, 385), (2103, 4096, 1024, 16.6, 17.0)])
def test_pairs_where_they_are_the_faster_form(M, N, K, one, two):
    assert _pair(M, N, K) == (two < one)


@pytest.mark.gpu
@pytest.mark.parametrize("M, N, K", [(24577, 264, 1096), (24800, 512, 1160), (29000, 776, 1032), (1409, 2312, 6152)])
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
@pytest.mark.parametrize("M, N, K", [(24577, 264, 1032), (5000, 1032, 1024), (5000, 1032, 200), (700, 6152, 72)])
def test_epilogues_that_take_longer_than_the_products(backend, M, N, K):
    """Bias, activation and residual with few k-blocks: 256-wide tiles whose loops are one lane's (K <= 1024), and the sizes beside them."""
    x, w, r, b = _bf((M, K), 1), _bf((N, K), 2, K ** -0.5), _bf((M, N), 3), _bf((N,), 4, 0.5)
    tx, tw, tb, tr = _put(x), _put(w), _put(b), _put(r)
    y = x.astype(np.float64) @ w.T.astype(np.float64)
    for bias, act, res in ((tb, 0, None), (tb, 1, None), (tb, 0, tr), (None, 0, tr), (None, 1, tr)):
        out = core.full((M, N), float("nan"), "bfloat16")
        lib.call("kd_linear_bf16_bias", _r(tx), _r(tw), _r(bias), _r(res), act, _r(out))
        want = y + b if bias is not None else y
        want = (vogozen.gelu_tanh(want) if act else want) + (r if res is not None else 0)
        _close(out.dataAsync(), want, 2.0 ** -8)
    res32 = core.full((M, N), float("nan"), "float32")
    lib.call("kd_linear_bf16", _r(tx), _r(tw), _r(Tensor(r)), 1, _r(res32))
    _close(res32.dataAsync(), y + r, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("epilogue", [2, 5])
def test_gated_epilogues_of_pairs(backend, epilogue):
    M, ff, K = 24800, 144, 840
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
    B, S, Hq, Hkv, K, d, max_s = 96, 257, 2, 1, 776, 128, 264
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
