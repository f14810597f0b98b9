"""bf16 linears whose tiles are shared by the CTAs of a cluster, each with a range of K: every width and number of CTAs, k-blocks
that do not divide evenly, remainders of K and N inside a shared tile, and every epilogue, against float64.  The form that a
case is there for is asserted, so that another choice of forms cannot empty the test."""
import ctypes

import numpy as np
import pytest

from kandle_b200 import core, lib, synth
from kandle_b200.core import Tensor
from kandle_b200.engine import interleave_gate_up
from oracle import vogozen

pytestmark = pytest.mark.gpu

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


def _plan(M, N, K, heads=0):
    w, s = ctypes.c_int(0), ctypes.c_int(0)
    lib.call("kd_debug_linear_plan", M, N, K, heads, 148, ctypes.byref(w), ctypes.byref(s))
    return w.value, s.value


def _close(got, want, rel, scale=None):
    """Within the rounding of the result (rel of its value) and of fp32 sums in any order (1e-5 of the largest)."""
    assert (np.abs(got - want) <= rel * np.abs(want) + 1e-5 * np.abs(want).max()).all()


# 34, 41, 49 and 65 k-blocks; the last of K holds 8 numbers; the last tile of N 8 columns (72, 1048, 2504, 2600) or all
@pytest.mark.parametrize("M, N, K, plan", [(97, 72, 2120, (64, 4)), (200, 1048, 2568, (64, 2)), (1, 2504, 3080, (64, 2)), (97, 6144, 3080, (128, 2)),
                                           (129, 2600, 4104, (128, 2)), (256, 200, 4104, (64, 4))])
def test_epilogues_of_shared_tiles(backend, M, N, K, plan):
    assert _plan(M, N, K) == plan
    x, w = _bf((M, K), 1), _bf((N, K), 2, K ** -0.5)
    tx, tw = _put(x), _put(w)
    y = x.astype(np.float64) @ w.T.astype(np.float64)
    outs = [core.full((M, N), float("nan"), "float32") for _ in range(2)]
    for o in outs:
        lib.call("kd_linear_bf16", _r(tx), _r(tw), None, 0, _r(o))
    got = outs[0].dataAsync()
    _close(got, y, 0)
    assert np.array_equal(got, outs[1].dataAsync())                    # the order of the sums is fixed
    r, b = _bf((M, N), 3), _bf((N,), 4, 0.5)
    out = core.full((M, N), float("nan"), "bfloat16")
    lib.call("kd_linear_bf16", _r(tx), _r(tw), _r(_put(r)), 1, _r(out))
    _close(out.dataAsync(), y + r, 2.0 ** -8)
    res = core.full((M, N), float("nan"), "float32")
    lib.call("kd_linear_ex", _r(tx), _r(tw), _r(Tensor(r)), F(1.0), _r(res), None)
    _close(res.dataAsync(), y + r, 0)
    lib.call("kd_linear_bf16_bias", _r(tx), _r(tw), _r(_put(b)), _r(_put(r)), 1, _r(out))
    _close(out.dataAsync(), vogozen.gelu_tanh(y + b) + r, 2.0 ** -8)
    lib.call("kd_linear_tanh", _r(tx), _r(tw), _r(out))
    _close(out.dataAsync(), np.tanh(y), 2.0 ** -8)
    n = N // 64 * 32
    head, tail = core.full((M, n), float("nan"), "bfloat16"), core.full((M, N - n), float("nan"), "float32")
    lib.call("kd_linear_ex", _r(tx), _r(tw), None, F(1.0), _r(head), _r(tail))
    _close(head.dataAsync(), y[:, :n], 2.0 ** -8)
    _close(tail.dataAsync(), y[:, n:], 0)


@pytest.mark.parametrize("M, ff, K, plan", [(97, 528, 2120, (64, 4)), (200, 528, 2568, (64, 2)), (129, 1296, 4104, (128, 2))])
@pytest.mark.parametrize("epilogue", [2, 5])
def test_gated_epilogues_of_shared_tiles(backend, M, ff, K, plan, epilogue):
    assert _plan(M, 2 * ff, K) == plan
    x, g, u = _bf((M, K), 5), _bf((ff, K), 6, 2 * K ** -0.5), _bf((ff, K), 7, K ** -0.5)
    out = core.full((M, ff), float("nan"), "bfloat16")
    lib.call("kd_linear_glu", _r(_put(x)), _r(_put(interleave_gate_up(g, u))), epilogue, _r(out))
    xd = x.astype(np.float64)
    act = vogozen.silu if epilogue == 2 else vogozen.gelu_tanh
    want = act(xd @ g.T) * (xd @ u.T)
    assert (np.abs(out.dataAsync() - want) <= 2.0 ** -8 * np.abs(want) + 2e-5 * np.abs(want).max()).all()


@pytest.mark.parametrize("B, S, Hq, Hkv, K, plan", [(1, 97, 4, 2, 2568, (128, 4)), (2, 70, 16, 4, 2568, (128, 2)), (1, 97, 32, 8, 2568, (128, 2))])
def test_heads_of_shared_tiles(backend, oracle, B, S, Hq, Hkv, K, plan):
    """Query/key norm, rotation and cache rows behind a shared tile (the widths of a 4B model among them)."""
    d, max_s, pos0 = 128, 192, 7
    n = (Hq + 2 * Hkv) * d
    assert _plan(B * S, n, K, 1) == plan
    x, w = _bf((B * S, K), 8), _bf((n, K), 9, K ** -0.5)
    qw, kw = (lib.round_to_bf16(1 + 0.1 * _bf((d,), s)) for s in (10, 11))
    cos_t, sin_t = core.empty((S, 64), "float32"), core.empty((S, 64), "float32")
    lib.call("kd_rope_table", _r(Tensor(oracle.rope_inv_freq(d, 1e6))), None, pos0, S, _r(cos_t), _r(sin_t))
    kc, vc = core.zeros((B, Hkv, max_s, d), "bfloat16"), core.zeros((B, Hkv, max_s, d), "bfloat16")
    q_out = core.full((B, S, Hq, d), float("nan"), "bfloat16")
    lib.call("kd_qkv_linear_norm_rope_cachewrite", _r(_put(x)), _r(_put(w)), _r(_put(qw)), _r(_put(kw)), F(1e-6), _r(cos_t), _r(sin_t), _r(kc), _r(vc), pos0, _r(q_out))
    y = (x.astype(np.float64) @ w.T.astype(np.float64)).astype(np.float32).reshape(B, S, -1, d).transpose(0, 2, 1, 3)
    cos, sin = oracle.rope_tables(np.arange(pos0, pos0 + S, dtype=np.int32), d, 1e6)
    heads = lambda part, weight: oracle.apply_rope(oracle.rms_norm(np.ascontiguousarray(part), weight, 1e-6), cos, sin)  # noqa: E731
    q, k, v = heads(y[:, :Hq], qw), heads(y[:, Hq:Hq + Hkv], kw), y[:, Hq + Hkv:]
    inside = slice(pos0, pos0 + S)
    for got, want in ((q_out.dataAsync().transpose(0, 2, 1, 3), q), (kc.dataAsync()[:, :, inside], k), (vc.dataAsync()[:, :, inside], v)):
        assert (np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-4 * np.abs(want).max()).all()
    for cache in (kc.dataAsync(), vc.dataAsync()):
        assert not cache[:, :, :pos0].any() and not cache[:, :, pos0 + S:].any()
