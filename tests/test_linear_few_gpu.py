"""bf16 linears of a few rows by all SMs (clusters of 1 to 8 CTAs share K, eight warps a CTA): remainders of N and K, warps without
columns, several passes of 32 weight rows, both row tiles, every epilogue, strided rows of x, against float64."""
import ctypes
import random

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


def _plan(M, N, K):
    a, b = ctypes.c_int(0), ctypes.c_int(0)
    lib.call("kd_debug_linear_few_plan", M, N, K, 148, ctypes.byref(a), ctypes.byref(b))
    return a.value, b.value


def _close(got, want, rel):
    """Within the rounding of the result (rel of its value) and of fp32 sums in any order (1e-5 of the largest)."""
    assert (np.abs(got - want) <= rel * np.abs(want) + 1e-5 * np.abs(want).max()).all()


# microseconds of the kernels for more rows, and of this one, from measuring both
@pytest.mark.parametrize("M, N, K, other, few", [(1, 2048, 2048, 9.0, 4.4), (1, 64, 2048, 7.5, 2.8), (8, 8192, 2048, 15.7, 14.8), (8, 12288, 2048, 17.5, 20.2),
                                                 (8, 2048, 6144, 17.9, 12.2), (8, 5120, 2560, 17.5, 14.1), (1, 5120, 2560, 16.2, 19.1), (8, 10240, 1536, 13.4, 15.6), (1, 10240, 1024, 10.5, 10.2),
                                                 (16, 10240, 768, 8.4, 9.1), (1, 4096, 4096, 15.6, 15.2),
                                                 (16, 4096, 4096, 13.0, 15.7), (16, 2048, 6144, 12.6, 13.5), (16, 1024, 6144, 11.6, 8.2), (1, 6144, 3072, 17.3, 20.1),
                                                 (32, 2048, 2048, 8.6, 6.7), (32, 1024, 2048, 7.9, 5.1), (32, 1024, 3072, 9.0, 5.9), (24, 1024, 3072, 9.0, 5.9),
                                                 (32, 512, 2048, 7.7, 4.3), (32, 2048, 3072, 9.5, 8.9), (32, 2560, 3072, 10.4, 11.1), (32, 4096, 1024, 6.5, 5.4),
                                                 (32, 4096, 2048, 9.3, 10.2), (20, 4096, 2048, 10.6, 9.8), (32, 8192, 1024, 8.6, 9.1), (24, 6144, 768, 7.3, 8.0),
                                                 (32, 1536, 6144, 11.9, 14.2), (17, 6144, 1024, 9.2, 8.0), (32, 10240, 512, 5.9, 7.1)])
def test_taken_where_it_is_the_faster_one(M, N, K, other, few):
    assert bool(_plan(M, N, K)[0]) == (few < other)


def test_plans_cover_every_row_and_column():
    rng, seen = random.Random(1), set()
    for _ in range(20000):
        M, N, K = rng.randint(1, 40), 8 * rng.randint(1, 1300), 8 * rng.randint(1, 900)
        S, R = _plan(M, N, K)
        if S:
            assert M <= 32 and K % 32 == 0 and S in (1, 2, 4, 8) and R % 32 == 0 and K // 32 >= 8 * S
            assert -(-N // R) <= (148 // S if M <= 16 else {1: 148, 2: 74, 4: 33, 8: 15}[S]) and 16 * (1 + (M > 16)) * (R + 4) * 4 < 200 * 1024
            seen.add(S)
    assert seen == {1, 2, 4, 8}


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 8, 16, 17, 32])
@pytest.mark.parametrize("N, K", [(64, 256), (40, 2048), (1032, 288), (2048, 2080), (200, 4096), (7000, 512), (4096, 1056), (1000, 3072), (520, 2560)])
def test_results(backend, M, N, K):
    assert _plan(M, N, K)[0]
    wide, w = _bf((M, K + 8), 1), _bf((N, K), 2, K ** -0.5)
    x = wide[:, :K]
    tx, tw = _put(wide).slice([slice(None), slice(0, K)]), _put(w)
    y = x.astype(np.float64) @ w.T.astype(np.float64)
    outs = [core.full((M, N), float("nan"), "float32") for _ in range(2)]
    for o in outs:
        lib.call("kd_linear_ex", _r(tx), _r(tw), None, F(1.0), _r(o), None)
    got = outs[0].dataAsync()
    _close(got, y, 0)
    assert np.array_equal(got, outs[1].dataAsync())
    res = Tensor(np.random.default_rng(3).standard_normal((M, N)).astype(np.float32))
    lib.call("kd_linear_ex", _r(tx), _r(tw), _r(res), F(1.0), _r(outs[1]), None)
    _close(outs[1].dataAsync(), y + res.dataAsync(), 0)
    out = core.full((M, N), float("nan"), "bfloat16")
    lib.call("kd_linear_ex", _r(tx), _r(tw), None, F(1.0), _r(out), None)
    _close(out.dataAsync(), y, 2.0 ** -8)
    dense, r16 = _put(x), _bf((M, N), 4)                                     # (the linear that prompts use)
    lib.call("kd_linear_bf16", _r(dense), _r(tw), _r(_put(r16)), 1, _r(out))
    _close(out.dataAsync(), y + r16, 2.0 ** -8)
    lib.call("kd_linear_tanh", _r(tx), _r(tw), _r(out))
    _close(out.dataAsync(), np.tanh(y), 2.0 ** -8)
    n = N // 64 * 32
    if n:
        head, tail = core.full((M, n), float("nan"), "bfloat16"), core.full((M, N - n), float("nan"), "float32")
        lib.call("kd_linear_ex", _r(tx), _r(tw), None, F(1.0), _r(head), _r(tail))
        _close(head.dataAsync(), y[:, :n], 2.0 ** -8)
        _close(tail.dataAsync(), y[:, n:], 0)


@pytest.mark.gpu
@pytest.mark.parametrize("M, ff, K", [(1, 48, 512), (16, 2048, 1024), (23, 528, 2080)])
@pytest.mark.parametrize("epilogue", [2, 5])
def test_gated_results(backend, M, ff, K, epilogue):
    assert _plan(M, 2 * ff, K)[0]
    x, g, u = _bf((M, K), 5), _bf((ff, K), 6, 2 * K ** -0.5), _bf((ff, K), 7, K ** -0.5)
    out = core.full((M, ff), float("nan"), "bfloat16")
    lib.call("kd_linear_glu", _r(_put(x)), _r(_put(interleave_gate_up(g, u))), epilogue, _r(out))
    if epilogue == 2:
        again = core.full((M, ff), float("nan"), "bfloat16")
        lib.call("kd_linear_bf16", _r(_put(x)), _r(_put(interleave_gate_up(g, u))), None, 2, _r(again))
        assert np.array_equal(again.dataAsync(), out.dataAsync())
    xd = x.astype(np.float64)
    want = (vogozen.silu if epilogue == 2 else vogozen.gelu_tanh)(xd @ g.T) * (xd @ u.T)
    assert (np.abs(out.dataAsync() - want) <= 2.0 ** -8 * np.abs(want) + 2e-5 * np.abs(want).max()).all()


@pytest.mark.gpu
def test_weights_fetched_before_the_wait(backend):
    """In a programmatic chain the weights are on their way before the kernel before is done; x, which that one writes, is not."""
    M, N = 8, 1024
    ws = [_bf((N, N), 20 + i, N ** -0.5) for i in range(3)]
    x = _bf((M, N), 30)
    a, tw = [_put(x)] + [core.full((M, N), float("nan"), "bfloat16") for _ in range(6)], [_put(w) for w in ws]
    want = x
    for i in range(6):
        want = lib.round_to_bf16((want.astype(np.float64) @ ws[i % 3].T.astype(np.float64)).astype(np.float32))
    lib.call("kd_set_pdl", 3)
    try:
        for i in range(6):
            lib.call("kd_linear_ex", _r(a[i]), _r(tw[i % 3]), None, F(1.0), _r(a[i + 1]), None)
    finally:
        lib.call("kd_set_pdl", 0)
    got = a[6].dataAsync()
    assert np.linalg.norm(got - want) <= 6 * 2.0 ** -8 * np.linalg.norm(want)
