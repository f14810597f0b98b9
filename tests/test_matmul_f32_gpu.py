"""fp32 matmul on the tensor cores (gemm_f32_split.cu) against float64: edges of its 128 x 64/128 x 64 tiles, K split over
a cluster, batches, alpha / beta / C, and numbers outside the range of the split."""
import ctypes

import numpy as np
import pytest

from kandle_b200 import core, lib
from kandle_b200.backend import CudaEvent
from kandle_b200.core import Tensor

pytestmark = pytest.mark.gpu


def _bound(a, b):
    """Every product and partial sum rounds at 2^-24 of at most sum |a||b|: four roundings' worth for the dropped terms
    (2^-26 each), the sums inside a k-block and the sums over k-blocks, which grow slower than their number."""
    return 4 * 2.0 ** -24 * (np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64).T)


def _rand(shape, seed):
    return np.random.default_rng(seed).standard_normal(shape).astype(np.float32)


# one row to several tiles, N and K beside multiples of 64 and 128, K of one block, split tiles (few tiles, deep K)
@pytest.mark.parametrize("m,n,k", [(1, 1, 64), (1, 130, 68), (127, 64, 64), (128, 128, 128), (129, 65, 132), (300, 257, 100), (64, 1024, 1024),
                                   (130, 192, 196), (512, 1024, 320), (97, 3072, 1024), (128, 300, 4096), (260, 20000, 72)])
def test_matmul_f32_tiles(backend, m, n, k):
    a, b = _rand((m, k), 1), _rand((n, k), 2)
    got = core.matmul(Tensor(a), Tensor(b), transposeB=True).dataAsync()
    err = np.abs(got - a.astype(np.float64) @ b.astype(np.float64).T)
    assert (err <= _bound(a, b)).all(), (err / _bound(a, b)).max()


def test_matmul_f32_batches_views_and_scalars(backend):
    a, b, c = _rand((2, 3, 70, 136), 3), _rand((3, 90, 136), 4), _rand((90,), 5)
    # rows of a wider buffer, a broadcast batch, C broadcast over rows
    wide = Tensor(np.concatenate([a, a], axis=-1))
    view = wide.slice(":, :, :, 136:272")
    got = core.matmul(view, Tensor(b), transposeB=True, alpha=0.5).dataAsync()
    ref = 0.5 * (a.astype(np.float64) @ b.astype(np.float64).transpose(0, 2, 1))
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max() * 2
    got = core.linear(Tensor(a[0, 0]), Tensor(b[0]), Tensor(c)).dataAsync()
    ref = a[0, 0].astype(np.float64) @ b[0].astype(np.float64).T + c
    assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max() * 2


@pytest.mark.parametrize("m,n,k", [(130, 70, 128), (130, 300, 1024)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3e38, -3.4e38, 0.0])
def test_matmul_f32_values_without_a_split(backend, m, n, k, value):
    a, b = _rand((m, k), 6), _rand((n, k), 7)
    a[3, 5] = value
    b[n - 1, k - 1] = value
    got = core.matmul(Tensor(a), Tensor(b), transposeB=True).dataAsync()
    with np.errstate(all="ignore"):
        exact = a.astype(np.float64) @ b.astype(np.float64).T
        ref = exact.astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
    ok = np.isfinite(ref)
    ok[3, n - 1] = False      # two huge terms: whether their sum overflows on the way depends on its order
    a[~np.isfinite(a)], b[~np.isfinite(b)] = 0, 0
    assert (np.abs(got[ok] - exact[ok]) <= 16 * _bound(a, b)[ok]).all()       # (plain fused multiply-adds: more roundings)


@pytest.mark.parametrize("scale", [1e-31, 1e-36, 1e-40])
def test_matmul_f32_tiny_operand(backend, scale):
    a, b = _rand((70, 256), 8) * np.float32(scale), _rand((130, 256), 9) * np.float32(1e20)
    got = core.matmul(Tensor(a), Tensor(b), transposeB=True).dataAsync()
    exact = a.astype(np.float64) @ b.astype(np.float64).T
    assert (np.abs(got - exact) <= 16 * _bound(a, b)).all()


@pytest.mark.parametrize("value", [1e-35, np.nan])
def test_matmul_f32_numbers_without_a_split_are_no_cliff(backend, value):
    """A number in every tile that sends it to plain multiply-adds: about 9 times the time of the split ones (that is the time
    of matmul_f32_kernel); the bound leaves room for a busy machine, and a scalar loop took 240 times."""
    a, b = _rand((512, 1024), 10), _rand((3072, 1024), 11)

    def once(x):
        ta, tb = Tensor(x), Tensor(b)
        start, stop = CudaEvent(), CudaEvent()
        best = np.inf
        for _ in range(4):
            start.record()
            for _ in range(4):
                core.matmul(ta, tb, transposeB=True).dispose()
            stop.record()
            best = min(best, start.elapsed_ms(stop))
        return best

    bad = a.copy()
    bad[::16, 3] = value
    assert once(bad) < 40 * once(a)


@pytest.mark.parametrize("m,n,k", [(130, 130, 1024), (300, 1000, 512)])
@pytest.mark.parametrize("sa,sb", [(1e-20, 1e-20), (3e-20, 1e-19), (1e-24, 1e-15)])
def test_matmul_f32_products_near_the_least_number(backend, m, n, k, sa, sb):
    """Operands inside the split's range whose products and sums are subnormal or nearly: K multiply-adds round by at most
    half of the least number, or 2^-25 of the partial sum, each, independently of one another."""
    a, b = _rand((m, k), 12) * np.float32(sa), _rand((n, k), 13) * np.float32(sb)
    got = core.matmul(Tensor(a), Tensor(b), transposeB=True).dataAsync()
    exact = a.astype(np.float64) @ b.astype(np.float64).T
    step = 0.5 * np.sqrt(k) * (2.0 ** -149 + 2.0 ** -24 * np.sqrt((exact ** 2).mean()))
    assert np.sqrt(((got - exact) ** 2).mean()) <= step


def _plan(batches, m, n, k):
    w, s = ctypes.c_int(0), ctypes.c_int(0)
    lib.call("kd_debug_matmul_f32_plan", batches, m, n, k, 148, ctypes.byref(w), ctypes.byref(s))
    return w.value, s.value


# 19, 10, 34, 18 k-blocks: ranges of unequal length, zeros behind the last numbers of K in the last range
@pytest.mark.parametrize("batches,m,n,k,plan", [(1, 130, 3000, 1160, (128, 2)), (3, 130, 1000, 584, (128, 2)), (1, 60, 100, 2116, (64, 4)), (1, 300, 1000, 1100, (128, 4))])
def test_matmul_f32_split_over_a_cluster(backend, batches, m, n, k, plan):
    assert _plan(batches, m, n, k) == plan
    a, b, c = _rand((batches, m, k), 14), _rand((batches, n, k), 15), _rand((n,), 16)
    exact = a.astype(np.float64) @ b.astype(np.float64).transpose(0, 2, 1)
    bound = np.stack([_bound(x, y) for x, y in zip(a, b)])
    assert (np.abs(core.matmul(Tensor(a), Tensor(b), transposeB=True, alpha=0.5).dataAsync() - 0.5 * exact) <= bound).all()
    assert (np.abs(core.linear(Tensor(a[0]), Tensor(b[0]), Tensor(c)).dataAsync() - exact[0] - c) <= 2 * bound[0]).all()
    a[0, 7, 3], a[0, m - 1, k - 1] = 1e-36, np.inf      # a range below the split's numbers, and one row that is not finite
    got = core.matmul(Tensor(a), Tensor(b), transposeB=True).dataAsync()
    with np.errstate(all="ignore"):
        exact = a.astype(np.float64) @ b.astype(np.float64).transpose(0, 2, 1)
    assert not np.isfinite(got[0, m - 1]).any() and np.array_equal(got[0, m - 1] > 0, exact[0, m - 1] > 0)
    exact[0, m - 1] = got[0, m - 1] = 0
    assert (np.abs(got - exact) <= 16 * bound).all()


def test_matmul_f32_out_of_range_in_late_tiles(backend):
    """More tiles than multiprocessors: a CTA's second and third tile, and none of the others."""
    m, n, k = 2500, 2400, 128
    assert _plan(1, m, n, k)[1] == 1 and -(-m // 128) * -(-n // 128) > 2 * 148
    a, b = _rand((m, k), 17), _rand((n, k), 18)
    clean = core.matmul(Tensor(a), Tensor(b), transposeB=True).dataAsync()
    bad = a.copy()
    bad[1900, 5], bad[2400, 60] = 1e-38, np.inf
    got = core.matmul(Tensor(bad), Tensor(b), transposeB=True).dataAsync()
    exact = a.astype(np.float64) @ b.astype(np.float64).T
    exact[1900] -= a[1900, 5].astype(np.float64) * b[:, 5]
    assert not np.isfinite(got[2400]).any()
    exact[2400] = got[2400] = 0
    assert (np.abs(got - exact) <= 16 * _bound(a, b)).all()
    rows = [i for i in range(m) if i // 128 not in (1900 // 128, 2400 // 128)]
    assert np.array_equal(got[rows], clean[rows])
