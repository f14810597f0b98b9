"""bf16 linears of up to 128 rows by tiles of 128 weight rows: steps of one and two k-blocks, an odd number of them, splits that end
inside a step, K that is no multiple of 64, remainders of N and of the rows, against float64."""
import ctypes

import numpy as np
import pytest

from kandle_b200 import core, lib
from kandle_b200.core import Tensor

pytestmark = pytest.mark.gpu


def _bf(shape, seed, sd):
    return lib.round_to_bf16((np.random.default_rng(seed).standard_normal(shape) * sd).astype(np.float32))


@pytest.mark.parametrize("M, N, K, splits", [(1, 128, 64, 1), (1, 136, 192, 1), (16, 256, 320, 2), (17, 72, 1088, 5), (32, 300, 2048, 9), (33, 640, 704, 3),
                                             (64, 128, 832, 13), (65, 264, 576, 2), (128, 130, 448, 4), (3, 200, 72, 2), (32, 129, 1000, 3), (5, 19200, 136, 1),
                                             (40, 19001, 320, 1), (100, 19200, 64, 1)])
def test_sums_of_every_split(backend, M, N, K, splits):
    x, w = _bf((M, K), 1, 1.0), _bf((N, K), 2, 1.0)
    tx, tw, out = Tensor(x, dtype="bfloat16"), Tensor(w, dtype="bfloat16"), core.empty((splits, M, N), "float32")
    lib.call("kd_linear_bf16_skinny", ctypes.byref(tx._handle.c()), ctypes.byref(tw._handle.c()), 0, ctypes.byref(out._handle.c()))
    each = -(-(-(-K // 64)) // splits) * 64
    got = out.dataAsync().reshape(splits, M, N)
    for s in range(splits):
        a, b = x[:, s * each:(s + 1) * each].astype(np.float64), w[:, s * each:(s + 1) * each].astype(np.float64)
        # fp32 sums of K exact products, in any order and with sums cut off instead of rounded: K 2^-23 of the sum of magnitudes
        assert (np.abs(got[s] - a @ b.T) <= each * 2.0 ** -23 * (np.abs(a) @ np.abs(b).T)).all()
