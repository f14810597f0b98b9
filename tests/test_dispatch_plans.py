"""Which form a call takes, checked without a GPU: the rules are host arithmetic (kd_debug_*_plan)."""
import ctypes
import random

import pytest

from kandle_b200 import lib

SMS = 148


def _two(entry, *args):
    a, b = ctypes.c_int(0), ctypes.c_int(0)
    lib.call(entry, *args, ctypes.byref(a), ctypes.byref(b))
    return a.value, b.value


# heads of all sequences, tokens, and what measuring both forms at that size gave (time of the records over the other form's)
@pytest.mark.parametrize("delta, bf16, dim, heads, tokens, ratio", [
    (1, 1, 128, 16, 8192, 0.27), (1, 1, 128, 16, 32, 0.56), (1, 1, 128, 64, 200, 0.78), (1, 1, 96, 96, 32, 1.14), (1, 1, 96, 96, 96, 0.84),
    (1, 1, 128, 64, 32, 1.07), (1, 1, 64, 272, 256, 1.04), (1, 1, 64, 192, 1000, 0.82), (1, 0, 64, 256, 32, 1.10), (1, 0, 96, 64, 32, 0.92),
    (1, 1, 256, 32, 32, 0.92), (1, 0, 256, 32, 1000, 0.40), (1, 1, 16, 512, 200, 0.69), (0, 1, 64, 32, 8192, 0.30), (0, 1, 64, 272, 32, 1.05),
    (0, 1, 64, 272, 600, 0.89), (0, 1, 96, 80, 48, 1.23), (0, 1, 128, 64, 64, 1.15), (0, 1, 128, 64, 600, 0.96), (0, 1, 96, 64, 32, 1.12),
    (0, 1, 192, 16, 32, 1.22), (0, 1, 192, 16, 200, 0.69), (0, 1, 192, 32, 256, 1.05), (0, 1, 256, 32, 1000, 1.22), (0, 0, 128, 64, 48, 1.16),
    (0, 0, 256, 32, 32, 1.24), (0, 0, 256, 32, 1000, 0.71), (0, 0, 192, 40, 48, 1.09), (0, 0, 64, 272, 32, 0.95)])
def test_records_where_they_are_the_shorter_form(delta, bf16, dim, heads, tokens, ratio):
    records, _ = _two("kd_debug_recurrence_plan", delta, bf16, dim, dim, heads, tokens, SMS)
    assert bool(records) == (ratio < 1)


def test_recurrences_outside_the_measured_range_take_one_kernel():
    rng = random.Random(1)
    for _ in range(3000):
        delta, bf16, dim, vdim = rng.randint(0, 1), rng.randint(0, 1), rng.randint(1, 256), rng.randint(1, 300)
        heads, tokens = rng.randint(1, 700), rng.randint(1, 64)
        records, ctas = _two("kd_debug_recurrence_plan", delta, bf16, dim, vdim, heads, tokens, SMS)
        assert ctas >= heads
        assert not (records and (tokens < 32 or ctas > 4 * SMS))


def test_linears_share_tiles_within_one_wave():
    """A CTA of a shared tile has one tile and at least two k-blocks, 256-wide tiles and more than two rows of tiles are not
    shared, and a head of 128 columns lies in one tile."""
    rng = random.Random(2)
    shared = set()
    for _ in range(20000):
        M, N, K, heads = rng.choice([1, 7, 97, 128, 129, 256, 257, 700]), 8 * rng.randint(1, 1300), 8 * rng.randint(1, 1300), rng.randint(0, 1)
        N = max(384, N // 128 * 128) if heads else N
        w, s = _two("kd_debug_linear_plan", M, N, K, heads, SMS)
        rows, kbs = -(-M // 128), -(-K // 64)
        assert w in ((128, 256) if heads else (64, 128, 256)) and s in (1, 2, 4)
        if s > 1:
            assert w < 256 and rows <= 2 and rows * -(-N // w) * s <= SMS and kbs >= 2 * s
            shared.add((w, s))
    assert shared == {(64, 2), (64, 4), (128, 2), (128, 4)}


def test_fp32_matmuls_split_k_within_one_wave():
    rng = random.Random(3)
    seen = set()
    for _ in range(20000):
        batches, M, N, K = rng.choice([1, 1, 3, 16]), rng.randint(1, 1500), rng.randint(1, 4000), 4 * rng.randint(16, 1100)
        w, s = _two("kd_debug_matmul_f32_plan", batches, M, N, K, SMS)
        assert w in (64, 128) and s in (1, 2, 4) and s <= -(-K // 64) and (w // 4) % s == 0
        assert s == 1 or batches * -(-M // 128) * -(-N // w) * s <= SMS
        seen.add((w, s))
    assert {(64, 4), (128, 1), (128, 2), (128, 4)} <= seen
