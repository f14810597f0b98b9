"""CPU checks of the contexts at which decode steps of a few sequences take the step kernel (kd_decode_step_max_context)."""
import ctypes

import pytest

from kandle_b200 import lib


def _most(sequences, hidden, inter, heads, kv_heads, **other):
    k = ctypes.c_int(-1)
    lib.call("kd_decode_step_max_context", sequences, hidden, inter, heads, kv_heads, other.get("dim", 128), 151936, 28, 148, ctypes.byref(k))
    return k.value


# microseconds a layer of the step kernel and of the kernels per layer, from measuring both; 0.6B and 4B widths: of a whole step, lm_head included
@pytest.mark.parametrize("shape, keys, step, layers", [
    ((1, 1024, 3072, 16, 8), 40000, 1566, 2146), ((2, 1024, 3072, 16, 8), 24000, 1819, 2037), ((2, 1024, 3072, 16, 8), 40000, 2691, 2573),
    ((3, 1024, 3072, 16, 8), 16000, 1895, 1984), ((3, 1024, 3072, 16, 8), 24000, 2560, 2384), ((4, 1024, 3072, 16, 8), 8000, 1610, 1676),
    ((4, 1024, 3072, 16, 8), 11000, 1971, 1871), ((5, 1024, 3072, 16, 8), 5000, 1504, 1541), ((5, 1024, 3072, 16, 8), 6000, 1676, 1621),
    ((6, 1024, 3072, 16, 8), 3000, 1385, 1416), ((6, 1024, 3072, 16, 8), 4000, 1565, 1524), ((1, 2560, 9728, 32, 8), 24000, 968, 1033),
    ((1, 2560, 9728, 32, 8), 32000, 1105, 1080), ((2, 2560, 9728, 32, 8), 6000, 879, 903), ((2, 2560, 9728, 32, 8), 8000, 955, 938),
    ((3, 2560, 9728, 32, 8), 1000, 799, 833), ((3, 2560, 9728, 32, 8), 3000, 919, 882), ((3, 4096, 12288, 32, 8), 300, 115.4, 108.6),
    ((2, 4096, 12288, 32, 8), 4000, 103.9, 116.5), ((4, 1024, 3072, 32, 8), 1000, 42.7, 46.9), ((4, 1024, 3072, 32, 8), 2000, 53.6, 49.7),
    ((6, 1024, 3072, 32, 8), 300, 45.5, 44.5), ((4, 512, 1536, 8, 2), 8000, 40.9, 49.0), ((4, 512, 1536, 8, 2), 16000, 61.9, 54.8),
    ((6, 1024, 3072, 8, 8), 4000, 48.9, 53.9), ((6, 1024, 3072, 8, 8), 8000, 68.8, 68.0), ((5, 2048, 6144, 16, 8), 4000, 63.2, 68.7),
    ((5, 2048, 6144, 16, 8), 8000, 85.7, 80.4)])
def test_the_step_kernel_is_taken_where_it_is_the_faster_form(shape, keys, step, layers):
    assert (keys <= _most(*shape)) == (step < layers)


def test_shapes_that_it_does_not_take_have_no_context():
    assert _most(7, 1024, 3072, 16, 8) == _most(0, 1024, 3072, 16, 8) == _most(4, 2560, 9728, 32, 8) == _most(1, 1024, 3072, 16, 8, dim=64) == 0
    assert _most(1, 1024, 3072, 16, 0) == 0
