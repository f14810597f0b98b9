"""bf16 attention on both sides of the line between one query tile a CTA (a single wave) and two that share K/V tiles: ragged last
tiles, absent second tiles, grouped and single heads, both head sizes, against the fp32 oracle on the same bf16 inputs."""
import numpy as np
import pytest

from kandle_b200 import core, lib, synth
from kandle_b200.core import Tensor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("b, hq, hkv, sq, skv, d", [
    (4, 16, 8, 130, 130, 128), (5, 16, 8, 130, 130, 128),            # 128 and 160 tiles, heads of a group in pairs
    (6, 12, 12, 200, 200, 64), (7, 12, 12, 257, 257, 64),            # 144, and 252 with three tiles a head: the last one alone
    (37, 2, 1, 129, 129, 64), (38, 2, 1, 129, 129, 64),              # 148 and 152
    (3, 24, 8, 300, 300, 128), (1, 48, 48, 300, 412, 128),           # odd groups: consecutive tiles of a head; more keys than queries
    (40, 4, 2, 100, 100, 128), (40, 4, 4, 100, 100, 128),            # one tile a head
    (9, 16, 8, 128, 128, 128), (10, 16, 8, 97, 97, 128), (12, 12, 6, 33, 33, 64), (1, 8, 2, 16, 16, 64)])     # ... of pairs of heads, 144, 160, 144 and 8 tiles
def test_one_and_two_query_tiles(backend, oracle, causal, b, hq, hkv, sq, skv, d):
    if causal and sq != skv:
        pytest.skip("the oracle aligns the mask at the first key")
    q, k, v = (lib.round_to_bf16(synth.normal(n, s)) for n, s in (("q", (b, hq, sq, d)), ("k", (b, hkv, skv, d)), ("v", (b, hkv, skv, d))))
    got = core.scaledDotProductAttention(*(Tensor(x, dtype="bfloat16") for x in (q, k, v)), None, 0.0, causal).dataAsync()
    ref = oracle.sdpa(q, k, v, is_causal=causal)
    assert np.linalg.norm(got - ref) <= 2.0 ** -7 * np.linalg.norm(ref)        # probabilities and results in bf16, 2^-9 each on average
    assert np.abs(got - ref).max() <= 2e-2 * np.abs(ref).max()
