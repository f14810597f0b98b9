"""GPU parity of kd_decode_step (a decode step of a few sequences as one kernel) against the fp32 oracle on the same
bf16-rounded weights, and of its cache rows against those that the kernels per layer write."""
import ctypes

import numpy as np
import pytest

from kandle_b200 import lib, synth
from kandle_b200.core import Tensor
from kandle_b200.engine import Qwen3Engine
from kandle_b200.model_utils import Qwen3Config

pytestmark = pytest.mark.gpu

# sequences, hidden, inter, heads, kv_heads, prompt: rows that leave one to six blocks of eight to a CTA, one and several
# segments of columns, one to six sequences, 1, 2 and 4 query heads to a KV head, contexts of one key, at the last unsplit one
# and beyond it, with unequal splits, and (24 and 32 KV heads leave a CTA all keys of a head) of more keys than the ring holds and
# of more stages than there are barriers; an lm_head of more rows than a CTA takes at once
CASES = [(1, 512, 512, 4, 2, 1), (1, 1536, 1024, 4, 4, 64), (2, 512, 1536, 8, 2, 97), (3, 1024, 3072, 16, 8, 130), (4, 512, 1024, 4, 2, 96),
         (1, 1024, 3072, 16, 8, 900), (2, 512, 4096, 8, 2, 33), (6, 1024, 3072, 16, 8, 300), (1, 2560, 9728, 32, 8, 200), (5, 2560, 1024, 32, 8, 70),
         (6, 512, 512, 24, 24, 1300), (4, 512, 1024, 64, 32, 1157)]
VOCABS = {(2, 512, 512, 4, 2, 40): 20011}
STEPS = 3


def _engine(c, paged=False):
    B, hidden, inter, heads, kv, prompt = c
    vocab = VOCABS.get(c, 1000)
    dims = dict(vocab=vocab, hidden=hidden, inter=inter, layers=2, heads=heads, kv_heads=kv, head_dim=128)
    w = {k: lib.round_to_bf16(v) for k, v in synth.qwen3_weights(std=0.03, norm_jitter=0.05, **dims).items()}
    cfg = Qwen3Config(vocabSize=vocab, hiddenSize=hidden, intermediateSize=inter, numHiddenLayers=2, numAttentionHeads=heads, numKeyValueHeads=kv,
                      headDim=128, dtype="bfloat16")
    return Qwen3Engine(cfg, w, B, -(-(prompt + STEPS) // 128) * 128, paged=paged), w


def _forced(eng, ids, prompt, use_graph):
    """Logits of the steps behind the prompt, which feed given tokens."""
    eng.prefill(np.ascontiguousarray(ids[:, :prompt]))
    out = []
    for t in range(STEPS):
        eng.start_decode(Tensor(ids[:, prompt + t].astype(np.int64)), use_graph)
        tokens = eng.decode_step().dataAsync()
        out.append(eng._decode["logits"].dataAsync()[0])
        assert np.array_equal(tokens, out[-1].argmax(-1))
    return np.stack(out, 1)


@pytest.mark.parametrize("c", CASES + list(VOCABS))
def test_step_kernel_follows_the_oracle(backend, oracle, c):
    B, hidden, inter, heads, kv, prompt = c
    eng, w = _engine(c)
    ids = synth.token_ids("step.ids", (B, prompt + STEPS), 1000)
    got = _forced(eng, ids, prompt, True)
    assert eng._decode["step"] is not None
    assert np.array_equal(got, _forced(eng, ids, prompt, False))           # bit for bit, replayed or not
    rows = [t.dataAsync()[:, :, prompt:prompt + STEPS] for t in eng.k_cache + eng.v_cache]
    eng.dispose()
    eng.use_step_kernel = False
    other = _forced(eng, ids, prompt, True)
    assert eng._decode["step"] is None
    for a, t in zip(rows, eng.k_cache + eng.v_cache):
        b = t.dataAsync()[:, :, prompt:prompt + STEPS]
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b)
    eng.dispose()
    ocfg = oracle.Qwen3Config(vocab_size=VOCABS.get(c, 1000), hidden_size=hidden, intermediate_size=inter, num_hidden_layers=2, num_attention_heads=heads,
                              num_key_value_heads=kv, head_dim=128)
    ref = oracle.Qwen3Oracle(ocfg, w).logits(ids)[:, prompt:]
    err, before = np.linalg.norm(got - ref), np.linalg.norm(other - ref)
    assert err <= 1e-2 * np.linalg.norm(ref) and err <= 1.2 * before       # bf16 activations: 2^-8 each


# (splits that begin inside a page and cross its end, over two and over twelve pages; whole caches of eleven pages)
@pytest.mark.parametrize("c", [(3, 512, 512, 4, 2, 150), (2, 512, 512, 8, 4, 1500), (6, 512, 512, 24, 24, 1300)])
def test_step_kernel_on_a_paged_cache(backend, c):
    B, prompt = c[0], c[-1]
    ids = synth.token_ids("step.ids", (B, prompt + STEPS), 1000)
    flat, paged = _engine(c)[0], _engine(c, paged=True)[0]
    a, b = _forced(flat, ids, prompt, True), _forced(paged, ids, prompt, True)
    assert flat._decode["step"] is not None and paged._decode["step"] is not None and np.array_equal(a, b)
    flat.dispose()
    paged.dispose()


def test_the_lowest_of_equal_logits_is_the_next_token(backend):
    eng, w = _engine((2, 512, 512, 4, 2, 9))
    rows = w["model.embed_tokens.weight"].copy()
    rows[500:] = rows[:500]
    eng.embed = Tensor(rows, dtype="bfloat16")
    got = _forced(eng, synth.token_ids("step.ids", (2, 9 + STEPS), 1000), 9, True)
    assert np.array_equal(got[..., :500], got[..., 500:])                  # (and _forced has compared the tokens)
    eng.dispose()
    eng.embed = Tensor(np.zeros_like(rows), dtype="bfloat16")
    assert not _forced(eng, synth.token_ids("step.ids", (2, 9 + STEPS), 1000), 9, True).any()
    eng.dispose()


def test_squares_beyond_fp32_count_as_the_kernels_per_layer_have_them(backend):
    """A row whose sum of squares overflows is scaled by 1 / infinity, in either form."""
    eng, w = _engine((2, 512, 512, 4, 2, 9))
    rows = w["model.embed_tokens.weight"].copy()
    rows[7] = np.where(rows[7] < 0, -1e25, 1e25)
    eng.embed = Tensor(rows, dtype="bfloat16")
    got = []
    for eng.use_step_kernel in (True, False):
        eng.prefill(synth.token_ids("step.ids", (2, 9), 6))
        eng.start_decode(Tensor(np.array([7, 3], np.int64)), False)
        assert (eng._decode["step"] is not None) == eng.use_step_kernel
        eng.decode_step()
        got.append(eng._decode["logits"].dataAsync()[0])
        eng.dispose()
    one, other = (g[:, np.arange(1000) != 7] for g in got)                 # (the products of row 7 with itself overflow as well)
    assert not one[0].any() and not other[0].any()
    assert np.linalg.norm(one[1] - other[1]) <= 1e-2 * np.linalg.norm(other[1])


def test_step_kernel_reports_bad_tokens_and_positions(backend):
    eng, _ = _engine((1, 512, 512, 4, 2, 5))
    eng.prefill(synth.token_ids("step.ids", (1, 5), 1000))
    for token, pos, code in ((1000, 5, 101), (1, 128, 102), (1, -1, 102)):
        eng.start_decode(Tensor(np.array([token], np.int64)), False)
        backend.upload(eng._decode["scalars"]._handle, np.array([pos, pos + 1], np.int32))
        eng.decode_step()
        with pytest.raises(lib.KandleCudaError, match=f"code {code}"):
            backend.synchronize()
        eng.pos = 5
    eng.start_decode(Tensor(np.array([1], np.int64)), False)               # and goes on
    eng.decode_step()
    backend.synchronize()
    eng.dispose()


def test_the_form_follows_the_position(backend):
    """An engine with room for far more positions than its requests have takes the step kernel, and goes over to the kernels per
    layer (and back, on the next prompt) at the context that the library names, replayed or not."""
    c = (2, 512, 512, 4, 2, 40)
    eng, _ = _engine(c)
    ids = synth.token_ids("step.ids", (2, 40 + STEPS), 20011)
    alone = _forced(eng, ids, 40, True)
    room = Qwen3Engine(eng.cfg, _engine(c)[1], 2, 40960)
    assert np.array_equal(_forced(room, ids, 40, True), alone)
    d = room._decode
    assert d["step_keys"] > 10000 and list(d["graph"]) == ["step"]
    d["step_keys"] = 41                                                    # (the last of the three steps is beyond it)
    for use_graph in (False, True, True):
        got = _forced(room, ids, 40, use_graph)
        assert np.array_equal(got[:, :2], alone[:, :2])
        assert 0 < np.linalg.norm(got[:, 2] - alone[:, 2]) <= 1e-2 * np.linalg.norm(alone[:, 2])
    assert list(d["graph"]) == ["step", "layers"]
    room.dispose()                                                         # the change, and its capture, in the middle of a run
    room.prefill(np.ascontiguousarray(ids[:, :40]))
    d = room.start_decode(Tensor(ids[:, 40].astype(np.int64)))
    d["step_keys"] = 41
    for t in range(STEPS):
        if t:
            backend.upload(d["ids"]._handle, ids[:, 40 + t].astype(np.int64))
        assert np.array_equal(d["ids"].dataAsync(), ids[:, 40 + t])
        room.decode_step()
        assert np.array_equal(d["logits"].dataAsync()[0], got[:, t])
    room.dispose()
    eng.dispose()


def test_pages_outside_the_pool_are_reported(backend):
    eng, _ = _engine((2, 512, 512, 4, 2, 150), paged=True)
    ids = synth.token_ids("step.ids", (2, 150), 1000)
    table = eng.block_table.dataAsync().astype(np.int32)
    eng.prefill(ids)
    first = Tensor(np.array([1, 2], np.int64))
    for b, place, page in ((0, 1, int(table.max()) + 1), (1, 0, -1), (1, 1, 1 << 30)):
        bad = table.copy()
        bad[b, place] = page
        eng.start_decode(first, False)
        backend.upload(eng.block_table._handle, bad)
        eng.decode_step()
        with pytest.raises(lib.KandleCudaError, match="code 103"):
            backend.synchronize()
        eng.pos = 150
    backend.upload(eng.block_table._handle, table)
    eng.start_decode(first, False)                                         # and goes on
    eng.decode_step()
    backend.synchronize()
    eng.dispose()


def test_shapes_that_keep_the_kernels_per_layer(backend):
    def taken(*shape):
        n = ctypes.c_uint64(0)
        lib.call("kd_decode_step_state_bytes", *shape, 148, ctypes.byref(n))
        return n.value > 0
    good = (1, 1024, 3072, 16, 8, 128, 1000, 2)
    assert taken(*good)
    for i, bad in ((0, 0), (0, 7), (1, 1000), (1, 1280), (2, 3080), (2, 3200), (3, 24), (3, 10), (3, 64), (5, 64), (6, 100), (7, 65)):
        assert not taken(*good[:i], bad, *good[i + 1:]), (i, bad)
    assert taken(3, 2560, 9728, 32, 8, 128, 1000, 2) and not taken(4, 2560, 9728, 32, 8, 128, 1000, 2)       # activations beside the ring
