"""Operators whose outputs are not cleared before their kernel runs must write every element of them: every operator gives the
same bits with new storage full of zeros and full of ones bits (NaN in every floating-point type, -1 in every integer)."""
import numpy as np
import pytest

import kandle_b200.backend as backend_module
from kandle_b200 import core, lib, synth
from kandle_b200.backend import CudaStorage
from kandle_b200.core import Tensor
from kandle_b200.model_utils import WhisperAudioEncoder, WhisperConfig
from kandle_b200.whisper_engine import WhisperEncoderEngine

pytestmark = pytest.mark.gpu


def _filled(byte):
    class Filled(CudaStorage):
        made = 0

        def __init__(self, nbytes, zero=True):
            super().__init__(nbytes, zero)
            if not zero:
                host = np.full(nbytes, byte, np.uint8)
                lib.call("kd_upload", self.handle, 0, host.ctypes.data, nbytes)
                Filled.made += 1
    return Filled


def _t(*shape, dtype="float32", seed="t"):
    return Tensor(synth.normal(seed, shape), dtype=dtype)


def _pair(dtype):
    return _t(3, 5, 37, dtype=dtype), _t(3, 1, 37, dtype=dtype, seed="u")


FLOATS = ("float32", "bfloat16", "float16")
CASES = {}
for _d in FLOATS:
    for _n in ("add", "sub", "mul", "div", "maximum"):
        CASES[f"{_n} {_d}"] = lambda n=_n, d=_d: getattr(core, n)(*_pair(d))
    for _n in ("neg", "cos", "sin", "silu", "gelu", "abs", "tanh", "sigmoid"):
        CASES[f"{_n} {_d}"] = lambda n=_n, d=_d: getattr(core, n)(_t(3, 5, 37, dtype=d))
    CASES[f"views {_d}"] = lambda d=_d: core.contiguous(_t(3, 5, 40, dtype=d).permute([1, 0, 2]).slice("..., 4:36"))
    CASES[f"cast {_d}"] = lambda d=_d: core.cast(_t(3, 5, 37).permute([2, 0, 1]), d)
    CASES[f"cat {_d}"] = lambda d=_d: core.cat([_t(3, n, 7, dtype=d) for n in (1, 4, 2)], 1)
    CASES[f"full {_d}"] = lambda d=_d: core.full((3, 37), 2.5, d)
    CASES[f"ones {_d}"] = lambda d=_d: core.ones((3, 37), d)
    CASES[f"zeros {_d}"] = lambda d=_d: core.zeros((3, 37), d)
    CASES[f"softmax {_d}"] = lambda d=_d: core.softmax(_t(9, 333, dtype=d))
    for _n in (24, 333, 768, 1024, 2048, 9000):
        CASES[f"rms_norm {_n} {_d}"] = lambda n=_n, d=_d: core.rmsNorm(_t(7, n, dtype=d), (n,), _t(n, dtype=d), 1e-6)
        CASES[f"layer_norm {_n} {_d}"] = lambda n=_n, d=_d: core.layerNorm(_t(7, n, dtype=d), (n,), _t(n, dtype=d), _t(n, dtype=d), 1e-5)
    for _k in (40, 64, 72, 1000):
        CASES[f"matmul {_k} {_d}"] = lambda k=_k, d=_d: core.matmul(_t(2, 130, k, dtype=d), _t(2, 72, k, dtype=d), transposeB=True)
        CASES[f"matmul n {_k} {_d}"] = lambda k=_k, d=_d: core.matmul(_t(70, k, dtype=d), _t(k, 33, dtype=d))
    CASES[f"linear {_d}"] = lambda d=_d: core.linear(_t(5, 40, 72, dtype=d), _t(48, 72, dtype=d), _t(48, dtype=d))
    CASES[f"matmul without k {_d}"] = lambda d=_d: core.matmul(_t(3, 0, dtype=d), _t(4, 0, dtype=d), transposeB=True)
    for _s, _h in ((5, 24), (70, 64), (33, 128)):
        for _c in (False, True):
            CASES[f"attention {_s} {_h} {_c} {_d}"] = lambda s=_s, h=_h, c=_c, d=_d: core.scaledDotProductAttention(
                _t(1, 4, s, h, dtype=d), _t(1, 2, s, h, dtype=d), _t(1, 2, s, h, dtype=d), None, 0.0, c)
    CASES[f"conv1d {_d}"] = lambda d=_d: core.conv1d(_t(2, 5, 31, dtype=d), _t(7, 5, 3, dtype=d), _t(7, dtype=d), 2, 1)
    CASES[f"argmax {_d}"] = lambda d=_d: core.argmax(_t(5, 33, 4, dtype=d), 1)
    CASES[f"embedding {_d}"] = lambda d=_d: core.embedding(Tensor(np.array([[3, 0], [6, 6]], np.int32)), _t(7, 24, dtype=d))
for _d in ("int32", "int64"):
    CASES[f"arange {_d}"] = lambda d=_d: core.arange(3, 40, 2, d)
    CASES[f"integers {_d}"] = lambda d=_d: core.add(core.arange(0, 37, 1, d), core.neg(core.arange(0, 37, 1, d)))
CASES["randn"] = lambda: (core.manualSeed(7), core.randn((3, 37)))[1]


def _whisper():
    enc = WhisperAudioEncoder(WhisperConfig(nMels=16, nAudioCtx=56, nAudioState=128, nAudioHead=2, nAudioLayer=2, dtype="bfloat16"))
    enc.loadStateDict({k: lib.round_to_bf16(v) for k, v in synth.whisper_encoder_weights(n_mels=16, state=128, layers=2, n_ctx=56, std=0.05).items()})
    return WhisperEncoderEngine(enc).forward(_t(3, 16, 111, dtype="bfloat16"))


CASES["whisper encoder"] = _whisper


@pytest.mark.parametrize("name", CASES)
def test_every_element_is_written(backend, monkeypatch, name):
    results = []
    for byte in (0x00, 0xFF):
        storage = _filled(byte)
        monkeypatch.setattr(backend_module, "CudaStorage", storage)
        try:
            results.append(CASES[name]().dataAsync())
        except (lib.KandleCudaError, ValueError, KeyError) as e:      # a type that this operator refuses
            results.append(np.array(type(e).__name__))
        assert storage.made or "without k" in name
    assert results[0].dtype == results[1].dtype and results[0].tobytes() == results[1].tobytes()
    assert results[0].dtype.kind == "U" or not np.isnan(results[0].astype(np.float64)).any()
