"""What this framework is used for, as cases that can be timed: each goes through the public entry points over the range
of sizes that a user meets, from one short request to the largest batches of the benchmark configurations.

  attention       scaledDotProductAttention as a single fp32 operator
  module_prefill  the operator-by-operator Qwen3 module in fp32, logits for every position
  qwen3_prefill   Qwen3Engine.prefill: prompts from host ids to next-token logits, cache filled
  qwen3_decode    Qwen3Engine decode steps behind a prompt, replayed from the captured graph
  whisper         WhisperEncoderEngine.forward over clips
  hybrid_prefill  HybridEngine.extend on a new prompt (Vogozen, Pedorax)
  hybrid_decode   HybridEngine decode steps behind a prompt

Weights are drawn by the engines themselves (RandomInit) or, for the modules, loaded from host arrays as a checkpoint
is.  A pass of decode steps starts behind the same prompt every time and feeds given tokens, so that its outputs do not
hang on ties between nearly equal logits.  `exact` has its own float64 form of every model.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import kandle_b200
from kandle_b200 import core
from kandle_b200.core import Tensor
from kandle_b200.engine import Qwen3Engine, RandomInit
from kandle_b200.hybrid_bench import SIZES, WINDOW, pedorax_config, vogozen_config
from kandle_b200.hybrid_engine import HybridEngine
from kandle_b200.model_utils import Qwen3Config, Qwen3ForCausalLM, WhisperAudioEncoder, WhisperConfig
from kandle_b200.whisper_engine import WhisperEncoderEngine

STD = 0.02
STEPS = 8        # decode steps of a pass
HYBRID_VOCAB = 32768

#: Qwen3 shapes: the 0.6B configuration whole, and the 4B widths in a quarter of its layers.
QWEN3 = {
    "0.6b": dict(vocab=151936, width=1024, ff=3072, layers=28, heads=16, kv_heads=8),
    "4b": dict(vocab=151936, width=2560, ff=9728, layers=9, heads=32, kv_heads=8),
}
#: Whisper-small's encoder.
WHISPER = dict(mels=80, width=768, heads=12, layers=12, positions=1500)
LAYERS = {"vogozen": 6, "pedorax": 4}


# ----------------------------------------------------------------------------- cases
def listed():
    return [
        # one attention call of an eager program, fp32: launch and latency
        {"name": "attention_f32_s128", "kind": "attention", "batch": 1, "heads": 16, "kv_heads": 8, "tokens": 128, "dim": 128, "causal": True},
        # the unmodified model code: fp32 modules, a prompt of 512, logits for all positions
        {"name": "module_f32_0.6b_1x512", "kind": "module_prefill", "batch": 1, "tokens": 512, "layers": 28},
        # a short question to an interactive service
        {"name": "qwen3_prefill_1x97", "kind": "qwen3_prefill", "model": "0.6b", "batch": 1, "tokens": 97},
        # a few requests of unequal documents padded to one odd length
        {"name": "qwen3_prefill_3x701", "kind": "qwen3_prefill", "model": "0.6b", "batch": 3, "tokens": 701},
        # the benchmark's batch of prompts
        {"name": "qwen3_prefill_32x2048", "kind": "qwen3_prefill", "model": "0.6b", "batch": 32, "tokens": 2048},
        # one user's answer being generated
        {"name": "qwen3_decode_1_at_300", "kind": "qwen3_decode", "model": "0.6b", "batch": 1, "tokens": 300},
        # the benchmark's decode batch
        {"name": "qwen3_decode_32_at_2176", "kind": "qwen3_decode", "model": "0.6b", "batch": 32, "tokens": 2176},
        # one 30 s clip being transcribed, and the benchmark's batch of clips
        {"name": "whisper_1_clip", "kind": "whisper", "clips": 1, "frames": 3000},
        {"name": "whisper_64_clips", "kind": "whisper", "clips": 64, "frames": 3000},
        # one long document read by a recurrent hybrid
        {"name": "vogozen_prefill_1x8192", "kind": "hybrid_prefill", "design": "vogozen", "size": "2k", "batch": 1, "tokens": 8192},
        # the hybrid's decode batch
        {"name": "vogozen_decode_32_at_2048", "kind": "hybrid_decode", "design": "vogozen", "size": "2k", "batch": 32, "tokens": 2048},
        # the other hybrid (latent attention, experts) on a batch of ordinary prompts
        {"name": "pedorax_prefill_8x1000", "kind": "hybrid_prefill", "design": "pedorax", "size": "1k", "batch": 8, "tokens": 1000},
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _prompts(rng, most_batch, least, most, most_tokens):
    tokens = _between(rng, least, most)
    return _between(rng, 1, max(1, min(most_batch, most_tokens // tokens))), tokens


def draw(rng):
    kind = rng.choice(["attention", "module_prefill", "qwen3_prefill", "qwen3_prefill", "qwen3_decode", "qwen3_decode", "whisper", "hybrid_prefill", "hybrid_decode"])
    if kind == "attention":
        kv = rng.choice([1, 2, 4, 8])
        return {"kind": kind, "batch": _between(rng, 1, 4), "heads": kv * rng.choice([1, 2, 4]), "kv_heads": kv, "tokens": _between(rng, 16, 1024),
                "dim": rng.choice([64, 128]), "causal": rng.random() < 0.7}
    if kind == "module_prefill":
        batch, tokens = _prompts(rng, 4, 8, 512, 512)
        return {"kind": kind, "batch": batch, "tokens": tokens, "layers": rng.choice([4, 8])}
    if kind in ("qwen3_prefill", "qwen3_decode"):
        model = rng.choice(["0.6b", "0.6b", "4b"])
        batch, tokens = _prompts(rng, 32, 16, 2300, 32768 if model == "0.6b" else 8192)
        return {"kind": kind, "model": model, "batch": batch, "tokens": tokens}
    if kind == "whisper":
        return {"kind": kind, "clips": _between(rng, 1, 48), "frames": _between(rng, 150, 3000)}
    design, size = rng.choice(["vogozen", "vogozen", "pedorax"]), rng.choice(["1k", "1k", "2k"])
    batch, tokens = _prompts(rng, 32, 16, 6000 if kind == "hybrid_prefill" else 2048, 12288)
    return {"kind": kind, "design": design, "size": size, "batch": batch, "tokens": tokens}


# ----------------------------------------------------------------------------- inputs
class _Device:
    """A device tensor of the framework as torch (and anything else that reads this interface) sees it."""

    def __init__(self, t: Tensor):
        kind, size = {"float32": ("<f4", 4), "bfloat16": ("<i2", 2), "int64": ("<i8", 8), "int32": ("<i4", 4)}[t.dtype]
        self.kept = t
        self.__cuda_array_interface__ = {"shape": tuple(t.shape), "typestr": kind, "data": (t._handle.storage.device_ptr() + t.offset * size, False),
                                         "strides": tuple(s * size for s in t.strides), "version": 2}


def _torch(t: Tensor) -> torch.Tensor:
    x = torch.as_tensor(_Device(t), device="cuda")
    return x.view(torch.bfloat16) if t.dtype == "bfloat16" else x


def _ids(seed, shape, vocab):
    return np.random.Generator(np.random.PCG64([seed, 1])).integers(0, vocab, size=shape, dtype=np.int32)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _attention_inputs(c, seed):
    g = _generator(seed)
    return [torch.randn(c["batch"], c[h], c["tokens"], c["dim"], generator=g, device="cuda") for h in ("heads", "kv_heads", "kv_heads")]


def _qwen3_config(m, dtype):
    return Qwen3Config(vocabSize=m["vocab"], hiddenSize=m["width"], intermediateSize=m["ff"], numHiddenLayers=m["layers"], numAttentionHeads=m["heads"],
                       numKeyValueHeads=m["kv_heads"], headDim=128, dtype=dtype)


def _module_weights(m, seed):
    """Checkpoint names -> fp32 tensors of the Qwen3 module."""
    g = _generator(seed)
    W, D = m["width"], 128
    shapes = {"self_attn.q_proj": (m["heads"] * D, W), "self_attn.k_proj": (m["kv_heads"] * D, W), "self_attn.v_proj": (m["kv_heads"] * D, W),
              "self_attn.o_proj": (W, m["heads"] * D), "mlp.gate_proj": (m["ff"], W), "mlp.up_proj": (m["ff"], W), "mlp.down_proj": (W, m["ff"])}
    normal = lambda s: torch.randn(s, generator=g, device="cuda") * STD  # noqa: E731
    w = {"model.embed_tokens.weight": normal((m["vocab"], W)), "model.norm.weight": torch.ones(W, device="cuda")}
    for i in range(m["layers"]):
        p = f"model.layers.{i}."
        w.update({p + n + ".weight": normal(s) for n, s in shapes.items()})
        w.update({p + n + ".weight": torch.ones(s, device="cuda") for n, s in (("self_attn.q_norm", D), ("self_attn.k_norm", D), ("input_layernorm", W),
                                                                              ("post_attention_layernorm", W))})
    return w


def _whisper_weights(seed):
    """Checkpoint names -> tensors of Whisper-small's encoder, rounded to bf16."""
    g = _generator(seed)
    E, w = WHISPER["width"], {}

    def put(name, *shape, mean=0.0):
        w[name] = (torch.randn(shape, generator=g, device="cuda") * STD + mean).bfloat16().float()

    def norm(name):
        put(name + ".weight", E, mean=1.0)
        put(name + ".bias", E)

    put("conv1.weight", E, WHISPER["mels"], 3), put("conv1.bias", E), put("conv2.weight", E, E, 3), put("conv2.bias", E)
    put("embed_positions.weight", WHISPER["positions"], E)
    for i in range(WHISPER["layers"]):
        p = f"layers.{i}."
        norm(p + "self_attn_layer_norm"), norm(p + "final_layer_norm")
        put(p + "self_attn.in_proj_weight", 3 * E, E), put(p + "self_attn.in_proj_bias", 3 * E)
        put(p + "self_attn.out_proj.weight", E, E), put(p + "self_attn.out_proj.bias", E)
        put(p + "fc1.weight", 4 * E, E), put(p + "fc1.bias", 4 * E), put(p + "fc2.weight", E, 4 * E), put(p + "fc2.bias", E)
    norm("layer_norm")
    return w


def _mel(c, seed):
    """Log-mel features after the extractor's scaling: about -1 to 1.5, quiet stretches at the floor."""
    x = torch.randn(c["clips"], WHISPER["mels"], c["frames"], generator=_generator(seed + 1), device="cuda") * 0.5
    return x.clamp(-0.8, 1.5).bfloat16()


def _host(w):
    return {k: v.cpu().numpy() for k, v in w.items()}


def _hybrid_config(c):
    make = {"vogozen": vogozen_config, "pedorax": pedorax_config}[c["design"]]
    return make(SIZES[c["size"]], LAYERS[c["design"]])


def _steps(c):
    """Places of the sequence that a pass fills: a prompt, or the steps behind one."""
    return (c["tokens"], c["tokens"] + STEPS) if c["kind"].endswith("decode") else (0, c["tokens"])


def _sequence_ids(c, seed):
    vocab = QWEN3[c["model"]]["vocab"] if "model" in c else HYBRID_VOCAB
    return _ids(seed, (c["batch"], _steps(c)[1]), vocab)


def prepare(case, seed):
    kandle_b200.init(0)
    c, kind = dict(case), case["kind"]
    s = {"case": c}
    if kind == "attention":
        s["qkv"] = [Tensor(x.cpu().numpy()) for x in _attention_inputs(c, seed)]
    elif kind == "module_prefill":
        m = dict(QWEN3["0.6b"], layers=c["layers"])
        s["model"] = Qwen3ForCausalLM(_qwen3_config(m, "float32"))
        s["model"].loadStateDict(_host(_module_weights(m, seed)))
        s["ids"] = Tensor(_ids(seed, (c["batch"], c["tokens"]), m["vocab"]))
    elif kind == "whisper":
        enc = WhisperAudioEncoder(WhisperConfig(nMels=WHISPER["mels"], nAudioCtx=WHISPER["positions"], nAudioState=WHISPER["width"],
                                                nAudioHead=WHISPER["heads"], nAudioLayer=WHISPER["layers"], dtype="bfloat16"))
        enc.loadStateDict(_host(_whisper_weights(seed)))
        s["engine"] = WhisperEncoderEngine(enc)
        s["mel"] = Tensor(_mel(c, seed).float().cpu().numpy(), dtype="bfloat16")
    else:
        B, P = c["batch"], c["tokens"]
        ids = _sequence_ids(c, seed)
        if kind.startswith("qwen3"):
            eng = Qwen3Engine(_qwen3_config(QWEN3[c["model"]], "bfloat16"), RandomInit(seed=seed, std=STD), B, P + 64)
        else:
            eng = HybridEngine(_hybrid_config(c), RandomInit(seed=seed, std=STD), B, P + 64)
        s.update(engine=eng, ids=np.ascontiguousarray(ids[:, :P]))
        if kind.endswith("decode"):
            eng.prefill(s["ids"])
            given = Tensor(np.ascontiguousarray(ids[:, P:].T).astype(np.int64))
            s["given"] = [given.slice([t, slice(None)]) for t in range(STEPS)]
            if kind.startswith("hybrid"):
                s["carried"] = eng.cache.snapshot()       # the recurrent state behind the prompt
            s["decode"] = eng.start_decode(s["given"][0])
            s["out"] = _kept(s, _torch(s["decode"]["logits"]).view(B, -1))
    return s


def _kept(s, logits):
    """A pass's outputs: logits, cache rows of its places, recurrent states."""
    eng, (a, b) = s["engine"], _steps(s["case"])
    out = {"logits": logits}
    if isinstance(eng, Qwen3Engine):
        for i in range(eng.L):
            out[f"k{i}"], out[f"v{i}"] = (_torch(t)[:, :, a:b] for t in (eng.k_cache[i], eng.v_cache[i]))
        return out
    for i in range(len(eng.mixers)):
        kept = eng.cache.of(i)
        for name in ("keys", "values"):
            if hasattr(kept, name):
                out[f"{name}{i}"] = _torch(getattr(kept, name))[:, :, a:b]
        if hasattr(kept, "rows"):
            out[f"rows{i}"] = _torch(kept.rows)[:, a:b]
        if hasattr(kept, "state"):
            out[f"state{i}"] = _torch(kept.state)
    return out


# ----------------------------------------------------------------------------- a pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "attention":
        return _torch(core.scaledDotProductAttention(*s["qkv"], None, 0.0, s["case"]["causal"]))
    if kind == "module_prefill":
        return _torch(s["model"](s["ids"]))
    if kind == "whisper":
        return _torch(s["engine"].forward(s["mel"]))
    eng, c = s["engine"], s["case"]
    if kind == "qwen3_prefill":
        eng.prefill(s["ids"])
        if "out" not in s:
            s["out"] = _kept(s, _torch(eng._bufs(c["batch"], c["tokens"])["logits"]).view(c["batch"], -1))
        return s["out"]
    if kind == "hybrid_prefill":
        eng.reset()
        logits = _torch(eng.extend(s["ids"]))
        if "out" not in s:
            s["out"] = _kept(s, None)
        return dict(s["out"], logits=logits)
    eng.pos = c["tokens"]
    if kind == "hybrid_decode":
        eng.cache.pos = c["tokens"]
        for t, saved in s["carried"]:
            core.copy_(t, saved)
    eng.start_decode(s["given"][0])
    for t in range(STEPS):
        if t:
            core.copy_(s["decode"]["ids"], s["given"][t])
        eng.decode_step()
    return s["out"]


# ----------------------------------------------------------------------------- work and tolerance
def _pairs(a, b, window=None):
    """Visible (query, key) pairs of queries a..b-1, causal, within a window."""
    return sum(min(i + 1, window or i + 1) for i in range(a, b))


def _qwen3_weights(m):
    """Numbers in the matrices of a layer."""
    return m["width"] * 128 * (2 * m["heads"] + 2 * m["kv_heads"]) + 3 * m["width"] * m["ff"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "attention":
        B, S, D = c["batch"], c["tokens"], c["dim"]
        return {"bytes": 4.0 * B * S * D * (2 * c["heads"] + 2 * c["kv_heads"]), "flops": 4.0 * B * c["heads"] * D * (_pairs(0, S) if c["causal"] else S * S)}
    if kind == "module_prefill":
        m, T = dict(QWEN3["0.6b"], layers=c["layers"]), c["batch"] * c["tokens"]
        flops = 2.0 * T * (m["layers"] * _qwen3_weights(m) + m["vocab"] * m["width"]) + 4.0 * c["batch"] * m["layers"] * m["heads"] * 128 * _pairs(0, c["tokens"])
        return {"bytes": 4.0 * (m["layers"] * _qwen3_weights(m) + m["vocab"] * m["width"] + T * m["vocab"]), "flops": flops}
    if kind == "whisper":
        E, L, F, B = WHISPER["width"], WHISPER["layers"], c["frames"], c["clips"]
        T = (F - 1) // 2 + 1
        weights = L * 12 * E * E + 3 * E * (WHISPER["mels"] + E)
        flops = 2.0 * B * (F * 3 * WHISPER["mels"] * E + T * 3 * E * E + T * L * 12 * E * E) + 4.0 * B * L * E * T * T
        return {"bytes": 2.0 * (weights + B * F * WHISPER["mels"] + B * T * E), "flops": flops}
    B, (a, b) = c["batch"], _steps(c)
    n, passes = b - a, STEPS if kind.endswith("decode") else 1     # tokens of a sequence, readings of the weights
    if kind.startswith("qwen3"):
        m = QWEN3[c["model"]]
        matrices = m["layers"] * _qwen3_weights(m)
        read = sum(range(a, b)) if passes > 1 else 0               # cache rows that the steps read
        rows = 2.0 * 2 * B * m["layers"] * m["kv_heads"] * 128
        flops = 2.0 * B * (n * matrices + passes * m["vocab"] * m["width"]) + 4.0 * B * m["layers"] * m["heads"] * 128 * _pairs(a, b)
        return {"bytes": passes * 2.0 * (matrices + m["vocab"] * m["width"]) + rows * (n + read), "flops": flops}
    z = SIZES[c["size"]]
    W, H, D = z["width"], z["heads"], 128
    matrices = active = state = rows = flops = 0.0
    for i in range(LAYERS[c["design"]]):
        if c["design"] == "vogozen":
            ff = 3 * W * z["top"] * z["ff"]
            if i % 3 == 0:
                mix = W * D * (2 * z["qheads"] + 2 * z["kv_heads"])
                row = 2.0 * 2 * z["kv_heads"] * D
                rows += B * row * (n + (sum(min(p, WINDOW) for p in range(a, b)) if passes > 1 else 0))
                flops += 4.0 * B * z["qheads"] * D * _pairs(a, b, WINDOW)
            elif i % 3 == 1:
                mix = 5 * W * W + 2 * 64 * W
                state += 4.0 * B * W * 64
                flops += 4.5 * B * n * W * 64
            else:
                mix = 5 * W * H * D + 2 * H * W
                state += 4.0 * B * H * D * D
                flops += 6.5 * B * n * H * D * D
            matrices, active = matrices + mix + ff, active + mix + ff
        else:
            expert = 3 * W * z["ff"]
            if i % 2 == 0:
                mix = W * H * D * 4 + 4 * D * W + H * W
                state += 4.0 * B * H * D * D
                flops += 6.5 * B * n * H * D * D
            else:
                mix = W * (H * 192 + z["rank"] + 64) + 2 * H * D * z["rank"] + W * H * D
                rows += 2.0 * B * (z["rank"] + 64) * (n + (sum(range(a, b)) if passes > 1 else 0))
                flops += 2.0 * B * H * (192 + 128) * _pairs(a, b)
            used = min(z["experts"], B * (n if passes == 1 else 1) * z["top"])
            matrices, active = matrices + mix + used * expert, active + mix + z["top"] * expert
    head = HYBRID_VOCAB * W
    return {"bytes": passes * (2.0 * (matrices + head) + 2 * state) + rows, "flops": 2.0 * B * (n * active + passes * head) + flops}


def tolerance(case):
    """Measured distance from `exact`: 2.7e-7 and 2.1e-6 in fp32; in bf16 0.006 to 0.015 (Qwen3, Whisper, Pedorax) and up to
    0.04 in the recurrent states of Vogozen's last layers, most of which two correct implementations share."""
    if case["kind"] in ("attention", "module_prefill"):
        return {"rel": 1e-5}
    return {"rel": 3e-2 if case.get("design") == "vogozen" else 2e-2}


# ----------------------------------------------------------------------------- the same in 64 bits
class _Philox:
    """Philox4x32-10 normals numbered as RandomInit numbers them, on the device."""

    def __init__(self, seed):
        self.seed, self.offset = seed, 0

    def __call__(self, *shape):
        n = math.prod(shape)
        parts = [self._normals(a, min(n, a + (1 << 24))) for a in range(0, n, 1 << 24)]
        self.offset += (n + 1) // 2
        return torch.cat(parts).view(shape)

    def _normals(self, a, b):
        i = torch.arange(a, b, dtype=torch.int64, device="cuda")
        low = 0xFFFFFFFF
        x = [((i >> 1) + self.offset) & low] + [torch.zeros_like(i) for _ in range(3)]
        k0, k1 = self.seed & low, (self.seed >> 32) & low
        for _ in range(10):
            h0, l0 = self._wide(0xD2511F53, x[0])
            h1, l1 = self._wide(0xCD9E8D57, x[2])
            x = [h1 ^ x[1] ^ k0, l1, h0 ^ x[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
        odd = (i & 1).bool()
        u1 = (torch.where(odd, x[2], x[0]) >> 8).float() * 2.0 ** -24
        u2 = (torch.where(odd, x[3], x[1]) >> 8).float() * 2.0 ** -24
        z = torch.sqrt(-2.0 * torch.log(u1.clamp_min(1e-10))) * torch.cos(6.283185307179586 * u2)
        return (z * STD).bfloat16()

    @staticmethod
    def _wide(m, x):
        """High and low word of the 64-bit product of two 32-bit numbers, without overflow."""
        low = m * (x & 0xFFFF)
        mid = m * (x >> 16) + (low >> 16)
        return mid >> 16, ((mid & 0xFFFF) << 16) | (low & 0xFFFF)


def _rms(x, eps=1e-6):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _rotate_half(x, cos, sin):
    u, v = x.chunk(2, -1)
    return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)


def _angles(tokens, freq):
    a = torch.arange(tokens, dtype=torch.float64, device="cuda")[:, None] * freq[None, :]
    return torch.cos(a), torch.sin(a)


def _attend(q, k, v, scale, causal=True, window=None, one=False):
    """q [H, S, d] against k, v [G, S, .]; one: the softmax denominator also holds a one."""
    H, S, _ = q.shape
    k, v = k.repeat_interleave(H // k.shape[0], 0), v.repeat_interleave(H // v.shape[0], 0)
    out = []
    for a in range(0, S, 1024):
        b = min(S, a + 1024)
        lo, hi = (max(0, a + 1 - window) if window else 0), (b if causal else S)
        s = q[:, a:b] @ k[:, lo:hi].transpose(1, 2) * scale
        i, j = torch.arange(a, b, device="cuda")[:, None], torch.arange(lo, hi, device="cuda")[None, :]
        if causal:
            s.masked_fill_(j > i, -math.inf)
        if window:
            s.masked_fill_(i - j >= window, -math.inf)
        if one:
            top = s.amax(-1, keepdim=True).clamp_min(0)
            e = torch.exp(s - top)
            p = e / (e.sum(-1, keepdim=True) + torch.exp(-top))
        else:
            p = torch.softmax(s, -1)
        out.append(p @ v[:, lo:hi])
    return torch.cat(out, 1)


def _qwen3_exact(m, embed, layer, ids, rows, all_logits=False):
    """layer(i): fp64 [wqkv, wo, gate, up, down].  Returns logits and keys, values of the places `rows`."""
    B, S = ids.shape
    H, G, D = m["heads"], m["kv_heads"], 128
    freq = torch.tensor([1.0 / math.pow(1e6, i / 64) for i in range(64)], device="cuda").float().double()
    cos, sin = _angles(S, freq)
    x = embed[torch.from_numpy(ids).long().cuda().view(-1)].double()
    out = {}
    for i in range(m["layers"]):
        wqkv, wo, gate, up, down = layer(i)
        keys, values = [], []
        for b in range(B):
            part = x[b * S:(b + 1) * S]
            q, k, v = (_rms(part) @ wqkv.T).view(S, H + 2 * G, D).transpose(0, 1).split([H, G, G])
            q, k = _rotate_half(_rms(q), cos, sin), _rotate_half(_rms(k), cos, sin)
            part += _attend(q, k, v, D ** -0.5).transpose(0, 1).reshape(S, H * D) @ wo.T
            n = _rms(part)
            part += (_silu(n @ gate.T) * (n @ up.T)) @ down.T
            keys.append(k[:, rows[0]:rows[1]])
            values.append(v[:, rows[0]:rows[1]])
        out[f"k{i}"], out[f"v{i}"] = torch.stack(keys), torch.stack(values)
    last = x if all_logits else x.view(B, S, -1)[:, -1]
    n, table = _rms(last), embed
    out["logits"] = torch.cat([n @ table[a:a + 16384].double().T for a in range(0, m["vocab"], 16384)], -1)
    return out


def _engine_layers(m, seed):
    """The engine's matrices as RandomInit draws them: the embedding, and for each layer q, k, v | o | gate and up rows in
    turn, 16 of each | down."""
    draw, W = _Philox(seed), m["width"]
    embed, layers = draw(m["vocab"], W), []
    for _ in range(m["layers"]):
        wqkv = torch.cat([draw(m[h] * 128, W) for h in ("heads", "kv_heads", "kv_heads")])
        wo, gu, down = draw(W, m["heads"] * 128), draw(2 * m["ff"], W).view(-1, 2, 16, W), draw(W, m["ff"])
        layers.append([wqkv, wo, gu[:, 0].reshape(-1, W), gu[:, 1].reshape(-1, W), down])
    return embed, layers


def _whisper_exact(c, seed):
    w = {k: v.double() for k, v in _whisper_weights(seed).items()}
    E, H = WHISPER["width"], WHISPER["heads"]
    F = torch.nn.functional

    def norm(x, name):
        return F.layer_norm(x, (E,), w[name + ".weight"], w[name + ".bias"], 1e-5)

    def linear(x, name):
        return x @ w[name + ".weight"].T + w[name + ".bias"]

    outs = []
    for mel in _mel(c, seed).double():
        taps = F.pad(mel, (1, 1)).unfold(1, 3, 1)                                    # [mels, L, 3]
        x = _gelu(torch.einsum("clk,ock->lo", taps, w["conv1.weight"]) + w["conv1.bias"])
        taps = F.pad(x.T, (1, 1)).unfold(1, 3, 2)
        x = _gelu(torch.einsum("clk,ock->lo", taps, w["conv2.weight"]) + w["conv2.bias"])
        T = x.shape[0]
        x = x + w["embed_positions.weight"][:T]
        for i in range(WHISPER["layers"]):
            p = f"layers.{i}."
            qkv = norm(x, p + "self_attn_layer_norm") @ w[p + "self_attn.in_proj_weight"].T + w[p + "self_attn.in_proj_bias"]
            q, k, v = qkv.view(T, 3, H, E // H).permute(1, 2, 0, 3)
            o = _attend(q, k, v, (E // H) ** -0.5, causal=False).transpose(0, 1).reshape(T, E)
            x = x + linear(o, p + "self_attn.out_proj")
            x = x + linear(_gelu(linear(norm(x, p + "final_layer_norm"), p + "fc1")), p + "fc2")
        outs.append(norm(x, "layer_norm"))
    return torch.stack(outs)


def _recurrence(step, B, S):
    out = [step(t) for t in range(S)]
    return torch.stack(out, 1)


def _delta(q, k, v, g, beta):
    """Gated delta rule, [B, S, H, .]; g broadcasts over the key channels."""
    B, S, H, d = q.shape
    state = torch.zeros(B, H, d, v.shape[-1], dtype=q.dtype, device="cuda")

    def step(t):
        state.mul_(g[:, t, :, :, None])
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", state, k[:, t]))
        state.addcmul_(k[:, t, :, :, None], u[:, :, None, :])
        return torch.einsum("bhdv,bhd->bhv", state, q[:, t])

    return _recurrence(step, B, S), state


def _wkv(r, k, v, decay, bonus):
    B, S, H, d = r.shape
    state = torch.zeros(B, H, d, d, dtype=r.dtype, device="cuda")

    def step(t):
        o = torch.einsum("bhij,bhi->bhj", state, r[:, t]) + (r[:, t] * bonus * k[:, t]).sum(-1, keepdim=True) * v[:, t]
        state.mul_(decay[:, t, :, :, None]).addcmul_(k[:, t, :, :, None], v[:, t, :, None, :])
        return o

    return _recurrence(step, B, S), state


def _conv_silu(x, taps):
    n = taps.shape[1]
    padded = torch.nn.functional.pad(x, (0, 0, n - 1, 0))
    return _silu(sum(padded[:, j:j + x.shape[1]] * taps[:, j] for j in range(n)))


def _unit(x):
    return x * torch.rsqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6)


def _delta_heads(cols, taps, B, S, H):
    q, k, v = (_conv_silu(x, t).view(B, S, H, 128) for x, t in zip(cols, taps))
    return _unit(q) * 128 ** -0.5, _unit(k), v


def _taps(rng, H):
    return [torch.from_numpy((rng.standard_normal((H * 128, 4)) * 0.5).astype(np.float32)).double().cuda() for _ in range(3)]


def _vogozen_exact(c, seed, ids):
    z, draw, rng = SIZES[c["size"]], _Philox(seed), np.random.Generator(np.random.PCG64(seed))
    W, H, G, HD, ff = z["width"], z["qheads"], z["kv_heads"], z["heads"], z["top"] * z["ff"]
    (B, S), (a, b) = ids.shape, _steps(c)
    x = draw(HYBRID_VOCAB, W)[torch.from_numpy(ids).long().cuda()].double()
    cos, sin = _angles(S, 1e6 ** (-2.0 * torch.arange(64, dtype=torch.float64, device="cuda") / 128))
    out = {}
    for i in range(LAYERS["vogozen"]):
        if i % 3 == 0:
            proj, wo = draw((H + 2 * G) * 128, W).double(), draw(W, H * 128).double()
            y, keys, values = torch.empty_like(x), [], []
            for s in range(B):
                q, k, v = (x[s] @ proj.T).split([H * 128, G * 128, G * 128], -1)
                q, k = (_rotate_half(_rms(t).view(S, -1, 128).transpose(0, 1), cos, sin) for t in (q, k))
                v = v.reshape(S, G, 128).transpose(0, 1)
                y[s] = _attend(q, k, v, 128 ** -0.5, window=WINDOW, one=True).transpose(0, 1).reshape(S, -1) @ wo.T
                keys.append(k[:, a:b])
                values.append(v[:, a:b])
            out[f"keys{i}"], out[f"values{i}"] = torch.stack(keys), torch.stack(values)
        elif i % 3 == 1:
            w4, w1, w2, wo = draw(4, W, W).double(), draw(64, W).double(), draw(W, 64).double(), draw(W, W).double()
            mix = (x + torch.nn.functional.pad(x, (0, 0, 1, 0))[:, :-1]) * 0.5
            r, k, v, gate = (mix @ w.T for w in w4)
            decay = torch.exp(-torch.exp(torch.tanh(mix @ w1.T) @ w2.T - 1.0))
            r, k, v, decay = (t.view(B, S, W // 64, 64) for t in (r, k, v, decay))
            o, out[f"state{i}"] = _wkv(r, k, v, decay, 0.5)
            y = (_rms(o).view(B, S, W) * _silu(gate)) @ wo.T
        else:
            taps, wo = _taps(rng, HD), draw(W, HD * 128).double()
            n = -(-(4 * HD * 128 + -(-HD // 8) * 8) // 32) * 32
            proj = draw(n + -(-HD // 8) * 8, W).double()
            p = x @ proj.T
            q, k, v, gate = p[..., :4 * HD * 128].chunk(4, -1)
            beta = torch.sigmoid(p[..., 4 * HD * 128:4 * HD * 128 + HD])
            g = torch.exp(-math.exp(-1.0) * torch.nn.functional.softplus(p[..., n:n + HD] - 3.0))
            o, out[f"state{i}"] = _delta(*_delta_heads((q, k, v), taps, B, S, HD), g[..., None], beta)
            y = (_rms(o) * _silu(gate).view(B, S, HD, 128)).view(B, S, -1) @ wo.T
        x = x + _rms(y)
        gu, down = draw(2 * ff, W).view(-1, 2, 16, W).double(), draw(W, ff).double()
        x = x + _rms((_gelu(x @ gu[:, 0].reshape(-1, W).T) * (x @ gu[:, 1].reshape(-1, W).T)) @ down.T)
    out["logits"] = _rms(x[:, -1]) @ draw(HYBRID_VOCAB, W).double().T
    return out


def _rotate_pairs(x, cos, sin):
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2)


def _pedorax_exact(c, seed, ids):
    z, draw, rng = SIZES[c["size"]], _Philox(seed), np.random.Generator(np.random.PCG64(seed))
    W, H, R, E, ff = z["width"], z["heads"], z["rank"], z["experts"], z["ff"]
    (B, S), (a, b) = ids.shape, _steps(c)
    embed = draw(HYBRID_VOCAB, W)
    x = embed[torch.from_numpy(ids).long().cuda()].double()
    cos, sin = _angles(S, 1e4 ** (-2.0 * torch.arange(32, dtype=torch.float64, device="cuda") / 64))
    up = lambda n, m: -(-n // m) * m  # noqa: E731
    expanded = (a or b) >= 64         # prompts of 64 tokens and more multiply by matrices of their own, drawn beside the others
    out = {}
    for i in range(LAYERS["pedorax"]):
        h = torch.tanh(0.5 * x)
        if i % 2 == 0:
            taps, wo = _taps(rng, H), draw(W, H * 128).double()
            n = up(3 * H * 128 + 256 + up(H, 8), 32)
            proj = draw(n + up(E, 8), W).double()
            a2, g2 = draw(H * 128, 128).double(), draw(H * 128, 128).double()
            p = h @ proj.T
            at = 3 * H * 128
            q, k, v = p[..., :at].chunk(3, -1)
            decay = p[..., at:at + 128] @ a2.T
            gate = torch.sigmoid(p[..., at + 128:at + 256] @ g2.T).view(B, S, H, 128)
            beta = torch.sigmoid(p[..., at + 256:at + 256 + H])
            g = torch.exp(-math.exp(-1.0) * torch.nn.functional.softplus(decay - 3.0)).view(B, S, H, 128)
            o, out[f"state{i}"] = _delta(*_delta_heads((q, k, v), taps, B, S, H), g, beta)
            y = (_rms(o) * gate).view(B, S, -1) @ wo.T
        else:
            n = up(up(H * 192, 8) + up(R + 64, 8), 32)
            proj, wo = draw(n + up(E, 8), W).double(), draw(W, H * 128).double()
            _, wuk_t, _, wuv, wukv = draw(H, 128, R), draw(H, R, 128), draw(H, R, 128), draw(H, 128, R), draw(2 * H * 128, R)
            absorbed = wuk_t.double().transpose(1, 2), wuv.double()                  # [H, 128, R] each
            whole = tuple(t.view(H, 128, R).double() for t in wukv.chunk(2))
            p = h @ proj.T
            y, kept = torch.empty_like(x), []
            for s in range(B):
                q = p[s, :, :H * 192].reshape(S, H, 192).transpose(0, 1)
                latent = _rms(p[s, :, H * 192:H * 192 + R])
                rot = _rotate_pairs(p[s, :, H * 192 + R:H * 192 + R + 64], cos, sin)
                q = torch.cat([q[..., :128], _rotate_pairs(q[..., 128:], cos, sin)], -1)

                def attend(uk, uv):
                    k = torch.cat([torch.einsum("tr,hdr->htd", latent, uk), rot.expand(H, S, 64)], -1)
                    return _attend(q, k, torch.einsum("tr,hdr->htd", latent, uv), 192 ** -0.5, one=True)

                o = attend(*(whole if expanded else absorbed))
                if a:
                    o[:, a:] = attend(*absorbed)[:, a:]
                y[s] = o.transpose(0, 1).reshape(S, -1) @ wo.T
                kept.append(torch.cat([latent, rot], -1)[a:b])
            out[f"rows{i}"] = torch.stack(kept)
        scores = torch.sigmoid(p[..., n:n + E]).view(B * S, E)
        grouped = scores.view(B * S, z["groups"], -1)
        best = grouped.topk(2, -1)[0].sum(-1).topk(z["keep"], -1)[1]
        allowed = torch.zeros(B * S, z["groups"], dtype=torch.bool, device="cuda").scatter_(1, best, True)
        masked = scores.masked_fill(~allowed.repeat_interleave(E // z["groups"], 1), -1.0)
        top, chosen = masked.topk(z["top"], -1)
        top = top / (top.sum(-1, keepdim=True) + 1e-20)
        gu, down = draw(E, 2 * ff, W).view(E, ff // 16, 2, 16, W), draw(E, W, ff)
        flat, y = h.view(B * S, W), y.view(B * S, W)
        for e in range(E):
            t, slot = (chosen == e).nonzero(as_tuple=True)
            g = (flat[t] @ gu[e, :, 0].reshape(ff, W).double().T).clamp_max(7.0)
            u = (flat[t] @ gu[e, :, 1].reshape(ff, W).double().T).clamp(-7.0, 7.0)
            y.index_add_(0, t, top[t, slot][:, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ down[e].double().T))
        x = x + y.view(B, S, W)
    out["logits"] = torch.tanh(0.5 * x[:, -1]) @ embed.double().T
    return out


def exact(case, seed):
    c, kind = dict(case), case["kind"]
    with torch.no_grad():
        if kind == "attention":
            return torch.stack([_attend(*(t.double() for t in qkv), c["dim"] ** -0.5, c["causal"]) for qkv in zip(*_attention_inputs(c, seed))])
        if kind == "module_prefill":
            m = dict(QWEN3["0.6b"], layers=c["layers"])
            w = _module_weights(m, seed)

            def layer(i):
                g = lambda n: w[f"model.layers.{i}.{n}.weight"].double()  # noqa: E731
                return (torch.cat([g(f"self_attn.{n}_proj") for n in "qkv"]), g("self_attn.o_proj"), g("mlp.gate_proj"), g("mlp.up_proj"), g("mlp.down_proj"))

            ids = _ids(seed, (c["batch"], c["tokens"]), m["vocab"])
            return _qwen3_exact(m, w["model.embed_tokens.weight"], layer, ids, (0, 0), True)["logits"].view(*ids.shape, -1)
        if kind == "whisper":
            return _whisper_exact(c, seed)
        ids = _sequence_ids(c, seed)
        if kind.startswith("qwen3"):
            m = QWEN3[c["model"]]
            embed, layers = _engine_layers(m, seed)
            return _qwen3_exact(m, embed, lambda i: [t.double() for t in layers[i]], ids, _steps(c))
        return (_vogozen_exact if c["design"] == "vogozen" else _pedorax_exact)(c, seed, ids)
