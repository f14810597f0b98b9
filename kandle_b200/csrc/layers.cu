// The layers of a prompt (Qwen3) and of Whisper's encoder as one call each: the same kernels in the same order as the calls of the
// engines, without the host language between them.  What bounds short inputs is the host: a launch cost 9 us (Qwen3Engine.prefill)
// to 17 us (WhisperEncoderEngine.forward) from Python, of which the library needs 3 to 4.
#include <algorithm>
#include <initializer_list>
#include <utility>

#include "common.cuh"
#include "kernels.cuh"

using namespace kd;

namespace {

// A dense view [n0, ...] of a storage, from element `offset` on.
kd_tensor dense(uint64_t storage, int dtype, int64_t offset, std::initializer_list<int64_t> shape) {
  kd_tensor t{};
  t.storage = storage;
  t.offset = offset;
  t.dtype = dtype;
  t.ndim = (int)shape.size();
  int64_t stride = 1;
  for (int i = t.ndim - 1; i >= 0; --i) {
    t.shape[i] = shape.begin()[i];
    t.strides[i] = stride;
    stride *= t.shape[i];
  }
  return t;
}

kd_tensor swapped(kd_tensor t, int a, int b) {
  std::swap(t.shape[a], t.shape[b]);
  std::swap(t.strides[a], t.strides[b]);
  return t;
}

kd_tensor narrowed(kd_tensor t, int dim, int64_t n) {
  t.shape[dim] = n;
  return t;
}

// A block of the caching allocator for as long as the calls that use it are being enqueued (the stream orders its reuse).
struct Scratch {
  uint64_t storage = 0;
  ~Scratch() { if (storage) kd_storage_release(storage); }
};

}  // namespace

KD_API int kd_qwen3_prompt_layers(const kd_tensor* const* layer_tensors, int n_layers, const kd_tensor* x, const kd_tensor* h, const kd_tensor* h1,
                                  const kd_tensor* q, const kd_tensor* attn, const kd_tensor* act, const kd_tensor* cos, const kd_tensor* sin,
                                  float eps, float scale) {
  KD_TRY(require_init());
  KD_REQUIRE(layer_tensors && x && h && h1 && q && attn && act && cos && sin, "null tensor");
  KD_REQUIRE(n_layers >= 1, "no layers");
  for (int i = 0; i < 10 * n_layers; ++i) KD_REQUIRE(layer_tensors[i], "null tensor in layer %d", i / 10);
  KD_REQUIRE(q->ndim == 4 && attn->ndim == 4 && is_contiguous(attn), "q and attn must be [B,S,Hq,128], attn contiguous");
  const int64_t B = q->shape[0], S = q->shape[1];
  const kd_tensor q_heads = swapped(*q, 1, 2), o_heads = swapped(*attn, 1, 2);
  const kd_tensor attn2 = dense(attn->storage, attn->dtype, attn->offset, {B * S, attn->shape[2] * attn->shape[3]});
  for (int l = 0; l < n_layers; ++l) {
    const kd_tensor* const* w = layer_tensors + 10 * l;       // in_norm, wqkv, q_norm, k_norm, wo, post_norm, wgu, wdown, K cache, V cache
    KD_REQUIRE(w[8]->ndim == 4 && w[9]->ndim == 4 && w[8]->shape[0] >= B && w[9]->shape[0] >= B && w[8]->shape[2] >= S && w[9]->shape[2] >= S,
               "caches of layer %d are smaller than the prompt", l);
    const kd_tensor kc = narrowed(*w[8], 0, B), vc = narrowed(*w[9], 0, B);
    const kd_tensor kp = narrowed(kc, 2, S), vp = narrowed(vc, 2, S);
    KD_TRY(kd_add_rmsnorm(h, nullptr, w[0], eps, nullptr, x));
    KD_TRY(kd_qkv_linear_norm_rope_cachewrite(x, w[1], w[2], w[3], eps, cos, sin, &kc, &vc, 0, q));
    KD_TRY(kd_flash_attention(&q_heads, &kp, &vp, &o_heads, scale, 1));
    KD_TRY(kd_linear_bf16(&attn2, w[4], h, KD_EPI_RESIDUAL, h1));
    KD_TRY(kd_add_rmsnorm(h1, nullptr, w[5], eps, nullptr, x));
    KD_TRY(kd_linear_bf16(x, w[6], nullptr, KD_EPI_SWIGLU, act));
    KD_TRY(kd_linear_bf16(act, w[7], h1, KD_EPI_RESIDUAL, h));
  }
  return KD_OK;
}

KD_API int kd_whisper_encoder_layers(const kd_tensor* const* layer_tensors, int n_layers, int heads, const float* eps, float scale, const kd_tensor* x,
                                     const kd_tensor* out) {
  KD_TRY(require_init());
  KD_REQUIRE(layer_tensors && eps && x && out, "null tensor");
  KD_REQUIRE(n_layers >= 1 && heads >= 1, "no layers or heads");
  KD_REQUIRE(x->ndim == 3 && out->ndim == 3 && x->dtype == KD_BF16 && out->dtype == KD_BF16 && is_contiguous(x) && is_contiguous(out), "x and out must be contiguous bf16 [B,T,E]");
  const int64_t B = x->shape[0], T = x->shape[1], E = x->shape[2], H = heads, D = E / H;
  for (int i = 0; i < 3; ++i) KD_REQUIRE(out->shape[i] == x->shape[i], "out must have the shape of x");
  KD_REQUIRE(D * H == E, "%lld channels do not divide over %d heads", (long long)E, heads);
  int64_t F = 0;
  for (int l = 0; l < n_layers; ++l) {
    // ln1 w, b; in_proj w, b; out_proj w, b; ln2 w, b; fc1 w, b; fc2 w, b (biases may be null)
    const kd_tensor* const* w = layer_tensors + 12 * l;
    KD_REQUIRE(w[2] && w[4] && w[8] && w[10] && w[8]->ndim == 2, "null matrix in layer %d", l);
    F = std::max(F, w[8]->shape[0]);
  }
  // norm | qkv | attention | first residual | two layer outputs | hidden, one behind the other on 256-byte boundaries
  if (B * T == 0) return KD_OK;
  const int64_t n = (B * T + 127) / 128 * 128;
  Scratch s;
  KD_TRY(kd_storage_alloc((uint64_t)n * (uint64_t)(8 * E + F) * 2, 0, &s.storage));
  auto at = [&](int64_t columns, int64_t width) { return dense(s.storage, KD_BF16, n * columns, {B, T, width}); };
  const kd_tensor y = at(0, E), qkv = at(E, 3 * E), attn = at(4 * E, E), x1 = at(5 * E, E), x2[2] = {at(6 * E, E), at(7 * E, E)};
  kd_tensor part[3];
  for (int j = 0; j < 3; ++j) {
    part[j] = dense(s.storage, KD_BF16, qkv.offset + j * E, {B, T, H, D});
    part[j].strides[0] = T * 3 * E;
    part[j].strides[1] = 3 * E;
    part[j] = swapped(part[j], 1, 2);
  }
  const kd_tensor o = swapped(dense(s.storage, KD_BF16, attn.offset, {B, T, H, D}), 1, 2);
  const kd_tensor* in = x;
  for (int l = 0; l < n_layers; ++l) {
    const kd_tensor* const* w = layer_tensors + 12 * l;
    const kd_tensor hidden = at(8 * E, w[8]->shape[0]);
    const kd_tensor* next = l == n_layers - 1 ? out : &x2[l & 1];
    KD_TRY(kd_layer_norm(in, w[0], w[1], eps[2 * l], &y));
    KD_TRY(kd_linear_bf16_bias(&y, w[2], w[3], nullptr, KD_ACT_NONE, &qkv));
    KD_TRY(kd_flash_attention(&part[0], &part[1], &part[2], &o, scale, 0));
    KD_TRY(kd_linear_bf16_bias(&attn, w[4], w[5], in, KD_ACT_NONE, &x1));
    KD_TRY(kd_layer_norm(&x1, w[6], w[7], eps[2 * l + 1], &y));
    KD_TRY(kd_linear_bf16_bias(&y, w[8], w[9], nullptr, KD_ACT_GELU, &hidden));
    KD_TRY(kd_linear_bf16_bias(&hidden, w[10], w[11], &x1, KD_ACT_NONE, next));
    in = next;
  }
  return KD_OK;
}
