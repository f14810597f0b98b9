// Map kernels: pointwise arithmetic, strided copy / cast, fill, arange.
//
// Replaces the reference's generated pointwise shaders (fast contiguous path + general strided
// path, rank <= 8; packages/backend-webgpu/src/kernels/pointwise/executor.ts:60-130) and the
// copy family (packages/backend-webgpu/src/kernels/copy/index.ts:15-30).  Arithmetic is fp32
// whatever the storage type and rounds once at the output, as the reference does for 16-bit
// storage (packages/backend-webgpu/src/base/dtype.ts:50-74).
//
// HBM-bound: the contiguous paths move 16 bytes per thread per access and size the grid as a
// multiple of the SM count.
#include "common.cuh"

namespace kd {

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }

// Expression table restated from packages/backend-webgpu/src/kernels/pointwise/ops.ts:
//   add a + alpha*b (:437-444), silu x/(1+exp(-clamp(x,+-88))) (:299),
//   gelu 0.5x(1+tanh(clamp(0.7978845608(x+0.044715x^3),+-20))) (:301), tanh clamp +-20 (:211),
//   sigmoid clamp +-88 (:297).  expf/tanhf/cosf/sinf are the accurate library versions.
__device__ __forceinline__ float apply_op(int op, float a, float b, float s) {
  switch (op) {
    case KD_OP_ADD: return a + s * b;
    case KD_OP_SUB: return a - s * b;
    case KD_OP_MUL: return a * b;
    case KD_OP_MUL_SCALAR: return a * s;
    case KD_OP_NEG: return -a;
    case KD_OP_COS: return cosf(a);
    case KD_OP_SIN: return sinf(a);
    case KD_OP_SILU: return a / (1.0f + expf(-clampf(a, -88.f, 88.f)));
    case KD_OP_GELU: {
      const float inner = 0.7978845608f * (a + 0.044715f * a * a * a);
      return 0.5f * a * (1.0f + tanhf(clampf(inner, -20.f, 20.f)));
    }
    case KD_OP_ABS: return fabsf(a);
    case KD_OP_DIV: return a / b;
    case KD_OP_MAXIMUM: return fmaxf(a, b);
    case KD_OP_TANH: return tanhf(clampf(a, -20.f, 20.f));
    case KD_OP_SIGMOID: return 1.0f / (1.0f + expf(-clampf(a, -88.f, 88.f)));
    default: return a;
  }
}

struct PwParams {
  int op;
  int ndim;
  int dt_a, dt_b, dt_o;
  int has_b;
  int int_mode;  // both operands integer: move values as int64 without a float round trip
  float scalar;
  int64_t n;
  int64_t shape[KD_MAX_DIMS];
  int64_t sa[KD_MAX_DIMS], sb[KD_MAX_DIMS], so[KD_MAX_DIMS];
};

__global__ void pointwise_strided_kernel(const void* __restrict__ a, const void* __restrict__ b, void* __restrict__ o,
                                         PwParams p) {
  pdl_wait();
  pdl_trigger();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += stride) {
    int64_t lin = i, oa = 0, ob = 0, oo = 0;
#pragma unroll 1
    for (int d = p.ndim - 1; d >= 0; --d) {
      const int64_t s = p.shape[d];
      const int64_t q = lin / s;
      const int64_t r = lin - q * s;
      oa += r * p.sa[d];
      ob += r * p.sb[d];
      oo += r * p.so[d];
      lin = q;
    }
    if (p.int_mode) {
      int64_t v;
      switch (p.dt_a) {
        case KD_I64: v = static_cast<const int64_t*>(a)[oa]; break;
        case KD_I32: v = static_cast<const int32_t*>(a)[oa]; break;
        default: v = static_cast<const uint8_t*>(a)[oa]; break;
      }
      switch (p.dt_o) {
        case KD_I64: static_cast<int64_t*>(o)[oo] = v; break;
        case KD_I32: static_cast<int32_t*>(o)[oo] = (int32_t)v; break;
        default: static_cast<uint8_t*>(o)[oo] = (uint8_t)v; break;
      }
      continue;
    }
    const float va = load_float(a, p.dt_a, oa);
    const float vb = p.has_b ? load_float(b, p.dt_b, ob) : 0.f;
    store_float(o, p.dt_o, oo, apply_op(p.op, va, vb, p.scalar));
  }
}

// Contiguous, same dtype for all operands: 16 bytes per thread per access.
template <typename T, int VEC>
__global__ void pointwise_contig_kernel(const T* __restrict__ a, const T* __restrict__ b, T* __restrict__ o, int op,
                                        int has_b, float scalar, int64_t n_vec, int64_t n) {
  struct alignas(16) Pack { T v[VEC]; };
  pdl_wait();
  pdl_trigger();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_vec; i += stride) {
    Pack pa = reinterpret_cast<const Pack*>(a)[i];
    Pack pb;
    if (has_b) pb = reinterpret_cast<const Pack*>(b)[i];
    Pack po;
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const float va = (float)pa.v[j];
      const float vb = has_b ? (float)pb.v[j] : 0.f;
      po.v[j] = (T)apply_op(op, va, vb, scalar);
    }
    reinterpret_cast<Pack*>(o)[i] = po;
  }
  // tail
  const int64_t tail0 = n_vec * VEC;
  for (int64_t i = tail0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const float va = (float)a[i];
    const float vb = has_b ? (float)b[i] : 0.f;
    o[i] = (T)apply_op(op, va, vb, scalar);
  }
}

// Floating-point operands whose rows come in pieces of four elements: every thread takes pieces of four, the output's
// dimensions merged where all operands allow it.  HBM-bound; pointwise_strided_kernel, one element a thread and a 64-bit
// division per dimension, took 325 us to widen 65536 x 1024 bf16 numbers (403 MB), and 10.5 us for the 2 MB slices, head
// permutations and broadcast products of rotary embeddings.
// n / d for n < 2^31 by a multiplication: division by an invariant integer after Granlund and Montgomery (1994), the
// multiplier rounded up.
struct FastDiv {
  uint32_t d, mul, shift;
  __device__ __forceinline__ uint32_t operator()(uint32_t n) const { return (__umulhi(n, mul) + n) >> shift; }
};

constexpr int PV_DIMS = 4;

struct PvParams {
  int op, ndim;                  // dimensions, innermost (in pieces) first
  int dt_a, dt_b, dt_o;
  int has_b, one_a, one_b;       // one: a row of this input is one number
  float scalar;
  uint32_t n;                    // pieces
  FastDiv shape[PV_DIMS];
  int64_t sa[PV_DIMS], sb[PV_DIMS], so[PV_DIMS];
};

__device__ __forceinline__ void load_piece(const void* base, int dt, int64_t at, int one, float (&v)[4]) {
  if (one) {
    v[0] = v[1] = v[2] = v[3] = load_float(base, dt, at);
  } else if (dt == KD_F32) {
    const float4 f = *reinterpret_cast<const float4*>(static_cast<const float*>(base) + at);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
    const uint2 u = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + at);
    const uint16_t h[4] = {(uint16_t)u.x, (uint16_t)(u.x >> 16), (uint16_t)u.y, (uint16_t)(u.y >> 16)};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = dt == KD_BF16 ? __uint_as_float((uint32_t)h[i] << 16) : __half2float(__ushort_as_half(h[i]));
  }
}

__global__ void __launch_bounds__(256) pointwise_pieces_kernel(const void* __restrict__ a, const void* __restrict__ b, void* __restrict__ o, PvParams p) {
  pdl_wait();
  pdl_trigger();
  for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < p.n; i += gridDim.x * 256) {
    uint32_t lin = i;
    int64_t oa = 0, ob = 0, oo = 0;
#pragma unroll
    for (int d = 0; d < PV_DIMS; ++d) {
      if (d < p.ndim) {
        const uint32_t q = d + 1 < p.ndim ? p.shape[d](lin) : 0;
        const int64_t r = lin - q * p.shape[d].d;
        oa += r * p.sa[d];
        ob += r * p.sb[d];
        oo += r * p.so[d];
        lin = q;
      }
    }
    float va[4], vb[4] = {0.f, 0.f, 0.f, 0.f}, y[4];
    load_piece(a, p.dt_a, oa, p.one_a, va);
    if (p.has_b) load_piece(b, p.dt_b, ob, p.one_b, vb);
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = apply_op(p.op, va[j], vb[j], p.scalar);
    if (p.dt_o == KD_F32) {
      *reinterpret_cast<float4*>(static_cast<float*>(o) + oo) = make_float4(y[0], y[1], y[2], y[3]);
    } else {
      uint16_t h[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = p.dt_o == KD_BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(y[j])) : __half_as_ushort(__float2half_rn(y[j]));
      *reinterpret_cast<uint2*>(static_cast<uint16_t*>(o) + oo) = make_uint2(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16);
    }
  }
}

static int grid_for(int64_t work_items, int threads) {
  const int sms = ctx().sm_count > 0 ? ctx().sm_count : 148;
  int64_t blocks = (work_items + threads - 1) / threads;
  const int64_t cap = (int64_t)sms * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static bool same_shape(const kd_tensor* a, const kd_tensor* b) {
  if (a->ndim != b->ndim) return false;
  for (int i = 0; i < a->ndim; ++i)
    if (a->shape[i] != b->shape[i]) return false;
  return true;
}

// Right-align `t` against `out` and produce broadcast strides (0 where t's extent is 1).
static int broadcast_strides(const kd_tensor* t, const kd_tensor* out, int64_t* st, const char* what) {
  const int shift = out->ndim - t->ndim;
  if (shift < 0) return fail(KD_ERR_INVALID, "%s has higher rank (%d) than the output (%d)", what, t->ndim, out->ndim);
  for (int d = 0; d < out->ndim; ++d) {
    if (d < shift) { st[d] = 0; continue; }
    const int64_t e = t->shape[d - shift];
    if (e == out->shape[d]) st[d] = t->strides[d - shift];
    else if (e == 1) st[d] = 0;
    else return fail(KD_ERR_INVALID, "%s extent %lld does not broadcast to %lld at dim %d", what, (long long)e,
                     (long long)out->shape[d], d);
  }
  return KD_OK;
}

static FastDiv fast_div(uint32_t d) {
  uint32_t shift = 0;
  while ((1ull << shift) < d) ++shift;
  return {d, (uint32_t)((((1ull << shift) - d) << 32) / d + 1), shift};
}

// Plans pointwise_pieces_kernel; false where the operands do not come in aligned pieces of four.
static bool plan_pieces(const PwParams& g, const void* a, const void* b, const void* o, PvParams* out) {
  PvParams p{};
  const int dts[3] = {g.dt_a, g.has_b ? g.dt_b : g.dt_a, g.dt_o};
  for (int dt : dts)
    if (!is_float_dtype(dt)) return false;
  if (g.n >= (1ll << 32) || g.ndim < 1) return false;      // (pieces are counted below 2^30)
  // Dimensions, innermost first, without those of one element; neighbours that are one run in every operand are merged.
  int64_t shape[KD_MAX_DIMS], st[3][KD_MAX_DIMS];
  int n = 0;
  for (int d = g.ndim - 1; d >= 0; --d) {
    if (g.shape[d] == 1) continue;
    const int64_t s[3] = {g.sa[d], g.has_b ? g.sb[d] : g.sa[d], g.so[d]};
    if (n > 0 && s[0] == st[0][n - 1] * shape[n - 1] && s[1] == st[1][n - 1] * shape[n - 1] && s[2] == st[2][n - 1] * shape[n - 1]) {
      shape[n - 1] *= g.shape[d];
      continue;
    }
    shape[n] = g.shape[d];
    for (int i = 0; i < 3; ++i) st[i][n] = s[i];
    ++n;
  }
  if (n == 0 || n > PV_DIMS || shape[0] % 4) return false;
  const void* ptr[3] = {a, g.has_b ? b : a, o};
  int one[3];
  for (int i = 0; i < 3; ++i) {
    one[i] = i < 2 && st[i][0] == 0;
    if (!one[i]) {
      if (st[i][0] != 1 || (reinterpret_cast<uintptr_t>(ptr[i]) & (4 * dtype_size(dts[i]) - 1))) return false;
      for (int d = 1; d < n; ++d)
        if (st[i][d] & 3) return false;
    }
  }
  p.op = g.op; p.ndim = n; p.dt_a = dts[0]; p.dt_b = dts[1]; p.dt_o = dts[2];
  p.has_b = g.has_b; p.one_a = one[0]; p.one_b = one[1]; p.scalar = g.scalar;
  p.n = (uint32_t)(g.n / 4);
  for (int d = 0; d < n; ++d) {
    p.shape[d] = fast_div((uint32_t)(d ? shape[d] : shape[0] / 4));
    const int64_t unit = d ? 1 : 4;
    p.sa[d] = st[0][d] * unit; p.sb[d] = st[1][d] * unit; p.so[d] = st[2][d] * unit;
  }
  *out = p;
  return true;
}

static int launch_pointwise(int op, const kd_tensor* a, const kd_tensor* b, float scalar, const kd_tensor* out) {
  KD_TRY(require_init());
  KD_REQUIRE(a && out, "null tensor");
  void *pa = nullptr, *pb = nullptr, *po = nullptr;
  KD_TRY(tensor_ptr(a, &pa));
  if (b) KD_TRY(tensor_ptr(b, &pb));
  KD_TRY(tensor_ptr(out, &po));
  const int64_t n = numel(out);
  if (n == 0) return KD_OK;
  cudaStream_t st = ctx().stream;

  const bool fast = is_contiguous(out) && is_contiguous(a) && same_shape(a, out) && a->dtype == out->dtype &&
                    (!b || (is_contiguous(b) && same_shape(b, out) && b->dtype == out->dtype)) && aligned16(pa) &&
                    aligned16(po) && (!b || aligned16(pb)) && (out->dtype == KD_F32 || out->dtype == KD_BF16);
  if (fast) {
    const int threads = 256;
    if (out->dtype == KD_F32) {
      const int64_t nv = n / 4;
      pointwise_contig_kernel<float, 4><<<grid_for(nv > 0 ? nv : n, threads), threads, 0, st>>>(
          (const float*)pa, (const float*)pb, (float*)po, op, b != nullptr, scalar, nv, n);
    } else {
      const int64_t nv = n / 8;
      pointwise_contig_kernel<__nv_bfloat16, 8><<<grid_for(nv > 0 ? nv : n, threads), threads, 0, st>>>(
          (const __nv_bfloat16*)pa, (const __nv_bfloat16*)pb, (__nv_bfloat16*)po, op, b != nullptr, scalar, nv, n);
    }
    return after_launch("pointwise_contig_kernel");
  }

  PwParams p{};
  p.op = op;
  p.ndim = out->ndim;
  p.dt_a = a->dtype;
  p.dt_b = b ? b->dtype : KD_F32;
  p.dt_o = out->dtype;
  p.has_b = b != nullptr;
  p.int_mode = (op < 0 && !is_float_dtype(a->dtype) && !is_float_dtype(out->dtype)) ? 1 : 0;
  p.scalar = scalar;
  p.n = n;
  for (int d = 0; d < out->ndim; ++d) {
    p.shape[d] = out->shape[d];
    p.so[d] = out->strides[d];
  }
  KD_TRY(broadcast_strides(a, out, p.sa, "input a"));
  if (b) KD_TRY(broadcast_strides(b, out, p.sb, "input b"));
  const int threads = 256;
  PvParams pv;
  if (plan_pieces(p, pa, pb, po, &pv)) {
    KD_CUDA_CHECK(launch_ex(pointwise_pieces_kernel, dim3(grid_for(pv.n, threads)), dim3(threads), 0, (const void*)pa, (const void*)pb, po, pv));
    return after_launch("pointwise_pieces_kernel");
  }
  KD_CUDA_CHECK(launch_ex(pointwise_strided_kernel, dim3(grid_for(n, threads)), dim3(threads), 0, (const void*)pa, (const void*)pb, po, p));
  return after_launch("pointwise_strided_kernel");
}

// ----------------------------------------------------------------------------- fill / arange
template <typename T>
__global__ void fill_kernel(T* __restrict__ p, T v, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) p[i] = v;
}

__global__ void fill_strided_kernel(void* __restrict__ p, int dt, float v, StridedIndex idx, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    store_float(p, dt, idx.offset_of(i), v);
}

__global__ void arange_kernel(void* __restrict__ p, int dt, double start, double step, int64_t n) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double v = start + (double)i * step;
    if (dt == KD_I32) static_cast<int32_t*>(p)[i] = (int32_t)v;
    else if (dt == KD_I64) static_cast<int64_t*>(p)[i] = (int64_t)v;
    else store_float(p, dt, i, (float)v);
  }
}

}  // namespace kd

using namespace kd;

KD_API int kd_pointwise(int op, const kd_tensor* a, const kd_tensor* b, float scalar, const kd_tensor* out) {
  KD_REQUIRE(op >= KD_OP_ADD && op <= KD_OP_SUB, "unknown pointwise op %d", op);
  const bool binary = (op == KD_OP_ADD || op == KD_OP_MUL || op == KD_OP_DIV || op == KD_OP_MAXIMUM || op == KD_OP_SUB);
  KD_REQUIRE(!binary || b != nullptr, "binary pointwise op %d needs two inputs", op);
  return launch_pointwise(op, a, binary ? b : nullptr, scalar, out);
}

KD_API int kd_copy(const kd_tensor* dst, const kd_tensor* src) {
  KD_TRY(require_init());
  KD_REQUIRE(dst && src, "null tensor");
  // Same dtype, both contiguous, same element count: a device memcpy.
  if (dst->dtype == src->dtype && is_contiguous(dst) && is_contiguous(src) && numel(dst) == numel(src) &&
      same_shape(dst, src)) {
    void *pd = nullptr, *ps = nullptr;
    KD_TRY(tensor_ptr(dst, &pd));
    KD_TRY(tensor_ptr(src, &ps));
    const int64_t n = numel(dst);
    if (n == 0) return KD_OK;
    KD_CUDA_CHECK(cudaMemcpyAsync(pd, ps, (size_t)n * dtype_size(dst->dtype), cudaMemcpyDeviceToDevice, ctx().stream));
    ctx().launches++;
    return KD_OK;
  }
  return launch_pointwise(-1 /* identity */, src, nullptr, 0.f, dst);
}

KD_API int kd_fill(const kd_tensor* dst, double value) {
  KD_TRY(require_init());
  KD_REQUIRE(dst, "null tensor");
  void* p = nullptr;
  KD_TRY(tensor_ptr(dst, &p));
  const int64_t n = numel(dst);
  if (n == 0) return KD_OK;
  cudaStream_t st = ctx().stream;
  const int threads = 256;
  if (is_contiguous(dst)) {
    if (value == 0.0) {
      KD_CUDA_CHECK(cudaMemsetAsync(p, 0, (size_t)n * dtype_size(dst->dtype), st));
      ctx().launches++;
      return KD_OK;
    }
    const int g = grid_for(n, threads);
    switch (dst->dtype) {
      case KD_F32: fill_kernel<float><<<g, threads, 0, st>>>((float*)p, (float)value, n); break;
      case KD_BF16: fill_kernel<__nv_bfloat16><<<g, threads, 0, st>>>((__nv_bfloat16*)p, __float2bfloat16_rn((float)value), n); break;
      case KD_F16: fill_kernel<__half><<<g, threads, 0, st>>>((__half*)p, __float2half_rn((float)value), n); break;
      case KD_I32: fill_kernel<int32_t><<<g, threads, 0, st>>>((int32_t*)p, (int32_t)value, n); break;
      case KD_I64: fill_kernel<int64_t><<<g, threads, 0, st>>>((int64_t*)p, (int64_t)value, n); break;
      default: fill_kernel<uint8_t><<<g, threads, 0, st>>>((uint8_t*)p, (uint8_t)value, n); break;
    }
    return after_launch("fill_kernel");
  }
  StridedIndex idx{};
  idx.ndim = dst->ndim;
  for (int d = 0; d < dst->ndim; ++d) { idx.shape[d] = dst->shape[d]; idx.strides[d] = dst->strides[d]; }
  fill_strided_kernel<<<grid_for(n, threads), threads, 0, st>>>(p, dst->dtype, (float)value, idx, n);
  return after_launch("fill_strided_kernel");
}

KD_API int kd_arange(const kd_tensor* dst, double start, double step) {
  KD_TRY(require_init());
  KD_REQUIRE(dst && dst->ndim == 1 && is_contiguous(dst), "arange needs a contiguous 1-D output");
  void* p = nullptr;
  KD_TRY(tensor_ptr(dst, &p));
  const int64_t n = numel(dst);
  if (n == 0) return KD_OK;
  arange_kernel<<<grid_for(n, 256), 256, 0, ctx().stream>>>(p, dst->dtype, start, step, n);
  return after_launch("arange_kernel");
}
