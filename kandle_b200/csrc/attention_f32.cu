// Key `flash_attention`, fp32 path on the CUDA cores (any storage dtype, fp32 math).
//
// Two kernels: attention_f32_tile_kernel for fp32 operands with heads of 64 or 128 channels in rows of 16-byte pieces,
// attention_f32_kernel for everything else.
//
// Same mathematics as the reference shader
// (packages/backend-webgpu/src/kernels/attention/builder.ts:138-329): score = dot(q,k)*scale,
// causal / out-of-range columns get -1e20, running max starts at -1e20, online-softmax
// rescaling per KV tile, final O/l.  The tiling is different: one warp owns one query row (the
// reference uses 8x4 tiles sized for 16 KB of workgroup memory and a serial per-row softmax),
// 16 rows per CTA share each 32-row K/V tile staged in shared memory, the softmax statistics
// live in registers and are combined with warp shuffles.  Unlike the reference kernel, operand
// strides are honoured (the reference assumes contiguous [B,H,S,D]).
#include "common.cuh"
#include "kernels.cuh"

namespace kd {


constexpr int ATT_WARPS = 16;
constexpr int ATT_TKV = 32;

template <int DPL>  // head dims per lane: head_dim <= 32*DPL, padded with zeros
__global__ void __launch_bounds__(ATT_WARPS * 32) attention_f32_kernel(const void* __restrict__ Q,
                                                                      const void* __restrict__ K,
                                                                      const void* __restrict__ V, void* __restrict__ O,
                                                                      AttnParams p) {
  constexpr int D = 32 * DPL;   // padded head dim; p.D is the real one
  extern __shared__ float smem[];
  float* Ks = smem;                          // [TKV][D+1]
  float* Vs = Ks + ATT_TKV * (D + 1);        // [TKV][D]
  float* Qs = Vs + ATT_TKV * D;              // [WARPS][D]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.y, b = blockIdx.z;
  const int hk = h / (p.Hq / p.Hkv);
  const int row0 = blockIdx.x * ATT_WARPS;
  const int row = row0 + warp;
  const bool row_ok = row < p.Sq;
  const float NEG = -1e20f;

  const int64_t q_off = (int64_t)b * p.sq[0] + (int64_t)h * p.sq[1] + (int64_t)row * p.sq[2];
  for (int d = lane; d < D; d += 32) Qs[warp * D + d] = (row_ok && d < p.D) ? load_float(Q, p.dt_q, q_off + d * p.sq[3]) : 0.f;

  float acc[DPL];
#pragma unroll
  for (int i = 0; i < DPL; ++i) acc[i] = 0.f;
  float m = NEG, l = 0.f;

  const int last_row = min(row0 + ATT_WARPS - 1, p.Sq - 1);
  const int kv_end = p.causal ? min(p.Skv, last_row + 1) : p.Skv;
  const int64_t k_base = (int64_t)b * p.sk[0] + (int64_t)hk * p.sk[1];
  const int64_t v_base = (int64_t)b * p.sv[0] + (int64_t)hk * p.sv[1];

  for (int j0 = 0; j0 < kv_end; j0 += ATT_TKV) {
    __syncthreads();
    for (int e = threadIdx.x; e < ATT_TKV * D; e += ATT_WARPS * 32) {
      const int r = e / D, d = e - r * D;
      const int j = j0 + r;
      float kv = 0.f, vv = 0.f;
      if (j < p.Skv && d < p.D) {
        kv = load_float(K, p.dt_k, k_base + (int64_t)j * p.sk[2] + d * p.sk[3]);
        vv = load_float(V, p.dt_v, v_base + (int64_t)j * p.sv[2] + d * p.sv[3]);
      }
      Ks[r * (D + 1) + d] = kv;
      Vs[r * D + d] = vv;
    }
    __syncthreads();
    if (!row_ok) continue;
    if (p.causal && j0 > row) continue;  // every column of this tile is masked for this row
    const int j = j0 + lane;
    float s;
    if (j >= p.Skv || (p.causal && j > row)) {
      s = NEG;
    } else {
      s = 0.f;
      const float* kr = Ks + lane * (D + 1);
      const float* qr = Qs + warp * D;
#pragma unroll 8
      for (int d = 0; d < D; ++d) s = fmaf(qr[d], kr[d], s);
      s *= p.scale;
    }
    const float m_new = fmaxf(m, warp_max(s));
    const float sf = expf(m - m_new);
    const float pj = expf(s - m_new);
    l = l * sf + warp_sum(pj);
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[i] *= sf;
#pragma unroll 4
    for (int jj = 0; jj < ATT_TKV; ++jj) {
      const float pv = __shfl_sync(0xffffffffu, pj, jj);
      const float* vr = Vs + jj * D + lane;
#pragma unroll
      for (int i = 0; i < DPL; ++i) acc[i] = fmaf(pv, vr[32 * i], acc[i]);
    }
    m = m_new;
  }
  if (row_ok) {
    const int64_t o_off = (int64_t)b * p.so[0] + (int64_t)h * p.so[1] + (int64_t)row * p.so[2];
#pragma unroll
    for (int i = 0; i < DPL; ++i)
      if (lane + 32 * i < p.D) store_float(O, p.dt_o, o_off + (int64_t)(lane + 32 * i) * p.so[3], acc[i] / l);
  }
}

// Register tiles: 128 threads own 8 R query rows and walk over tiles of 64 keys; a thread holds R rows x 4 keys of the scores
// and R rows x D / 16 channels of the output, 16 lanes share a row.  Keys arrive while the values of the tile before are
// used, and the other way round (cp.async).  A warp's rows lie inside one block of 32, so the 32-key blocks that
// attention_f32_kernel passes over (all masked, or past the end) are passed over here too: infinities among masked values
// stay out of the sums.
// Bound: shared-memory reads, (R + 4) 16-byte reads for 16 R multiply-adds; attention_f32_kernel, one row a warp, reads two
// numbers a multiply-add.  16 heads of 128 channels, causal, replayed from a graph: 128 queries 12.3 us (28.5 before), 300 33.9
// (108), 1000 136 (803); launched one by one 128 queries take 14.5.
template <int D, int R>
__global__ void __launch_bounds__(128) attention_f32_tile_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V,
                                                                 float* __restrict__ O, AttnParams p) {
  constexpr int ROWS = 8 * R, TK = 64, LDK = D + 4, LDP = TK + 4, OC = D / 64;
  extern __shared__ __align__(16) float smem[];
  float* Ks = smem;                 // [TK][LDK]
  float* Vs = Ks + TK * LDK;        // [TK][D]
  float* Qs = Vs + TK * D;          // [ROWS][LDK]
  float* Ps = Qs + ROWS * LDK;      // [ROWS][LDP]
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int h = blockIdx.x % p.Hq, b = blockIdx.x / p.Hq, hk = h / (p.Hq / p.Hkv);
  const int row0 = (int)(gridDim.y - 1 - blockIdx.y) * ROWS;      // the longest rows first
  const float NEG = -1e20f;
  auto copy = [&](float* dst, int ld, const float* src, int64_t src_ld, int first, int rows, int end) {
    for (int e = tid; e < rows * (D / 4); e += 128) {
      const int r = e / (D / 4), c = (e % (D / 4)) * 4;
      const bool in = first + r < end;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + r * ld + c)),
                   "l"(src + (in ? first + r : 0) * src_ld + c), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const float* Kh = K + (int64_t)b * p.sk[0] + (int64_t)hk * p.sk[1];
  const float* Vh = V + (int64_t)b * p.sv[0] + (int64_t)hk * p.sv[1];
  const int kv_end = p.causal ? min(p.Skv, min(row0 + ROWS, p.Sq)) : p.Skv;
  copy(Qs, LDK, Q + (int64_t)b * p.sq[0] + (int64_t)h * p.sq[1], p.sq[2], row0, ROWS, p.Sq);
  copy(Ks, LDK, Kh, p.sk[2], 0, TK, p.Skv);
  copy(Vs, D, Vh, p.sv[2], 0, TK, p.Skv);

  float acc[R][OC * 4], m[R], l[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m[i] = NEG;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < OC * 4; ++c) acc[i][c] = 0.f;
  }
  const int first_row = row0 + ty * R, warp_row = row0 + (tid >> 5) * 2 * R;

  for (int j0 = 0; j0 < kv_end; j0 += TK) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");      // keys (the values may still be on their way)
    __syncthreads();
    // 32-key blocks of this tile that the warp's rows see
    auto seen = [&](int j) { return j < kv_end && (!p.causal || j <= (warp_row | 31)); };
    const int n_keys = seen(j0 + 32) ? 64 : seen(j0) ? 32 : 0;
    if (n_keys) {
      float s[R][4];
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
      for (int d = 0; d < D; d += 4) {
        float4 q[R], k[4];
#pragma unroll
        for (int i = 0; i < R; ++i) q[i] = *reinterpret_cast<const float4*>(Qs + (ty * R + i) * LDK + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * LDK + d);
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) s[i][j] = fmaf(q[i].w, k[j].w, fmaf(q[i].z, k[j].z, fmaf(q[i].y, k[j].y, fmaf(q[i].x, k[j].x, s[i][j]))));
      }
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int row = first_row + i;
        float top = NEG;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = j0 + tx + 16 * j;
          s[i][j] = key >= p.Skv || (p.causal && key > row) ? NEG : s[i][j] * p.scale;
          if (16 * j < n_keys) top = fmaxf(top, s[i][j]);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float m_new = fmaxf(m[i], top), sf = expf(m[i] - m_new);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e = 16 * j < n_keys ? expf(s[i][j] - m_new) : 0.f;
          Ps[(ty * R + i) * LDP + tx + 16 * j] = e;
          sum += e;
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        l[i] = l[i] * sf + sum;
        m[i] = m_new;
#pragma unroll
        for (int c = 0; c < OC * 4; ++c) acc[i][c] *= sf;
      }
    }
    __syncthreads();                                          // the keys are used up
    if (j0 + TK < kv_end) copy(Ks, LDK, Kh, p.sk[2], j0 + TK, TK, p.Skv);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");      // values
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < n_keys; k += 4) {
      float4 e[R];
#pragma unroll
      for (int i = 0; i < R; ++i) e[i] = *reinterpret_cast<const float4*>(Ps + (ty * R + i) * LDP + k);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        float4 v[OC];
#pragma unroll
        for (int c = 0; c < OC; ++c) v[c] = *reinterpret_cast<const float4*>(Vs + (k + kk) * D + c * 64 + tx * 4);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const float w = kk == 0 ? e[i].x : kk == 1 ? e[i].y : kk == 2 ? e[i].z : e[i].w;
#pragma unroll
          for (int c = 0; c < OC; ++c) {
            acc[i][c * 4] = fmaf(w, v[c].x, acc[i][c * 4]);
            acc[i][c * 4 + 1] = fmaf(w, v[c].y, acc[i][c * 4 + 1]);
            acc[i][c * 4 + 2] = fmaf(w, v[c].z, acc[i][c * 4 + 2]);
            acc[i][c * 4 + 3] = fmaf(w, v[c].w, acc[i][c * 4 + 3]);
          }
        }
      }
    }
    __syncthreads();                                          // the values are used up
    if (j0 + TK < kv_end) copy(Vs, D, Vh, p.sv[2], j0 + TK, TK, p.Skv);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float* out = O + (int64_t)b * p.so[0] + (int64_t)h * p.so[1];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int row = first_row + i;
    if (row >= p.Sq) continue;
#pragma unroll
    for (int c = 0; c < OC; ++c)
      *reinterpret_cast<float4*>(out + (int64_t)row * p.so[2] + c * 64 + tx * 4) =
          make_float4(acc[i][c * 4] / l[i], acc[i][c * 4 + 1] / l[i], acc[i][c * 4 + 2] / l[i], acc[i][c * 4 + 3] / l[i]);
  }
}

template <int D, int R>
static int launch_attention_tile(const void* pq, const void* pk, const void* pv, void* po, const AttnParams& p) {
  constexpr int SMEM = (64 * (D + 4) + 64 * D + 8 * R * (D + 4) + 8 * R * 68) * 4;
  static bool configured[64] = {false};
  if (!configured[ctx().device & 63]) {
    KD_CUDA_CHECK(cudaFuncSetAttribute(attention_f32_tile_kernel<D, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    configured[ctx().device & 63] = true;
  }
  dim3 grid((unsigned)(p.Hq * p.B), (unsigned)((p.Sq + 8 * R - 1) / (8 * R)));
  attention_f32_tile_kernel<D, R><<<grid, 128, SMEM, ctx().stream>>>((const float*)pq, (const float*)pk, (const float*)pv, (float*)po, p);
  return after_launch("attention_f32_tile_kernel");
}

// 16-byte pieces of every row of all four operands.
static bool attention_tile_fits(const void* pq, const void* pk, const void* pv, const void* po, const AttnParams& p) {
  if (p.dt_q != KD_F32 || p.dt_k != KD_F32 || p.dt_v != KD_F32 || p.dt_o != KD_F32 || (p.D != 64 && p.D != 128)) return false;
  if ((reinterpret_cast<uintptr_t>(pq) | reinterpret_cast<uintptr_t>(pk) | reinterpret_cast<uintptr_t>(pv) | reinterpret_cast<uintptr_t>(po)) & 15) return false;
  for (const int64_t* st : {p.sq, p.sk, p.sv, p.so}) {
    if (st[3] != 1) return false;
    for (int d = 0; d < 3; ++d)
      if (st[d] & 3) return false;
  }
  return (int64_t)p.Hq * p.B < (1ll << 31) && p.Sq < 65535 * 16;
}

template <int D>
static int launch_attention_tile_rows(const void* pq, const void* pk, const void* pv, void* po, const AttnParams& p) {
  // Rows a CTA: 32 (half the key reads a row) where there are more than 16 and that leaves a CTA for every SM, 16 otherwise.
  // Causal, heads of 128, launched one by one: 16 heads of 128 queries 14.5 us with 16 rows, 16.5 with 32; 64 heads of 512
  // queries 215 and 148 us (64 rows: 178).  256 heads of 64, one query, one key: 4.9 us with 16 rows, 6.1 with 32 (attention_f32_kernel 5.0).
  if (p.Sq > 16 && (int64_t)p.Hq * p.B * ((p.Sq + 31) / 32) >= ctx().sm_count) return launch_attention_tile<D, 4>(pq, pk, pv, po, p);
  return launch_attention_tile<D, 2>(pq, pk, pv, po, p);
}

static void to4(const kd_tensor* t, int64_t* ext, int64_t* st) {
  for (int i = 0; i < 4; ++i) { ext[i] = 1; st[i] = 0; }
  const int shift = 4 - t->ndim;
  for (int d = 0; d < t->ndim; ++d) { ext[d + shift] = t->shape[d]; st[d + shift] = t->strides[d]; }
}

// Validates the operands of flash_attention and fills AttnParams (shared by all attention paths).
int attention_params(const kd_tensor* q, const kd_tensor* k, const kd_tensor* v, const kd_tensor* out, float scale,
                     int is_causal, AttnParams* p) {
  KD_REQUIRE(q && k && v && out, "null tensor");
  KD_REQUIRE(q->ndim >= 2 && q->ndim <= 4 && k->ndim == q->ndim && v->ndim == q->ndim && out->ndim == q->ndim,
             "flash_attention operands must all have the same rank (2, 3 or 4)");
  int64_t eq[4], ek[4], ev[4], eo[4];
  to4(q, eq, p->sq); to4(k, ek, p->sk); to4(v, ev, p->sv); to4(out, eo, p->so);
  KD_REQUIRE(ek[0] == eq[0] && ev[0] == eq[0] && eo[0] == eq[0], "flash_attention: batch sizes differ");
  KD_REQUIRE(ek[3] == eq[3] && ev[3] == eq[3] && eo[3] == eq[3], "flash_attention: head dims differ");
  KD_REQUIRE(ev[1] == ek[1] && ev[2] == ek[2], "flash_attention: K and V shapes differ");
  KD_REQUIRE(eo[1] == eq[1] && eo[2] == eq[2], "flash_attention: output shape differs from Q");
  KD_REQUIRE(ek[1] > 0 && eq[1] % ek[1] == 0, "flash_attention: %lld query heads is not a multiple of %lld KV heads",
             (long long)eq[1], (long long)ek[1]);
  KD_REQUIRE(is_float_dtype(q->dtype) && is_float_dtype(k->dtype) && is_float_dtype(v->dtype) && is_float_dtype(out->dtype),
             "flash_attention needs floating-point tensors");
  p->B = (int)eq[0]; p->Hq = (int)eq[1]; p->Hkv = (int)ek[1]; p->Sq = (int)eq[2]; p->Skv = (int)ek[2]; p->D = (int)eq[3];
  p->dt_q = q->dtype; p->dt_k = k->dtype; p->dt_v = v->dtype; p->dt_o = out->dtype;
  p->scale = scale;
  p->causal = is_causal ? 1 : 0;
  return KD_OK;
}

template <int DPL>
static int launch_attention_f32(const void* pq, const void* pk, const void* pv, void* po, const AttnParams& p) {
  constexpr int D = 32 * DPL;
  const size_t smem = sizeof(float) * (ATT_TKV * (D + 1) + ATT_TKV * D + ATT_WARPS * D);
  if (smem > 48 * 1024)
    KD_CUDA_CHECK(cudaFuncSetAttribute(attention_f32_kernel<DPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  dim3 grid((p.Sq + ATT_WARPS - 1) / ATT_WARPS, p.Hq, p.B);
  attention_f32_kernel<DPL><<<grid, ATT_WARPS * 32, smem, ctx().stream>>>(pq, pk, pv, po, p);
  return after_launch("attention_f32_kernel");
}

int attention_f32_dispatch(const kd_tensor* q, const kd_tensor* k, const kd_tensor* v, const kd_tensor* out,
                           const AttnParams& p) {
  void *pq = nullptr, *pk = nullptr, *pv = nullptr, *po = nullptr;
  KD_TRY(tensor_ptr(q, &pq));
  KD_TRY(tensor_ptr(k, &pk));
  KD_TRY(tensor_ptr(v, &pv));
  KD_TRY(tensor_ptr(out, &po));
  if (p.B == 0 || p.Hq == 0 || p.Sq == 0) return KD_OK;
  KD_REQUIRE(p.Skv > 0, "flash_attention: empty key/value sequence");
  KD_REQUIRE(p.Hq <= 65535 && p.B <= 65535, "flash_attention: too many heads or batches for one launch");
  KD_REQUIRE(p.D >= 1, "flash_attention: empty head dimension");
  // A few rows of heads of 128 against a few keys: the general kernel is through sooner (16 heads, one query: 1 key 5.4 us,
  // 5.9 in tiles; 4 keys 5.5, 5.9; 8 keys 5.8, 5.9; 256 heads, 1 key: 10.0, 7.9)
  const bool few = p.D == 128 && p.Skv <= 6 && p.Sq <= ATT_WARPS && (int64_t)p.Hq * p.B <= ctx().sm_count;
  if (!few && attention_tile_fits(pq, pk, pv, po, p))
    return p.D == 64 ? launch_attention_tile_rows<64>(pq, pk, pv, po, p) : launch_attention_tile_rows<128>(pq, pk, pv, po, p);
  if (p.D <= 32) return launch_attention_f32<1>(pq, pk, pv, po, p);
  if (p.D <= 64) return launch_attention_f32<2>(pq, pk, pv, po, p);
  if (p.D <= 128) return launch_attention_f32<4>(pq, pk, pv, po, p);
  if (p.D <= 256) return launch_attention_f32<8>(pq, pk, pv, po, p);
  return fail(KD_ERR_UNSUPPORTED, "flash_attention: head_dim %d exceeds 256", p.D);
}

}  // namespace kd
