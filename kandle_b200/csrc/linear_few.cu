// bf16 linears of a few rows (1 to 32, the decode steps of the engines that mix layer types): y[m, n] = sum_k x[m, k] W[n, k].
//
// What bounds them: a step of such an engine is a chain of some 60 kernels, and a linear reads 2 to 50 MB of weights (0.3 to 8 us at
// HBM's rate).  The tcgen05 kernels took 8 to 18 us for them: 16 to 40 tiles of 64 or 128 weight rows with a long walk over K
// each, or shared tiles whose tensor memory has to be allocated, drained, exchanged and freed.  Here
//   - all SMs stream: a cluster of 1 to 8 CTAs has R weight rows, each CTA a range of K, each of its eight warps every eighth group
//     of 32 columns.  A lane reads the 16 bytes of a weight row that it multiplies itself, straight into registers, four
//     steps (8 KB a warp, 64 KB an SM) ahead; in a programmatic chain (kd_set_pdl(3)) the first four before the wait.
//   - mma.sync m16n8k16 multiplies 8 weight rows x 32 columns at a time by 16 or 32 rows of x, whose columns it reads from shared
//     memory in the order in which the lane holds the weights.
//   - the eight warps' sums meet in shared memory after every 32 weight rows, the CTAs' through distributed shared memory
//     once, at the end, each CTA finishing a part of the columns.
// Measured: see lf_plan.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "sm100.cuh"

namespace kd {

constexpr int LF_WARPS = 8, LF_THREADS = LF_WARPS * 32, LF_ROWS = 32, LF_STEPS = 4;

struct FewParams {
  const __nv_bfloat16 *x, *w;
  int64_t ldx, ldo, ld_tail, ldr;
  int M, N, K, R;             // R: weight rows of a cluster, a multiple of 32
  int epi;                    // 0 plain, 1 + residual (fp32), 2 silu(gate) up, 5 gelu(gate) up, 6 tanh
  int out_f32, early_w;
  void* out;
  const void* resid;          // of the output's type
  float* tail;                // columns from tail_col on, fp32
  int tail_col;
};

__device__ __forceinline__ uint4 lf_weights(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void lf_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float4 lf_peer(const float* p, uint32_t rank) {
  const uint32_t a = sm100::smem_u32(p);
  uint32_t r;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r) : "memory");
  return v;
}
__device__ __forceinline__ void lf_cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float lf_silu(float x) { return x / (1.0f + __expf(-x)); }
__device__ __forceinline__ float lf_gelu(float x) { return x / (1.0f + __expf(-1.5957691216f * (x + 0.044715f * x * x * x))); }
__device__ __forceinline__ float lf_tanh(float x) { return 1.0f - 2.0f / (1.0f + __expf(2.0f * x)); }

// Results of a cluster, from its CTAs' sums (part [16 MT][R + 4] in each).
template <int MT>
__device__ __forceinline__ void lf_finish(const FewParams& p, const float* part, int ldp, int S, int rank, int n0, int rows, int t) {
  if (S > 1) lf_cluster_sync();
  const bool glu = p.epi == 2 || p.epi == 5;
  const int cols = (glu ? rows / 2 : rows), groups = (cols + 3) / 4, g0 = groups * rank / S, g1 = groups * (rank + 1) / S;
  auto sum = [&](int m, int c) {
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = 0; r < S; ++r) {
      const float4 v = S > 1 ? lf_peer(part + m * ldp + c, (uint32_t)r) : *reinterpret_cast<const float4*>(part + m * ldp + c);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    return s;
  };
  for (int i = t; i < p.M * (g1 - g0); i += LF_THREADS) {
    const int m = i / (g1 - g0), c = (g0 + i - m * (g1 - g0)) * 4;
    float4 y;
    int64_t n = n0 + c;
    if (glu) {
      const int row = c / 16 * 32 + c % 16;          // 16 gate rows, then their 16 up rows
      const float4 g = sum(m, row), u = sum(m, row + 16);
      y = p.epi == 2 ? make_float4(lf_silu(g.x) * u.x, lf_silu(g.y) * u.y, lf_silu(g.z) * u.z, lf_silu(g.w) * u.w)
                     : make_float4(lf_gelu(g.x) * u.x, lf_gelu(g.y) * u.y, lf_gelu(g.z) * u.z, lf_gelu(g.w) * u.w);
      n = n0 / 2 + c;
    } else {
      y = sum(m, c);
      if (p.epi == 6) y = make_float4(lf_tanh(y.x), lf_tanh(y.y), lf_tanh(y.z), lf_tanh(y.w));
      if (p.epi == 1) {
        if (p.out_f32) {
          const float4 r = *reinterpret_cast<const float4*>(static_cast<const float*>(p.resid) + m * p.ldr + n);
          y = make_float4(y.x + r.x, y.y + r.y, y.z + r.z, y.w + r.w);
        } else {
          const uint2 r = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(p.resid) + m * p.ldr + n);
          y = make_float4(y.x + __uint_as_float(r.x << 16), y.y + __uint_as_float(r.x & 0xffff0000u), y.z + __uint_as_float(r.y << 16),
                          y.w + __uint_as_float(r.y & 0xffff0000u));
        }
      }
      if (p.tail && n >= p.tail_col) {
        *reinterpret_cast<float4*>(p.tail + m * p.ld_tail + (n - p.tail_col)) = y;
        continue;
      }
    }
    if (p.out_f32) {
      *reinterpret_cast<float4*>(static_cast<float*>(p.out) + m * p.ldo + n) = y;
    } else {
      __nv_bfloat162 a = __floats2bfloat162_rn(y.x, y.y), b = __floats2bfloat162_rn(y.z, y.w);
      *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.out) + m * p.ldo + n) =
          make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    }
  }
  if (S > 1) lf_cluster_sync();                      // nobody leaves while its sums may be read
}

// MT: tiles of 16 rows of x; S: CTAs of a cluster
template <int MT>
__global__ void __launch_bounds__(LF_THREADS, 1) linear_few_kernel(const FewParams p, const int S) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, t = threadIdx.x;
  const int rank = (int)blockIdx.x % S, n0 = (int)blockIdx.x / S * p.R;
  const int chunks = p.K / 32, c0 = chunks * rank / S, nc = chunks * (rank + 1) / S - c0;      // groups of 32 columns of this CTA
  const int rows = min(p.R, p.N - n0), passes = (rows + LF_ROWS - 1) / LF_ROWS;
  const int stride = (((p.K / 32 + S - 1) / S) | 1) * 64;          // bytes of a row of x (two rows' pieces meet no bank twice)
  uint8_t* xs = smem;                                              // [16 MT][stride]
  float* red = reinterpret_cast<float*>(xs + 16 * MT * stride);    // [warp][16 MT][32 + 4]
  float* part = red + LF_WARPS * 16 * MT * (LF_ROWS + 4);          // [16 MT][R + 4]
  const int ldp = p.R + 4;

  // steps of a warp: 32 rows x one of its groups of columns
  const int mine = warp < nc ? (nc - warp + LF_WARPS - 1) / LF_WARPS : 0, steps = passes * mine;
  uint4 w[LF_STEPS][4];
  int next_pass = 0, next_i = 0;
  auto fetch = [&](uint4 (&v)[4]) {
    const int64_t col = (int64_t)(c0 + warp + next_i * LF_WARPS) * 32 + (lane & 3) * 8;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int row = min(n0 + next_pass * LF_ROWS + b * 8 + (lane >> 2), p.N - 1);       // (beyond the edge: results nobody stores)
      v[b] = lf_weights(p.w + (int64_t)row * p.K + col);
    }
    if (++next_i == mine) {
      next_i = 0;
      ++next_pass;
    }
  };
  if (!p.early_w) pdl_wait();
#pragma unroll
  for (int i = 0; i < LF_STEPS; ++i)
    if (i < steps) fetch(w[i]);
  if (p.early_w) pdl_wait();
  pdl_trigger();

  // x: this CTA's columns
  for (int i = t; i < 16 * MT * nc * 4; i += LF_THREADS) {
    const int m = i / (nc * 4), j = i - m * (nc * 4);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (m < p.M) v = *reinterpret_cast<const uint4*>(p.x + m * p.ldx + c0 * 32 + j * 8);
    *reinterpret_cast<uint4*>(xs + m * stride + j * 16) = v;
  }
  __syncthreads();

  const uint8_t* xf = xs + (lane >> 2) * stride + (lane & 3) * 16 + warp * 64;
  float acc[4][MT][4];
  auto clear = [&] {
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[b][m][e] = 0.f;
  };
  // 32 rows are done: the warps' sums of this CTA
  auto meet = [&](int pass) {
    float* r = red + warp * 16 * MT * (LF_ROWS + 4);
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        *reinterpret_cast<float2*>(r + (m * 16 + (lane >> 2)) * (LF_ROWS + 4) + b * 8 + (lane & 3) * 2) = make_float2(acc[b][m][0], acc[b][m][1]);
        *reinterpret_cast<float2*>(r + (m * 16 + (lane >> 2) + 8) * (LF_ROWS + 4) + b * 8 + (lane & 3) * 2) = make_float2(acc[b][m][2], acc[b][m][3]);
      }
    clear();
    __syncthreads();
    for (int i = t; i < 16 * MT * LF_ROWS / 4; i += LF_THREADS) {
      const int m = i / (LF_ROWS / 4), c = i % (LF_ROWS / 4) * 4;
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < LF_WARPS; ++k) {
        const float4 v = *reinterpret_cast<const float4*>(red + (k * 16 * MT + m) * (LF_ROWS + 4) + c);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      *reinterpret_cast<float4*>(part + m * ldp + pass * LF_ROWS + c) = s;
    }
    __syncthreads();
  };
  clear();
  int pass = 0, i_in = 0;
  auto step = [&](uint4 (&v)[4], int s) {
    const uint8_t* a = xf + i_in * (LF_WARPS * 64);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint4 lo = *reinterpret_cast<const uint4*>(a + m * 16 * stride), hi = *reinterpret_cast<const uint4*>(a + (m * 16 + 8) * stride);
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        lf_mma(acc[b][m], lo.x, hi.x, lo.y, hi.y, v[b].x, v[b].y);
        lf_mma(acc[b][m], lo.z, hi.z, lo.w, hi.w, v[b].z, v[b].w);
      }
    }
    if (s + LF_STEPS < steps) fetch(v);
    if (++i_in == mine) {
      i_in = 0;
      meet(pass++);
    }
  };
  for (int s = 0; s < steps; s += LF_STEPS) {
#pragma unroll
    for (int u = 0; u < LF_STEPS; ++u)
      if (s + u < steps) step(w[u], s + u);
  }
  for (; pass < passes; ++pass) meet(pass);          // (a warp without columns)

  lf_finish<MT>(p, part, ldp, S, rank, n0, rows, t);
}

struct FewPlan { int S, R, smem; };

// How the call is split: the fewest CTAs a cluster that fill the SMs and leave a CTA at most 32 KB of x to read (all of x passes through
// every cluster).  With more than 16 rows an SM holds one CTA (registers), and clusters of four and eight leave SMs over: 33 and 15 of
// them fit 148 SMs.  A cluster is not doubled there where that many more do not fit, as long as x allows it (32 x 1024 x 3072, rows
// x N x K: 16 clusters of eight 12.5 us, 32 of four 5.9; 32 x 2560 x 512: 40 of two 4.7, 80 CTAs alone 3.5).
// S = 0: not taken.  Taken are the sizes at which this kernel is the faster one (us in a chain with kd_set_pdl(3): tcgen05
// kernels, this one).  Up to 16 rows: 1 x 2048 x 2048 9.0, 4.4; 1 x 64 x 2048 7.5, 2.8; 8 x 4096 x 2048 10.9, 8.3; 8 x 8192 x 2048 15.7, 14.8;
// 8 x 2048 x 6144 17.9, 12.2; 8 x 5120 x 2560 17.5, 14.1; 1 x 10240 x 1024 10.5, 10.2; not: 16 x 10240 x 768 8.4, 9.1; 8 x 10240 x 1536 13.4, 15.6; 16 x 4096 x 4096 13.0, 15.7; 16 x 2048 x 6144
// 12.6, 13.5; 1 x 5120 x 2560 16.2, 19.1 (registers hold too little of a long stream).  More: 32 x 2048 x 2048 8.6, 6.7; 32 x 1024 x 3072 9.0,
// 5.9; 32 x 2048 x 3072 9.5, 8.9; 32 x 6144 x 1024 8.5, 8.5; 20 x 4096 x 2048 10.6, 9.8; not: 32 x 4096 x 2048 9.3, 10.2; 32 x 8192 x 1024 8.6,
// 9.1; 32 x 2560 x 3072 10.4, 11.1; 24 x 6144 x 768 7.3, 8.0.
static FewPlan lf_plan(int64_t M, int64_t N, int64_t K, int sms) {
  FewPlan f{0, 0, 0};
  if (M < 1 || M > 32 || N < 32 || N % 8 || K < 256 || K % 32) return f;
  const int64_t weights = N * K, x = M * K * 2, mega = 1ll << 20, kb = 1024;
  if (M <= 16) {
    if (weights > (N > 8192 ? (M <= 8 ? 12 : 6) : x > 128 * kb ? 9 : 18) * mega) return f;
    if (weights > 12 * mega && K > 2048 && ((x < 32 * kb && (N > 4096 || K > 4096)) || x > 96 * kb)) return f;
  } else {
    if (K > 4096 || N > 8192 || weights > (x > 128 * kb ? 6 : 8) * mega || M * weights > 192 * mega) return f;
    if (N > 4096 && K > 512 && K < 1024 && M > 20) return f;
  }
  const int tiles = (int)((N + LF_ROWS - 1) / LF_ROWS), mt = M <= 16 ? 1 : 2;
  const auto fit = [&](int S) { return std::max(1, sms / S - (mt == 1 || S < 4 ? 0 : S == 4 ? 4 : 3)); };      // clusters at a time
  const auto rounds = [&](int S) { return (tiles + fit(S) - 1) / fit(S); };
  int S = 1;
  while (S < 8 && K / 32 >= 16 * S && (tiles * S < sms * 2 / 3 || x / S > 32 * kb)) {
    if (mt == 2 && rounds(2 * S) >= 2 * rounds(S) && x / S <= (S == 2 ? 48 : 64) * kb) break;
    S *= 2;
  }
  const int R = LF_ROWS * rounds(S);
  const int64_t smem = 16 * mt * (((((K / 32 + S - 1) / S) | 1) * 64) + LF_WARPS * (LF_ROWS + 4) * 4 + (R + 4) * 4);
  if (smem > 200 * kb) return f;
  return FewPlan{S, R, (int)smem};
}

bool linear_few_rows(int64_t M, int64_t N, int64_t K) { return lf_plan(M, N, K, ctx().sm_count).S > 0; }

int linear_few(const void* x, int64_t ldx, const void* w, void* out, int64_t ldo, int out_f32, const void* resid, int64_t ldr, int M, int N, int K, int epi,
               float* tail, int tail_col, int64_t ld_tail) {
  const FewPlan f = lf_plan(M, N, K, ctx().sm_count);
  KD_REQUIRE(f.S > 0, "linear_few: %d x %d x %d is not taken", M, N, K);
  FewParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x);
  p.w = static_cast<const __nv_bfloat16*>(w);
  p.ldx = ldx; p.ldo = ldo; p.ldr = ldr; p.ld_tail = ld_tail;
  p.M = M; p.N = N; p.K = K; p.R = f.R;
  p.epi = epi;
  p.out_f32 = out_f32;
  p.early_w = ctx().pdl_weights;
  p.out = out;
  p.resid = resid;
  p.tail = tail;
  p.tail_col = tail_col;
  const auto kernel = M <= 16 ? linear_few_kernel<1> : linear_few_kernel<2>;
  static bool configured[64] = {false};
  if (!configured[ctx().device & 63]) {
    for (const auto k : {linear_few_kernel<1>, linear_few_kernel<2>})
      KD_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    configured[ctx().device & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((N + f.R - 1) / f.R * f.S));
  cfg.blockDim = dim3(LF_THREADS);
  cfg.dynamicSmemBytes = f.smem;
  cfg.stream = ctx().stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)f.S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctx().pdl ? 2 : 1;
  KD_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, p, f.S));
  return after_launch("linear_few_kernel");
}

}  // namespace kd

// Test support: CTAs of a cluster and its weight rows for a linear of a few rows, zeros where another kernel takes it.
KD_API int kd_debug_linear_few_plan(int64_t M, int64_t N, int64_t K, int sms, int* ctas, int* rows) {
  if (!ctas || !rows || sms <= 0) return kd::fail(KD_ERR_INVALID, "bad argument");
  const kd::FewPlan f = kd::lf_plan(M, N, K, sms);
  *ctas = f.S;
  *rows = f.R;
  return KD_OK;
}
