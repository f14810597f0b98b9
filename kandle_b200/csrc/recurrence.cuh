// Shared by the recurrent layers whose state is a [dim, vdim] fp32 matrix per head (delta_rule.cu, wkv.cu):
// elementary functions, packed arithmetic, the state held in registers, and the kernel that walks through the prompts of
// a few heads (second half).
//
// Many heads (delta_rule_kernel, wkv_kernel):
// A warp owns 32 / LPC groups of 8 state columns; the LPC lanes of a group share the rows, 16 a lane: lane j
// holds rows (i LPC + j) 4 + e (i < 4, e < 4), as s[column][row pair].  State in memory is
// [B, heads, rows, columns] with rows = 16 LPC and columns padded to a multiple of 8.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "sm100.cuh"

namespace kd {

constexpr int REC_CONSUMERS = 8, REC_HELPERS = 8;       // warps that hold the state; warps that prepare its inputs
constexpr int REC_THREADS = (REC_CONSUMERS + REC_HELPERS) * 32;
// Decays below this are applied to the state at once; products of four larger ones keep 1 / P in range.
constexpr float REC_SMALL_DECAY = 1e-6f;

template <typename T> __device__ __forceinline__ float rec_f(T v);
template <> __device__ __forceinline__ float rec_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float rec_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// In bf16 mode (FAST) the elementary functions are the special-function unit's, accurate to a few fp32
// roundings for these arguments; the fp32 mode uses the accurate library functions.
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcpf(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float REC_LOG2E = 1.4426950408889634f;
template <bool FAST> __device__ __forceinline__ float rec_sigmoid(float x) {
  return FAST ? rcpf(1.0f + ex2f(-REC_LOG2E * x)) : 1.0f / (1.0f + expf(-x));
}

// Four consecutive channels of a row as they lie in memory.
template <typename T> struct Raw4;
template <> struct Raw4<__nv_bfloat16> {
  uint2 u;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { u = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void get(float (&v)[4]) const {
    v[0] = __uint_as_float(u.x << 16); v[1] = __uint_as_float(u.x & 0xffff0000u);
    v[2] = __uint_as_float(u.y << 16); v[3] = __uint_as_float(u.y & 0xffff0000u);
  }
  __device__ __forceinline__ void set(const float (&v)[4]) {      // of values that bf16 holds exactly
    u.x = (__float_as_uint(v[0]) >> 16) | (__float_as_uint(v[1]) & 0xffff0000u);
    u.y = (__float_as_uint(v[2]) >> 16) | (__float_as_uint(v[3]) & 0xffff0000u);
  }
};
template <> struct Raw4<float> {
  float4 f;
  __device__ __forceinline__ void load(const float* p) { f = *reinterpret_cast<const float4*>(p); }
  __device__ __forceinline__ void get(float (&v)[4]) const { v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; }
  __device__ __forceinline__ void set(const float (&v)[4]) { f = make_float4(v[0], v[1], v[2], v[3]); }
};

// Rows of this lane's 8 columns; src points at (row 4 j, first column), null: zeros.
template <int LPC>
__device__ __forceinline__ void state_load(float2 (&s)[8][8], const float* src, int ld) {
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int r = 0; r < 8; ++r) s[c][r] = make_float2(0.f, 0.f);
  if (!src) return;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const float4 v = *reinterpret_cast<const float4*>(src + (int64_t)(i * LPC * 4 + e) * ld + w * 4);
        const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (e & 1) s[w * 4 + c][i * 2 + (e >> 1)].y = vv[c];
          else s[w * 4 + c][i * 2 + (e >> 1)].x = vv[c];
        }
      }
}

template <int LPC>
__device__ __forceinline__ void state_store(const float2 (&s)[8][8], float* dst, int ld) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const int r = i * 2 + (e >> 1);
        const float4 v = (e & 1) ? make_float4(s[w * 4][r].y, s[w * 4 + 1][r].y, s[w * 4 + 2][r].y, s[w * 4 + 3][r].y)
                                 : make_float4(s[w * 4][r].x, s[w * 4 + 1][r].x, s[w * 4 + 2][r].x, s[w * 4 + 3][r].x);
        *reinterpret_cast<float4*>(dst + (int64_t)(i * LPC * 4 + e) * ld + w * 4) = v;
      }
}

// Rows times d (quads of the row vector, starting at this lane's).
template <int LPC>
__device__ __forceinline__ void state_scale(float2 (&s)[8][8], const float4* d4) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 d = d4[i * LPC];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      s[c][2 * i] = mul2(s[c][2 * i], make_float2(d.x, d.y));
      s[c][2 * i + 1] = mul2(s[c][2 * i + 1], make_float2(d.z, d.w));
    }
  }
}

// Sums x and y over the group's lanes; lane j ends with columns j 8 / LPC .. (8 / LPC of them, at least one) in front.
template <int LPC>
__device__ __forceinline__ void group_sums(int j, float (&x)[8], float (&y)[8]) {
  int n = 8;
#pragma unroll
  for (int m = LPC / 2; m > 0; m >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = j & m;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < n) {
          const float sx = up ? x[i] : x[i + n], kx = up ? x[i + n] : x[i];
          const float sy = up ? y[i] : y[i + n], ky = up ? y[i + n] : y[i];
          x[i] = kx + __shfl_xor_sync(0xffffffffu, sx, m);
          y[i] = ky + __shfl_xor_sync(0xffffffffu, sy, m);
        }
    } else {
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], m);
      y[0] += __shfl_xor_sync(0xffffffffu, y[0], m);
    }
  }
}

// ----------------------------------------------------------------------------- few heads
// Where the heads of a call leave most of the chip idle (REC_LEAST_TOKENS has the rule), a prompt takes two kernels.  The
// layer's own prepare kernel turns every four tokens of a head into one record of what the walk needs (the vectors with the
// decays in them, and the 4 x 4 products between the tokens), all tokens side by side; then recurrence_kernel walks through
// the records with the state in registers:
//   read     D = S^T k_t, O = S^T q_t for all four tokens at once, against the state before them
//   solve    u_t = beta_t (v_t - D_t - sum_{s<t} (k_t . k_s) u_s)   (WKV: u_t = v_t)
//   output   o_t = O_t + sum_{s<=t} (q_t . k_s) u_s
//   write    S += sum_t k_t u_t^T, then rows times the decay of the four tokens
// so that sums over lanes and the dependent chain come once in four tokens.  Decays: with P_t their product from the group's
// first token to t, the record holds k_t P_t and q_t P_t to read, k_t / P_t to write and P_3.  Where a decay is so small
// that 1 / P could leave the range of fp32 (below 1e-6), the record holds the plain vectors and the walk takes the four
// tokens one by one with their decays.
//
// Mapping: a lane holds rec_rows rows of 4 columns, a CTA has up to four such warps and one that copies records into a ring
// in shared memory.  Bound: the chain of a group (shared memory -> products -> sums over lanes -> solve -> write), about
// 1200 cycles whatever the split over lanes; a warp issues every third to fourth cycle of it.
// Sums x over LPC lanes; lane j ends with values j N / LPC .. (N / LPC of them, at least one) in front.
template <int N, int LPC>
__device__ __forceinline__ void lanes_sum(int j, float (&x)[N]) {
  int n = N;
#pragma unroll
  for (int m = LPC / 2; m > 0; m >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = j & m;
#pragma unroll
      for (int i = 0; i < N / 2; ++i)
        if (i < n) {
          const float send = up ? x[i] : x[i + n], keep = up ? x[i + n] : x[i];
          x[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
        }
    } else {
      x[0] += __shfl_xor_sync(0xffffffffu, x[0], m);
    }
  }
}

// ----------------------------------------------------------------------------- records
// Floats of a record: (delta) k P [4][dk]; q P [4][dk], k / P [4][dk], P_3 [dk], M [4][4], step sizes [4], flag [4].
// M[t][s]: q_t . k_s for s <= t, k_s . k_t (read side of s, write side of t) for s > t.
__host__ __device__ constexpr int rec_floats(bool delta, int dk) { return (delta ? 13 : 9) * dk + 24; }
constexpr int REC_M = -24, REC_BETA = -8, REC_FLAG = -4;      // from a record's end

struct RecStream {
  int units, H, S, vdim, dk_pad, dv_pad;
  int t0, groups;                // first token and groups of four of this launch
  int dvc, tiles;                // columns of a CTA, and CTAs a head
  int stages;
  float* rec;                    // [units][groups][rec_floats]
  float* direct;                 // [units][groups][4][dk]: decays of groups whose flag is set (others: not written)
  float* v;                      // [units][tiles][groups][dvc][4]
  float* state;                  // [units][dk_pad][dv_pad]
  float* o;                      // [B, S, H, vdim]
  int* err;
};

constexpr int REC_STAGE_GROUPS = 2, REC_MAX_STAGES = 8;
// A lane holds rec_rows rows of REC_COLS columns: a column's rows lie over all 32 lanes where there are enough.
constexpr int REC_COLS = 4, REC_WARPS = 4;
__host__ __device__ constexpr int rec_rows(int dk) { return dk <= 128 ? 4 : dk / 32; }

template <int DK, bool DELTA>
__global__ void __launch_bounds__(REC_WARPS * 32 + 32, 2)
recurrence_kernel(RecStream p) {
  constexpr int R = rec_rows(DK), C = REC_COLS, LPC = DK / R, V = R / 4, REC = rec_floats(DELTA, DK);
  constexpr int N = 4 * C, OWN = N >= LPC ? N / LPC : 1, REP = N >= LPC ? 1 : LPC / N;
  constexpr int CPW = C * (32 / LPC);
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(8) uint64_t full[REC_MAX_STAGES], empty[REC_MAX_STAGES];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, consumers = (blockDim.x >> 5) - 1;
  const int unit = blockIdx.x, tile = blockIdx.y;
  const int stage_floats = REC_STAGE_GROUPS * (REC + p.dvc * 4);
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) { sm100::mbar_init(&full[s], 1); sm100::mbar_init(&empty[s], consumers); }
    abort_word = 0;
    sm100::fence_mbar_init();
  }
  __syncthreads();
  pdl_wait();
  pdl_trigger();

  if (warp == consumers) {
    if (lane == 0) {
      const float* rec = p.rec + (int64_t)unit * p.groups * REC;
      const float* v = p.v + ((int64_t)unit * p.tiles + tile) * p.groups * p.dvc * 4;
      int stage = 0;
      uint32_t phase = 0;
      for (int g = 0; g < p.groups; g += REC_STAGE_GROUPS) {
        if (!sm100::mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.err, 231)) break;
        const int n = min(REC_STAGE_GROUPS, p.groups - g);
        float* dst = sm + stage * stage_floats;
        sm100::mbar_arrive_expect_tx(&full[stage], (uint32_t)(n * (REC + p.dvc * 4) * 4));
        sm100::bulk_load(dst, rec + (int64_t)g * REC, (uint32_t)(n * REC * 4), &full[stage]);
        sm100::bulk_load(dst + REC_STAGE_GROUPS * REC, v + (int64_t)g * p.dvc * 4, (uint32_t)(n * p.dvc * 16), &full[stage]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      // A CTA does not end before its copies: consumers that give up, now or later, leave the wait for them to this warp.
      for (int s = 0; s < p.stages; ++s) {
        const long long since = clock64();
        while (!sm100::mbar_try_wait(&full[s], s < stage ? phase : phase ^ 1) && clock64() - since < 1000000) {}
      }
    }
    return;
  }

  const int j = lane % LPC, cg = lane / LPC;
  const int lcol = warp * CPW + cg * C, col = tile * p.dvc + lcol;
  float2 s[C][R / 2];            // rows (i LPC + j) 4 + e (i < V, e < 4) of columns col .. col + C - 1, as [column][row pair]
  float* srow = p.state + ((int64_t)unit * p.dk_pad + j * 4) * p.dv_pad + col;
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int i = 0; i < V; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float* src = srow + (int64_t)(i * LPC * 4 + 2 * e) * p.dv_pad + c;
        s[c][2 * i + e] = col + c < p.dv_pad ? make_float2(src[0], src[p.dv_pad]) : make_float2(0.f, 0.f);
      }

  struct Vec { float4 x[V]; };   // this lane's rows of a vector
  auto load = [&](const float* vec) {
    Vec r;
#pragma unroll
    for (int i = 0; i < V; ++i) r.x[i] = reinterpret_cast<const float4*>(vec)[i * LPC + j];
    return r;
  };
  // x[c] = this lane's part of (state column c) . (row vector)
  auto dot = [&](const Vec& k, float* x) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      float2 a;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        a = i ? fma2(s[c][2 * i], make_float2(k.x[i].x, k.x[i].y), a) : mul2(s[c][0], make_float2(k.x[0].x, k.x[0].y));
        a = fma2(s[c][2 * i + 1], make_float2(k.x[i].z, k.x[i].w), a);
      }
      x[c] = a.x + a.y;
    }
  };
  auto add = [&](const Vec& k, const float* u) {
#pragma unroll
    for (int i = 0; i < V; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        s[c][2 * i] = fma2(make_float2(k.x[i].x, k.x[i].y), make_float2(u[c], u[c]), s[c][2 * i]);
        s[c][2 * i + 1] = fma2(make_float2(k.x[i].z, k.x[i].w), make_float2(u[c], u[c]), s[c][2 * i + 1]);
      }
  };
  auto scale = [&](const Vec& d) {
#pragma unroll
    for (int i = 0; i < V; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        s[c][2 * i] = mul2(s[c][2 * i], make_float2(d.x[i].x, d.x[i].y));
        s[c][2 * i + 1] = mul2(s[c][2 * i + 1], make_float2(d.x[i].z, d.x[i].w));
      }
  };

  const int b = unit / p.H, h = unit - b * p.H;
  const int64_t o_ld = (int64_t)p.H * p.vdim;
  float* out = p.o + (int64_t)b * p.S * o_ld + (int64_t)h * p.vdim + col;
  int stage = 0;
  uint32_t phase = 0;
  // The vectors that a group reads with are fetched while the group before writes.
  constexpr int QV = DELTA ? 4 * DK : 0;
  Vec kr[DELTA ? 4 : 1], qr[4];
  float flag;
  auto fetch = [&](const float* rec) {
    flag = rec[REC + REC_FLAG];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if constexpr (DELTA) kr[t] = load(rec + t * DK);
      qr[t] = load(rec + QV + t * DK);
    }
  };
  bool ok = __all_sync(0xffffffffu, sm100::mbar_wait(&full[0], 0, abort_flag, p.err, 232));
  if (ok) fetch(sm);
  int at = 0;
  // One record.  RAGGED: the last of a prompt, with tokens past the end.  A copy of the code: the masks cost every record 3 %
  // (8192 tokens, 16 heads of 128: 1538 us, 1589 with masks), the copy a call that needs it 1.3 us.
  auto walk = [&](int g, auto ragged) {
    constexpr bool RAGGED = decltype(ragged)::value;
    const float* base = sm + stage * stage_floats;
    const float* rec = base + at * REC;
    const float* kw = rec + QV + 4 * DK;
    const float* M = rec + REC + REC_M;
    const float* vv = base + REC_STAGE_GROUPS * REC + (at * p.dvc + lcol) * 4;
    const int t0 = p.t0 + g * 4;
    const bool last = at + 1 == REC_STAGE_GROUPS || g + 1 == p.groups;      // of this stage
    const int next_stage = !last ? stage : stage + 1 == p.stages ? 0 : stage + 1;
    const uint32_t next_phase = last && next_stage == 0 ? phase ^ 1 : phase;
    auto fetch_next = [&] {
      if (g + 1 == p.groups) return;
      if (last) ok = __all_sync(0xffffffffu, sm100::mbar_wait(&full[next_stage], next_phase, abort_flag, p.err, 232));
      if (ok) fetch(last ? sm + next_stage * stage_floats : rec + REC);
    };
    if (flag == 0.f) {
      float u[4][C], y[N];
      if constexpr (DELTA) {
        float x[N];
#pragma unroll
        for (int t = 0; t < 4; ++t) dot(kr[t], x + t * C);
        lanes_sum<N, LPC>(j, x);
#pragma unroll
        for (int i = 0; i < N; ++i) u[i / C][i % C] = __shfl_sync(0xffffffffu, x[N >= LPC ? i % OWN : 0], cg * LPC + (N >= LPC ? i / OWN : i * REP));
      }
#pragma unroll
      for (int t = 0; t < 4; ++t) dot(qr[t], y + t * C);
      Vec w[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) w[t] = load(kw + t * DK);
      const Vec post = load(kw + 4 * DK);
      lanes_sum<N, LPC>(j, y);
      if constexpr (DELTA) {
        const float4 m0 = *reinterpret_cast<const float4*>(M), m1 = *reinterpret_cast<const float4*>(M + 4), m2 = *reinterpret_cast<const float4*>(M + 8);
        const float4 beta = *reinterpret_cast<const float4*>(rec + REC + REC_BETA);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(vv + c * 4);
          // (the tokens' own products are summed first: small next to v - D, they round less)
          u[0][c] = beta.x * (v.x - u[0][c]);
          u[1][c] = beta.y * ((v.y - u[1][c]) - m0.y * u[0][c]);
          u[2][c] = beta.z * ((v.z - u[2][c]) - fmaf(m1.z, u[1][c], m0.z * u[0][c]));
          u[3][c] = beta.w * ((v.w - u[3][c]) - fmaf(m2.w, u[2][c], fmaf(m1.w, u[1][c], m0.w * u[0][c])));
        }
        // (tokens past the end write nothing, not even zero times an infinity)
        if constexpr (RAGGED) {
#pragma unroll
          for (int t = 1; t < 4; ++t)
#pragma unroll
            for (int c = 0; c < C; ++c) u[t][c] = t0 + t < p.S ? u[t][c] : 0.f;
        }
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const float4 v = *reinterpret_cast<const float4*>(vv + c * 4);
          u[0][c] = v.x; u[1][c] = v.y; u[2][c] = v.z; u[3][c] = v.w;
        }
      }
#pragma unroll
      for (int i = 0; i < OWN; ++i) {
        const int n = N >= LPC ? j * OWN + i : j / REP, t = n / C, c = n % C;
        const float4 m = *reinterpret_cast<const float4*>(M + t * 4);
        float us[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          us[k] = u[k][0];
#pragma unroll
          for (int cc = 1; cc < C; ++cc) us[k] = c == cc ? u[k][cc] : us[k];
        }
        float own = m.x * us[0];
        own = t >= 1 ? fmaf(m.y, us[1], own) : own;
        own = t >= 2 ? fmaf(m.z, us[2], own) : own;
        own = t >= 3 ? fmaf(m.w, us[3], own) : own;
        const float o = y[i] + own;
        if (j % REP == 0 && t0 + t < p.S && col + c < p.vdim) out[(t0 + t) * o_ld + c] = o;
      }
      fetch_next();
#pragma unroll
      for (int t = 0; t < 4; ++t) add(w[t], u[t]);
      scale(post);
    } else {
      const float* direct = p.direct + ((int64_t)unit * p.groups + g) * 4 * DK;
#pragma unroll 1
      for (int t = 0; t < 4 && t0 + t < p.S; ++t) {
        float x[C], u[C];
        auto sum = [&] {
#pragma unroll
          for (int c = 0; c < C; ++c)
#pragma unroll
            for (int m = LPC / 2; m > 0; m >>= 1) x[c] += __shfl_xor_sync(0xffffffffu, x[c], m);
        };
        if constexpr (DELTA) {
          scale(load(direct + t * DK));
          dot(load(rec + t * DK), x);
          sum();
#pragma unroll
          for (int c = 0; c < C; ++c) u[c] = rec[REC + REC_BETA + t] * (vv[c * 4 + t] - x[c]);
          add(load(kw + t * DK), u);
          dot(load(rec + QV + t * DK), x);
          sum();
        } else {
          dot(load(rec + QV + t * DK), x);
          sum();
#pragma unroll
          for (int c = 0; c < C; ++c) {
            u[c] = vv[c * 4 + t];
            x[c] = fmaf(M[t * 5], u[c], x[c]);
          }
          scale(load(direct + t * DK));
          add(load(kw + t * DK), u);
        }
#pragma unroll
        for (int c = 0; c < C; ++c)
          if (j == 0 && col + c < p.vdim) out[(t0 + t) * o_ld + c] = x[c];
      }
      fetch_next();
    }
    if (last) {
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&empty[stage]);
      at = 0;
    } else {
      ++at;
    }
    stage = next_stage;
    phase = next_phase;
  };
  const int whole = DELTA && p.t0 + p.groups * 4 > p.S ? p.groups - 1 : p.groups;      // (WKV: zero values, no masks)
  for (int g = 0; ok && g < whole; ++g) walk(g, std::false_type());
  if constexpr (DELTA)
    if (ok && whole < p.groups) walk(whole, std::true_type());
#pragma unroll
  for (int c = 0; c < C; ++c)
#pragma unroll
    for (int i = 0; i < V; ++i)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (col + c < p.dv_pad) {
          float* dst = srow + (int64_t)(i * LPC * 4 + 2 * e) * p.dv_pad + c;
          dst[0] = s[c][2 * i + e].x;
          dst[p.dv_pad] = s[c][2 * i + e].y;
        }
}

// Bytes of records that a portion of a prompt may take: they are written and read back inside the L2 cache.  They lie in the
// library's workspace, which the first such call grows to 96 MB (1.5 times) for good.
constexpr int64_t REC_SCRATCH = 64 << 20;
// ... but at least this many groups a portion, or loading and storing the states would count (that is below
// REC_SCRATCH but for many heads of few value channels: 321 MB for 592 heads of 256 key and 16 value channels).
constexpr int REC_LEAST_GROUPS = 32;

// Least tokens of a call that take records, by [delta rule][16-bit inputs][key channels 32, 64, 128, 256][CTAs of the walk
// in units of SMs, rounded up, 1 .. 4]; 0: none do.  Both forms measured for 10 to 592 CTAs and 32 to 1000 tokens; a number
// stands where the records were the shorter from there on (time of the records over the one-kernel form's):
//   delta, bf16  64 channels, 4: 0.92 to 1.07, no gain.  128, 3: 1.05 at 32 tokens, 0.97 at 40; 4: 1.14 at 32, 0.95 at 64
//   delta, fp32  64, 4: 1.10 at 32, 0.96 at 40
//   WKV, bf16    64, 4: 1.07 at 32, 0.97 at 48.  128, 3: 1.10 at 32, 0.98 at 48; 4: 1.38 at 32, 0.97 at 256.
//                256, 2: 1.23 at 32, 0.95 at 64; 3: 1.58 at 32, 1.06 at 600; 4: 1.79 and 1.31
//   WKV, fp32    128, 4: 1.28 at 32, 0.97 at 96.  256, 3: 1.11 at 32, 0.97 at 40; 4: 1.27 at 32, 0.89 at 96
//   elsewhere    0.12 to 0.95; 16 tokens: 30 us against 28 (delta rule, 16 heads of 128)
constexpr int REC_LEAST_TOKENS[2][2][4][4] = {
    {{{32, 32, 32, 32}, {32, 32, 32, 32}, {32, 32, 32, 96}, {32, 32, 40, 96}},
     {{32, 32, 32, 32}, {32, 32, 32, 48}, {32, 32, 48, 256}, {32, 64, 0, 0}}},
    {{{32, 32, 32, 32}, {32, 32, 32, 40}, {32, 32, 32, 32}, {32, 32, 32, 32}},
     {{32, 32, 32, 32}, {32, 32, 32, 0}, {32, 32, 40, 64}, {32, 32, 32, 32}}}};
// Warps of a CTA and CTAs of a head whose state has dk rows and dv_pad columns.
inline void recurrence_shape(int dk, int dv_pad, int* warps, int* tiles) {
  const int cpw = REC_COLS * 32 * rec_rows(dk) / dk, all = (dv_pad + cpw - 1) / cpw;
  *warps = all > REC_WARPS ? REC_WARPS : all;
  *tiles = (dv_pad + *warps * cpw - 1) / (*warps * cpw);
}
inline bool recurrence_takes_records(bool delta, bool half, int dk, int64_t ctas, int S, int sms) {
  const int64_t waves = (ctas + sms - 1) / sms;
  if (waves < 1 || waves > 4) return false;
  const int least = REC_LEAST_TOKENS[delta][half][dk <= 32 ? 0 : dk <= 64 ? 1 : dk <= 128 ? 2 : 3][waves - 1];
  return least > 0 && S >= least;
}

template <int DK, bool DELTA>
static int launch_recurrence_kernel(const RecStream& p, int warps) {
  const int smem = p.stages * REC_STAGE_GROUPS * (rec_floats(DELTA, DK) + p.dvc * 4) * 4;
  static bool configured[64] = {false};
  if (!configured[ctx().device & 63]) {
    KD_CUDA_CHECK(cudaFuncSetAttribute(recurrence_kernel<DK, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
    configured[ctx().device & 63] = true;
  }
  KD_CUDA_CHECK(launch_ex(recurrence_kernel<DK, DELTA>, dim3(p.units, p.tiles), dim3((warps + 1) * 32), (size_t)smem, p));
  return after_launch("recurrence_kernel");
}

// Walks through a prompt in portions; prepare(portion) launches the layer's prepare kernel for one.  *handled = 0: the
// heads fill the chip by themselves, or there is no room for records, and the caller's one-kernel form is to run.
template <int DK, bool DELTA, bool HALF, typename Prepare>
static int launch_recurrence(RecStream p, int* handled, Prepare&& prepare) {
  *handled = 0;
  const int sms = ctx().sm_count;
  int warps;
  recurrence_shape(DK, p.dv_pad, &warps, &p.tiles);
  p.dvc = warps * (REC_COLS * 32 * rec_rows(DK) / DK);
  const int64_t ctas = (int64_t)p.units * p.tiles;
  if (!recurrence_takes_records(DELTA, HALF, DK, ctas, p.S, sms)) return KD_OK;
  const int stage_bytes = REC_STAGE_GROUPS * (rec_floats(DELTA, DK) + p.dvc * 4) * 4;
  const int room = (ctas <= sms ? 200 : ctas <= 2 * sms ? 100 : 50) * 1024 / stage_bytes;
  p.stages = room < 2 ? 2 : room > REC_MAX_STAGES ? REC_MAX_STAGES : room;
  p.err = ctx().error_flag;
  const int64_t rec = rec_floats(DELTA, DK), group = rec + 4 * DK + (int64_t)p.tiles * p.dvc * 4, all = (p.S + 3) / 4;
  int64_t portion = REC_SCRATCH / (group * 4 * p.units);
  if (portion < REC_LEAST_GROUPS) portion = REC_LEAST_GROUPS;
  if (portion > all) portion = all;
  const int64_t parts = (all + portion - 1) / portion, even = (all + parts - 1) / parts;
  void* ws = nullptr;
  if (get_workspace((uint64_t)(even * group * p.units) * 4, &ws) != KD_OK) return KD_OK;
  *handled = 1;
  for (int64_t g = 0; g < all; g += even) {
    p.t0 = (int)(g * 4);
    p.groups = (int)(all - g < even ? all - g : even);
    p.rec = static_cast<float*>(ws);
    p.direct = p.rec + rec * p.groups * p.units;
    p.v = p.direct + (int64_t)4 * DK * p.groups * p.units;
    KD_TRY(prepare(p));
    KD_TRY((launch_recurrence_kernel<DK, DELTA>(p, warps)));
  }
  return KD_OK;
}

}  // namespace kd
