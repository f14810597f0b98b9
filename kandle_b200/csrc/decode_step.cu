// A whole decode step of a Qwen3-architecture decoder for a few sequences (1..6) as ONE persistent kernel: embedding, every
// layer's QKV projection, q/k-norm + RoPE + cache write, attention over the cache, o_proj, SwiGLU MLP, and the lm_head.
//
// It computes what decode_layer.cu and the kernels around it compute (packages/model-utils/src/qwen3/decoder_layer.ts:191-241,
// attention/gqa.ts:246-322, mlp/swiglu.ts:119-134, rope.ts:546-644, kv-cache.ts:164-212, qwen3/for_causal_lm.ts:475-508) and
// needs nothing but vectors between SMs: a step of one sequence moves 1.2 GB of weights and 2 to 12 KB per hand-over.
//
// What bounds it: HBM, the bytes of the weights, as long as the hand-overs stay hidden; there are five per layer (six where
// the keys of a head are split) and each is a round trip through L2, so with the weights of a small layer (31 MB: 5 us) it is
// the chain of hand-overs and of the instructions between them, of which a warp issues one in 5 to 7 cycles.  So:
//   - Weights never wait for activations.  Four warps copy the rows that the CTA will multiply into a ring of units (8 rows x
//     512 columns; attention: 32 keys, 32 values) in shared memory, across phases and layers, as far ahead as the ring
//     reaches (about 190 KB).  All but the newest position's cache rows are older than the step and travel the same way.
//   - A hand-over is one store and one load.  A number is handed on as a 64-bit word that holds it and a tag (step, layer);
//     the reader polls the words it needs until their tags match, so there is no counter, fence or second round trip for the
//     data.  Tags differ from one use of a word to the next, and a word is never overwritten before its readers are
//     done: whoever writes it again has, through the phases between, seen a result of every reader.
//     The words of a phase leave a CTA in one store instruction: a line that all CTAs poll moves with each store into it.
//   - A CTA owns the same rows of every matrix, so that the residual stays in its shared memory; a warp owns every 16th group
//     of 32 columns and polls only those of the activations; one barrier per phase, where the warps' partial sums meet.
//   - Up to six units are one stage (one wait, one release), whose loads and products are straight-line code for the
//     number of row blocks.
// mma.sync (m16n8k16) does the products: 8 weight rows x 32 columns at a time against up to 6 sequences.  tcgen05 needs 128
// rows of one operand in shared memory and a trip through tensor memory, which here only adds latency: an SM multiplies
// 830 such tiles a layer, under 2 % of its time.
//
// Measured on B200, Qwen3-0.6B without the lm_head, us a step at a context of 300 (kernels per layer in brackets): 1 sequence 446
// (1042), 2 478 (1061), 4 584 (1069), 6 757 (1102); 4B widths, 9 layers: 1 472 (687), 2 554 (685).  7 and 8 sequences, where
// registers run out, were 943 and 985 (1091, 1102) there and slower than the kernels per layer at 1200 keys: not taken.
// Contexts that one CTA takes whole and keys of a split: 96 and 32 (446 us at 300 keys; 96 and 96: 464, 192 and 96: 464).
//
// All CTAs wait for one another, so the launch is cooperative, and every wait is bounded (codes 541-545): a CTA that
// gives up goes on to the end without waiting, so that the step's ticket and tag stay in order.
#include <algorithm>
#include <climits>
#include <cstddef>
#include <type_traits>

#include "chain_common.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "sm100.cuh"

namespace kd {

constexpr int DS_WARPS = 16, DS_WORKERS = DS_WARPS * 32, DS_THREADS = DS_WORKERS + 128;     // the last four warps copy
// Registers: 640 threads are launched with 96 each; the last warpgroup gives back what the workers take (512 x 112 + 128 x 32 = 640 x 96).
constexpr int DS_REGS_WORK = 112, DS_REGS_COPY = 32;
constexpr int DS_RB = 6;                  // blocks of 8 weight rows that a pass accumulates
constexpr int DS_ROWS = DS_RB * 8;
constexpr int DS_SEG = DS_WARPS * 32;     // columns of a unit
constexpr int DS_UNIT_ROW = DS_SEG * 2 + 64;      // (an odd number of half lines: two rows' pieces meet no bank twice)
constexpr int DS_UNIT = 8 * DS_UNIT_ROW;
constexpr int DS_COPY_WARPS = 4;          // (a warp issues its lanes' copies one by one: one warp alone kept up with 2.7 TB/s)
constexpr int DS_STAGE = 6;               // units of a stage at most
constexpr int DS_BARS = 32;               // stages on their way at most (units of the ring, at least)
constexpr int DS_KEYS = 32;               // keys of a unit
constexpr int DS_MAX_LAYERS = 64, DS_MAX_M = 6, DS_MAX_SPLITS = 32, DS_MAX_UNITS = 24;
constexpr int DS_MAX_N = 1 << 23;         // rows of a matrix
constexpr int DS_UNSPLIT_KEYS = 96;       // contexts that one CTA takes whole: the hand-over of a split costs as much as three steps over keys

typedef unsigned long long u64;

struct DsLayer {
  const __nv_bfloat16 *in_norm, *wqkv, *q_norm, *k_norm, *wo, *post_norm, *wgu, *wdown;
  __nv_bfloat16 *kc, *vc;
};

struct DsParams {
  DsLayer layer[DS_MAX_LAYERS];
  const __nv_bfloat16 *embed, *final_norm, *head;
  const int64_t* ids;
  const float* inv_freq;
  int *pos, *ctx;             // advanced at the end of the step
  float* logits;              // [M][V]
  const int* table;           // paged cache (null: contiguous)
  int* err;
  unsigned* state;            // [0] steps done, [1] tickets of the step that runs
  u64* best;                  // [M] largest logit so far of the step that runs (ds_key), zero between steps
  int64_t* next;              // [M] greedy next tokens, or null
  u64 *qkv, *part, *attn, *h1, *act, *h2;     // tagged words
  int64_t kc_b, kc_h, kc_s;
  float eps, scale_log2;
  int M, H, I, Hq, Hkv, L, V, max_s, max_pages, splits, units;
  unsigned last_page;         // of the pools
  int x_stride, h_rows;       // bytes of a sequence's activations; rows of the residual that a CTA may own
};

// ---- tagged words
__device__ __forceinline__ void ds_st(u64* p, uint32_t v, uint32_t tag) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((u64)v | ((u64)tag << 32)) : "memory");
}
__device__ __forceinline__ ulonglong2 ds_ld2(const u64* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool ds_ok(const ulonglong2& v, uint32_t tag) { return (uint32_t)(v.x >> 32) == tag && (uint32_t)(v.y >> 32) == tag; }
__device__ __forceinline__ float ds_f(u64 v) { return __uint_as_float((uint32_t)v); }

// Waits for words until their tags match are bounded; after a CTA has given up nothing waits any more.
__device__ __noinline__ bool ds_give_up(long long t0, volatile int* abort_flag, int* err, int code) {
  if (*abort_flag) return true;
  if (clock64() - t0 <= sm100::WAIT_CYCLE_LIMIT) return false;
  *abort_flag = 1;
  if (atomicCAS(err, 0, code) == 0) { err[1] = (int)blockIdx.x; err[2] = (int)threadIdx.x; }
  return true;
}
// N pairs of words, the i-th at at(i) where wanted(i).  All loads of a round are on their way before the first is looked at: a
// round trip through L2 is what this costs.
template <int N, typename At, typename Wanted>
__device__ __forceinline__ void ds_take(ulonglong2 (&v)[N], At at, Wanted wanted, uint32_t tag, volatile int* abort_flag, int* err, int code) {
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (wanted(i)) v[i] = ds_ld2(at(i));
  const long long t0 = clock64();
  for (int n = 1;; ++n) {
    bool all = true;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (wanted(i) && !ds_ok(v[i], tag)) all = false;
    if (all || ((n & 255) == 0 && ds_give_up(t0, abort_flag, err, code))) return;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (wanted(i)) v[i] = ds_ld2(at(i));
  }
}

// D[8 sequences (of 16 rows), 8 weight rows] += X[., 32] W[8, 32]^T, a lane's 16 bytes of each: the columns of the two
// products are taken in the same order on both sides.
__device__ __forceinline__ void ds_mma(float (&d)[4], const uint4& x, const uint4& w) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %8, %5, %8}, {%9, %10}, {%0, %1, %2, %3};\n\t"
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%6, %8, %7, %8}, {%11, %12}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(x.x), "r"(x.y), "r"(x.z), "r"(x.w), "r"(0u), "r"(w.x), "r"(w.y), "r"(w.z), "r"(w.w));
}
__device__ __forceinline__ float ds_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float ds_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
__device__ __forceinline__ uint32_t ds_pack(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// A logit and its column as a number that is larger for the larger logit and, among equals, the lower column; 0 for what is no maximum
// of anything (argmax_kernel's rule: compared with the lowest float by `greater than`).
__device__ __forceinline__ u64 ds_key(float v, int column) {
  if (!(v > -3.402823466e38f)) return 0;
  const uint32_t b = __float_as_uint(v + 0.0f);          // (-0 is 0)
  return (u64)(b & 0x80000000u ? ~b : b | 0x80000000u) << 32 | (0xffffffffu - (uint32_t)column);
}
// 1 / sqrt(s), with a Newton step: as exact as the division; 0 for squares beyond the range of fp32, as the division gives.
__device__ __forceinline__ float ds_inv_sqrt(float s) {
  const float y = rsqrtf(s);
  return y == 0.f ? 0.f : y * (1.5f - 0.5f * s * y * y);
}
template <int LANES>
__device__ __forceinline__ float ds_sum(float v) {        // over groups of lanes
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void ds_bar() { asm volatile("bar.sync 1, 512;" ::: "memory"); }      // all but the copying warp

// Where CTA c's share of n items begins (n * 256 fits 32 bits: DS_MAX_N).
__device__ __forceinline__ int ds_lo_of(int n, int c, int G) { return (int)((uint32_t)n * (uint32_t)c / (uint32_t)G); }

// Keys of a head that split s of a step at position pos reads from the cache.
struct DsKeys { int splits, k0, k1; };
__device__ __forceinline__ DsKeys ds_keys(int pos, int max_splits, int s) {
  DsKeys r;
  r.splits = pos <= DS_UNSPLIT_KEYS ? 1 : min(max_splits, (pos + DS_KEYS - 1) / DS_KEYS);
  const int per = (pos + r.splits - 1) / r.splits;
  r.k0 = min(pos, s * per);
  r.k1 = s < r.splits ? min(pos, r.k0 + per) : r.k0;
  return r;
}

enum { DS_QKV = 0, DS_ATT, DS_O, DS_GU, DS_DOWN, DS_HEAD, DS_DONE };

// What threads look up again and again, in shared memory: the layers' pointers, and each phase's rows of this CTA (gate/up:
// intermediate channels).
struct DsTable {
  int n0[DS_DONE], nn[DS_DONE];
  DsLayer layer[DS_MAX_LAYERS];
};

__device__ __forceinline__ int ds_columns(const DsParams& p, int phase) { return phase == DS_O ? p.Hq * 128 : phase == DS_DOWN ? p.I : p.H; }
__device__ __forceinline__ void ds_next(int& l, int& phase, int L) {
  if (phase == DS_DOWN && l < L - 1) {
    phase = DS_QKV;
    ++l;
  } else {
    ++phase;
  }
}
// A page outside the pool (reported at the start of the step) is taken for the last one.
__device__ __forceinline__ int64_t ds_cache_row(const DsParams& p, int b, int g, int key) {
  if (p.table) return (int64_t)min((unsigned)p.table[(int64_t)b * p.max_pages + key / 128], p.last_page) * p.kc_b + g * p.kc_h + (key % 128) * p.kc_s;
  return b * p.kc_b + g * p.kc_h + key * p.kc_s;
}

// Where a stage of n units begins in a ring of `units`: a stage does not wrap.
__device__ __forceinline__ int ds_stage_at(int at, int n, int units) { return at + n > units ? 0 : at; }
// Segments of columns that a stage takes with nrb row blocks.
__host__ __device__ constexpr int ds_stage_segs(int nrb) { return nrb == 1 ? 2 : 1; }

// M sequences
template <int GROUP, int M>
__global__ void __launch_bounds__(DS_THREADS, 1) decode_step_kernel(const __grid_constant__ DsParams p) {
  using namespace sm100;
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, t = threadIdx.x;
  const int cta = blockIdx.x, G = gridDim.x;
  // [units][activations][2 x partial sums][2 x sums of squares][residual][attention][cos, sin][barriers][table]
  uint8_t* at = smem + p.units * DS_UNIT;
  uint8_t* xs = at;                                          // [sequence][x_stride]
  at += M * p.x_stride;
  const int red_warp = M * DS_ROWS + 2;                      // (16 warps' sums of two rows lie in 32 banks)
  float* red = reinterpret_cast<float*>(at);                 // [2][warp][sequence][48]
  at += 2 * DS_WARPS * red_warp * 4;
  float* ssq = reinterpret_cast<float*>(at);                 // [2][sequence][warp]
  at += 2 * M * DS_WARPS * 4;
  float* hid = reinterpret_cast<float*>(at);                 // [sequence][own rows]
  at += (M * p.h_rows * 4 + 15) / 16 * 16;
  float* att_o = reinterpret_cast<float*>(at);               // [warp][GROUP][128]
  float* att_ml = att_o + DS_WARPS * GROUP * 128;            // [GROUP][2][warp]
  float* q_s = att_ml + DS_WARPS * GROUP * 2;                // [GROUP][128], then the new key and value
  uint32_t* out_s = reinterpret_cast<uint32_t*>(q_s + (GROUP + 2) * 128);   // [sequence][64] results of a phase; attention: [GROUP][64]
  float* rot = reinterpret_cast<float*>(out_s + (M > GROUP ? M : GROUP) * 64);      // cos [64], sin [64]
  uint64_t* full = reinterpret_cast<uint64_t*>(rot + 128);
  uint64_t* empty = full + DS_BARS;
  uint8_t* stage_units = reinterpret_cast<uint8_t*>(empty + DS_BARS);       // [copying warp][stage]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(stage_units + DS_COPY_WARPS * DS_BARS);
  DsTable& tab = *reinterpret_cast<DsTable*>(stage_units + DS_COPY_WARPS * DS_BARS + 16);

  const int pos_given = *p.pos;
  const bool pos_ok = pos_given >= 0 && pos_given < p.max_s;
  const int pos = pos_ok ? pos_given : 0;                    // (an error below)
  const uint32_t tag0 = p.state[0] * (uint32_t)(p.L + 1);
  if (t < DS_DONE) {
    const int n = t == DS_QKV ? (p.Hq + 2 * p.Hkv) * 128 : t == DS_GU ? p.I / 2 : t == DS_HEAD ? p.V : p.H, unit = t == DS_GU ? 2 : 1;
    const int lo = ds_lo_of(n, cta, G);
    tab.n0[t] = unit * lo;
    tab.nn[t] = unit * (ds_lo_of(n, cta + 1, G) - lo);
  }
  for (int i = t; i < p.L * (int)(sizeof(DsLayer) / 8); i += DS_THREADS)
    reinterpret_cast<u64*>(tab.layer)[i] = reinterpret_cast<const u64*>(p.layer)[i];
  if (t == 0) {
    *abort_flag = 0;
    for (int i = 0; i < DS_BARS; ++i) {
      mbar_init(&full[i], DS_COPY_WARPS);
      mbar_init(&empty[i], DS_WARPS);
    }
    fence_mbar_init();
    if (!pos_ok && cta == 0 && atomicCAS(p.err, 0, 102) == 0) { p.err[1] = pos_given; p.err[2] = p.max_s; }
  }
  if (p.table && cta < M)                                    // the step's pages of a sequence
    for (int i = t; i <= pos / 128; i += DS_THREADS) {
      const int page = p.table[(int64_t)cta * p.max_pages + i];
      if ((unsigned)page > p.last_page && atomicCAS(p.err, 0, 103) == 0) { p.err[1] = cta; p.err[2] = page; }
    }
  __syncthreads();

  // attention: (sequence, KV head), share of its keys
  const int item = cta / p.splits, split = cta - item * p.splits;
  const bool has_item = item < M * p.Hkv;
  const int att_b = has_item ? item / p.Hkv : 0, att_g = has_item ? item - att_b * p.Hkv : 0;
  const DsKeys keys = ds_keys(pos, p.splits, split);
  const bool attends = has_item && split < keys.splits;

  if (warp >= DS_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(DS_REGS_COPY));
    // ------------------------------------------------------------ the copying warps: they go through the same stages, and each
    // copies every fourth row (key) of a unit.  Each announces its own bytes (there may be none) on every stage's `full`: a stage
    // is not there before all four have come to it, so none falls behind by more than a ring of stages, and the parity of
    // `empty` is enough for it (a warp that had no part in a stage could miss two phases of a barrier and wait for a third).
    const int copier = warp - DS_WARPS;
    stage_units += copier * DS_BARS;
    int stage = 0, tail = 0, free = p.units, unit = 0;       // stages begun, stages given back, units free, next unit
    bool ok = true;
    auto claim = [&](int n) {                                // room for a stage, when its readers have left it
      const int begin = ds_stage_at(unit, n, p.units), need = n + (begin < unit ? p.units - unit : 0);
      while (free < need) {
        // (readers that have given up release stages that are not there yet: such a release is none)
        ok = mbar_wait(&empty[tail % DS_BARS], (uint32_t)(tail / DS_BARS) & 1u, abort_flag, p.err, 544) && !*abort_flag;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) return -1;
        free += stage_units[tail % DS_BARS];
        ++tail;
      }
      if (lane == 0) stage_units[stage % DS_BARS] = (uint8_t)need;
      __syncwarp();
      free -= need;
      unit = begin + n;
      ++stage;
      return begin;
    };
    // this warp's part of the claimed stage: `bytes` in each of its lanes that copy
    auto announce = [&](bool copies, uint32_t bytes) {
      const uint32_t lanes = __popc(__ballot_sync(0xffffffffu, copies));
      if (lane == 0) mbar_arrive_expect_tx(&full[(stage - 1) % DS_BARS], lanes * bytes);      // (before or after the copies land)
    };
    for (int l = 0, phase = DS_QKV; ok && phase != DS_DONE; ds_next(l, phase, p.L)) {
      const DsLayer& w = tab.layer[l];
      if (phase == DS_ATT) {
        if (!attends) continue;
        for (int key = keys.k0; ok && key < keys.k1; key += DS_KEYS) {
          const int n = min(DS_KEYS, keys.k1 - key), begin = claim(2);
          if (begin < 0) break;
          // one copy of keys and one of values where the rows lie side by side (8000 keys, 6 sequences: a copy per row kept the
          // step at 3.2 ms)
          const bool whole = p.kc_s == 128 && (!p.table || key % 128 + n <= 128);
          const bool copies = whole ? lane == 0 && copier < 2 : lane < n && lane % DS_COPY_WARPS == copier;
          announce(copies, whole ? n * 256u : 512u);
          if (copies) {
            const int64_t row = ds_cache_row(p, att_b, att_g, key + lane);
            uint64_t* bar = &full[(stage - 1) % DS_BARS];
            uint8_t* to = smem + begin * DS_UNIT + lane * 256;
            const uint32_t bytes = whole ? n * 256u : 256u;
            if (!whole || copier == 0) bulk_load(to, w.kc + row, bytes, bar);
            if (!whole || copier == 1) bulk_load(to + DS_UNIT, w.vc + row, bytes, bar);
          }
        }
        continue;
      }
      const int K = ds_columns(p, phase), nseg = K / DS_SEG, n0 = tab.n0[phase], nn = tab.nn[phase], per = phase == DS_GU ? 4 : 8;
      const __nv_bfloat16* W = phase == DS_QKV ? w.wqkv : phase == DS_O ? w.wo : phase == DS_GU ? w.wgu : phase == DS_DOWN ? w.wdown : p.head;
      for (int r0 = 0; ok && r0 < nn; r0 += DS_RB * per) {
        const int nrb = (min(nn - r0, DS_RB * per) + per - 1) / per, segs = ds_stage_segs(nrb);
        for (int s0 = 0; ok && s0 < nseg; s0 += segs) {
          const int n = min(segs, nseg - s0) * nrb;          // unit u: segment u / nrb, block u % nrb
          // unit u: segment u of one block, or block u of one segment; two of its rows are this warp's
          const int u = lane >> 1, rr = copier + DS_COPY_WARPS * (lane & 1), sg = nrb == 1 ? u : 0, rb = nrb == 1 ? 0 : u;
          // a block: 8 rows, or four channels' gate rows and their up rows (16 gate rows, then their 16 up rows)
          const int i = r0 + rb * per + (phase == DS_GU ? rr & 3 : rr), c = n0 + i;
          const int row = phase == DS_GU ? c + (c & ~15) + ((rr & 4) << 2) : c;
          const int begin = claim(n);
          if (begin < 0) break;
          announce(u < n && i < nn, DS_SEG * 2);
          if (u < n && i < nn)
            bulk_load(smem + (begin + u) * DS_UNIT + rr * DS_UNIT_ROW, W + (int64_t)row * K + (s0 + sg) * DS_SEG, DS_SEG * 2, &full[(stage - 1) % DS_BARS]);
        }
      }
    }
    // No copy is on its way when the CTA ends, whoever has given up.  The copying warps agree on the last stage that one of them
    // has begun, announce nothing for those that they have not come to, and wait for all that none has seen released (fewer
    // than there are barriers), within one limit.
    __syncwarp();
    volatile int* mine = reinterpret_cast<volatile int*>(stage_units);       // (its entries are not needed any more)
    if (lane == 0) {
      mine[0] = stage;
      mine[1] = tail;
    }
    asm volatile("bar.sync 2, 128;" ::: "memory");
    int last = stage, first = tail;
    for (int i = 0; i < DS_COPY_WARPS; ++i) {
      const volatile int* of = mine + (i - copier) * (DS_BARS / 4);
      last = max(last, of[0]);
      first = max(first, of[1]);
    }
    if (lane == 0)
      for (int i = stage; i < last; ++i) mbar_arrive(&full[i % DS_BARS]);
    volatile int never = 0;
    for (int i = first; i < last; ++i)
      if (!mbar_wait(&full[i % DS_BARS], (uint32_t)(i / DS_BARS) & 1u, &never, p.err, 544)) break;
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(DS_REGS_WORK));
    int stage = 0, unit = 0;
    if (t < 64) {
      const float ang = (float)pos * p.inv_freq[t];          // as rope_table_kernel
      rot[t] = cosf(ang);
      rot[64 + t] = sinf(ang);
    }
    auto token = [&](int m) -> const __nv_bfloat16* {        // embedding row of a sequence's token, null if there is none
      const int64_t id = p.ids[m];
      return id >= 0 && id < p.V ? p.embed + id * p.H : nullptr;
    };
    const int h0 = tab.n0[DS_O], nh = tab.nn[DS_O];
    for (int m = 0; m < M; ++m) {
      const __nv_bfloat16* e = token(m);
      if (!e && cta == 0 && t == 0 && atomicCAS(p.err, 0, 101) == 0) { p.err[1] = m; p.err[2] = (int)p.ids[m]; }
      for (int i = t; i < nh; i += DS_WORKERS) hid[m * p.h_rows + i] = e ? __bfloat162float(e[h0 + i]) : 0.f;
    }
    ds_bar();

    int flip = 0;                                            // which of the two reduction buffers
    u64 top = 0;                                             // of the logits that this thread has stored, all of sequence t / 64
    const float inv_h = 1.0f / (float)p.H;
    const int nqkv = (p.Hq + 2 * p.Hkv) * 128;
    const bool x_mine = (lane >> 2) < M;
    const uint8_t* x_frag = xs + (x_mine ? (lane >> 2) * p.x_stride : 0) + (lane & 3) * 16 + warp * 64;
    const uint8_t* w_frag = smem + (lane >> 2) * DS_UNIT_ROW + (lane & 3) * 16 + warp * 64;

    // The next stage, of n units: waits until it is there, gives its first unit.
    auto begin_stage = [&](int n) {
      const int begin = ds_stage_at(unit, n, p.units);
      mbar_wait(&full[stage % DS_BARS], (uint32_t)(stage / DS_BARS) & 1u, abort_flag, p.err, 545);
      unit = begin + n;
      return begin;
    };
    auto end_stage = [&] {
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[stage % DS_BARS]);
      ++stage;
    };

    // This warp's columns of fp32 activations, times the norm weights, as bf16; their sums of squares.  A lane takes two columns
    // of one of two segments.
    auto take_hidden = [&](const u64* src, uint32_t tag, const __nv_bfloat16* nw) {
      float ss[M];
#pragma unroll
      for (int m = 0; m < M; ++m) ss[m] = 0.f;
      for (int k = (lane >> 4) * DS_SEG + warp * 32 + (lane & 15) * 2; k < p.H; k += 2 * DS_SEG) {
        const uint32_t nwv = *reinterpret_cast<const uint32_t*>(nw + k);
        ulonglong2 v[M];
        if (src) {
          ds_take(v, [&](int m) { return src + m * p.H + k; }, [](int) { return true; }, tag, abort_flag, p.err, 541);
        } else {
#pragma unroll
          for (int m = 0; m < M; ++m)
            {
              const __nv_bfloat16* e = token(m);
              const uint32_t x = e ? *reinterpret_cast<const uint32_t*>(e + k) : 0u;
              v[m] = make_ulonglong2(x << 16, x & 0xffff0000u);
            }
        }
#pragma unroll
        for (int m = 0; m < M; ++m)
          {
            const float a = ds_f(v[m].x), b = ds_f(v[m].y);
            ss[m] += a * a + b * b;
            *reinterpret_cast<uint32_t*>(xs + m * p.x_stride + k * 2) = ds_pack(a * ds_lo(nwv), b * ds_hi(nwv));
          }
      }
#pragma unroll
      for (int m = 0; m < M; ++m)
        {
          const float s = warp_sum(ss[m]);
          if (lane == 0) ssq[(flip * M + m) * DS_WARPS + warp] = s;
        }
      __syncwarp();
    };
    // The same of bf16 activations, handed on in pairs: a lane takes four columns of one of four segments.
    auto take_pairs = [&](const u64* src, int K, uint32_t tag) {
      for (int k = (lane >> 3) * DS_SEG + warp * 32 + (lane & 7) * 4; k < K; k += 8 * DS_SEG) {
        ulonglong2 v[2 * M];
        const bool two = k + 4 * DS_SEG < K;
        const u64* a = src + k / 2;
        const auto wanted = [&](int i) { return i < M || two; };
        ds_take(v, [&](int i) { return a + (i % M) * (K / 2) + (i < M ? 0 : 2 * DS_SEG); }, wanted, tag, abort_flag, p.err, 542);
#pragma unroll
        for (int i = 0; i < 2 * M; ++i)
          if (wanted(i)) *reinterpret_cast<uint2*>(xs + (i % M) * p.x_stride + k * 2 + (i < M ? 0 : 8 * DS_SEG)) = make_uint2((uint32_t)v[i].x, (uint32_t)v[i].y);
      }
      __syncwarp();
    };

    // One pass: NRB blocks of 8 rows of this CTA against this warp's columns; its partial sums into red[flip].
    auto multiply = [&](auto blocks, int nseg) {
      constexpr int NRB = decltype(blocks)::value, SEGS = ds_stage_segs(NRB), ACC = NRB == 1 ? 2 : 1;
      float acc[ACC][NRB][4];
#pragma unroll
      for (int a = 0; a < ACC; ++a)
#pragma unroll
        for (int r = 0; r < NRB; ++r)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[a][r][i] = 0.f;
      const uint8_t* xa = x_frag;
      for (int left = nseg; left > 0; left -= SEGS) {
        const int ns = min(left, SEGS);
        uint4 x[SEGS], w[SEGS * NRB];
#pragma unroll
        for (int s = 0; s < SEGS; ++s)
          if (s < ns) x[s] = *reinterpret_cast<const uint4*>(xa + s * DS_SEG * 2);
        xa += SEGS * DS_SEG * 2;
        const uint8_t* wa = w_frag + begin_stage(ns * NRB) * DS_UNIT;
#pragma unroll
        for (int s = 0; s < SEGS; ++s)
          if (s < ns) {
            if (!x_mine) x[s] = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int r = 0; r < NRB; ++r) w[s * NRB + r] = *reinterpret_cast<const uint4*>(wa + (s * NRB + r) * DS_UNIT);
          }
#pragma unroll
        for (int s = 0; s < SEGS; ++s)
          if (s < ns) {
#pragma unroll
            for (int r = 0; r < NRB; ++r) ds_mma(acc[s % ACC][r], x[s], w[s * NRB + r]);
          }
        end_stage();
      }
      float* mine = red + (flip * DS_WARPS + warp) * red_warp + (M == 1 ? 0 : (lane >> 2) * DS_ROWS) + (lane & 3) * 2;
      if (x_mine) {
#pragma unroll
        for (int r = 0; r < NRB; ++r)
          *reinterpret_cast<float2*>(mine + r * 8) = make_float2(acc[0][r][0] + (ACC == 2 ? acc[ACC - 1][r][0] : 0.f), acc[0][r][1] + (ACC == 2 ? acc[ACC - 1][r][1] : 0.f));
      }
    };
    // Sum of a row over the warps, in half a warp (lane % 16 = warp whose share it reads).
    auto total = [&](int m, int row) { return ds_sum<16>(red[(flip * DS_WARPS + (lane & 15)) * red_warp + m * DS_ROWS + row]); };
    auto inv_rms = [&](int at_flip, int m) {
      return ds_inv_sqrt(ds_sum<16>(ssq[(at_flip * M + m) * DS_WARPS + (lane & 15)]) * inv_h + p.eps);
    };

    for (int l = 0, phase = DS_QKV; phase != DS_DONE; ds_next(l, phase, p.L)) {
      const DsLayer& w = tab.layer[l];
      const uint32_t tag = tag0 + (uint32_t)l + 1u;
      if (phase == DS_ATT) {
        if (!attends) continue;
        const int b = att_b, g = att_g;
        if (warp < GROUP || (split == 0 && warp < GROUP + 2)) {
          // a head per warp: q heads of the group, then (the CTA that takes the new position) key and value
          const int head = warp < GROUP ? g * GROUP + warp : warp == GROUP ? p.Hq + g : p.Hq + p.Hkv + g;
          const u64* src = p.qkv + b * nqkv + head * 128 + 4 * lane;
          const uint2 nw = reinterpret_cast<const uint2*>(warp < GROUP ? w.q_norm : w.k_norm)[lane];
          ulonglong2 v[2];
          ds_take(v, [&](int i) { return src + 2 * i; }, [](int) { return true; }, tag, abort_flag, p.err, 543);
          float y[4] = {ds_f(v[0].x), ds_f(v[0].y), ds_f(v[1].x), ds_f(v[1].y)};
          if (warp <= GROUP) {
            const float sc = ds_inv_sqrt(warp_sum(y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3]) * (1.f / 128.f) + p.eps);
            y[0] = (y[0] * sc) * ds_lo(nw.x);
            y[1] = (y[1] * sc) * ds_hi(nw.x);
            y[2] = (y[2] * sc) * ds_lo(nw.y);
            y[3] = (y[3] * sc) * ds_hi(nw.y);
            const float4 cs = *reinterpret_cast<const float4*>(rot + (4 * lane & 63)), sn = *reinterpret_cast<const float4*>(rot + 64 + (4 * lane & 63));
            const float c4[4] = {cs.x, cs.y, cs.z, cs.w}, s4[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              // out[d] = y[d] cos - y[d+64] sin; out[d+64] = y[d+64] cos + y[d] sin
              const float other = __shfl_xor_sync(0xffffffffu, y[i], 16);
              y[i] = lane < 16 ? y[i] * c4[i] - other * s4[i] : y[i] * c4[i] + other * s4[i];
            }
          }
          const uint32_t lo = ds_pack(y[0], y[1]), hi = ds_pack(y[2], y[3]);
          if (warp >= GROUP && pos_ok && (!p.table || (unsigned)p.table[(int64_t)b * p.max_pages + pos / 128] <= p.last_page))
            *reinterpret_cast<uint2*>((warp == GROUP ? w.kc : w.vc) + ds_cache_row(p, b, g, pos) + 4 * lane) = make_uint2(lo, hi);
          *reinterpret_cast<float4*>(q_s + warp * 128 + 4 * lane) = make_float4(ds_lo(lo), ds_hi(lo), ds_lo(hi), ds_hi(hi));
        }
        ds_bar();
        // each half warp walks keys of its own, a lane eight channels
        const int half = lane >> 4, d0 = (lane & 15) * 8;
        float q[GROUP][8], o[GROUP][8], mx[GROUP], sum[GROUP];
#pragma unroll
        for (int h = 0; h < GROUP; ++h) {
          mx[h] = -1e30f;
          sum[h] = 0.f;
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            const float4 v = *reinterpret_cast<const float4*>(q_s + h * 128 + d0 + e);
            q[h][e] = v.x; q[h][e + 1] = v.y; q[h][e + 2] = v.z; q[h][e + 3] = v.w;
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) o[h][e] = 0.f;
        }
        auto key_step = [&](const float (&k)[8], const float (&v)[8], bool ok) {
          float s[GROUP];
#pragma unroll
          for (int h = 0; h < GROUP; ++h) {
            const float a = (q[h][0] * k[0] + q[h][1] * k[1]) + (q[h][2] * k[2] + q[h][3] * k[3]);
            s[h] = a + ((q[h][4] * k[4] + q[h][5] * k[5]) + (q[h][6] * k[6] + q[h][7] * k[7]));
          }
#pragma unroll
          for (int x = 8; x > 0; x >>= 1)
#pragma unroll
            for (int h = 0; h < GROUP; ++h) s[h] += __shfl_xor_sync(0xffffffffu, s[h], x);
#pragma unroll
          for (int h = 0; h < GROUP; ++h) {
            const float x = ok ? s[h] * p.scale_log2 : -1e30f, nm = fmaxf(mx[h], x), f = exp2f(mx[h] - nm), e1 = ok ? exp2f(x - nm) : 0.f;
            mx[h] = nm;
            sum[h] = sum[h] * f + e1;
#pragma unroll
            for (int e = 0; e < 8; ++e) o[h][e] = o[h][e] * f + e1 * v[e];
          }
        };
        if (warp == DS_WARPS - 1 && split == 0) {            // (the warp with the fewest keys)
          float k[8], v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            k[e] = q_s[GROUP * 128 + d0 + e];
            v[e] = q_s[(GROUP + 1) * 128 + d0 + e];
          }
          key_step(k, v, half == 0);
        }
        for (int key = keys.k0; key < keys.k1; key += DS_KEYS) {
          const uint8_t* a = smem + begin_stage(2) * DS_UNIT + (lane & 15) * 16;
          const int mine = 2 * warp + half;
          const bool ok = key + mine < keys.k1;
          if (key + 2 * warp < keys.k1) {
            a += (ok ? mine : 0) * 256;
            const uint4 kr = *reinterpret_cast<const uint4*>(a), vr = *reinterpret_cast<const uint4*>(a + DS_UNIT);
            const float k[8] = {ds_lo(kr.x), ds_hi(kr.x), ds_lo(kr.y), ds_hi(kr.y), ds_lo(kr.z), ds_hi(kr.z), ds_lo(kr.w), ds_hi(kr.w)};
            const float v[8] = {ds_lo(vr.x), ds_hi(vr.x), ds_lo(vr.y), ds_hi(vr.y), ds_lo(vr.z), ds_hi(vr.z), ds_lo(vr.w), ds_hi(vr.w)};
            key_step(k, v, ok);
          }
          end_stage();
        }
#pragma unroll
        for (int h = 0; h < GROUP; ++h) {
          const float om = __shfl_xor_sync(0xffffffffu, mx[h], 16), nm = fmaxf(mx[h], om);
          const float f = exp2f(mx[h] - nm);
          float s = sum[h] * f;
          s += __shfl_xor_sync(0xffffffffu, s, 16);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            o[h][e] *= f;
            o[h][e] += __shfl_xor_sync(0xffffffffu, o[h][e], 16);
          }
          float4* out = reinterpret_cast<float4*>(att_o + (warp * GROUP + h) * 128 + d0);
          if (half == 0) {
            out[0] = make_float4(o[h][0], o[h][1], o[h][2], o[h][3]);
            out[1] = make_float4(o[h][4], o[h][5], o[h][6], o[h][7]);
          }
          if (lane == 0) {
            att_ml[(h * 2) * DS_WARPS + warp] = nm;
            att_ml[(h * 2 + 1) * DS_WARPS + warp] = s;
          }
        }
        ds_bar();
        {
          // two channels of a head in PARTS lanes, each with the shares of 16 / PARTS warps
          constexpr int PARTS = 8 / GROUP, EACH = DS_WARPS / PARTS;
          const int part = t % PARTS, i = t / PARTS, h = i / 64, d = (i % 64) * 2;
          float ml[EACH], nm = -1e30f, s = 0.f, a = 0.f, c = 0.f;
#pragma unroll
          for (int x = 0; x < EACH; ++x) {
            ml[x] = att_ml[(h * 2) * DS_WARPS + part * EACH + x];
            nm = fmaxf(nm, ml[x]);
          }
#pragma unroll
          for (int x = PARTS / 2; x > 0; x >>= 1) nm = fmaxf(nm, __shfl_xor_sync(0xffffffffu, nm, x));
#pragma unroll
          for (int x = 0; x < EACH; ++x) {
            const float f = exp2f(ml[x] - nm);
            const float2 ov = *reinterpret_cast<const float2*>(att_o + ((part * EACH + x) * GROUP + h) * 128 + d);
            s += f * att_ml[(h * 2 + 1) * DS_WARPS + part * EACH + x];
            a += f * ov.x;
            c += f * ov.y;
          }
#pragma unroll
          for (int x = PARTS / 2; x > 0; x >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, x);
            a += __shfl_xor_sync(0xffffffffu, a, x);
            c += __shfl_xor_sync(0xffffffffu, c, x);
          }
          if (part == 0) {
            if (keys.splits == 1) {
              const float r = 1.0f / s;
              ds_st(p.attn + b * p.Hq * 64 + (g * GROUP + h) * 64 + d / 2, ds_pack(a * r, c * r), tag);
            } else {
              u64* out = p.part + ((item * p.splits + split) * GROUP + h) * 130;
              ds_st(out + d, __float_as_uint(a), tag);
              ds_st(out + d + 1, __float_as_uint(c), tag);
              if (d == 0) {
                ds_st(out + 128, __float_as_uint(nm), tag);
                ds_st(out + 129, __float_as_uint(s), tag);
              }
            }
          }
        }
        if (keys.splits > 1) {
          // the CTAs of a head share its channels; a lane reads one split
          const int p0 = ds_lo_of(GROUP * 64, split, keys.splits), p1 = ds_lo_of(GROUP * 64, split + 1, keys.splits);
          for (int i = p0 + warp; i < p1; i += DS_WARPS) {
            const int h = i / 64, d = (i % 64) * 2;
            float nm = -1e30f, s = 0.f, a = 0.f, c = 0.f;
            if (lane < keys.splits) {
              const u64* src = p.part + ((item * p.splits + lane) * GROUP + h) * 130;
              ulonglong2 v[2];
              ds_take(v, [&](int i) { return src + (i ? 128 : d); }, [](int) { return true; }, tag, abort_flag, p.err, 543);
              a = ds_f(v[0].x);
              c = ds_f(v[0].y);
              nm = ds_f(v[1].x);
              s = ds_f(v[1].y);
            }
            __syncwarp();
            const float all = warp_max(nm), f = exp2f(nm - all);
            s *= f;
            a *= f;
            c *= f;
#pragma unroll
            for (int x = 16; x > 0; x >>= 1) {
              s += __shfl_xor_sync(0xffffffffu, s, x);
              a += __shfl_xor_sync(0xffffffffu, a, x);
              c += __shfl_xor_sync(0xffffffffu, c, x);
            }
            const float r = 1.0f / s;
            if (lane == 0) out_s[i] = ds_pack(a * r, c * r);
          }
          ds_bar();
          if (p0 + t < p1) ds_st(p.attn + b * p.Hq * 64 + g * GROUP * 64 + p0 + t, out_s[p0 + t], tag);
        }
        continue;
      }
      const bool hidden = phase == DS_QKV || phase == DS_GU || phase == DS_HEAD;
      const int K = ds_columns(p, phase), n0 = tab.n0[phase], nn = tab.nn[phase], norm_flip = flip;
      if (hidden) {
        const u64* src = phase == DS_GU ? p.h1 : phase == DS_HEAD || l > 0 ? p.h2 : nullptr;
        take_hidden(src, phase == DS_QKV ? tag - 1u : tag, phase == DS_QKV ? w.in_norm : phase == DS_GU ? w.post_norm : p.final_norm);
      } else {
        take_pairs(phase == DS_O ? p.attn : p.act, K, tag);
      }
      const int per = phase == DS_GU ? 4 : 8;
      for (int b = 0; b < nn; b += DS_RB * per) {
        const int n = min(DS_RB * per, nn - b);
        switch ((n + per - 1) / per) {
          case 1: multiply(std::integral_constant<int, 1>(), K / DS_SEG); break;
          case 2: multiply(std::integral_constant<int, 2>(), K / DS_SEG); break;
          case 3: multiply(std::integral_constant<int, 3>(), K / DS_SEG); break;
          case 4: multiply(std::integral_constant<int, 4>(), K / DS_SEG); break;
          case 5: multiply(std::integral_constant<int, 5>(), K / DS_SEG); break;
          default: multiply(std::integral_constant<int, 6>(), K / DS_SEG); break;
        }
        ds_bar();
        // results: half a warp per row (gate/up: gate and up of two channels, one after the other)
        if (phase == DS_GU) {
          const int c = 2 * warp, row = (c / 4) * 8 + (c & 3) + ((lane >> 4) << 2);     // blocks of four gate rows and their up rows
          if (c < n) {
#pragma unroll
            for (int m = 0; m < M; ++m) {
              const float rs = inv_rms(norm_flip, m);
              const float v0 = total(m, row) * rs, v1 = total(m, row + 1) * rs;
              const float u0 = __shfl_down_sync(0xffffffffu, v0, 16), u1 = __shfl_down_sync(0xffffffffu, v1, 16);
              if (lane == 0) out_s[m * 64 + warp] = ds_pack(chain_silu(v0) * u0, chain_silu(v1) * u1);
            }
          }
        } else {
          for (int r2 = 2 * warp; r2 < n; r2 += 2 * DS_WARPS) {
            const int r = r2 + (lane >> 4);
            const bool out = (lane & 15) == 0 && r < n;
#pragma unroll
            for (int m = 0; m < M; ++m) {
              const float v = total(m, r);
              if (hidden) {
                const float y = v * inv_rms(norm_flip, m);
                if (out) out_s[m * 64 + r] = __float_as_uint(y);
              } else if (out) {
                float& h = hid[m * p.h_rows + b + r];                   // (always this thread's)
                h += v;
                out_s[m * 64 + r] = __float_as_uint(h);
              }
            }
          }
        }
        // together: stored by the warps that sum them, a step of one sequence took 550 us instead of 443
        ds_bar();
        const int m = t >> 6, r = t & 63, words = phase == DS_GU ? n / 2 : n;
        if (m < M && r < words) {
          const uint32_t v = out_s[m * 64 + r];
          if (phase == DS_HEAD) {
            const u64 key = ds_key(__uint_as_float(v), n0 + b + r);
            p.logits[(size_t)m * p.V + n0 + b + r] = __uint_as_float(v);
            top = key > top ? key : top;
          } else {
            u64* dst = phase == DS_QKV ? p.qkv + m * nqkv + n0 + b : phase == DS_GU ? p.act + m * (p.I / 2) + (n0 + b) / 2 : (phase == DS_O ? p.h1 : p.h2) + m * p.H + n0 + b;
            ds_st(dst + r, v, tag);
          }
        }
        flip ^= 1;
      }
    }
    if (p.next) {
#pragma unroll
      for (int x = 16; x > 0; x >>= 1) {
        const u64 o = __shfl_xor_sync(0xffffffffu, top, x);
        top = o > top ? o : top;
      }
      if (lane == 0 && (t >> 6) < M) atomicMax(p.best + (t >> 6), top);
    }
  }

  __syncthreads();
  if (warp == 0) {
    unsigned n = 0;
    if (lane == 0) {
      __threadfence();                             // (this CTA's shares of `best`, ordered before its ticket)
      n = atomicAdd(p.state + 1, 1u);
      __threadfence();
    }
    n = __shfl_sync(0xffffffffu, n, 0);
    if (n == (unsigned)G - 1) {                    // every CTA has read the step's position, tokens and tag
      if (p.next && lane < M) {
        const u64 key = atomicExch(p.best + lane, 0ull);
        p.next[lane] = key ? (int64_t)(0xffffffffu - (uint32_t)key) : 0;
      }
      if (lane == 0) {
        p.state[1] = 0u;
        p.state[0] += 1u;
        *p.pos += 1;
        *p.ctx += 1;
      }
    }
  }
}

// ----------------------------------------------------------------------------- host side
struct DsShape { int M, H, I, Hq, Hkv, D, V, L; };

struct DsPlan {
  int units, splits, x_stride, h_rows;
  size_t smem;
  size_t words[6];            // qkv, part, attn, h1, act, h2
  size_t state_bytes;
};

// Whether a step of this shape is taken, and how.  G: CTAs that are resident together.
static bool ds_plan(const DsShape& s, int G, DsPlan* out) {
  const int group = s.Hkv > 0 && s.Hq % s.Hkv == 0 ? s.Hq / s.Hkv : 0;
  const int nqkv = (s.Hq + 2 * s.Hkv) * 128, kq = s.Hq * 128;
  if (s.D != 128 || s.M < 1 || s.M > DS_MAX_M || s.L < 1 || s.L > DS_MAX_LAYERS || G < 1 || G > 256) return false;
  if ((group != 1 && group != 2 && group != 4) || s.M * s.Hkv > G) return false;
  // every CTA has rows in every phase
  if (s.H % DS_SEG || s.I % DS_SEG || kq % DS_SEG || s.H < G || s.I / 2 < G || nqkv < G || s.V < G || s.V > DS_MAX_N || nqkv > DS_MAX_N) return false;
  DsPlan p = {};
  p.x_stride = std::max({s.H, kq, s.I}) * 2 + 64;      // (like a unit's rows)
  p.h_rows = (s.H + G - 1) / G;
  p.splits = std::min(DS_MAX_SPLITS, G / (s.M * s.Hkv));
  const size_t rest = (size_t)s.M * p.x_stride + (size_t)2 * DS_WARPS * (s.M * DS_ROWS + 2) * 4 + 2 * s.M * DS_WARPS * 4 +
                      ((size_t)s.M * p.h_rows * 4 + 15) / 16 * 16 + (size_t)DS_WARPS * group * 130 * 4 + (size_t)(group + 2) * 512 + (size_t)std::max(s.M, group) * 256 + 512 +
                      DS_BARS * (16 + DS_COPY_WARPS) + 16 + offsetof(DsTable, layer) + s.L * sizeof(DsLayer);
  p.units = rest < 227 * 1024 ? std::min<int>(DS_MAX_UNITS, (int)((227 * 1024 - rest) / DS_UNIT)) : 0;
  if (p.units < 2 * DS_STAGE - 1) return false;      // a stage does not wrap: the units that it skips and its own are all it can ask for
  p.smem = p.units * DS_UNIT + rest;
  const size_t m = s.M;
  const size_t words[6] = {m * nqkv, (size_t)G * group * 130, m * kq / 2, m * s.H, m * s.I / 2, m * s.H};
  p.state_bytes = 256;
  for (int i = 0; i < 6; ++i) {
    p.words[i] = (words[i] + 31) / 32 * 32;
    p.state_bytes += p.words[i] * sizeof(u64);
  }
  *out = p;
  return true;
}

// The longest context at which the step kernel is faster than the kernels per layer.  Those read the cache at HBM's rate; here a CTA
// walks its share of a head's keys at 15, 17.6 and 33 to 59 ns a key for 1, 2 and 4 query heads (with 4, registers run out
// beyond three sequences), which is slower wherever the heads do not fill the SMs.  Against that stands what a layer saves
// in launches and hand-overs: 31 us for one sequence, less for more, and for three less by what they cost beside large weights
// (the ring shrinks by their activations).  Measured, us a layer here / kernels per layer: 1024 wide, 16 query heads on 8: 1 sequence
// at 40000 keys 56 / 78, 2 at 16000 49 / 65, 3 at 16000 67 / 72, 4 at 8000 57 / 61, 16000 92 / 81, 6 at 2000 42 / 49, 8000 79 / 70; 32
// on 8: 1 at 16000 51 / 64, 40000 96 / 81, 2 at 4000 40 / 53, 16000 92 / 67, 5 at 300 43 / 45, 1000 55 / 47; 512 wide, 8 on 2: 4 at 8000 41 / 49, 16000 62 / 55; 2560 wide: 3 at 1000
// 74 / 82, 4000 92 / 88; 4096 wide: 2 at 4000 104 / 117, 3 at 300 115 / 109.
static int ds_max_context(const DsShape& s, int G) {
  DsPlan plan;
  if (!ds_plan(s, G, &plan)) return 0;
  const int group = s.Hq / s.Hkv;
  const double weights = 2e-6 * s.H * (2.0 * s.Hq * 128 + 2.0 * s.Hkv * 128 + 3.0 * s.I);      // MB of a layer
  const double saved[2][DS_MAX_M] = {{31, 23, 23 - 0.06 * weights, 18, 15, 7},
                                      {31, 23, 23 - 0.06 * weights, 24 - 32.0 / plan.splits, 15 - 22.0 / plan.splits, 3.7}};      // us
  const double walk[DS_MAX_M] = {33.5, 38.5, 40, 47.5, 59, 56};      // ns a key
  const double gain = 1e3 * saved[group == 4][s.M - 1];
  const double loss = (group == 1 ? 15.0 : group == 2 ? 17.6 : walk[s.M - 1]) / plan.splits - s.M * s.Hkv * 512 / 6900.0;
  if (gain <= 0) return 0;
  return loss * 1e9 <= gain ? INT_MAX : (int)std::min<double>(gain / loss, INT_MAX);
}

typedef void (*DsKernel)(const DsParams);
template <int GROUP>
static DsKernel ds_kernel(int M) {
  static const DsKernel kernels[DS_MAX_M] = {decode_step_kernel<GROUP, 1>, decode_step_kernel<GROUP, 2>, decode_step_kernel<GROUP, 3>,
                                             decode_step_kernel<GROUP, 4>, decode_step_kernel<GROUP, 5>, decode_step_kernel<GROUP, 6>};
  return kernels[M - 1];
}

static bool ds_dense(const kd_tensor* t, int dtype, int64_t n) { return t && t->dtype == dtype && is_contiguous(t) && numel(t) == n; }

static int ds_ptr(const kd_tensor* t, const char* what, void** out) {
  KD_TRY(tensor_ptr(t, out));
  KD_REQUIRE((reinterpret_cast<uintptr_t>(*out) & 15) == 0, "decode step: %s must be 16-byte aligned", what);
  return KD_OK;
}

}  // namespace kd

using namespace kd;

KD_API int kd_decode_step_state_bytes(int sequences, int hidden, int inter, int q_heads, int kv_heads, int head_dim, int vocab, int layers,
                                      int grid, uint64_t* bytes_out) {
  KD_REQUIRE(bytes_out, "null argument");
  if (grid <= 0) {
    KD_TRY(require_init());
    grid = ctx().sm_count;
  }
  DsPlan plan;
  *bytes_out = ds_plan(DsShape{sequences, hidden, inter, q_heads, kv_heads, head_dim, vocab, layers}, grid, &plan) ? plan.state_bytes : 0;
  return KD_OK;
}

KD_API int kd_decode_step_max_context(int sequences, int hidden, int inter, int q_heads, int kv_heads, int head_dim, int vocab, int layers,
                                      int grid, int* keys_out) {
  KD_REQUIRE(keys_out, "null argument");
  if (grid <= 0) {
    KD_TRY(require_init());
    grid = ctx().sm_count;
  }
  *keys_out = ds_max_context(DsShape{sequences, hidden, inter, q_heads, kv_heads, head_dim, vocab, layers}, grid);
  return KD_OK;
}

KD_API int kd_decode_step(const kd_tensor* const* layer_tensors, int n_layers, const kd_tensor* embed, const kd_tensor* final_norm,
                          const kd_tensor* ids, const kd_tensor* inv_freq, const kd_tensor* pos, const kd_tensor* ctx_len, float eps,
                          float scale, const kd_tensor* block_table, const kd_tensor* state, const kd_tensor* logits, const kd_tensor* next_ids) {
  KD_TRY(require_init());
  KD_REQUIRE(layer_tensors && embed && final_norm && ids && inv_freq && pos && ctx_len && state && logits, "null tensor");
  KD_REQUIRE(n_layers >= 1 && n_layers <= DS_MAX_LAYERS, "decode step: %d layers; this path takes 1..%d", n_layers, DS_MAX_LAYERS);
  for (int i = 0; i < 10 * n_layers; ++i) KD_REQUIRE(layer_tensors[i], "decode step: null tensor in layer %d", i / 10);
  KD_REQUIRE(embed->ndim == 2 && ids->ndim == 1 && layer_tensors[1]->ndim == 2 && layer_tensors[4]->ndim == 2 && layer_tensors[7]->ndim == 2,
             "decode step: embedding and matrices must be 2-D, ids 1-D");
  Context& c = ctx();
  const kd_tensor* kc0 = layer_tensors[8];
  KD_REQUIRE(kc0->ndim == 4 && kc0->shape[0] >= 1, "decode step: caches must be 4-D, with rows");
  DsShape s;
  s.M = (int)ids->shape[0];
  s.V = (int)embed->shape[0];
  s.H = (int)embed->shape[1];
  s.I = (int)layer_tensors[7]->shape[1];
  s.Hq = (int)(layer_tensors[4]->shape[1] / 128);
  s.Hkv = (int)kc0->shape[1];
  s.D = (int)kc0->shape[3];
  s.L = n_layers;
  DsPlan plan;
  KD_REQUIRE(ds_plan(s, c.sm_count, &plan), "decode step: this path does not take %d sequences of these widths", s.M);
  const int nqkv = (s.Hq + 2 * s.Hkv) * 128;
  KD_REQUIRE(scale > 0.f, "decode step: scale must be positive");
  KD_REQUIRE(ds_dense(embed, KD_BF16, (int64_t)s.V * s.H) && ds_dense(final_norm, KD_BF16, s.H), "decode step: embedding [V,H] and final norm [H] must be contiguous bf16");
  KD_REQUIRE(ds_dense(ids, KD_I64, s.M) && ds_dense(inv_freq, KD_F32, 64) && pos->dtype == KD_I32 && numel(pos) == 1 && ctx_len->dtype == KD_I32 && numel(ctx_len) == 1,
             "decode step: ids int64 [M], inv_freq fp32 [64], position and context length int32 scalars");
  KD_REQUIRE(ds_dense(logits, KD_F32, (int64_t)s.M * s.V), "decode step: logits must be contiguous fp32 [M,V]");
  KD_REQUIRE(!next_ids || ds_dense(next_ids, KD_I64, s.M), "decode step: next_ids must be int64 [M]");
  KD_REQUIRE(is_contiguous(state) && (uint64_t)numel(state) * dtype_size(state->dtype) >= plan.state_bytes, "decode step: state must hold %llu bytes",
             (unsigned long long)plan.state_bytes);
  if (block_table)
    KD_REQUIRE(block_table->dtype == KD_I32 && block_table->ndim == 2 && is_contiguous(block_table) && block_table->shape[0] >= s.M && kc0->shape[2] == 128,
               "decode step: block_table must be a contiguous int32 [B>=M, max_pages] tensor and the pools must have pages of 128 rows");
  else
    KD_REQUIRE(kc0->shape[0] >= s.M, "decode step: caches hold fewer sequences than ids");
  static thread_local DsParams p;       // (larger than a stack frame should be)
  p = DsParams{};
  for (int l = 0; l < n_layers; ++l) {
    const kd_tensor* const* t = layer_tensors + 10 * l;
    const int64_t n[8] = {s.H, (int64_t)nqkv * s.H, 128, 128, (int64_t)s.H * s.Hq * 128, s.H, (int64_t)2 * s.I * s.H, (int64_t)s.H * s.I};
    void* q[10];
    for (int i = 0; i < 8; ++i) {
      KD_REQUIRE(ds_dense(t[i], KD_BF16, n[i]), "decode step: weight %d of layer %d must be contiguous bf16 with %lld elements", i, l, (long long)n[i]);
      KD_TRY(ds_ptr(t[i], "a weight", &q[i]));
    }
    KD_REQUIRE(t[1]->ndim == 2 && t[1]->shape[1] == s.H && t[4]->ndim == 2 && t[4]->shape[0] == s.H && t[6]->ndim == 2 && t[6]->shape[1] == s.H && t[7]->ndim == 2 &&
                   t[7]->shape[0] == s.H,
               "decode step: matrices of layer %d must be [rows, columns]", l);
    for (int i = 8; i < 10; ++i) {
      KD_REQUIRE(t[i]->dtype == KD_BF16 && t[i]->ndim == 4 && t[i]->strides[3] == 1, "decode step: caches must be bf16 with unit head_dim stride");
      for (int d = 0; d < 4; ++d)
        KD_REQUIRE(t[i]->shape[d] == kc0->shape[d] && t[i]->strides[d] == kc0->strides[d] && (d == 3 || t[i]->strides[d] % 8 == 0),
                   "decode step: all caches need one shape and strides that are multiples of 8");
      KD_TRY(ds_ptr(t[i], "a cache", &q[i]));
    }
    const auto w = [&](int i) { return static_cast<const __nv_bfloat16*>(q[i]); };
    p.layer[l] = DsLayer{w(0), w(1), w(2), w(3), w(4), w(5), w(6), w(7), static_cast<__nv_bfloat16*>(q[8]), static_cast<__nv_bfloat16*>(q[9])};
  }
  void *pe, *pf, *pi, *pv, *pp, *pc, *ps, *pl, *pt = nullptr, *pn = nullptr;
  KD_TRY(ds_ptr(embed, "the embedding", &pe));
  KD_TRY(ds_ptr(final_norm, "the final norm", &pf));
  KD_TRY(tensor_ptr(ids, &pi));
  KD_TRY(tensor_ptr(inv_freq, &pv));
  KD_TRY(tensor_ptr(pos, &pp));
  KD_TRY(tensor_ptr(ctx_len, &pc));
  KD_TRY(ds_ptr(state, "the state", &ps));
  KD_TRY(tensor_ptr(logits, &pl));
  if (block_table) KD_TRY(tensor_ptr(block_table, &pt));
  if (next_ids) KD_TRY(tensor_ptr(next_ids, &pn));
  p.embed = p.head = static_cast<const __nv_bfloat16*>(pe);
  p.final_norm = static_cast<const __nv_bfloat16*>(pf);
  p.ids = static_cast<const int64_t*>(pi);
  p.inv_freq = static_cast<const float*>(pv);
  p.pos = static_cast<int*>(pp);
  p.ctx = static_cast<int*>(pc);
  p.logits = static_cast<float*>(pl);
  p.table = static_cast<const int*>(pt);
  p.max_pages = block_table ? (int)block_table->shape[1] : 0;
  p.last_page = (unsigned)(kc0->shape[0] - 1);
  p.max_s = block_table ? p.max_pages * 128 : (int)kc0->shape[2];
  p.err = c.error_flag;
  p.state = static_cast<unsigned*>(ps);
  p.best = reinterpret_cast<u64*>(static_cast<char*>(ps) + 64);
  p.next = static_cast<int64_t*>(pn);
  u64* words = reinterpret_cast<u64*>(static_cast<char*>(ps) + 256);
  u64** to[6] = {&p.qkv, &p.part, &p.attn, &p.h1, &p.act, &p.h2};
  for (int i = 0; i < 6; ++i) {
    *to[i] = words;
    words += plan.words[i];
  }
  p.kc_b = kc0->strides[0];
  p.kc_h = kc0->strides[1];
  p.kc_s = kc0->strides[2];
  p.eps = eps;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.M = s.M; p.H = s.H; p.I = s.I; p.Hq = s.Hq; p.Hkv = s.Hkv; p.L = s.L; p.V = s.V;
  p.splits = plan.splits;
  p.units = plan.units;
  p.x_stride = plan.x_stride;
  p.h_rows = plan.h_rows;
  const int group = s.Hq / s.Hkv;
  const DsKernel kernel = group == 1 ? ds_kernel<1>(s.M) : group == 2 ? ds_kernel<2>(s.M) : ds_kernel<4>(s.M);
  KD_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(c.sm_count);
  cfg.blockDim = dim3(DS_THREADS);
  cfg.dynamicSmemBytes = plan.smem;
  cfg.stream = c.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  KD_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, p));
  return after_launch("decode_step_kernel");
}
