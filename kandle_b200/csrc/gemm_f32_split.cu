// fp32 GEMM on the bf16 tensor cores: out[M,N] = alpha A[M,K] B[N,K]^T (+ beta C), fp32 in, fp32 out.
//
// tcgen05 has no fp32 input format, but an fp32 number is the exact sum of three bf16 numbers (8 + 8 + 8 bits of
// significand): x = h + m + l, each the rounded rest of the one before.  A product of two such sums has nine terms; the
// six largest (hh, hm, mh, hl, lh, mm) hold everything down to 2^-26 of the product, the other three are dropped.  All
// products of bf16 pairs are exact in fp32, so what remains is the rounding of the sums:
//   * the tensor core's own accumulation does not round to nearest, so the hh terms stay in tensor memory for one k-block
//     of 64 only; the accumulating warps then add that block to fp32 registers with ordinary rounded additions;
//   * the five small terms are 2^-8 of hh, their sum stays in tensor memory for the whole of K.
// Measured against float64 (N(0,1) by N(0,0.02^2) operands, relative 2-norm): 1.0e-7 at K = 1024, 1.7e-7 at K = 4096; a
// chain of K fused multiply-adds (matmul_f32_kernel) has 5.7e-7 at K = 1024 and 9.9e-7 at K = 3072.
//
// Range: a split needs room below it.  Numbers with 2^-100 <= |x| < 2^127, and zero, split exactly.  The converting warps
// keep the least of a tile; a tile with a smaller one, and 32 rows with a sum that is not finite (so does every infinity,
// NaN or number from 2^127 on end), are computed again by their accumulating warps with plain fused multiply-adds, in the
// order of matmul_f32_kernel.  One such number costs its tiles, a denormal weight every row of tiles: 512 x 3072 x 1024 takes
// 38 us, 356 with every tile computed again (matmul_f32_kernel 367); 2048 x 4096 x 4096 463 and 5512 us (7510).
// Where an operand has numbers below 2^-50, the small terms of a product may be subnormal and lose bits to the tensor core;
// that shows in sums below 2^-100 (8.9e-16, 7.9e-31), and 32 rows with such a sum are computed again likewise.  Operands of
// 1e-20 at K = 1024: 4.0e-6 relative, 1.7e-5 by the split alone; of 1e-19 and 3e-20: 3.0e-7, 6.0e-7.
//
// Structure (one persistent CTA per SM, 640 threads):
//   warps 0-7    global fp32 -> registers (next k-block in flight) -> three bf16 planes per operand in shared memory,
//                128-byte swizzle.  No TMA: the numbers pass through registers anyway.
//   warps 8-15   accumulate: one row and BN/2 columns per thread; hh blocks through two TMEM buffers.
//   warp 16      one thread issues 24 tcgen05.mma per k-block (M=128, N=BN, K=16).
//                (warps 17-19 idle: registers move between groups of four warps)
// Bound: the split, about 35 instructions per 4 numbers of either operand and 1.8 us per 128 x 128 x 64 block, against
// 0.8 us of MMA.  2048 x 4096 x 4096 takes 463 us = 148 TFLOP/s; matmul_f32_kernel reaches about 9.  Where the tiles
// are too few for the SMs, K is shared: a cluster of 2 or 4 CTAs, each a range of k-blocks, adds its sums up through shared
// memory in a fixed order.
#include "common.cuh"
#include "kernels.cuh"
#include "sm100.cuh"

namespace kd {

using namespace sm100;

struct SplitParams {
  const float* A;
  const float* B;
  const void* C;
  float* O;
  int M, N, K;
  int lda, ldb;
  int64_t a_b0, a_b1, b_b0, b_b1, c_b0, c_b1, c_m, c_n, o_b0, o_b1, o_m;
  int b1;
  int dt_c, has_c;
  int vec_out;           // output rows are 16-byte aligned
  float alpha, beta;
  int m_tiles, n_tiles, m_inner;
  int splits;            // CTAs of a cluster that share a tile, each with a range of k-blocks (then a CTA has one tile)
  int total;
  int* err;
};

constexpr int FS_CONV = 256, FS_ACC = 256, FS_THREADS = FS_CONV + FS_ACC + 128;
// Registers a thread: launched with 96 (640 threads: 61440); 256 x 104 + 256 x 104 + 128 x 56 after the exchange are 60416.
constexpr int FS_REGS_CONV = 104, FS_REGS_ACC = 104, FS_REGS_MMA = 56;
constexpr int FS_BM = 128, FS_BK = 64;
constexpr int FS_WARP_ACC = FS_CONV / 32, FS_WARP_MMA = (FS_CONV + FS_ACC) / 32;
constexpr int FS_PLANE_A = FS_BM * FS_BK * 2;
// Microseconds of a k-block of a 128 x 64 and a 128 x 128 tile, and of the exchange of a split tile's sums (measured at M = 512:
// N = K = 1024 takes 32.9, 39.1 us with 64- and 128-wide tiles, 28.8, 20.7 us with 128-wide ones split in 2 and 4).
constexpr double FS_US_64 = 1.6, FS_US_128 = 1.9, FS_US_EXCHANGE = 6.0;
constexpr int FS_ROWS = FS_CONV / 16;      // rows of 64 numbers per pass of the converting warps

// Two numbers to their bf16 parts, packed like the numbers (first in the low half).
__device__ __forceinline__ uint32_t cvt_pair(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ float low_half(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float high_half(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// h, m, l of a pair
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = cvt_pair(a, b);
  uint64_t rest;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%1, %2};\n\tmov.b64 y, {%3, %4};\n\tadd.rn.f32x2 %0, x, y;\n\t}"
      : "=l"(rest) : "f"(a), "f"(b), "f"(-low_half(h)), "f"(-high_half(h)));
  float ra, rb;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(ra), "=f"(rb) : "l"(rest));
  m = cvt_pair(ra, rb);
  asm("{\n\t.reg .b64 y;\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 %0, %1, y;\n\t}" : "=l"(rest) : "l"(rest), "f"(-low_half(m)), "f"(-high_half(m)));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(ra), "=f"(rb) : "l"(rest));
  l = cvt_pair(ra, rb);
}
// Smallest |x| that is not zero, as twice the bits less one (a zero becomes the largest value).
__device__ __forceinline__ uint32_t least(uint32_t now, float a, float b) {
  return min(now, min(2u * __float_as_uint(a) - 1u, 2u * __float_as_uint(b) - 1u));
}
constexpr uint32_t FS_LEAST = 2u * (27u << 23) - 1u;      // 2^-100
// From 2^-50 on in both operands, the kept terms of a product that matter are normal numbers.
constexpr uint32_t FS_LOW = 2u * (77u << 23) - 1u;        // 2^-50
constexpr float FS_LOW_SUM = 0x1p-100f;

template <int REGS>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS)); }
template <int REGS>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS)); }
// Barrier of a cluster.  It wants its warps converged: one lane alone issues the products, rows past the output store nothing.
__device__ __forceinline__ void cluster_arrive_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

template <int BN>
__global__ void __launch_bounds__(FS_THREADS, 1) gemm_f32_split_kernel(SplitParams p) {
  constexpr int PLANE_B = BN * FS_BK * 2;
  constexpr int STAGE = 3 * (FS_PLANE_A + PLANE_B);
  constexpr int STAGES = 2;
  constexpr int A_PASSES = FS_BM / FS_ROWS, B_PASSES = BN / FS_ROWS;
  constexpr uint32_t TMEM_COLS = 4 * BN;                     // hh 0, hh 1, small terms of even and odd tiles
  constexpr uint32_t IDESC = make_idesc_bf16(FS_BM, BN, 0, 0);
  constexpr int COLS = BN / 2;                               // columns of an accumulating thread

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE);
  uint64_t* empty = full + STAGES;
  uint64_t* hh_full = empty + STAGES;
  uint64_t* hh_empty = hh_full + 2;
  uint64_t* rest_full = hh_empty + 2;
  uint64_t* rest_empty = rest_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rest_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // a tile with numbers below the range of the split, and one with numbers below FS_LOW: its ordinal + 1.  The converting
  // warps are at most four tiles ahead of the accumulating ones (two stages, two buffers of small terms).
  volatile int* bad_tile = abort_flag + 1;
  volatile int* low_tile = bad_tile + 8;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], FS_CONV / 32); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&hh_full[b], 1); mbar_init(&hh_empty[b], FS_ACC / 32);
      mbar_init(&rest_full[b], 1); mbar_init(&rest_empty[b], FS_ACC / 32);
    }
    *abort_flag = 0;
    for (int i = 0; i < 16; ++i) bad_tile[i] = 0;
    fence_mbar_init();
  }
  if (warp == FS_WARP_MMA) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  const int all_kb = (p.K + FS_BK - 1) / FS_BK;
  const int rank = (int)(blockIdx.x % p.splits);
  const int kb0 = all_kb * rank / p.splits, num_kb = all_kb * (rank + 1) / p.splits - kb0;
  const int first = blockIdx.x / p.splits, step = gridDim.x / p.splits;
  const int per_batch = p.m_tiles * p.n_tiles;
  auto locate = [&](int tile, int& z, int& m0, int& n0) {
    z = tile / per_batch;
    const int t = tile - z * per_batch;
    const int m = p.m_inner ? t % p.m_tiles : t / p.n_tiles, n = p.m_inner ? t / p.m_tiles : t % p.n_tiles;
    m0 = m * FS_BM;
    n0 = n * BN;
  };
  auto batch = [&](int z, int64_t s0, int64_t s1) { return (int64_t)(z / p.b1) * s0 + (int64_t)(z % p.b1) * s1; };

  auto store = [&](int z, int row, int col, const float (&s)[4]) {
    float* o = p.O + batch(z, p.o_b0, p.o_b1) + (int64_t)row * p.o_m + col;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = p.alpha * s[i];
      if (p.has_c && col + i < p.N)
        v[i] += p.beta * load_float(p.C, p.dt_c, batch(z, p.c_b0, p.c_b1) + (int64_t)row * p.c_m + (int64_t)(col + i) * p.c_n);
    }
    if (p.vec_out && col + 4 <= p.N) {
      *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (col + i < p.N) o[i] = v[i];
    }
  };
  auto issue = [&]() {
    int stage = 0, buffer = 0, ordinal = 0;
    uint32_t phase = 0, hh_phase = 0;
    const uint64_t desc_hi = make_smem_desc_sw128(0, 16, 1024);     // (addresses below 256 KB: the low word has room for them)
    bool ok = true;
    for (int tile = first; ok && tile < p.total; tile += step, ++ordinal) {
      const int parity = ordinal & 1;
      if (!mbar_wait(&rest_empty[parity], ((uint32_t)(ordinal >> 1) & 1) ^ 1, abort_flag, p.err, 224)) break;
      const uint32_t rest = tmem_base + (uint32_t)((2 + parity) * BN);
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(&hh_empty[buffer], hh_phase ^ 1, abort_flag, p.err, 225) || !mbar_wait(&full[stage], phase, abort_flag, p.err, 226)) { ok = false; break; }
        tc_fence_after();
        // Descriptors advance by whole 16-byte units in their low words.  The low words pass through an empty asm: as
        // loop invariants the 48 descriptors would take more registers than the warp has.
        uint32_t a0 = smem_u32(smem + stage * STAGE) >> 4, b0 = a0 + (3 * FS_PLANE_A >> 4);
        asm volatile("" : "+r"(a0), "+r"(b0));
        auto product = [&](uint32_t d, int pa, int pb, bool fresh) {
#pragma unroll
          for (int k = 0; k < FS_BK / 16; ++k)
            umma_ss(d, desc_hi | (a0 + ((pa * FS_PLANE_A + k * 32) >> 4)), desc_hi | (b0 + ((pb * PLANE_B + k * 32) >> 4)), IDESC, fresh && k == 0 ? 0u : 1u);
        };
        product(tmem_base + (uint32_t)(buffer * BN), 0, 0, true);
        umma_commit(&hh_full[buffer]);
        product(rest, 1, 1, kb == 0);
        product(rest, 0, 2, false);
        product(rest, 2, 0, false);
        product(rest, 0, 1, false);
        product(rest, 1, 0, false);
        umma_commit(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        buffer ^= 1;
        if (buffer == 0) hh_phase ^= 1;
      }
      if (ok) umma_commit(&rest_full[parity]);
    }
  };

  if (warp < FS_WARP_ACC) {
    regs_inc<FS_REGS_CONV>();
    const int r = threadIdx.x >> 4, k4 = (threadIdx.x & 15) * 4;
    // this thread's place in a plane: row r of every pass of 16 rows, 8 bytes of 16-byte piece k4 / 8
    const uint32_t place = (uint32_t)(r * 128 + ((((threadIdx.x & 15) >> 1) ^ (r & 7)) << 4) + (threadIdx.x & 1) * 8);
    float4 buf[A_PASSES + B_PASSES];
    const float *pa = nullptr, *pb = nullptr;
    const int k_last = p.K - kb0 * FS_BK - 4 - k4;      // the last piece of a row, from here
    int rows_a = 0, rows_b = 0;      // last row of this tile, from row r on
    auto seek = [&](int tile) {
      int z, m0, n0;
      locate(tile, z, m0, n0);
      rows_a = p.M - 1 - m0 - r;
      rows_b = p.N - 1 - n0 - r;
      pa = p.A + batch(z, p.a_b0, p.a_b1) + (int64_t)(m0 + r) * p.lda + kb0 * FS_BK + k4;
      pb = p.B + batch(z, p.b_b0, p.b_b1) + (int64_t)(n0 + r) * p.ldb + kb0 * FS_BK + k4;
    };
    // Rows past the operand repeat its last one (their products are not stored), pieces past K its last piece (zeroed
    // before the split): no load is predicated.
    auto fetch = [&](int i, int kb) {
      const int at = min(kb * FS_BK, k_last);
      const float* src = i < A_PASSES ? pa + min(i * FS_ROWS, rows_a) * p.lda : pb + min((i - A_PASSES) * FS_ROWS, rows_b) * p.ldb;
      buf[i] = __ldg(reinterpret_cast<const float4*>(src + at));
    };
    int tile = first;
    if (tile < p.total) {
      seek(tile);
#pragma unroll
      for (int i = 0; i < A_PASSES + B_PASSES; ++i) fetch(i, 0);
    }
    int stage = 0, ordinal = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (; ok && tile < p.total; tile += step, ++ordinal) {
      uint32_t small = 0xffffffffu;
      for (int kb = 0; kb < num_kb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.err, 221));
        if (!ok) break;
        if (kb * FS_BK > k_last) {
#pragma unroll
          for (int i = 0; i < A_PASSES + B_PASSES; ++i) buf[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        int next = kb + 1;
        if (next == num_kb) {
          next = 0;
          seek(tile + step < p.total ? tile + step : tile);      // (after the last tile: loads that nothing uses)
        }
        uint8_t* st = smem + stage * STAGE + place;
#pragma unroll
        for (int i = 0; i < A_PASSES + B_PASSES; ++i) {
          const float4 v = buf[i];
          fetch(i, next);
          small = least(least(small, v.x, v.y), v.z, v.w);
          uint2 h, m, l;
          split_pair(v.x, v.y, h.x, m.x, l.x);
          split_pair(v.z, v.w, h.y, m.y, l.y);
          constexpr int PIECE = FS_ROWS * 128;
          uint8_t* d = st + (i < A_PASSES ? i * PIECE : 3 * FS_PLANE_A + (i - A_PASSES) * PIECE);
          const int plane = i < A_PASSES ? FS_PLANE_A : PLANE_B;
          *reinterpret_cast<uint2*>(d) = h;
          *reinterpret_cast<uint2*>(d + plane) = m;
          *reinterpret_cast<uint2*>(d + 2 * plane) = l;
        }
        if (kb + 1 == num_kb && small < FS_LOW) {
          low_tile[ordinal & 7] = ordinal + 1;
          if (small < FS_LEAST) bad_tile[ordinal & 7] = ordinal + 1;
        }
        fence_async_proxy();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[stage]);      // (an arrival of every thread takes longer than the products)
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp < FS_WARP_MMA) {
    regs_inc<FS_REGS_ACC>();
    const int q = warp & 3, half = (warp - FS_WARP_ACC) >> 2;
    const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * COLS);
    int buffer = 0, ordinal = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = first; ok && tile < p.total; tile += step, ++ordinal) {
      float acc[COLS];
#pragma unroll
      for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
      for (int kb = 0; kb < num_kb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&hh_full[buffer], phase, abort_flag, p.err, 222));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < COLS; c += 16) {
          uint32_t x[16];
          tmem_ld_32x16(t_row + buffer * BN + c, x);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(x[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&hh_empty[buffer]);
        buffer ^= 1;
        if (buffer == 0) phase ^= 1;
      }
      if (!ok) break;
      const int parity = ordinal & 1;
      ok = __all_sync(0xffffffffu, mbar_wait(&rest_full[parity], (uint32_t)(ordinal >> 1) & 1, abort_flag, p.err, 223));
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < COLS; c += 16) {
        uint32_t x[16];
        tmem_ld_32x16(t_row + (2 + parity) * BN + c, x);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c + i] += __uint_as_float(x[i]);
      }
      // infinity, NaN and numbers from 2^127 on leave no finite sum behind (their parts hold infinity less infinity)
      const float least_sum = low_tile[ordinal & 7] == ordinal + 1 ? FS_LOW_SUM : 0.f;
      bool again = bad_tile[ordinal & 7] == ordinal + 1;
#pragma unroll
      for (int i = 0; i < COLS; ++i) again |= !(fabsf(acc[i]) < INFINITY) | (fabsf(acc[i]) < least_sum);
      again = __any_sync(0xffffffffu, again);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&rest_empty[parity]);
      int z, m0, n0;
      locate(tile, z, m0, n0);
      // Where sums go: the output, or (split tiles) this CTA's share in the stages that no copy or product uses any more;
      // 16-byte pieces of a row trade places so that eight rows meet eight bank groups.
      auto put = [&](int r, int c, const float (&v)[4]) {
        if (p.splits > 1) *reinterpret_cast<float4*>(smem + r * (BN * 4) + (((c >> 2) ^ (r & 7)) << 4)) = make_float4(v[0], v[1], v[2], v[3]);
        else if (m0 + r < p.M) store(z, m0 + r, n0 + c, v);
      };
      if (again) {
        // Plain fused multiply-adds for the warp's 32 rows, 8 rows x 4 columns a lane, straight from global memory: the lines of
        // the tile's operands, 24 KB, stay in the L1 cache while their 32 k are used.  Rows past an operand repeat its last one.
        // A load takes the cache a cycle per line and eight lanes: eight neighbours share two rows of A and four of B.
        int l = lane;
        asm volatile("" : "+r"(l));      // (what follows from l is not to be kept in registers through the main loop)
        const int r0 = q * 32 + ((l & 1) | (l >> 2 & 2)), c0 = half * COLS + ((l >> 1 & 3) | (l >> 2 & 4)) * 4, k_end = min(p.K, (kb0 + num_kb) * FS_BK);
        const float* A = p.A + batch(z, p.a_b0, p.a_b1) + (int64_t)m0 * p.lda;
        const float* B = p.B + batch(z, p.b_b0, p.b_b1) + (int64_t)n0 * p.ldb;
#pragma unroll 1
        for (int c = c0; c < half * COLS + COLS; c += 32) {
          float v[8][4];
          int oa[8], ob[4];
#pragma unroll
          for (int i = 0; i < 8; ++i) oa[i] = min(r0 + 4 * i, p.M - 1 - m0) * p.lda;
#pragma unroll
          for (int j = 0; j < 4; ++j) ob[j] = min(c + j, p.N - 1 - n0) * p.ldb;
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = 0.f;
#pragma unroll 1
          for (int k = kb0 * FS_BK; k < k_end; k += 4) {
            float4 b[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = __ldg(reinterpret_cast<const float4*>(B + k + ob[j]));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 a = __ldg(reinterpret_cast<const float4*>(A + k + oa[i]));
#pragma unroll
              for (int j = 0; j < 4; ++j) v[i][j] = fmaf(a.w, b[j].w, fmaf(a.z, b[j].z, fmaf(a.y, b[j].y, fmaf(a.x, b[j].x, v[i][j]))));
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) put(r0 + 4 * i, c, v[i]);
        }
      } else {
#pragma unroll
        for (int c = 0; c < COLS; c += 4) {
          const float v[4] = {acc[c], acc[c + 1], acc[c + 2], acc[c + 3]};
          put(q * 32 + lane, half * COLS + c, v);
        }
      }
    }
  } else {
    regs_dec<FS_REGS_MMA>();
    if (warp == FS_WARP_MMA && lane == 0) issue();
  }

  if (p.splits > 1) {
    // every CTA of the cluster adds up its share of the columns, in the order of the k ranges
    cluster_arrive_wait();
    if (warp >= FS_WARP_ACC && warp < FS_WARP_MMA && first < p.total) {
      int z, m0, n0;
      locate(first, z, m0, n0);
      const int pieces = BN / 4 / p.splits;       // 16-byte pieces of a row that this CTA finishes
      for (int i = threadIdx.x - FS_CONV; i < FS_BM * pieces; i += FS_ACC) {
        const int r = i / pieces, c = rank * pieces + i % pieces;
        if (m0 + r >= p.M) continue;
        const uint32_t at = smem_u32(smem + r * (BN * 4) + ((c ^ (r & 7)) << 4));
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < p.splits; ++s) {
          const float4 x = ld_cluster_f4(at, (uint32_t)s);
          v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
        }
        store(z, m0 + r, n0 + c * 4, v);
      }
    }
    cluster_arrive_wait();     // the others may still be reading this CTA's shared memory
  }
  tc_fence_before();
  __syncthreads();
  if (warp == FS_WARP_MMA) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int BN>
static int launch_split(SplitParams& p, int64_t batches) {
  constexpr int SMEM = 2 * 3 * (FS_PLANE_A + BN * FS_BK * 2) + 1024 + 256;
  static bool configured[64] = {false};
  if (!configured[ctx().device & 63]) {
    KD_CUDA_CHECK(cudaFuncSetAttribute(gemm_f32_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    configured[ctx().device & 63] = true;
  }
  p.m_tiles = (p.M + FS_BM - 1) / FS_BM;
  p.n_tiles = (p.N + BN - 1) / BN;
  p.total = (int)(batches * p.m_tiles * p.n_tiles);
  if (p.splits > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.total * p.splits));
    cfg.blockDim = dim3(FS_THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = ctx().stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    KD_CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel<BN>, p));
    return after_launch("gemm_f32_split_kernel");
  }
  const int grid = p.total < ctx().sm_count ? (int)p.total : ctx().sm_count;
  KD_CUDA_CHECK(launch_ex(gemm_f32_split_kernel<BN>, dim3(grid), dim3(FS_THREADS), (size_t)SMEM, p));
  return after_launch("gemm_f32_split_kernel");
}

// Tile width and split of K with the shortest estimate: rounds of CTAs over the SMs, each with its k-blocks and a fixed part.
static int split_tile(int64_t batches, int64_t M, int64_t N, int64_t K, int64_t sms, int* splits) {
  const int64_t m_tiles = (M + FS_BM - 1) / FS_BM, kbs = (K + FS_BK - 1) / FS_BK;
  double best = 1e30;
  int bn = 128;
  *splits = 1;
  for (int w = 64; w <= 128; w += 64) {
    const int64_t tiles = batches * m_tiles * ((N + w - 1) / w);
    for (int s = 1; s <= 4 && s <= kbs; s *= 2) {
      if (s > 1 && tiles * s > sms) break;       // (a CTA of a split tile has one tile)
      const double cost = (double)((tiles * s + sms - 1) / sms) * ((kbs + s - 1) / s) * (w == 64 ? FS_US_64 : FS_US_128) + (s > 1 ? FS_US_EXCHANGE : 0.0);
      if (cost < best) { best = cost; bn = w; *splits = s; }
    }
  }
  return bn;
}

int gemm_f32_split(const F32Gemm& g, int* handled) {
  *handled = 0;
  const uintptr_t base = reinterpret_cast<uintptr_t>(g.a) | reinterpret_cast<uintptr_t>(g.b);
  // 16-byte pieces of both operands along K, output rows with unit stride
  if (g.a_k != 1 || g.b_k != 1 || g.o_n != 1 || (base & 15) || g.K % 4) return KD_OK;
  if ((g.a_m | g.b_n | g.a_b0 | g.a_b1 | g.b_b0 | g.b_b1) & 3) return KD_OK;
  if (g.a_m < 0 || g.b_n < 0 || g.a_m >= (1 << 23) || g.b_n >= (1 << 23)) return KD_OK;      // (offsets inside a tile are 32-bit)
  if (g.M > (1 << 30) || g.N > (1 << 30) || g.K > (1 << 30) || g.b0 * g.b1 > (1 << 20)) return KD_OK;
  if (g.b0 * g.b1 * ((g.M + FS_BM - 1) / FS_BM) * ((g.N + 63) / 64) > (1 << 30)) return KD_OK;     // (tiles are counted in 32 bits)
  // a k-block of 64 is the unit of work: below one the padding outweighs the faster products
  if (g.K < FS_BK) return KD_OK;
  SplitParams p{};
  p.A = static_cast<const float*>(g.a); p.B = static_cast<const float*>(g.b); p.C = g.c; p.O = static_cast<float*>(g.o);
  p.M = (int)g.M; p.N = (int)g.N; p.K = (int)g.K;
  p.lda = (int)g.a_m; p.ldb = (int)g.b_n;
  p.a_b0 = g.a_b0; p.a_b1 = g.a_b1; p.b_b0 = g.b_b0; p.b_b1 = g.b_b1;
  p.c_b0 = g.c_b0; p.c_b1 = g.c_b1; p.c_m = g.c_m; p.c_n = g.c_n;
  p.o_b0 = g.o_b0; p.o_b1 = g.o_b1; p.o_m = g.o_m;
  p.b1 = (int)g.b1;
  p.dt_c = g.dt_c; p.has_c = g.has_c; p.alpha = g.alpha; p.beta = g.beta;
  p.vec_out = (reinterpret_cast<uintptr_t>(g.o) & 15) == 0 && ((g.o_m | g.o_b0 | g.o_b1) & 3) == 0;
  // tiles that share the larger operand run side by side, so that it is read from HBM once
  p.m_inner = g.N >= g.M;
  p.err = ctx().error_flag;
  const int64_t batches = g.b0 * g.b1;
  const int bn = split_tile(batches, g.M, g.N, g.K, ctx().sm_count, &p.splits);
  *handled = 1;
  return bn == 64 ? launch_split<64>(p, batches) : launch_split<128>(p, batches);
}

}  // namespace kd

using namespace kd;

KD_API int kd_debug_matmul_f32_plan(int64_t batches, int64_t M, int64_t N, int64_t K, int sms, int* width, int* splits) {
  KD_REQUIRE(width && splits && batches > 0 && M > 0 && N > 0 && K >= FS_BK && sms > 0, "bad argument");
  *width = split_tile(batches, M, N, K, sms, splits);
  return KD_OK;
}
