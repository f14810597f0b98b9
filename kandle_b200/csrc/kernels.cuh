// Internal entry points shared between translation units.
#pragma once
#include "common.cuh"

namespace kd {

struct AttnParams {
  int B, Hq, Hkv, Sq, Skv, D;
  int64_t sq[4], sk[4], sv[4], so[4];
  int dt_q, dt_k, dt_v, dt_o;
  float scale;
  int causal;
};

// fp32 GEMM on the tensor cores (three bf16 parts per operand); strides in elements: A(m,k), B(k,n), C(m,n), O(m,n) and two
// batch dimensions each.  Sets *handled = 1 when it took the call.
struct F32Gemm {
  const void *a, *b, *c;
  void* o;
  int64_t M, N, K, b0, b1;
  int64_t a_b0, a_b1, a_m, a_k, b_b0, b_b1, b_k, b_n, c_b0, c_b1, c_m, c_n, o_b0, o_b1, o_m, o_n;
  int dt_c, has_c;
  float alpha, beta;
};
int gemm_f32_split(const F32Gemm& g, int* handled);

int matmul_f32_dispatch(const kd_matmul_cfg* cfg, const kd_tensor* a, const kd_tensor* b, const kd_tensor* c,
                        const kd_tensor* out);
// Tensor-core GEMM; sets *handled = 1 when it took the call (bf16 operands in a supported layout).
int matmul_tc_try(const kd_matmul_cfg* cfg, const kd_tensor* a, const kd_tensor* b, const kd_tensor* c,
                  const kd_tensor* out, int* handled);

int attention_params(const kd_tensor* q, const kd_tensor* k, const kd_tensor* v, const kd_tensor* out, float scale,
                     int is_causal, AttnParams* p);
int attention_f32_dispatch(const kd_tensor* q, const kd_tensor* k, const kd_tensor* v, const kd_tensor* out,
                           const AttnParams& p);
// out[M, N or N/2] = epilogue(A[M,K] * W[N,K]^T) on tcgen05; device pointers, ld* in elements.
int gemm_bf16(const void* A, int64_t lda, const void* W, int64_t ldw, void* out, int64_t ldo, int out_f32,
              const void* resid, int64_t ldr, int M, int N, int K, int epi);
int gemm_bf16_bias_act(const void* A, int64_t lda, const void* W, int64_t ldw, void* out, int64_t ldo, int out_f32,
              const void* resid, int64_t ldr, int M, int N, int K, int epi, const void* bias, int act, float* tail = nullptr,
              int tail_col = 0, int64_t ld_tail = 0);
// Grouped form: rows [group_off[g], group_off[g+1]) of A against W[g] [N,K] (group_off null: R / groups rows each);
// epi: KD_EPI_NONE, KD_EPI_CLAMPED_GLU or KD_EPI_GEGLU over interleaved rows.
int gemm_bf16_grouped(const void* A, const void* W, void* out, const int* group_off, int R, int groups, int N, int K, int epi, float limit);
// Tensor-core attention; sets *handled = 1 when it took the call.
int attention_tc_try(const kd_tensor* q, const kd_tensor* k, const kd_tensor* v, const kd_tensor* out,
                     const AttnParams& p, int* handled);

int gemm_bf16_qkv_rope(const void* A, int64_t lda, const void* W, int64_t ldw, int M, int K, int S, int Hq, int Hkv, int pos0,
                       float eps, const float* cos_t, const float* sin_t, const void* qw, const void* kw, void* q_out,
                       void* k_cache, void* v_cache, int64_t kc_b, int64_t kc_h, int64_t kc_s);
int gemm_skinny_auto_splits(int N, int K);
// x [Mb<=128,K] * W[N,K]^T -> fp32 partials [splits][Mb][N], or bf16 [Mb][N] when out_bf16 != NULL (splits == 1).
// groups > 1: as many independent problems, x [groups][Mb][K], W [groups][N][K], bf16 out [groups][Mb][N].
// glu (bf16 output [Mb][N/2], interleaved rows): 0 none, 1 silu(gate) * up, 2 gelu(gate) * up.
int gemm_bf16_skinny(const void* x, int64_t ldx, const void* W, int64_t ldw, int Mb, int N, int K, int splits,
                     float* out_f32, void* out_bf16, int glu, float alpha = 1.0f, float* tail = nullptr, int tail_row = 0,
                     int ld_tail = 0, int groups = 1);
// x [M <= 32, K] * W[N, K]^T by all SMs at once (linear_few.cu), where linear_few_rows says so.  Pointers 16-byte aligned, W dense.  epi: KD_EPI_NONE,
// KD_EPI_RESIDUAL (resid of the output's type, ldr), KD_EPI_SWIGLU, KD_EPI_GEGLU, or LINEAR_FEW_TANH; columns from tail_col on go to `tail` in fp32.
constexpr int LINEAR_FEW_TANH = 6;
bool linear_few_rows(int64_t M, int64_t N, int64_t K);
int linear_few(const void* x, int64_t ldx, const void* w, void* out, int64_t ldo, int out_f32, const void* resid, int64_t ldr, int M, int N, int K, int epi,
               float* tail = nullptr, int tail_col = 0, int64_t ld_tail = 0);
size_t attention_decode_scratch_bytes(int B, int Hkv, int group, int splits, int D);
int attention_decode(const kd_tensor* q, const kd_tensor* k, const kd_tensor* v, const kd_tensor* out, float scale,
                     const int* ctx_dev, int ctx_host, const int* block_table, int max_pages, int splits,
                     void* scratch, size_t scratch_bytes);

int attention_decode_static(const kd_tensor* q, const kd_tensor* k, const kd_tensor* v, const kd_tensor* out, float scale,
                            const int* ctx_dev, int ctx_host, int splits);

int attention_decode_static_fill(int byte_value);

// One token per sequence against cache rows [B,G,maxS,D] (D = 64 or 128, bf16): the newest `window` keys (0: all) up to
// the position, and a per-head sink (fp32 [H], or null).  q and out are dense [B,H,D].
struct WindowDecode {
  int B, H, G, D, max_s, window;
  float scale;
  const float* sink;
  const int* pos_dev;       // position of the token: device scalar, or
  int pos_host;
  int64_t kc[3], vc[3];     // cache strides: sequence, head, row
};
int attention_decode_window(const void* q, const void* k, const void* v, void* out, const WindowDecode& d);
// Prompts and portions: queries from position q_off on, `window` keys each (0: all), optional sink.
int attention_prefill2_window(const void* q, const void* k, const void* v, void* out, const AttnParams& a, int q_off, int window, const float* sink);

}  // namespace kd
