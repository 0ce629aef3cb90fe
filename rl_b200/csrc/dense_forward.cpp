// Inference pass of packed whole sequences through dense decoder layers (norm, fused q/k/v projection, rotation, causal attention, output
// projection, norm, gated unit), enqueued by one call.
//
// Small passes were bound by the host: eight launches a layer, each some 25 us of Python (16 layers of the 1B model on 240 tokens: 5.4 ms for 2.9 ms
// of device work). Enqueued from here a launch takes 2 to 3 us. The kernels and the rules that choose them are those of the layer-by-layer path.
// So the results are the same bit for bit, which prompts that are prefilled in parts rely on. (The decode step's fusions of norms and gated unit into the
// projections round at other places: two kernels a layer less, but another result for the same prompt.)
//
// Counterpart in the reference: the model forward behind get_logprobs and the prefill of its generation workers
// (nemo_rl/models/policy/workers/dtensor_policy_worker.py, nemo_rl/models/generation/vllm/vllm_worker.py:570-597).
#include <cstdint>

#define RLB_EXTERN extern "C"
RLB_EXTERN int rlb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out, float* rstd, long long rows, int d, long long x_stride,
                               long long y_stride, float eps, void* stream);
RLB_EXTERN int rlb_gemm_takes_skinny(int M, int N, int K);
RLB_EXTERN int rlb_gemm_skinny(const void* X, const void* W, void* Y, int M, int N, int K, long long ldx, long long ldw, long long ldy, int out_fp32,
                               const float* bias, const void* residual, long long ldr, int split, int* status, void* stream);
RLB_EXTERN int rlb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_mn_major,
                             int b_mn_major, int out_fp32, int accumulate, const float* bias, const void* residual, long long ldr, int* status, int max_ctas,
                             void* stream);
RLB_EXTERN int rlb_qk_rmsnorm_fwd(const void* x, const void* wq, const void* wk, void* out, float* rstd, long long rows, int Hq, int Hkv, int D,
                                  long long x_stride, long long out_stride, float eps, void* stream);
RLB_EXTERN int rlb_rope(void* x, const int* pos, const float* inv_freq, long long rows, int heads, int D, long long row_stride, int backward, void* stream);
RLB_EXTERN int rlb_rope_kv_cache_write(void* qkv, const int* pos, const float* inv_freq, const long long* slots, void* k_cache, void* v_cache, long long T,
                                       int Hq, int Hkv, int D, int block_size, long long row_stride, long long num_blocks, int* status, void* stream);
RLB_EXTERN int rlb_flash_attn_fwd(const void* qkv, long long qkv_stride, const int* cu_seqlens, int num_seqs, int T, int Hq, int Hkv, int D, float scale,
                                  void* out, long long out_stride, float* lse, int max_tiles, int* status, void* stream);
RLB_EXTERN int rlb_flash_attn_fwd_d64(const void* qkv, long long qkv_stride, const int* cu_seqlens, int num_seqs, int T, int Hq, int Hkv, int D, float scale,
                                      void* out, long long out_stride, float* lse, int max_tiles, int* status, void* stream);
RLB_EXTERN int rlb_swiglu_fwd(const void* gu, void* y, long long rows, int F, void* stream);

// The caller's arrays (ops/dense_forward.py mirrors both).
struct RlbDenseLayer {
  const void *norm1, *qkv, *o, *norm2, *gate_up, *down;      // contiguous bf16
  const void *q_norm, *k_norm;                               // or null
  const float* qkv_bias;                                     // or null
  const float* inv_freq;
  void *k_cache, *v_cache;                                   // with `slots`
};
struct RlbDenseForward {
  const RlbDenseLayer* layers;
  const void* h;                  // [T, d]
  void *out, *mid;                // [T, d]: the residual stream after a layer and after its attention
  void *x, *qkv, *att, *gate_up, *act;
  const int *positions, *cu_seqlens;
  const long long* slots;         // where keys and values go in the caches, or null
  int* status;
  int L, T, B, d, Hq, Hkv, D, F, block_size;
  long long num_blocks;
  float eps, scale;
};

namespace {
int linear(const RlbDenseForward& p, const void* x, const void* w, void* y, int N, int K, const float* bias, const void* residual, void* stream) {
  if (rlb_gemm_takes_skinny(p.T, N, K)) return rlb_gemm_skinny(x, w, y, p.T, N, K, K, K, N, 0, bias, residual, residual ? N : 0, 0, p.status, stream);
  return rlb_gemm_bf16(x, w, y, p.T, N, K, K, K, N, 0, 0, 0, 0, bias, residual, residual ? N : 0, p.status, 0, stream);
}
}  // namespace

extern "C" __attribute__((visibility("default"))) int rlb_dense_forward(const RlbDenseForward* desc, void* stream) {
  const RlbDenseForward& p = *desc;
  if (p.T <= 0 || p.L <= 0) return 0;
  if (p.D != 64 && p.D != 128) return -2;
  const int heads = p.Hq + 2 * p.Hkv, width = heads * p.D;
  const void* h = p.h;
  int rc = 0;
#define RLB_TRY(call) \
  do { if ((rc = (call)) != 0) return rc; } while (0)
  for (int l = 0; l < p.L; ++l) {
    const RlbDenseLayer& w = p.layers[l];
    RLB_TRY(rlb_rmsnorm_fwd(h, nullptr, w.norm1, p.x, nullptr, nullptr, p.T, p.d, p.d, p.d, p.eps, stream));
    RLB_TRY(linear(p, p.x, w.qkv, p.qkv, width, p.d, w.qkv_bias, nullptr, stream));
    if (w.q_norm) RLB_TRY(rlb_qk_rmsnorm_fwd(p.qkv, w.q_norm, w.k_norm, p.qkv, nullptr, p.T, p.Hq, p.Hkv, p.D, width, width, p.eps, stream));
    if (p.slots)
      RLB_TRY(rlb_rope_kv_cache_write(p.qkv, p.positions, w.inv_freq, p.slots, w.k_cache, w.v_cache, p.T, p.Hq, p.Hkv, p.D, p.block_size, width, p.num_blocks,
                                      p.status, stream));
    else
      RLB_TRY(rlb_rope(p.qkv, p.positions, w.inv_freq, p.T, p.Hq + p.Hkv, p.D, width, 0, stream));
    RLB_TRY((p.D == 128 ? rlb_flash_attn_fwd : rlb_flash_attn_fwd_d64)(p.qkv, width, p.cu_seqlens, p.B, p.T, p.Hq, p.Hkv, p.D, p.scale, p.att,
                                                                       static_cast<long long>(p.Hq) * p.D, nullptr, (p.T + 127) / 128 + p.B, p.status, stream));
    RLB_TRY(linear(p, p.att, w.o, p.mid, p.d, p.Hq * p.D, nullptr, h, stream));
    RLB_TRY(rlb_rmsnorm_fwd(p.mid, nullptr, w.norm2, p.x, nullptr, nullptr, p.T, p.d, p.d, p.d, p.eps, stream));
    RLB_TRY(linear(p, p.x, w.gate_up, p.gate_up, 2 * p.F, p.d, nullptr, nullptr, stream));
    RLB_TRY(rlb_swiglu_fwd(p.gate_up, p.act, p.T, p.F, stream));
    RLB_TRY(linear(p, p.act, w.down, p.out, p.d, p.F, nullptr, p.mid, stream));
    h = p.out;
  }
#undef RLB_TRY
  return 0;
}
