// Causal self-attention over packed (variable-length) sequences on the 5th-generation tensor cores:
// forward and backward, grouped-query heads, head dimension 128, bf16 in / fp32 accumulate.
//
// Inputs are read in place from the fused projection buffer qkv[T, (Hq + 2*Hkv) * 128] ([q | k | v] per token, after
// RoPE) through 2-D TMA tensor maps; `cu_seqlens[B+1]` marks sequence boundaries. The same kernels serve training
// (packed micro-batches) and the prefill of the generation engine.
//
// Forward, one CTA per (128-row query tile, query head), two CTAs per SM, the longest tiles first:
//   warp 0      TMA producer: Q once, then K tiles of 64 keys through a 3-stage ring and V tiles through a 2-stage ring
//   warp 1      tcgen05.mma issuer: S = Q K^T (128x64x128) into one of two TMEM buffers, one tile ahead of the softmax, then
//               O += P V (128x128x64) with P read from TMEM
//   warps 2..5  softmax: one thread per query row reads its 64 scores from TMEM (no shuffles), keeps the running
//               max / sum in the exp2 domain, writes P in bf16 over the scores it has read, and rescales the O accumulator in
//               TMEM only when the row maximum moved by more than 2^8 (stale maxima are exact because the final normalisation
//               uses the same reference).
// Bound by the tensor core (768 cycles per tile and CTA with heads of 128: eight steps of the scores, which take 64 cycles although only 64 columns wide, and
// four of the output; 512 with heads of 64) and the exponentials (512), so both have to run all the time: the next tile's scores are computed under this
// one's softmax, and two CTAs cover each other's hand-offs. Measured, 32 query and 8 KV heads of 128
// (before: one score buffer, P through shared memory): 16 x 4096 tokens 3.77 -> 2.24 ms (984 TFLOP/s); 64 x 1280 2.02 -> 1.18 ms. Since then, by the order of the tiles and an elected issuer: 4 x 4096 670 -> 546 us, 1 x 7600 541 -> 422.
// Output: O[T, Hq*128] bf16 and the per-row log-sum-exp lse[Hq, T] (natural log) for the backward pass.
//
// Backward (flash_attention_bwd.cu) is two kernels without atomics: one per (128-key tile, kv head) accumulating dK / dV over all query
// tiles and the G query heads of the group, one per (128-row query tile, query head) accumulating dQ over key tiles. Both
// recompute S and P from Q, K and lse.
//
// Replaces flash-attn 2 / cuDNN fused attention in the reference's policy workers
// (nemo_rl/models/automodel/setup.py:321-325, nemo_rl/models/megatron/setup.py:1114-1140).
#include "attention_tiles.cuh"

#include <math.h>

namespace {
using namespace rlb;

constexpr int BQ = 128;   // query rows per CTA
constexpr int BKV = 64;   // keys per pipeline stage
#ifndef RLB_HD
#define RLB_HD 128        // head dimension of this translation unit; flash_attention_d64.cu includes this file with 64
#endif
#ifndef RLB_NAME
#define RLB_NAME(x) x     // exported names get a suffix in the other instantiations (rlb_flash_attn_fwd_d64, ...)
#endif
constexpr int HD = RLB_HD;
static_assert(HD == 64 || HD == 128, "head dimension: 64 or 128");
constexpr int ATOMS = HD / 64;            // [rows x 64] swizzle atoms per operand tile along the head dimension
constexpr int K_STAGES = 3;
constexpr int V_STAGES = 2;
constexpr int Q_BYTES = BQ * HD * 2;         // 32 KB at HD 128: two [128 x 64] swizzle atoms
constexpr int Q_ATOM = BQ * 64 * 2;
constexpr int KV_ATOM = BKV * 64 * 2;
constexpr int K_BYTES = BKV * HD * 2;        // 16 KB: two [64 x 64] atoms
constexpr int V_BYTES = BKV * HD * 2;        // 16 KB: two boxes of 64 head-dim columns
constexpr int FWD_SMEM = Q_BYTES + K_STAGES * K_BYTES + V_STAGES * V_BYTES + 256;  // 2 CTAs fit in 227 KB
constexpr int FWD_THREADS = 192;
constexpr int TMEM_COLS_FWD = 256;  // S of even and odd tiles at columns 0 and 64 (P in the first 32 of each), O at column 128
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_THRESHOLD = 8.0f;  // in log2 units

__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

struct FwdParams {
  const int* cu_seqlens;
  int num_seqs;
  int T;
  int Hq, Hkv;
  float scale_log2;  // softmax scale * log2(e)
  __nv_bfloat16* out;
  long long out_stride;
  float* lse;  // [Hq, T]
  int* status;
  int longest_first;
};

__global__ void __launch_bounds__(FWD_THREADS, 2)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv,
                 FwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (smem_u32(smem) & 1023u) {  // the swizzled tiles need a 1024-byte aligned base; report instead of misreading
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, RLB_ERR_BAD_ARG);
    return;
  }
  uint8_t* q_s = smem;
  uint8_t* k_s = q_s + Q_BYTES;
  uint8_t* v_s = k_s + K_STAGES * K_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + V_STAGES * V_BYTES);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;    // [3]
  uint64_t* k_empty = bars + 4;   // [3]
  uint64_t* v_full = bars + 7;    // [2]
  uint64_t* v_empty = bars + 9;   // [2] also: the product with this V tile is in O
  uint64_t* s_full = bars + 11;   // [2]
  uint64_t* p_full = bars + 13;   // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* tile_info = reinterpret_cast<int*>(tmem_slot + 2);  // seq_start, seq_len, tile_in_seq, valid

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = p.longest_first ? blockIdx.x : blockIdx.y;
  const int kv_head = head / (p.Hq / p.Hkv);

  if (warp == 0) {
    int start = 0, len = 0, tis = 0;
    const bool ok = p.longest_first ? locate_longest_first(p.cu_seqlens, p.num_seqs, BQ, blockIdx.y, gridDim.y, true, start, len, tis)
                                    : locate_tile(p.cu_seqlens, p.num_seqs, BQ, gridDim.x - 1 - blockIdx.x, start, len, tis);      // late tiles of a sequence see the most keys
    if (lane == 0) {
      tile_info[0] = start;
      tile_info[1] = len;
      tile_info[2] = tis;
      tile_info[3] = ok ? 1 : 0;
    }
  } else if (threadIdx.x == 64) {      // (while the first warp waits for the sequences' bounds)
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_kv);
    mbar_init(smem_u32(q_full), 1);
    for (int s = 0; s < K_STAGES; ++s) {
      mbar_init(smem_u32(&k_full[s]), 1);
      mbar_init(smem_u32(&k_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&v_full[s]), 1);
      mbar_init(smem_u32(&v_empty[s]), 1);
      mbar_init(smem_u32(&s_full[s]), 1);
      mbar_init(smem_u32(&p_full[s]), 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  __syncthreads();
  if (!tile_info[3]) return;  // uniform: past the last tile (before any TMEM allocation)
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS_FWD);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_o = tmem_base + 128;

  const int seq_start = tile_info[0], seq_len = tile_info[1];
  const int q0 = tile_info[2] * BQ;                       // first query row, relative to the sequence
  const int q_rows = min(BQ, seq_len - q0);
  const int n_kv = (q0 + q_rows + BKV - 1) / BKV;         // causal: keys up to the tile's last row
  const int q_col = head * HD;
  const int k_col = (p.Hq + kv_head) * HD;
  const int v_col = (p.Hq + p.Hkv + kv_head) * HD;

  if (warp == 0) {
    if (elect_one()) {
      mbar_arrive_expect_tx(smem_u32(q_full), Q_BYTES);
#pragma unroll
      for (int a = 0; a < ATOMS; ++a)
        tma_load_2d(smem_u32(q_s + a * Q_ATOM), &tmap_q, smem_u32(q_full), q_col + a * 64, seq_start + q0);
      bool ok = true;
      for (int j = 0; j < n_kv && ok; ++j) {
        const int row = seq_start + j * BKV, ks = j % K_STAGES, vs = j % V_STAGES;
        ok = mbar_wait(smem_u32(&k_empty[ks]), ((j / K_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        mbar_arrive_expect_tx(smem_u32(&k_full[ks]), K_BYTES);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a)
          tma_load_2d(smem_u32(k_s + ks * K_BYTES + a * KV_ATOM), &tmap_kv, smem_u32(&k_full[ks]), k_col + a * 64, row);
        ok = mbar_wait(smem_u32(&v_empty[vs]), ((j / V_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        mbar_arrive_expect_tx(smem_u32(&v_full[vs]), V_BYTES);
#pragma unroll
        for (int a = 0; a < ATOMS; ++a)
          tma_load_2d(smem_u32(v_s + vs * V_BYTES + a * KV_ATOM), &tmap_kv, smem_u32(&v_full[vs]), v_col + a * 64, row);
      }
      if (!ok) {      // loads in flight land within microseconds: they must not outlive the CTA
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 1000000ull) {}
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(BQ, BKV, false, false);
      constexpr uint32_t idesc_o = make_idesc_bf16(BQ, HD, false, true);
      // S = Q K^T of tile j over the head dimension: steps of 16, swizzle atoms of 64. Its buffer held P of tile j - 2, whose product has
      // to be complete.
      auto scores = [&](int j) -> bool {
        const int ks = j % K_STAGES;
        if (j > 1 && !mbar_wait(smem_u32(&v_empty[j % V_STAGES]), ((j - 2) / V_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) return false;
        if (!mbar_wait(smem_u32(&k_full[ks]), (j / K_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t qa = smem_u32(q_s) + (kk / 4) * Q_ATOM + (kk % 4) * 32;
          const uint32_t ka = smem_u32(k_s + ks * K_BYTES) + (kk / 4) * KV_ATOM + (kk % 4) * 32;
          umma_f16(tmem_base + (j & 1) * 64, make_smem_desc_sw128(qa, 16, 1024), make_smem_desc_sw128(ka, 16, 1024), idesc_s, kk != 0 ? 1u : 0u);
        }
        umma_commit(smem_u32(&s_full[j & 1]));
        umma_commit(smem_u32(&k_empty[ks]));
        return true;
      };
      bool ok = mbar_wait(smem_u32(q_full), 0, abort_flag, p.status, RLB_ERR_WAIT_FULL) && (n_kv == 0 || scores(0));
      for (int j = 0; j < n_kv && ok; ++j) {
        const int vs = j % V_STAGES;
        if (j + 1 < n_kv && !scores(j + 1)) break;
        if (!mbar_wait(smem_u32(&p_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG)) break;
        if (!mbar_wait(smem_u32(&v_full[vs]), (j / V_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) break;
        tc_fence_after();
        // O += P V over the 64 keys: 4 steps of 16 key rows, 8 columns of P each
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk)
          umma_f16_ts(tmem_o, tmem_base + (j & 1) * 64 + kk * 8, make_smem_desc_sw128(smem_u32(v_s + vs * V_BYTES) + kk * (16 * 128), KV_ATOM, 1024), idesc_o,
                      (j | kk) != 0 ? 1u : 0u);
        umma_commit(smem_u32(&v_empty[vs]));
      }
    }
  } else {
    // ------------------------------------------------------------ softmax: thread = query row
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int qi = q0 + r;  // row index inside the sequence
    float m_ref = -INFINITY;  // reference maximum used for the exponentials (log2 domain)
    float l = 0.f;
    bool ok = true;
    // scores are compared before scaling; a negative scale turns the comparison round
    const bool neg = p.scale_log2 < 0.f;
    const float hidden = neg ? INFINITY : -INFINITY;
    for (int j = 0; j < n_kv; ++j) {
      const uint32_t tmem_s = tmem_base + (j & 1) * 64 + lane_addr;
      if (!mbar_wait(smem_u32(&s_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t s0[32], s1[32];
      tmem_ld_32x32b_x32(tmem_s, s0);
      tmem_ld_32x32b_x32(tmem_s + 32, s1);
      tmem_ld_wait();
      const int k0 = j * BKV;
      if (k0 + BKV - 1 > q0) {  // tile touches the causal boundary of some row
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (k0 + i > qi) s0[i] = __float_as_uint(hidden);
          if (k0 + 32 + i > qi) s1[i] = __float_as_uint(hidden);
        }
      }
      float best[4] = {__uint_as_float(s0[0]), __uint_as_float(s0[1]), __uint_as_float(s1[0]), __uint_as_float(s1[1])};
      if (!neg) {
#pragma unroll
        for (int i = 2; i < 32; i += 2) {
          best[0] = fmaxf(best[0], __uint_as_float(s0[i]));
          best[1] = fmaxf(best[1], __uint_as_float(s0[i + 1]));
          best[2] = fmaxf(best[2], __uint_as_float(s1[i]));
          best[3] = fmaxf(best[3], __uint_as_float(s1[i + 1]));
        }
        best[0] = fmaxf(fmaxf(best[0], best[1]), fmaxf(best[2], best[3]));
      } else {
#pragma unroll
        for (int i = 2; i < 32; i += 2) {
          best[0] = fminf(best[0], __uint_as_float(s0[i]));
          best[1] = fminf(best[1], __uint_as_float(s0[i + 1]));
          best[2] = fminf(best[2], __uint_as_float(s1[i]));
          best[3] = fminf(best[3], __uint_as_float(s1[i + 1]));
        }
        best[0] = fminf(fminf(best[0], best[1]), fminf(best[2], best[3]));
      }
      const float mx = best[0] * p.scale_log2;
      // Lazy rescale: move the reference only when the maximum grew by more than the threshold.
      float factor = 1.f;
      bool need = false;
      if (mx > m_ref + RESCALE_THRESHOLD || m_ref == -INFINITY) {
        const float m_new = fmaxf(mx, m_ref);
        if (m_new != -INFINITY) {
          factor = (m_ref == -INFINITY) ? 0.f : exp2f(m_ref - m_new);
          need = m_ref != -INFINITY;  // nothing accumulated yet: no O to rescale
          m_ref = m_new;
        }
      }
      const float mr = (m_ref == -INFINITY) ? 0.f : -m_ref;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[32];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float e0 = exp2f(fmaf(__uint_as_float(s0[2 * i]), p.scale_log2, mr)), e1 = exp2f(fmaf(__uint_as_float(s0[2 * i + 1]), p.scale_log2, mr));
        const float f0 = exp2f(fmaf(__uint_as_float(s1[2 * i]), p.scale_log2, mr)), f1 = exp2f(fmaf(__uint_as_float(s1[2 * i + 1]), p.scale_log2, mr));
        sum[0] += e0;
        sum[1] += e1;
        sum[2] += f0;
        sum[3] += f1;
        pk[i] = pack_bf16x2(e0, e1);
        pk[16 + i] = pack_bf16x2(f0, f1);
      }
      l = l * factor + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      tmem_st_32x32b_x32(tmem_s, pk);      // over the scores that this thread has read
      if (__any_sync(0xffffffffu, need)) {
        // O may be touched only after the previous P V product has completed (the next one waits for p_full)
        if (!mbar_wait(smem_u32(&v_empty[(j - 1) % V_STAGES]), ((j - 1) / V_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(tmem_o + lane_addr + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
          tmem_st_32x32b_x32(tmem_o + lane_addr + c * 32, o);
        }
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[j & 1]));
    }
    if (ok && mbar_wait(smem_u32(&v_empty[(n_kv - 1) % V_STAGES]), ((n_kv - 1) / V_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) {
      tc_fence_after();
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      const bool row_ok = r < q_rows;
      __nv_bfloat16* dst = p.out + static_cast<long long>(seq_start + qi) * p.out_stride + head * HD;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(tmem_o + lane_addr + c * 32, o);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 v;
            v.x = pack_bf16x2(__uint_as_float(o[q * 8 + 0]) * inv_l, __uint_as_float(o[q * 8 + 1]) * inv_l);
            v.y = pack_bf16x2(__uint_as_float(o[q * 8 + 2]) * inv_l, __uint_as_float(o[q * 8 + 3]) * inv_l);
            v.z = pack_bf16x2(__uint_as_float(o[q * 8 + 4]) * inv_l, __uint_as_float(o[q * 8 + 5]) * inv_l);
            v.w = pack_bf16x2(__uint_as_float(o[q * 8 + 6]) * inv_l, __uint_as_float(o[q * 8 + 7]) * inv_l);
            *reinterpret_cast<uint4*>(dst + c * 32 + q * 8) = v;
          }
        }
      }
      if (row_ok && p.lse)
        p.lse[static_cast<long long>(head) * p.T + seq_start + qi] = (m_ref + log2f(l)) * (1.f / LOG2E);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS_FWD);
  }
}

// delta[h, t] = sum_d dO[t, h, d] * O[t, h, d]: eight elements a thread, so many lanes a head (a warp per head moved 8 bytes a lane: 4000 tokens of 32
// heads of 128 26 us, now 20; of 64 23 and 14).
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                                                         float* __restrict__ delta, int T, int Hq, long long do_stride, long long o_stride) {
  constexpr int LANES = HD / 8;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x, head = i / LANES;
  const int piece = static_cast<int>(i % LANES);
  const bool in = head < static_cast<long long>(T) * Hq;
  const int t = in ? static_cast<int>(head / Hq) : 0, h = in ? static_cast<int>(head % Hq) : 0;
  const uint4 a = *reinterpret_cast<const uint4*>(dout + t * do_stride + h * HD + piece * 8), b = *reinterpret_cast<const uint4*>(out + t * o_stride + h * HD + piece * 8);
  const uint32_t x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
  float s = 0.f;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 u = unpack_bf16x2(x[q]), v = unpack_bf16x2(y[q]);
    s += u.x * v.x + u.y * v.y;
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (in && piece == 0) delta[static_cast<long long>(h) * T + t] = s;
}

int g_fwd_configured = 0;

}  // namespace

// qkv: [T, (Hq+2Hkv)*128] bf16 with row stride `qkv_stride` (elements); out: [T, Hq*128]; lse: [Hq, T] or null.
// cu_seqlens: device int32 [num_seqs + 1]. max_tiles: an upper bound on the number of 128-row query tiles
// (ceil(T / 128) + num_seqs is always enough).
RLB_API int RLB_NAME(rlb_flash_attn_fwd)(const void* qkv, long long qkv_stride, const int* cu_seqlens, int num_seqs, int T,
                               int Hq, int Hkv, int D, float scale, void* out, long long out_stride, float* lse,
                               int max_tiles, int* status, void* stream) {
  if (T <= 0 || num_seqs <= 0) return 0;
  if (D != HD || Hq % Hkv || qkv_stride % 8 || out_stride % 8) return -2;
  CUtensorMap tq, tkv;
  const long long C = static_cast<long long>(Hq + 2 * Hkv) * HD;
  int rc = rlb_make_tmap_2d(&tq, qkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, T, qkv_stride * 2, 64, BQ,
                            CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return -100 - rc;
  rc = rlb_make_tmap_2d(&tkv, qkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, T, qkv_stride * 2, 64, BKV,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return -100 - rc;
  if (!g_fwd_configured) {
    cudaError_t e = cudaFuncSetAttribute(flash_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    g_fwd_configured = 1;
  }
  FwdParams p;
  p.cu_seqlens = cu_seqlens;
  p.num_seqs = num_seqs;
  p.T = T;
  p.Hq = Hq;
  p.Hkv = Hkv;
  // (hidden scores are infinite: they must not meet a factor of zero, nor one that the kernel would flush to zero)
  p.scale_log2 = fabsf(scale) < 1e-30f ? copysignf(1e-30f, scale) : scale * LOG2E;
  p.out = reinterpret_cast<__nv_bfloat16*>(out);
  p.out_stride = out_stride;
  p.lse = lse;
  p.status = status;
  // Up to ten waves of two CTAs per SM the order of falling work over all sequences and heads saves most of the last one (one sequence of 7600 tokens,
  // 32 heads of 128: 543 -> 488 us; 8 x 500 71 -> 69); with more there is little to save, and neighbouring tiles of a head find their keys in the
  // nearer cache (16 x 1200: 323 us, longest first 336).
  p.longest_first = static_cast<long long>(max_tiles) * Hq <= 10 * 2 * 148;
  const dim3 grid = p.longest_first ? dim3(Hq, max_tiles) : dim3(max_tiles, Hq);
  flash_fwd_kernel<<<grid, FWD_THREADS, FWD_SMEM, static_cast<cudaStream_t>(stream)>>>(tq, tkv, p);
  return static_cast<int>(cudaGetLastError());
}

RLB_API int RLB_NAME(rlb_attn_delta)(const void* dout, const void* out, float* delta, int T, int Hq, long long do_stride,
                           long long o_stride, void* stream) {
  if (T <= 0) return 0;
  if ((do_stride % 8) || (o_stride % 8) || ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(out)) & 15)) return -3;      // (as the gradient's loads want it)
  const long long blocks = (static_cast<long long>(T) * Hq * (HD / 8) + 255) / 256;
  attn_delta_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(dout), reinterpret_cast<const __nv_bfloat16*>(out), delta, T, Hq,
      do_stride, o_stride);
  return static_cast<int>(cudaGetLastError());
}
