// Backward of the packed causal attention (see flash_attention.cu for the forward and the data layout).
//
// Two kernels, no atomics, S and P recomputed from Q, K and the saved log-sum-exp:
//   flash_bwd_dq_kernel   one CTA per (128-row query tile, query head); loops over 64-key tiles:
//                         S = Q K^T, dP = dO V^T, dS = P o (dP - delta) * scale, dQ += dS K
//   flash_bwd_dkv_kernel  one CTA per (128-key tile, kv head); loops over the G query heads of the group and over
//                         64-row query tiles at or below the diagonal, working on transposed tiles so that the key
//                         index is the TMEM lane: S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q
// All five products run on tcgen05 with fp32 accumulators in TMEM. A tile loaded by TMA with the 128-byte swizzle
// ([rows x 64 columns] boxes) serves both as a K-major and as an MN-major operand: the bytes are the same, only the
// shared-memory descriptor differs, so Q, K, V and dO are each loaded once per use.
// Scores live in two TMEM buffers each; two groups of four warps take the tiles in turn and write P and dS in bf16 over the
// scores they have read, from where the second products take them as TMEM operands. The scores of tile j + 1 are computed while tile j is in
// the warps' hands, so that the tensor core (768 cycles a tile in dQ, 1024 in dK / dV) and the exponentials (512) overlap.
// Measured, 32 query and 8 KV heads of 128, causal (before: one score buffer, one group, P and dS through shared memory): 16 x 4096 tokens
// 15.4 -> 11.0 ms (499 TFLOP/s of the five products that a gradient needs); 64 x 1280 7.7 -> 5.5 ms; 8 x (513, 700, 333) 0.83 -> 0.65 ms; with
// heads of 64 11.1 -> 8.8, 5.4 -> 4.4 and 0.59 -> 0.52 ms.
// delta[h, t] = sum_d dO * O is computed beforehand by rlb_attn_delta.
#include "attention_tiles.cuh"

#include <math.h>

namespace {
using namespace rlb;

#ifndef RLB_HD
#define RLB_HD 128        // head dimension of this translation unit; flash_attention_bwd_d64.cu includes this file with 64
#endif
#ifndef RLB_NAME
#define RLB_NAME(x) x
#endif
constexpr int HD = RLB_HD;
static_assert(HD == 64 || HD == 128, "head dimension: 64 or 128");
constexpr int ATOMS = HD / 64;   // [rows x 64] swizzle atoms per operand tile along the head dimension
constexpr float LOG2E = 1.4426950408889634f;
constexpr int BWD_THREADS = 320;      // TMA, MMA, two groups of four warps

__device__ __forceinline__ void named_bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// 32 accumulator columns of a lane as bf16.
__device__ __forceinline__ void store_row32(__nv_bfloat16* dst, const uint32_t (&o)[32]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 v;
    v.x = pack_bf16x2(__uint_as_float(o[q * 8 + 0]), __uint_as_float(o[q * 8 + 1]));
    v.y = pack_bf16x2(__uint_as_float(o[q * 8 + 2]), __uint_as_float(o[q * 8 + 3]));
    v.z = pack_bf16x2(__uint_as_float(o[q * 8 + 4]), __uint_as_float(o[q * 8 + 5]));
    v.w = pack_bf16x2(__uint_as_float(o[q * 8 + 6]), __uint_as_float(o[q * 8 + 7]));
    *reinterpret_cast<uint4*>(dst + q * 8) = v;
  }
}
// Loads in flight land within microseconds: after a wait that ran out they must not outlive the CTA.
__device__ __forceinline__ void let_loads_land() {
  const unsigned long long t0 = globaltimer_ns();
  while (globaltimer_ns() - t0 < 1000000ull) {}
}

struct BwdParams {
  const int* cu_seqlens;
  int num_seqs;
  int T;
  int Hq, Hkv;
  float scale;
  float scale_log2;
  const float* lse;    // [Hq, T] natural log
  const float* delta;  // [Hq, T]
  __nv_bfloat16* dqkv;
  long long dqkv_stride;
  int* status;
};

// ------------------------------------------------------------------------------------------------ dQ
constexpr int DQ_BQ = 128, DQ_BKV = 64;
constexpr int DQ_Q_BYTES = DQ_BQ * HD * 2;     // 32 KB
constexpr int DQ_KV_BYTES = DQ_BKV * HD * 2;   // 16 KB
constexpr int DQ_Q_ATOM = DQ_BQ * 128, DQ_KV_ATOM = DQ_BKV * 128;   // bytes of one [rows x 64] bf16 atom
constexpr int DQ_K_STAGES = 4, DQ_V_STAGES = 3;   // K is needed again by the second product, V only by the first
constexpr int DQ_SMEM = 2 * DQ_Q_BYTES + (DQ_K_STAGES + DQ_V_STAGES) * DQ_KV_BYTES + 256;

__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv,
                    const __grid_constant__ CUtensorMap tmap_do, BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* q_s = smem;
  uint8_t* do_s = q_s + DQ_Q_BYTES;
  uint8_t* k_s = do_s + DQ_Q_BYTES;
  uint8_t* v_s = k_s + DQ_K_STAGES * DQ_KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + DQ_V_STAGES * DQ_KV_BYTES);
  uint64_t* q_full = bars;         // Q and dO
  uint64_t* k_full = bars + 1;     // [4]
  uint64_t* k_empty = bars + 5;    // [4]
  uint64_t* v_full = bars + 9;     // [3]
  uint64_t* v_empty = bars + 12;   // [3]
  uint64_t* s_full = bars + 15;    // [2]
  uint64_t* p_full = bars + 17;    // [2]
  uint64_t* dq_done = bars + 19;   // [2] the second product of the buffer's tile is complete
  uint64_t* all_done = bars + 21;  // every product is
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 22);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* info = reinterpret_cast<int*>(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.x % p.Hq;
  const int kv_head = head / (p.Hq / p.Hkv);
  if (warp == 0) {
    int start = 0, len = 0, tis = 0;
    const bool ok = locate_longest_first(p.cu_seqlens, p.num_seqs, DQ_BQ, blockIdx.x / p.Hq, gridDim.x / p.Hq, true, start, len, tis) && (smem_u32(smem) & 1023u) == 0;
    if (lane == 0) {
      info[0] = start; info[1] = len; info[2] = tis; info[3] = ok ? 1 : 0;
      mbar_init(smem_u32(q_full), 1);
      for (int i = 1; i < 17; ++i) mbar_init(smem_u32(&bars[i]), 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(smem_u32(&p_full[i]), 4);
        mbar_init(smem_u32(&dq_done[i]), 1);
      }
      mbar_init(smem_u32(all_done), 1);
      *abort_flag = 0;
      mbar_fence_init();
      fence_proxy_async();
    }
  }
  __syncthreads();
  if (!info[3]) return;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // S of even / odd tiles at columns 0 / 64 (dS in the first 32 of each), dP at 128 / 192, dQ at 256
  const uint32_t tmem_dq = tmem_base + 256;
  const int seq_start = info[0], seq_len = info[1];
  const int q0 = info[2] * DQ_BQ;
  const int q_rows = min(DQ_BQ, seq_len - q0);
  const int n_kv = (q0 + q_rows + DQ_BKV - 1) / DQ_BKV;
  const int q_col = head * HD, k_col = (p.Hq + kv_head) * HD, v_col = (p.Hq + p.Hkv + kv_head) * HD;

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(smem_u32(q_full), 2 * DQ_Q_BYTES);
      for (int a = 0; a < ATOMS; ++a) {
        tma_load_2d(smem_u32(q_s + a * DQ_Q_ATOM), &tmap_q, smem_u32(q_full), q_col + a * 64, seq_start + q0);
        tma_load_2d(smem_u32(do_s + a * DQ_Q_ATOM), &tmap_do, smem_u32(q_full), head * HD + a * 64, seq_start + q0);
      }
      bool ok = true;
      for (int j = 0; j < n_kv && ok; ++j) {
        const int row = seq_start + j * DQ_BKV, ks = j % DQ_K_STAGES, vs = j % DQ_V_STAGES;
        ok = mbar_wait(smem_u32(&k_empty[ks]), ((j / DQ_K_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        mbar_arrive_expect_tx(smem_u32(&k_full[ks]), DQ_KV_BYTES);
        for (int a = 0; a < ATOMS; ++a)
          tma_load_2d(smem_u32(k_s + ks * DQ_KV_BYTES + a * DQ_KV_ATOM), &tmap_kv, smem_u32(&k_full[ks]), k_col + a * 64, row);
        ok = mbar_wait(smem_u32(&v_empty[vs]), ((j / DQ_V_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        mbar_arrive_expect_tx(smem_u32(&v_full[vs]), DQ_KV_BYTES);
        for (int a = 0; a < ATOMS; ++a)
          tma_load_2d(smem_u32(v_s + vs * DQ_KV_BYTES + a * DQ_KV_ATOM), &tmap_kv, smem_u32(&v_full[vs]), v_col + a * 64, row);
      }
      if (!ok) let_loads_land();
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16(DQ_BQ, DQ_BKV, false, false);
      constexpr uint32_t idesc_dq = make_idesc_bf16(DQ_BQ, HD, false, true);
      // S and dP of tile j; their buffers are free once the second product of tile j - 2 is complete
      auto scores = [&](int j) -> bool {
        const int ks = j % DQ_K_STAGES, vs = j % DQ_V_STAGES;
        if (j > 1 && !mbar_wait(smem_u32(&dq_done[j & 1]), ((j - 2) >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) return false;
        if (!mbar_wait(smem_u32(&k_full[ks]), (j / DQ_K_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        if (!mbar_wait(smem_u32(&v_full[vs]), (j / DQ_V_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        const uint32_t s_at = tmem_base + (j & 1) * 64, dp_at = tmem_base + 128 + (j & 1) * 64;
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t off_a = (kk / 4) * DQ_Q_ATOM + (kk % 4) * 32;
          const uint32_t off_b = (kk / 4) * DQ_KV_ATOM + (kk % 4) * 32;
          umma_f16(s_at, make_smem_desc_sw128(smem_u32(q_s) + off_a, 16, 1024),
                   make_smem_desc_sw128(smem_u32(k_s + ks * DQ_KV_BYTES) + off_b, 16, 1024), idesc_s, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t off_a = (kk / 4) * DQ_Q_ATOM + (kk % 4) * 32;
          const uint32_t off_b = (kk / 4) * DQ_KV_ATOM + (kk % 4) * 32;
          umma_f16(dp_at, make_smem_desc_sw128(smem_u32(do_s) + off_a, 16, 1024),
                   make_smem_desc_sw128(smem_u32(v_s + vs * DQ_KV_BYTES) + off_b, 16, 1024), idesc_s, kk != 0);
        }
        umma_commit(smem_u32(&s_full[j & 1]));
        umma_commit(smem_u32(&v_empty[vs]));
        return true;
      };
      bool ok = mbar_wait(smem_u32(q_full), 0, abort_flag, p.status, RLB_ERR_WAIT_FULL) && (n_kv == 0 || scores(0));
      for (int j = 0; j < n_kv && ok; ++j) {
        if (j + 1 < n_kv && !scores(j + 1)) break;
        if (!mbar_wait(smem_u32(&p_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG)) break;
        tc_fence_after();
        const uint32_t ka = smem_u32(k_s + (j % DQ_K_STAGES) * DQ_KV_BYTES);
#pragma unroll
        for (int kk = 0; kk < DQ_BKV / 16; ++kk)
          umma_f16_ts(tmem_dq, tmem_base + (j & 1) * 64 + kk * 8, make_smem_desc_sw128(ka + kk * 2048, DQ_KV_ATOM, 1024), idesc_dq, (j | kk) != 0);
        umma_commit(smem_u32(&k_empty[j % DQ_K_STAGES]));
        umma_commit(smem_u32(&dq_done[j & 1]));
        if (j + 1 == n_kv) umma_commit(smem_u32(all_done));
      }
    }
  } else {
    const int group = (warp - 2) >> 2;      // takes the tiles of this parity
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int qi = q0 + r;
    const bool row_ok = r < q_rows;
    const long long stat_idx = static_cast<long long>(head) * p.T + seq_start + qi;
    const float lse2 = row_ok ? p.lse[stat_idx] * LOG2E : INFINITY;      // (rows behind the sequence: weights of zero)
    const float dlt = row_ok ? p.delta[stat_idx] : 0.f;
    bool ok = true;
    for (int j = group; j < n_kv; j += 2) {
      const uint32_t s_at = tmem_base + group * 64 + lane_addr, dp_at = s_at + 128;
      if (!mbar_wait(smem_u32(&s_full[group]), (j >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int k0 = j * DQ_BKV;
      const bool diag = k0 + DQ_BKV - 1 > q0;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t s[32], dpv[32];
        tmem_ld_32x32b_x32(s_at + c * 32, s);
        tmem_ld_32x32b_x32(dp_at + c * 32, dpv);
        tmem_ld_wait();
        if (diag) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float w = k0 + c * 32 + i <= qi ? exp2f(__uint_as_float(s[i]) * p.scale_log2 - lse2) : 0.f;
            s[i] = __float_as_uint(w * (__uint_as_float(dpv[i]) - dlt) * p.scale);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            s[i] = __float_as_uint(exp2f(__uint_as_float(s[i]) * p.scale_log2 - lse2) * (__uint_as_float(dpv[i]) - dlt) * p.scale);
        }
        uint32_t pk[16];      // over scores that this thread has read
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
        tmem_st_32x32b_x16(s_at + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[group]));
    }
    // A barrier of its own: a group may be two phases of the other group's dq_done behind, where a wait for that parity passes at once.
    if (ok && mbar_wait(smem_u32(all_done), 0, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) {
      tc_fence_after();
      __nv_bfloat16* dst = p.dqkv + static_cast<long long>(seq_start + qi) * p.dqkv_stride + q_col;
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) {      // each group writes half of the columns
        const int col = group * (HD / 2) + c * 32;
        uint32_t o[32];
        tmem_ld_32x32b_x32(tmem_dq + lane_addr + col, o);
        tmem_ld_wait();
        if (row_ok) store_row32(dst + col, o);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------ dK / dV
constexpr int KV_BKV = 128, KV_BQ = 64;
constexpr int KV_K_BYTES = KV_BKV * HD * 2;      // 32 KB (two [128 x 64] atoms)
constexpr int KV_Q_BYTES = KV_BQ * HD * 2;       // 16 KB (two [64 x 64] atoms)
constexpr int KV_K_ATOM = KV_BKV * 128, KV_Q_ATOM = KV_BQ * 128;
constexpr int KV_STAGES = 4;
constexpr int KV_STAT_BYTES = 2 * 2 * 2 * KV_BQ * 4; // per group, double buffered: lse2 and delta of the 64 query rows
constexpr int KV_SMEM = 2 * KV_K_BYTES + 2 * KV_STAGES * KV_Q_BYTES + KV_STAT_BYTES + 256;

__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmap_kv128, const __grid_constant__ CUtensorMap tmap_q64,
                     const __grid_constant__ CUtensorMap tmap_do64, BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* k_s = smem;
  uint8_t* v_s = k_s + KV_K_BYTES;
  uint8_t* q_s = v_s + KV_K_BYTES;                    // [stages]
  uint8_t* do_s = q_s + KV_STAGES * KV_Q_BYTES;       // [stages]
  float* stat_s = reinterpret_cast<float*>(do_s + KV_STAGES * KV_Q_BYTES);  // [group][2][lse2 | delta][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(stat_s) + KV_STAT_BYTES);
  uint64_t* kv_full = bars;
  uint64_t* qdo_full = bars + 1;    // [4]
  uint64_t* qdo_empty = bars + 5;   // [4]
  uint64_t* s_full = bars + 9;      // [2]
  uint64_t* p_full = bars + 11;     // [2]
  uint64_t* acc_done = bars + 13;   // [2]
  uint64_t* all_done = bars + 15;   // every product is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* info = reinterpret_cast<int*>(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_head = blockIdx.x % p.Hkv;
  const int G = p.Hq / p.Hkv;
  if (warp == 0) {
    int start = 0, len = 0, tis = 0;
    const bool ok = locate_longest_first(p.cu_seqlens, p.num_seqs, KV_BKV, blockIdx.x / p.Hkv, gridDim.x / p.Hkv, false, start, len, tis) && (smem_u32(smem) & 1023u) == 0;
    if (lane == 0) {
      info[0] = start; info[1] = len; info[2] = tis; info[3] = ok ? 1 : 0;
      for (int i = 0; i < 11; ++i) mbar_init(smem_u32(&bars[i]), 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(smem_u32(&p_full[i]), 4);
        mbar_init(smem_u32(&acc_done[i]), 1);
      }
      mbar_init(smem_u32(all_done), 1);
      *abort_flag = 0;
      mbar_fence_init();
      fence_proxy_async();
    }
  }
  __syncthreads();
  if (!info[3]) return;
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // S^T of even / odd tiles at columns 0 / 64, dP^T at 128 / 192 (P^T and dS^T in the first 32 of each), dV at 256, dK at 384
  const uint32_t tmem_dv = tmem_base + 256, tmem_dk = tmem_base + 384;
  const int seq_start = info[0], seq_len = info[1];
  const int kv0 = info[2] * KV_BKV;
  const int kv_rows = min(KV_BKV, seq_len - kv0);
  const int qt_first = kv0 / KV_BQ;                           // first 64-row query tile at or below the diagonal
  const int qt_count = (seq_len + KV_BQ - 1) / KV_BQ - qt_first;
  const int n_iter = qt_count * G;                            // (query head of the group, query tile) pairs
  const int k_col = (p.Hq + kv_head) * HD, v_col = (p.Hq + p.Hkv + kv_head) * HD;

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(smem_u32(kv_full), 2 * KV_K_BYTES);
      for (int a = 0; a < ATOMS; ++a) {
        tma_load_2d(smem_u32(k_s + a * KV_K_ATOM), &tmap_kv128, smem_u32(kv_full), k_col + a * 64, seq_start + kv0);
        tma_load_2d(smem_u32(v_s + a * KV_K_ATOM), &tmap_kv128, smem_u32(kv_full), v_col + a * 64, seq_start + kv0);
      }
      bool ok = true;
      for (int it = 0; it < n_iter && ok; ++it) {
        const int st = it % KV_STAGES;
        ok = mbar_wait(smem_u32(&qdo_empty[st]), ((it / KV_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        const int g = it / qt_count, qt = qt_first + it % qt_count;
        const int head = kv_head * G + g;
        const int row = seq_start + qt * KV_BQ;
        mbar_arrive_expect_tx(smem_u32(&qdo_full[st]), 2 * KV_Q_BYTES);
        for (int a = 0; a < ATOMS; ++a) {
          tma_load_2d(smem_u32(q_s + st * KV_Q_BYTES + a * KV_Q_ATOM), &tmap_q64, smem_u32(&qdo_full[st]), head * HD + a * 64, row);
          tma_load_2d(smem_u32(do_s + st * KV_Q_BYTES + a * KV_Q_ATOM), &tmap_do64, smem_u32(&qdo_full[st]), head * HD + a * 64, row);
        }
      }
      if (!ok) let_loads_land();
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc_st = make_idesc_bf16(KV_BKV, KV_BQ, false, false);  // [128 keys] x [64 queries]
      constexpr uint32_t idesc_acc = make_idesc_bf16(KV_BKV, HD, false, true);     // += [128 x 64] * [64 x 128]
      auto scores = [&](int it) -> bool {
        const int st = it % KV_STAGES;
        if (it > 1 && !mbar_wait(smem_u32(&acc_done[it & 1]), ((it - 2) >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) return false;
        if (!mbar_wait(smem_u32(&qdo_full[st]), (it / KV_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        const uint32_t s_at = tmem_base + (it & 1) * 64, dp_at = tmem_base + 128 + (it & 1) * 64;
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t off_a = (kk / 4) * KV_K_ATOM + (kk % 4) * 32;
          const uint32_t off_b = (kk / 4) * KV_Q_ATOM + (kk % 4) * 32;
          umma_f16(s_at, make_smem_desc_sw128(smem_u32(k_s) + off_a, 16, 1024),
                   make_smem_desc_sw128(smem_u32(q_s + st * KV_Q_BYTES) + off_b, 16, 1024), idesc_st, kk != 0);
        }
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint32_t off_a = (kk / 4) * KV_K_ATOM + (kk % 4) * 32;
          const uint32_t off_b = (kk / 4) * KV_Q_ATOM + (kk % 4) * 32;
          umma_f16(dp_at, make_smem_desc_sw128(smem_u32(v_s) + off_a, 16, 1024),
                   make_smem_desc_sw128(smem_u32(do_s + st * KV_Q_BYTES) + off_b, 16, 1024), idesc_st, kk != 0);
        }
        umma_commit(smem_u32(&s_full[it & 1]));
        return true;
      };
      bool ok = mbar_wait(smem_u32(kv_full), 0, abort_flag, p.status, RLB_ERR_WAIT_FULL) && (n_iter == 0 || scores(0));
      for (int it = 0; it < n_iter && ok; ++it) {
        const int st = it % KV_STAGES;
        if (it + 1 < n_iter && !scores(it + 1)) break;
        if (!mbar_wait(smem_u32(&p_full[it & 1]), (it >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG)) break;
        tc_fence_after();
        // the query tile read as an MN-major operand: 16 query rows per step, 64-column groups 8 KB apart
#pragma unroll
        for (int kk = 0; kk < KV_BQ / 16; ++kk)
          umma_f16_ts(tmem_dv, tmem_base + (it & 1) * 64 + kk * 8, make_smem_desc_sw128(smem_u32(do_s + st * KV_Q_BYTES) + kk * 2048, KV_Q_ATOM, 1024), idesc_acc, (it | kk) != 0);
#pragma unroll
        for (int kk = 0; kk < KV_BQ / 16; ++kk)
          umma_f16_ts(tmem_dk, tmem_base + 128 + (it & 1) * 64 + kk * 8, make_smem_desc_sw128(smem_u32(q_s + st * KV_Q_BYTES) + kk * 2048, KV_Q_ATOM, 1024), idesc_acc, (it | kk) != 0);
        umma_commit(smem_u32(&qdo_empty[st]));
        umma_commit(smem_u32(&acc_done[it & 1]));
        if (it + 1 == n_iter) umma_commit(smem_u32(all_done));
      }
    }
  } else {
    const int group = (warp - 2) >> 2;      // takes the tiles of this parity
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;   // key row of this thread
    const int ct = (threadIdx.x - 64) & 127;     // 0..127 among the group's threads
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int kj = kv0 + r;
    // statistics of a tile's 64 query rows (threads 0..63: lse, 64..127: delta); rows behind the sequence get weights of zero
    auto statistic = [&](int it) -> float {
      if (it >= n_iter) return 0.f;
      const int g = it / qt_count, qi = (qt_first + it % qt_count) * KV_BQ + (ct & 63);
      const long long idx = static_cast<long long>(kv_head * G + g) * p.T + seq_start + qi;
      if (qi >= seq_len) return ct < 64 ? INFINITY : 0.f;
      return ct < 64 ? p.lse[idx] * LOG2E : p.delta[idx];
    };
    float next = statistic(group);
    bool ok = true;
    for (int it = group; it < n_iter; it += 2) {
      const int qbase = (qt_first + it % qt_count) * KV_BQ;
      float* st_lse = stat_s + (group * 2 + ((it >> 1) & 1)) * 2 * KV_BQ;
      st_lse[ct] = next;
      next = statistic(it + 2);
      named_bar_sync(1 + group, 128);
      ok = ok && mbar_wait(smem_u32(&s_full[group]), (it >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL);
      if (!ok) continue;      // every warp of the group meets every barrier, also after a wait that ran out
      tc_fence_after();
      const uint32_t s_at = tmem_base + group * 64 + lane_addr, dp_at = s_at + 128;
      const bool diag = qbase < kv0 + KV_BKV - 1;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t s[32], dpv[32];
        tmem_ld_32x32b_x32(s_at + c * 32, s);
        tmem_ld_32x32b_x32(dp_at + c * 32, dpv);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(st_lse + c * 32 + i), d4 = *reinterpret_cast<const float4*>(st_lse + KV_BQ + c * 32 + i);
          const float ll[4] = {l4.x, l4.y, l4.z, l4.w}, dl[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            float w = exp2f(__uint_as_float(s[i + h]) * p.scale_log2 - ll[h]);
            if (diag && qbase + c * 32 + i + h < kj) w = 0.f;
            s[i + h] = __float_as_uint(w);
            dpv[i + h] = __float_as_uint(w * (__uint_as_float(dpv[i + h]) - dl[h]) * p.scale);
          }
        }
        uint32_t pk[16];      // over scores that this thread has read
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
        tmem_st_32x32b_x16(s_at + c * 16, pk);
#pragma unroll
        for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(__uint_as_float(dpv[2 * i]), __uint_as_float(dpv[2 * i + 1]));
        tmem_st_32x32b_x16(dp_at + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&p_full[group]));
    }
    // (a barrier of its own, as for dQ)
    if (ok && n_iter > 0 && mbar_wait(smem_u32(all_done), 0, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) {
      tc_fence_after();
      // the first group writes dK, the second dV
      __nv_bfloat16* dst = p.dqkv + static_cast<long long>(seq_start + kj) * p.dqkv_stride + (group == 0 ? k_col : v_col);
      const uint32_t src = (group == 0 ? tmem_dk : tmem_dv) + lane_addr;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(src + c * 32, o);
        tmem_ld_wait();
        if (r < kv_rows) store_row32(dst + c * 32, o);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

int g_bwd_configured = 0;

}  // namespace

// dqkv[T, (Hq+2Hkv)*128] = gradient of the packed causal attention w.r.t. the fused [q | k | v] buffer.
// lse and delta are [Hq, T] fp32 (lse from the forward pass, delta from rlb_attn_delta).
// max_q_tiles / max_kv_tiles: upper bounds on the number of 128-row tiles (ceil(T/128) + num_seqs is enough for both).
RLB_API int RLB_NAME(rlb_flash_attn_bwd)(const void* qkv, long long qkv_stride, const void* dout, long long do_stride,
                               const float* lse, const float* delta, const int* cu_seqlens, int num_seqs, int T, int Hq,
                               int Hkv, int D, float scale, void* dqkv, long long dqkv_stride, int max_q_tiles,
                               int max_kv_tiles, int* status, void* stream) {
  if (T <= 0 || num_seqs <= 0) return 0;
  if (D != HD || Hq % Hkv || qkv_stride % 8 || do_stride % 8 || dqkv_stride % 8) return -2;
  const long long C = static_cast<long long>(Hq + 2 * Hkv) * HD;
  CUtensorMap tq128, tq64, tkv64, tkv128, tdo128, tdo64;
  int rc = 0;
  rc |= rlb_make_tmap_2d(&tq128, qkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, T, qkv_stride * 2, 64, 128, CU_TENSOR_MAP_SWIZZLE_128B);
  rc |= rlb_make_tmap_2d(&tq64, qkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, T, qkv_stride * 2, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  tkv64 = tq64;
  tkv128 = tq128;
  rc |= rlb_make_tmap_2d(&tdo128, dout, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, static_cast<long long>(Hq) * HD, T, do_stride * 2, 64, 128, CU_TENSOR_MAP_SWIZZLE_128B);
  rc |= rlb_make_tmap_2d(&tdo64, dout, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, static_cast<long long>(Hq) * HD, T, do_stride * 2, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return -100 - rc;
  if (!g_bwd_configured) {
    cudaError_t e = cudaFuncSetAttribute(flash_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DQ_SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    e = cudaFuncSetAttribute(flash_bwd_dkv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KV_SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    g_bwd_configured = 1;
  }
  BwdParams p;
  p.cu_seqlens = cu_seqlens;
  p.num_seqs = num_seqs;
  p.T = T;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.scale = scale;
  p.scale_log2 = scale * LOG2E;
  p.lse = lse;
  p.delta = delta;
  p.dqkv = reinterpret_cast<__nv_bfloat16*>(dqkv);
  p.dqkv_stride = dqkv_stride;
  p.status = status;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int most = (T + KV_BKV - 1) / KV_BKV + num_seqs;
  if (max_kv_tiles > most) max_kv_tiles = most;      // (blocks without a tile end at once, but take their turn)
  flash_bwd_dq_kernel<<<max_q_tiles * Hq, BWD_THREADS, DQ_SMEM, s>>>(tq128, tkv64, tdo128, p);
  flash_bwd_dkv_kernel<<<max_kv_tiles * Hkv, BWD_THREADS, KV_SMEM, s>>>(tkv128, tq64, tdo64, p);
  return static_cast<int>(cudaGetLastError());
}
