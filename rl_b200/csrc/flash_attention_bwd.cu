// Backward of the packed causal attention (see flash_attention.cu for the forward and the data layout).
//
// Two kernels, no atomics, S and P recomputed from Q, K and the saved log-sum-exp:
//   flash_bwd_dq_kernel   one CTA per (128-row query tile, query head); loops over 128-key tiles:
//                         S = Q K^T, dP = dO V^T, dS = P o (dP - delta) * scale, dQ += dS K
//   flash_bwd_dkv_kernel  one CTA per (128-key tile, kv head); loops over the G query heads of the group and over
//                         128-row query tiles at or below the diagonal, working on transposed tiles so that the key
//                         index is the TMEM lane: S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q
// All five products run on tcgen05 with fp32 accumulators in TMEM. A tile loaded by TMA with the 128-byte swizzle
// ([rows x 64 columns] boxes) serves both as a K-major and as an MN-major operand: the bytes are the same, only the
// shared-memory descriptor differs, so Q, K, V and dO are each loaded once per use.
// Two groups of four warps take half of a tile's columns each and write P and dS in bf16 over scores that they have read, from where the second products
// take them as TMEM operands. Scores go to a place as soon as the warps have read what it held, so that the next tile's are there when the warps get to
// them: in dQ one place for S and two for dP; in dK / dV, where the accumulators leave two, S and dP swap them with every tile.
// Tiles are 128 x 128 because a product of 128 x 64 x 16 takes the tensor core as long as one of 128 x 128 x 16 (64 cycles): 1536 of its cycles a tile in dQ
// and 2048 in dK / dV. The exponentials take 1024, the warps' whole chain some 2200: that chain bounds both kernels now. The products are
// issued by an elected thread: by lane 0 each took 105 cycles to issue, more than to execute.
// Measured, 32 query and 8 KV heads of 128, causal, dQ + dK / dV (before: tiles of 64, each group its own, lane 0 issuing), us: 4 x 4096 tokens
// 1433 + 1501 -> 774 + 951 (796 TFLOP/s of the five products that a gradient needs); 1 x 7600 1176 + 1327 -> 590 + 801; 16 x 1280 738 + 670 ->
// 475 + 471; 4 x 1000 129 + 116 -> 89 + 79; 16 x 300 114 + 74 -> 94 + 68.
// What lies behind a sequence's end is left out, by warps of 32 rows and by halves of the other side: sequences of up to 64 tokens, half of a tile, took up to a
// fifth longer than with tiles of 64 without that. 64 x 64 tokens 155 -> 139 us, 256 x 16 507 -> 440 (tiles of 64: 144 and 476).
// delta[h, t] = sum_d dO * O is computed beforehand by rlb_attn_delta.
#include "attention_tiles.cuh"

#include <math.h>
#include <type_traits>

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

// A step of 16 in the contraction is 32 bytes along the swizzled rows of a K-major operand; the address field of a descriptor counts 16 bytes.
__device__ __forceinline__ uint64_t desc_at(uint64_t base, int bytes) { return base + static_cast<uint64_t>(bytes >> 4); }
constexpr int TILE = 128;                  // query rows and keys of a tile
constexpr int TILE_BYTES = TILE * HD * 2;  // 32 KB
constexpr int ATOM = TILE * 128;           // bytes of one [rows x 64] bf16 atom
constexpr int HALF = TILE / 2;             // columns of a tile that a group of four warps takes

// D (+)= A B^T over HD, both operands K-major tiles in shared memory.
__device__ __forceinline__ void scores_mma(uint32_t d, uint32_t a_s, uint32_t b_s) {
  constexpr uint32_t idesc = make_idesc_bf16(TILE, TILE, false, false);
  const uint64_t a = make_smem_desc_sw128(a_s, 16, 1024), b = make_smem_desc_sw128(b_s, 16, 1024);
#pragma unroll
  for (int kk = 0; kk < HD / 16; ++kk) {
    const int off = (kk / 4) * ATOM + (kk % 4) * 32;
    umma_f16(d, desc_at(a, off), desc_at(b, off), idesc, kk != 0);
  }
}
// D[TILE x HD] (+)= A B with A [TILE x TILE] in TMEM, the two groups' halves 64 columns apart, and B a tile of rows read as an MN-major operand: 16 rows per
// step, 64-column groups an atom apart. BOTH: the second half holds something, too (else nothing was written there).
template <bool BOTH>
__device__ __forceinline__ void gradient_mma(uint32_t d, uint32_t a, uint32_t b_s, bool add) {
  constexpr uint32_t idesc = make_idesc_bf16(TILE, HD, false, true);
  const uint64_t b = make_smem_desc_sw128(b_s, ATOM, 1024);
#pragma unroll
  for (int kk = 0; kk < (BOTH ? TILE : HALF) / 16; ++kk) umma_f16_ts(d, a + (kk / 4) * HALF + (kk % 4) * 8, desc_at(b, kk * 2048), idesc, add || kk != 0);
}
__device__ __forceinline__ void load_rows(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col, int row) {
  mbar_arrive_expect_tx(smem_u32(bar), TILE_BYTES);
  for (int a = 0; a < ATOMS; ++a) tma_load_2d(smem_u32(dst + a * ATOM), map, smem_u32(bar), col + a * 64, row);
}
// This thread's 32 values as bf16 over 16 columns of scores that it has read.
__device__ __forceinline__ void store_bf16(uint32_t at, const float* v) {
  uint32_t pk[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
  tmem_st_32x32b_x16(at, pk);
}
// This thread's 64 scores; `read` hears from the warp that their place may be written again.
__device__ __forceinline__ void load_scores(uint32_t at, float* v, uint64_t* read, int lane) {
  uint32_t a[32], b[32];
  tmem_ld_32x32b_x32(at, a);
  tmem_ld_32x32b_x32(at + 32, b);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(a[i]), v[32 + i] = __uint_as_float(b[i]);
  if (read) {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(read));
  }
}
// The same from a warp that has nothing to read or store.
__device__ __forceinline__ void pass_on(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(bar));
}
// After a warp's stores to TMEM: its arrival at a barrier that the MMA warp waits for.
__device__ __forceinline__ void hand_over(uint64_t* bar, int lane) {
  tmem_st_wait();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(bar));
}

// ------------------------------------------------------------------------------------------------ dQ
constexpr int DQ_K_STAGES = 3, DQ_V_STAGES = 2;   // K is needed again by the second product, V only by the first
constexpr int DQ_SMEM = (2 + DQ_K_STAGES + DQ_V_STAGES) * TILE_BYTES + 256;

__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const __grid_constant__ CUtensorMap tmap_do, BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* q_s = smem;
  uint8_t* do_s = q_s + TILE_BYTES;
  uint8_t* k_s = do_s + TILE_BYTES;
  uint8_t* v_s = k_s + DQ_K_STAGES * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + DQ_V_STAGES * TILE_BYTES);
  uint64_t* q_full = bars;         // [2] Q, dO
  uint64_t* k_full = bars + 2;     // [3]
  uint64_t* k_empty = bars + 5;    // [3]
  uint64_t* v_full = bars + 8;     // [2]
  uint64_t* v_empty = bars + 10;   // [2]
  uint64_t* s_full = bars + 12;
  uint64_t* dp_full = bars + 13;   // [2]
  uint64_t* dq_done = bars + 15;   // the second product of a tile is complete
  uint64_t* all_done = bars + 16;  // every product is
  uint64_t* s_read = bars + 17;
  uint64_t* ds_full = bars + 18;   // [2]: a group may be done with the next tile before the other is with this one
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* info = reinterpret_cast<int*>(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.x;
  const int kv_head = head / (p.Hq / p.Hkv);
  if (warp == 0) {
    int start = 0, len = 0, tis = 0;
    const bool ok = locate_longest_first(p.cu_seqlens, p.num_seqs, TILE, blockIdx.z * gridDim.y + blockIdx.y, gridDim.y * gridDim.z, true, start, len, tis) && (smem_u32(smem) & 1023u) == 0;
    if (lane == 0) {
      info[0] = start; info[1] = len; info[2] = tis; info[3] = ok ? 1 : 0;
    }
  } else if (threadIdx.x == 64) {      // (while the first warp waits for the sequences' bounds)
    prefetch_tmap(&tmap_qkv);
    prefetch_tmap(&tmap_do);
    for (int i = 0; i < 17; ++i) mbar_init(smem_u32(&bars[i]), 1);
    mbar_init(smem_u32(s_read), 8);
    for (int i = 0; i < 2; ++i) mbar_init(smem_u32(&ds_full[i]), 8);
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
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
  // S at column 0, dP of even / odd tiles at 128 / 256 (each group's dS over the first half of its dP), dQ at 384
  const uint32_t tmem_dp = tmem_base + 128, tmem_dq = tmem_base + 384;
  const int seq_start = info[0], seq_len = info[1];
  const int q0 = info[2] * TILE;
  const int q_rows = min(TILE, seq_len - q0);
  const int n_kv = (q0 + q_rows + TILE - 1) / TILE;
  const int q_col = head * HD, k_col = (p.Hq + kv_head) * HD, v_col = (p.Hq + p.Hkv + kv_head) * HD;

  if (warp == 0) {
    if (elect_one()) {
      load_rows(q_s, &tmap_qkv, &q_full[0], q_col, seq_start + q0);
      bool ok = true;
      for (int j = 0; j < n_kv && ok; ++j) {
        const int row = seq_start + j * TILE, ks = j % DQ_K_STAGES, vs = j % DQ_V_STAGES;
        ok = mbar_wait(smem_u32(&k_empty[ks]), ((j / DQ_K_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        load_rows(k_s + ks * TILE_BYTES, &tmap_qkv, &k_full[ks], k_col, row);
        if (j == 0) load_rows(do_s, &tmap_do, &q_full[1], head * HD, seq_start + q0);
        ok = mbar_wait(smem_u32(&v_empty[vs]), ((j / DQ_V_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        load_rows(v_s + vs * TILE_BYTES, &tmap_qkv, &v_full[vs], v_col, row);
      }
      if (!ok) let_loads_land();
    }
  } else if (warp == 1) {
    const int cut = __shfl_sync(0xffffffffu, (q0 + q_rows - 1) % TILE < HALF ? 1 : 0, 0);      // 1: the last tile has keys in its first half only
    if (elect_one()) {
      auto scores = [&](int j) -> bool {      // S of tile j
        const int ks = j % DQ_K_STAGES;
        if (!mbar_wait(smem_u32(&k_full[ks]), (j / DQ_K_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        scores_mma(tmem_base, smem_u32(q_s), smem_u32(k_s + ks * TILE_BYTES));
        umma_commit(smem_u32(s_full));
        return true;
      };
      auto dprobs = [&](int j) -> bool {      // dP of tile j
        const int vs = j % DQ_V_STAGES;
        if (!mbar_wait(smem_u32(&v_full[vs]), (j / DQ_V_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        scores_mma(tmem_dp + (j & 1) * TILE, smem_u32(do_s), smem_u32(v_s + vs * TILE_BYTES));
        umma_commit(smem_u32(&dp_full[j & 1]));
        umma_commit(smem_u32(&v_empty[vs]));
        return true;
      };
      bool ok = mbar_wait(smem_u32(&q_full[0]), 0, abort_flag, p.status, RLB_ERR_WAIT_FULL) && scores(0) &&
                mbar_wait(smem_u32(&q_full[1]), 0, abort_flag, p.status, RLB_ERR_WAIT_FULL) && dprobs(0);
      auto product = [&](int j, auto both) -> bool {      // of tile j; the next tile's before it
        if (j + 1 < n_kv) {      // scores as soon as the warps have read the last ones, dP in the place of the last dS but one
          if (!mbar_wait(smem_u32(s_read), j & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG) || !scores(j + 1)) return false;
          if (j > 0 && !mbar_wait(smem_u32(dq_done), (j - 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY)) return false;
          if (!dprobs(j + 1)) return false;
        }
        if (!mbar_wait(smem_u32(&ds_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG)) return false;
        tc_fence_after();
        gradient_mma<decltype(both)::value>(tmem_dq, tmem_dp + (j & 1) * TILE, smem_u32(k_s + (j % DQ_K_STAGES) * TILE_BYTES), j != 0);
        umma_commit(smem_u32(&k_empty[j % DQ_K_STAGES]));
        umma_commit(smem_u32(dq_done));
        if (j + 1 == n_kv) umma_commit(smem_u32(all_done));
        return true;
      };
      for (int j = 0; j < n_kv - cut && ok; ++j) ok = product(j, std::true_type{});
      if (cut && ok) product(n_kv - 1, std::false_type{});
    }
  } else {
    const int warp_u = __shfl_sync(0xffffffffu, warp, 0);      // (the compiler sees that a branch on it is one of the whole warp)
    const int group = (warp_u - 2) >> 2;      // takes this half of a tile's keys
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int qi = q0 + r;
    const bool row_ok = r < q_rows;
    const long long stat_idx = static_cast<long long>(head) * p.T + seq_start + qi;
    const float lse2 = row_ok ? p.lse[stat_idx] * LOG2E : INFINITY;      // (rows behind the sequence: weights of zero)
    const float dlt = row_ok ? p.delta[stat_idx] : 0.f;
    const uint32_t s_at = tmem_base + group * HALF + lane_addr;
    // Tiles that have something for this warp: none where all of its rows are behind the sequence (what the products make of them is not stored), not the last
    // one where its half of the keys is.
    const int n_live = (warp_u & 3) * 32 >= q_rows ? 0 : q0 + q_rows > (n_kv - 1) * TILE + group * HALF ? n_kv : n_kv - 1;
    bool ok = true;
    for (int j = 0; j < n_live; ++j) {
      const uint32_t dp_at = tmem_dp + (j & 1) * TILE + group * HALF + lane_addr;
      if (!mbar_wait(smem_u32(s_full), j & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int k0 = j * TILE + group * HALF;
      const bool diag = k0 + HALF - 1 > q0;
      float w[HALF];
      load_scores(s_at, w, s_read, lane);
#pragma unroll
      for (int i = 0; i < HALF; ++i) w[i] = exp2f(w[i] * p.scale_log2 - lse2);
      if (diag) {
#pragma unroll
        for (int i = 0; i < HALF; ++i) w[i] = k0 + i <= qi ? w[i] : 0.f;
      }
      if (!mbar_wait(smem_u32(&dp_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t dpv[32];
        tmem_ld_32x32b_x32(dp_at + c * 32, dpv);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) w[c * 32 + i] *= (__uint_as_float(dpv[i]) - dlt) * p.scale;
        store_bf16(dp_at + c * 16, w + c * 32);
      }
      hand_over(&ds_full[j & 1], lane);
    }
    for (int j = n_live; j < n_kv && ok; ++j) {
      ok = mbar_wait(smem_u32(s_full), j & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL);
      if (ok) pass_on(s_read, lane);
      ok = ok && mbar_wait(smem_u32(&dp_full[j & 1]), (j >> 1) & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL);
      if (ok) pass_on(&ds_full[j & 1], lane);
    }
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
constexpr int KV_Q_STAGES = 3, KV_DO_STAGES = 2;      // (Q is needed by the first product and the last, dO by the two between)
constexpr int KV_STAT_BYTES = 2 * 2 * 2 * HALF * 4;   // per group, double buffered: lse2 and delta of its 64 query rows
constexpr int KV_SMEM = (2 + KV_Q_STAGES + KV_DO_STAGES) * TILE_BYTES + KV_STAT_BYTES + 256;

__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const __grid_constant__ CUtensorMap tmap_do, BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* k_s = smem;
  uint8_t* v_s = k_s + TILE_BYTES;
  uint8_t* q_s = v_s + TILE_BYTES;                    // [stages]
  uint8_t* do_s = q_s + KV_Q_STAGES * TILE_BYTES;     // [stages]
  float* stat_s = reinterpret_cast<float*>(do_s + KV_DO_STAGES * TILE_BYTES);  // [group][2][lse2 | delta][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(stat_s) + KV_STAT_BYTES);
  uint64_t* kv_full = bars;         // [2] K, V
  uint64_t* q_full = bars + 2;      // [3]
  uint64_t* q_empty = bars + 5;     // [3]
  uint64_t* do_full = bars + 8;     // [2]
  uint64_t* do_empty = bars + 10;   // [2]
  uint64_t* s_full = bars + 12;
  uint64_t* dp_full = bars + 13;
  uint64_t* dk_done = bars + 14;
  uint64_t* all_done = bars + 15;   // every product is complete
  uint64_t* p_full = bars + 16;
  uint64_t* dp_read = bars + 17;
  uint64_t* ds_full = bars + 18;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* info = reinterpret_cast<int*>(tmem_slot + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv_head = blockIdx.x;
  const int G = p.Hq / p.Hkv;
  if (warp == 0) {
    int start = 0, len = 0, tis = 0;
    const bool ok = locate_longest_first(p.cu_seqlens, p.num_seqs, TILE, blockIdx.z * gridDim.y + blockIdx.y, gridDim.y * gridDim.z, false, start, len, tis) && (smem_u32(smem) & 1023u) == 0;
    if (lane == 0) {
      info[0] = start; info[1] = len; info[2] = tis; info[3] = ok ? 1 : 0;
    }
  } else if (threadIdx.x == 64) {      // (while the first warp waits for the sequences' bounds)
    prefetch_tmap(&tmap_qkv);
    prefetch_tmap(&tmap_do);
    for (int i = 0; i < 16; ++i) mbar_init(smem_u32(&bars[i]), 1);
    mbar_init(smem_u32(p_full), 8);
    mbar_init(smem_u32(dp_read), 8);
    mbar_init(smem_u32(ds_full), 8);
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
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
  // S^T of even tiles at column 0 and dP^T at 128, of odd tiles the other way round (each group's P^T and dS^T over its half of the scores), dV at 256, dK at 384
  const uint32_t tmem_dv = tmem_base + 256, tmem_dk = tmem_base + 384;
  const int seq_start = info[0], seq_len = info[1];
  const int kv0 = info[2] * TILE;
  const int kv_rows = min(TILE, seq_len - kv0);
  const int qt_first = info[2];                               // first query tile at or below the diagonal
  const int qt_count = (seq_len + TILE - 1) / TILE - qt_first;
  const int n_iter = qt_count * G;                            // (query head of the group, query tile) pairs
  const int k_col = (p.Hq + kv_head) * HD, v_col = (p.Hq + p.Hkv + kv_head) * HD;

  if (warp == 0) {
    if (elect_one()) {
      load_rows(k_s, &tmap_qkv, &kv_full[0], k_col, seq_start + kv0);
      bool ok = true;
      for (int it = 0; it < n_iter && ok; ++it) {
        const int qs = it % KV_Q_STAGES, os = it % KV_DO_STAGES;
        const int g = it / qt_count, qt = qt_first + it % qt_count;
        const int col = (kv_head * G + g) * HD, row = seq_start + qt * TILE;
        ok = mbar_wait(smem_u32(&q_empty[qs]), ((it / KV_Q_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        load_rows(q_s + qs * TILE_BYTES, &tmap_qkv, &q_full[qs], col, row);
        if (it == 0) load_rows(v_s, &tmap_qkv, &kv_full[1], v_col, seq_start + kv0);
        ok = mbar_wait(smem_u32(&do_empty[os]), ((it / KV_DO_STAGES) & 1) ^ 1, abort_flag, p.status, RLB_ERR_WAIT_EMPTY);
        if (!ok) break;
        load_rows(do_s + os * TILE_BYTES, &tmap_do, &do_full[os], col, row);
      }
      if (!ok) let_loads_land();
    }
  } else if (warp == 1) {
    const int cut = __shfl_sync(0xffffffffu, (seq_len - 1) % TILE < HALF ? 1 : 0, 0);      // 1: the last query tile has rows in its first half only
    if (elect_one()) {
      auto scores = [&](int it) -> bool {      // S^T
        const int qs = it % KV_Q_STAGES;
        if (!mbar_wait(smem_u32(&q_full[qs]), (it / KV_Q_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        scores_mma(tmem_base + (it & 1) * TILE, smem_u32(k_s), smem_u32(q_s + qs * TILE_BYTES));
        umma_commit(smem_u32(s_full));
        return true;
      };
      auto dprobs = [&](int it) -> bool {      // dP^T
        const int os = it % KV_DO_STAGES;
        if (!mbar_wait(smem_u32(&do_full[os]), (it / KV_DO_STAGES) & 1, abort_flag, p.status, RLB_ERR_WAIT_FULL)) return false;
        tc_fence_after();
        scores_mma(tmem_base + (~it & 1) * TILE, smem_u32(v_s), smem_u32(do_s + os * TILE_BYTES));
        umma_commit(smem_u32(dp_full));
        return true;
      };
      bool ok = n_iter > 0 && mbar_wait(smem_u32(&kv_full[0]), 0, abort_flag, p.status, RLB_ERR_WAIT_FULL) && scores(0) &&
                mbar_wait(smem_u32(&kv_full[1]), 0, abort_flag, p.status, RLB_ERR_WAIT_FULL) && dprobs(0);
      auto products = [&](int it, auto both) -> bool {
        const int qs = it % KV_Q_STAGES, os = it % KV_DO_STAGES;
        if (!mbar_wait(smem_u32(p_full), it & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG)) return false;
        tc_fence_after();
        gradient_mma<decltype(both)::value>(tmem_dv, tmem_base + (it & 1) * TILE, smem_u32(do_s + os * TILE_BYTES), it != 0);
        umma_commit(smem_u32(&do_empty[os]));      // (dP^T of this tile was issued before)
        // the next scores take the place of this tile's dP as soon as the warps have read it, the next dP that of its P and dS
        if (it + 1 < n_iter && !(mbar_wait(smem_u32(dp_read), it & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG) && scores(it + 1))) return false;
        if (!mbar_wait(smem_u32(ds_full), it & 1, abort_flag, p.status, RLB_ERR_WAIT_FLAG)) return false;
        tc_fence_after();
        gradient_mma<decltype(both)::value>(tmem_dk, tmem_base + (it & 1) * TILE + 32, smem_u32(q_s + qs * TILE_BYTES), it != 0);
        umma_commit(smem_u32(&q_empty[qs]));
        umma_commit(smem_u32(dk_done));
        if (it + 1 == n_iter) umma_commit(smem_u32(all_done));
        return it + 1 == n_iter || (mbar_wait(smem_u32(dk_done), it & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_EMPTY) && dprobs(it + 1));
      };
      for (int it = 0; it < n_iter && ok;) {      // a head's query tiles
        for (const int whole = it + qt_count - cut; it < whole && ok; ++it) ok = products(it, std::true_type{});
        if (cut && ok) ok = products(it++, std::false_type{});
      }
    }
  } else {
    const int warp_u = __shfl_sync(0xffffffffu, warp, 0);      // (the compiler sees that a branch on it is one of the whole warp)
    const int group = (warp_u - 2) >> 2;      // takes this half of a tile's query rows
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;   // key row of this thread
    const int ct = (threadIdx.x - 64) & 127;     // 0..127 among the group's threads
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const int kj = kv0 + r;
    // statistics of the group's 64 query rows (threads 0..63: lse, 64..127: delta); rows behind the sequence get weights of zero
    auto statistic = [&](int it) -> float {
      if (it >= n_iter) return 0.f;
      const int g = it / qt_count, qi = (qt_first + it % qt_count) * TILE + group * HALF + (ct & 63);
      const long long idx = static_cast<long long>(kv_head * G + g) * p.T + seq_start + qi;
      if (qi >= seq_len) return ct < 64 ? INFINITY : 0.f;
      return ct < 64 ? p.lse[idx] * LOG2E : p.delta[idx];
    };
    float next = statistic(0);
    // Query tiles of a head that have something for this warp: none where all of its keys are behind the sequence, not the last one where its half of the rows is.
    const int n_live = (warp_u & 3) * 32 >= kv_rows ? 0 : seq_len > (qt_first + qt_count - 1) * TILE + group * HALF ? qt_count : qt_count - 1;
    bool ok = true;
    // The statistics of tile `it` in their place and its scores computed. Every warp of the group meets every barrier, also after a wait that ran out.
    auto begin = [&](int it) {
      stat_s[(group * 2 + (it & 1)) * 2 * HALF + ct] = next;
      next = statistic(it + 1);
      named_bar_sync(1 + group, 128);
      ok = ok && mbar_wait(smem_u32(s_full), it & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL);
    };
    for (int it = 0; it < n_iter;) {
      const int live_end = it + n_live, head_end = it + qt_count;
      int qbase = qt_first * TILE + group * HALF;
      for (; it < live_end; ++it, qbase += TILE) {
        begin(it);
        if (!ok) continue;
        const float* st_lse = stat_s + (group * 2 + (it & 1)) * 2 * HALF;
        tc_fence_after();
        const uint32_t s_at = tmem_base + (it & 1) * TILE + group * HALF + lane_addr, dp_at = tmem_base + (~it & 1) * TILE + group * HALF + lane_addr;
        float w[HALF];
        load_scores(s_at, w, nullptr, lane);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 l4 = *reinterpret_cast<const float4*>(st_lse + c * 32 + i);
            w[c * 32 + i] = exp2f(w[c * 32 + i] * p.scale_log2 - l4.x);
            w[c * 32 + i + 1] = exp2f(w[c * 32 + i + 1] * p.scale_log2 - l4.y);
            w[c * 32 + i + 2] = exp2f(w[c * 32 + i + 2] * p.scale_log2 - l4.z);
            w[c * 32 + i + 3] = exp2f(w[c * 32 + i + 3] * p.scale_log2 - l4.w);
          }
          if (qbase < kv0 + TILE - 1) {      // on the diagonal
#pragma unroll
            for (int i = 0; i < 32; ++i) w[c * 32 + i] = qbase + c * 32 + i < kj ? 0.f : w[c * 32 + i];
          }
          store_bf16(s_at + c * 16, w + c * 32);
        }
        hand_over(p_full, lane);
        ok = mbar_wait(smem_u32(dp_full), it & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL);
        if (!ok) continue;
        tc_fence_after();
        float dpv[HALF];
        load_scores(dp_at, dpv, dp_read, lane);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 d4 = *reinterpret_cast<const float4*>(st_lse + HALF + c * 32 + i);
            w[c * 32 + i] *= (dpv[c * 32 + i] - d4.x) * p.scale;
            w[c * 32 + i + 1] *= (dpv[c * 32 + i + 1] - d4.y) * p.scale;
            w[c * 32 + i + 2] *= (dpv[c * 32 + i + 2] - d4.z) * p.scale;
            w[c * 32 + i + 3] *= (dpv[c * 32 + i + 3] - d4.w) * p.scale;
          }
          store_bf16(s_at + 32 + c * 16, w + c * 32);
        }
        hand_over(ds_full, lane);
      }
      for (; it < head_end; ++it) {
        begin(it);
        if (ok) pass_on(p_full, lane);
        ok = ok && mbar_wait(smem_u32(dp_full), it & 1, abort_flag, p.status, RLB_ERR_WAIT_TMEM_FULL);
        if (ok) pass_on(dp_read, lane);
        if (ok) pass_on(ds_full, lane);
      }
    }
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
// max_q_tiles / max_kv_tiles: upper bounds on the number of 128-row tiles (ceil(T/128) + num_seqs is enough for both; blocks without a tile end at once, but take their turn).
RLB_API int RLB_NAME(rlb_flash_attn_bwd)(const void* qkv, long long qkv_stride, const void* dout, long long do_stride,
                               const float* lse, const float* delta, const int* cu_seqlens, int num_seqs, int T, int Hq,
                               int Hkv, int D, float scale, void* dqkv, long long dqkv_stride, int max_q_tiles,
                               int max_kv_tiles, int* status, void* stream) {
  if (T <= 0 || num_seqs <= 0) return 0;
  if (D != HD || Hq % Hkv || qkv_stride % 8 || do_stride % 8 || dqkv_stride % 8) return -2;
  const long long C = static_cast<long long>(Hq + 2 * Hkv) * HD;
  CUtensorMap tqkv, tdo;
  int rc = 0;
  rc |= rlb_make_tmap_2d(&tqkv, qkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, C, T, qkv_stride * 2, 64, TILE, CU_TENSOR_MAP_SWIZZLE_128B);
  rc |= rlb_make_tmap_2d(&tdo, dout, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, static_cast<long long>(Hq) * HD, T, do_stride * 2, 64, TILE, CU_TENSOR_MAP_SWIZZLE_128B);
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
  // Heads are the fast dimension; tiles take two where they are more than one can count.
  auto grid = [](int heads, int tiles) { return tiles <= 65535 ? dim3(heads, tiles) : dim3(heads, 65535, (tiles + 65534) / 65535); };
  flash_bwd_dq_kernel<<<grid(Hq, max_q_tiles), BWD_THREADS, DQ_SMEM, s>>>(tqkv, tdo, p);
  flash_bwd_dkv_kernel<<<grid(Hkv, max_kv_tiles), BWD_THREADS, KV_SMEM, s>>>(tqkv, tdo, p);
  return static_cast<int>(cudaGetLastError());
}
