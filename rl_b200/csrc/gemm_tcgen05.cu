// bf16 GEMM on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM, operands staged
// by TMA into 128B-swizzled shared memory).
//
//   C[M,N] = op(A) * op(B)^T      A: [M,K] (K-major) or stored as [K,M] (MN-major)
//                                  B: [N,K] (K-major) or stored as [K,N] (MN-major)
//
// The three operand layouts cover a linear layer's forward (K,K), input gradient (K,MN) and
// weight gradient (MN,MN) without transposing anything in memory.
//
// Persistent kernel, one pair of CTAs (cta_group::2) per two SMs and 256 x 256 tile, 192 threads each:
//   warp 0      TMA producer (one elected lane): this CTA's 128 rows of A and 128 of the 256 rows of B
//   warp 1      TMEM allocator; in the pair's first CTA also the tcgen05.mma issuer (one elected lane) for both
//   warps 2..5  epilogue of this CTA's 128 rows: tcgen05.ld -> registers -> (shared memory ->) global
// A 6-deep shared-memory ring feeds 256x256x16 MMAs; two 256-column TMEM accumulators let the
// epilogue of tile i overlap the main loop of tile i+1. Where tiles of 256 rows would leave the last wave nearly empty (takes_pairs) the same
// kernel runs with one CTA per 128 x 256 tile and a 4-deep ring.
//
// Why pairs: one CTA's 128 x 256 tile fills and reads 192 bytes of shared memory per cycle of tensor time, above the 128
// that an SM has; a pair shares the B operand, which brings that to 128 and the L2 reads of a tile from 48 to 32 KB per k-block.
// Measured in short runs, one CTA per tile -> pairs (5120 rows, d 4096, ffn 14336): forward gate_up 938 -> 850 us (1415 TFLOP/s), input
// gradient of down 520 -> 441 us, weight gradient of gate_up 1177 -> 950 us, at 700 rows 630 -> 311 us (its rows are written whole, see
// store_piece). Over seconds the board's power limit, not the kernel, sets the rate of the forward products.
//
// Epilogues:
//   EPI_STORE    C = acc (+ bias) (+ C), bf16 or fp32
//   EPI_LOGPROB  for a vocab projection: per (row, n-tile) online-softmax partials (max, sum-exp,
//                sum of z*exp) and the target logit; logits are never written. A small second
//                kernel folds the partials into logprob / entropy / logsumexp per row.
//   EPI_LOGPROB_KEEP  the same, and the scaled logits are written in fp32 for the backward pass (dlogits_kept_kernel)
//   EPI_LAYER    products of a parallel mixer layer (LayerEpilogue in common.cuh): squared ReLU on a column range, or
//                residual update + dynamic-tanh norm
//   EPI_LINEAR   products of post-norm layers (LinearEpi in common.cuh): bias, then clamped gated unit or gated token input
//   EPI_DLOGITS  recomputes the logits tile and writes coef[row]*(onehot - softmax)*inv_temp in
//                bf16, the gradient that the dH / dW GEMMs consume.
// Replaces the cuBLAS calls behind nn.Linear and the chunked hidden->logprob path of the reference
// (nemo_rl/distributed/model_utils.py:2137-2316).
#include "common.cuh"
#include "out_piece.cuh"

#include <cstdlib>

#include <math.h>
#include <stdio.h>

namespace {

using namespace rlb;

constexpr int CTA_M = 128;    // rows of one CTA
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = CTA_M * BK * 2;  // 16 KB
constexpr int SMEM_BARRIER_BYTES = 256;
constexpr int NUM_THREADS = 192;
constexpr int TMEM_COLS = 512;
constexpr int GROUP_ROWS = 2048;  // rasterisation: the m-tiles of so many rows share each sweep over n

// A tile of a pair of CTAs, or of one.
template <bool PAIR>
struct Tile {
  static constexpr int CTAS = PAIR ? 2 : 1;
  static constexpr int BM = CTAS * CTA_M;
  static constexpr int CTA_N = BN / CTAS;                  // rows of B that each CTA loads
  static constexpr int STAGES = PAIR ? 6 : 4;
  static constexpr int STAGE_BYTES = A_STAGE_BYTES + CTA_N * BK * 2;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 4 * OUT_WARP_BYTES + SMEM_BARRIER_BYTES + 1024;  // +1024: manual alignment
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
};

enum { EPI_STORE = 0, EPI_LOGPROB = 1, EPI_DLOGITS = 2, EPI_LAYER = 3, EPI_LINEAR = 4, EPI_LOGPROB_KEEP = 5 };

struct EpiParams {
  void* C;              // output (EPI_STORE, EPI_DLOGITS), scaled logits (EPI_LOGPROB_KEEP)
  long long ldc;        // leading dimension of C in elements
  const float* bias;    // [N] or null
  const void* residual; // bf16 [M, ldr] added to the result (the residual stream), or null
  long long ldr;
  int out_fp32;         // EPI_STORE: 1 -> fp32 output
  int accumulate;       // EPI_STORE: 1 -> C += acc
  // vocab-projection epilogues
  const int* targets;   // [M] target column per row (global vocab id - vocab_offset), <0 or >=N: not here
  float inv_temp;
  float* part_max;      // [num_n_tiles, M]
  float* part_sum;      // [num_n_tiles, M]
  float* part_zsum;     // [num_n_tiles, M]
  float* target_logit;  // [M], written only by the tile that owns the target column
  const float* lse;     // [M] log-sum-exp of the scaled logits (EPI_DLOGITS)
  const float* coef;    // [M] upstream gradient of the log-probability (EPI_DLOGITS)
  const float* ent_coef;  // [M] upstream gradient of the entropy, or null (EPI_DLOGITS)
  const float* entropy;   // [M] entropy per row, needed with ent_coef
  LayerEpilogue layer;    // EPI_LAYER
};

template <int BM>
__device__ __forceinline__ void tile_coords(int tile, int num_m, int num_n, int& m_blk, int& n_blk) {
  constexpr int GROUP_M = GROUP_ROWS / BM;
  const int per_group = GROUP_M * num_n;
  const int group = tile / per_group;
  const int first_m = group * GROUP_M;
  const int rows = min(GROUP_M, num_m - first_m);
  const int in_group = tile - group * per_group;
  m_blk = first_m + in_group % rows;
  n_blk = in_group / rows;
}

__device__ __forceinline__ void unpack8(const uint4 r, float (&v)[8]) {
  const float2 a = unpack_bf16x2(r.x), b = unpack_bf16x2(r.y), c = unpack_bf16x2(r.z), d = unpack_bf16x2(r.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
__device__ __forceinline__ float4 square_relu4(float4 v) {
  v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f);
  return make_float4(v.x * v.x, v.y * v.y, v.z * v.z, v.w * v.w);
}

// Gradient of a logit whose scaled value is z: d logprob_t / dz_j = 1[j=t] - p_j ;  dH/dz_j = -p_j (logp_j + H)
__device__ __forceinline__ float dlogit(float z, bool is_target, float lse, float g, float ge, float ent, float inv_temp) {
  const float logp = z - lse;
  const float p = __expf(logp);
  float d = g * ((is_target ? 1.f : 0.f) - p);
  d -= ge * p * (logp + ent);
  return d * inv_temp;
}

// A load of this CTA's operands, signalling `bar`: with PAIR the first CTA's barrier.
template <bool PAIR>
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  if constexpr (PAIR) tma_load_2d_pair(dst, map, bar, c0, c1);
  else tma_load_2d(dst, map, bar, c0, c1);
}
template <bool PAIR>
__device__ __forceinline__ void commit_tile(uint32_t bar) {
  if constexpr (PAIR) umma_commit_pair(bar);
  else umma_commit(bar);
}

template <bool PAIR, bool A_MN, bool B_MN, int EPI>
__global__ void __cluster_dims__(Tile<PAIR>::CTAS, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 int M, int N, int K, EpiParams ep, int* status) {
  constexpr int BM = Tile<PAIR>::BM, CTA_N = Tile<PAIR>::CTA_N, STAGES = Tile<PAIR>::STAGES, STAGE_BYTES = Tile<PAIR>::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  // 128B swizzle needs 1024-byte aligned stage buffers.
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_smem = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_smem + 4 * OUT_WARP_BYTES);
  uint64_t* full_bar = bars;                 // [STAGES]
  uint64_t* empty_bar = bars + STAGES;       // [STAGES]
  uint64_t* tfull_bar = bars + 2 * STAGES;   // [2]
  uint64_t* tempty_bar = bars + 2 * STAGES + 2;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0;      // in the pair; the first CTA's barriers count the loads of both
  const int first = blockIdx.x / Tile<PAIR>::CTAS, step = gridDim.x / Tile<PAIR>::CTAS;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&tfull_bar[a]), 1);
      mbar_init(smem_u32(&tempty_bar[a]), 4 * Tile<PAIR>::CTAS);  // one arrive per epilogue warp
    }
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(smem_u32(tmem_slot), TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();      // both CTAs' barriers exist before either signals the other's
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int num_m = (M + BM - 1) / BM;
  const int num_n = (N + BN - 1) / BN;
  const int num_tiles = num_m * num_n;
  const int num_k = (K + BK - 1) / BK;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step) {
        int m_blk, n_blk;
        tile_coords<BM>(tile, num_m, num_n, m_blk, n_blk);
        const int row0 = m_blk * BM + rank * CTA_M, brow0 = n_blk * BN + rank * CTA_N;
        for (int kb = 0; kb < num_k; ++kb) {
          if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag, status, RLB_ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          const uint32_t bar = PAIR ? mapa_shared(smem_u32(&full_bar[stage]), 0) : smem_u32(&full_bar[stage]);
          const uint32_t a_dst = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t b_dst = a_dst + A_STAGE_BYTES;
          if (rank == 0) mbar_arrive_expect_tx(smem_u32(&full_bar[stage]), Tile<PAIR>::CTAS * STAGE_BYTES);
          if (!A_MN) {
            load_tile<PAIR>(a_dst, &tmap_a, bar, kb * BK, row0);
          } else {
#pragma unroll
            for (int j = 0; j < CTA_M / 64; ++j)
              load_tile<PAIR>(a_dst + j * (BK * 128), &tmap_a, bar, row0 + j * 64, kb * BK);
          }
          if (!B_MN) {
            load_tile<PAIR>(b_dst, &tmap_b, bar, kb * BK, brow0);
          } else {
#pragma unroll
            for (int j = 0; j < CTA_N / 64; ++j)
              load_tile<PAIR>(b_dst + j * (BK * 128), &tmap_b, bar, brow0 + j * 64, kb * BK);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok) {      // loads in flight land within microseconds: they must not outlive the CTA
        const unsigned long long t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 1000000ull) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, A_MN, B_MN);
      uint32_t stage = 0, phase = 0;
      uint32_t local_tile = 0;
      bool ok = true;
      for (int tile = first; tile < num_tiles && ok; tile += step, ++local_tile) {
        const uint32_t acc = local_tile & 1;
        const uint32_t acc_phase = (local_tile >> 1) & 1;
        if (!mbar_wait(smem_u32(&tempty_bar[acc]), acc_phase ^ 1, abort_flag, status, RLB_ERR_WAIT_TMEM_EMPTY)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = 0; kb < num_k; ++kb) {
          if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag, status, RLB_ERR_WAIT_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * STAGE_BYTES);
          const uint32_t b_addr = a_addr + A_STAGE_BYTES;
          const uint64_t a_desc = A_MN ? make_smem_desc_sw128(a_addr, BK * 128, 1024)
                                       : make_smem_desc_sw128(a_addr, 16, 1024);
          const uint64_t b_desc = B_MN ? make_smem_desc_sw128(b_addr, BK * 128, 1024)
                                       : make_smem_desc_sw128(b_addr, 16, 1024);
          // Advance along K inside the stage: 32 B per MMA for a K-major tile (inside the swizzle
          // atom), 16 k-rows of 128 B for an MN-major tile.
          constexpr uint32_t a_step = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
          constexpr uint32_t b_step = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            if constexpr (PAIR) umma_f16_pair(tmem_d, a_desc + kk * a_step, b_desc + kk * b_step, idesc, (kb | kk) != 0 ? 1u : 0u);
            else umma_f16(tmem_d, a_desc + kk * a_step, b_desc + kk * b_step, idesc, (kb | kk) != 0 ? 1u : 0u);
          }
          commit_tile<PAIR>(smem_u32(&empty_bar[stage]));  // stage reusable, in both CTAs, once these MMAs have read it
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) commit_tile<PAIR>(smem_u32(&tfull_bar[acc]));  // accumulator complete
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5)
    const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 belong to this warp
    const uint32_t buf = smem_u32(out_smem) + quarter * OUT_WARP_BYTES;
    uint32_t local_tile = 0;
    bool ok = true;
    for (int tile = first; tile < num_tiles && ok; tile += step, ++local_tile) {
      int m_blk, n_blk;
      tile_coords<BM>(tile, num_m, num_n, m_blk, n_blk);
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_phase = (local_tile >> 1) & 1;
      if (!mbar_wait(smem_u32(&tfull_bar[acc]), acc_phase, abort_flag, status, RLB_ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const int row0 = m_blk * BM + rank * CTA_M + quarter * 32, row = row0 + lane;
      const bool row_ok = row < M;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN;
      const int col0 = n_blk * BN;

      if (EPI == EPI_STORE) {
        for (int c = 0; c < BN / OUT_COLS && col0 + c * OUT_COLS < N; ++c) {
          uint32_t r[64];
          tmem_ld_32x32b_x32(taddr + c * OUT_COLS, *reinterpret_cast<uint32_t(*)[32]>(r));
          tmem_ld_32x32b_x32(taddr + c * OUT_COLS + 32, *reinterpret_cast<uint32_t(*)[32]>(r + 32));
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < OUT_COLS / 4; ++q)
            st_shared_f4(out_chunk(buf, lane, q), __uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
          store_piece(ep, buf, row0, col0 + c * OUT_COLS, M, N, lane);
        }
      } else if (EPI == EPI_LAYER) {
        // Through shared memory like store_piece. With one row to a lane the epilogue was longer than the main loop of short contractions and
        // than the fp32 stream of long ones: 11200 x 11264 x 2048 with the squared ReLU 452 -> 350 us (plain store 358), 11200 x 2048 x
        // 10240 onto the stream 404 -> 337 (with embeddings and step 453 -> 344), 700 rows of it 130 -> 88. The norm's loop is kept small:
        // unrolled over the rows, with branches in tanh, the same layout was slower than a row to a lane.
        const LayerEpilogue& le = ep.layer;
        const float alpha = le.x ? __bfloat162float(*le.alpha) : 0.f;
        const int q = (lane & 7) * 2, r0 = lane >> 3;      // eight lanes a row, eight columns each
        for (int c = 0; c < BN / OUT_COLS && col0 + c * OUT_COLS < N; ++c) {
          uint32_t t[64];
          tmem_ld_32x32b_x32(taddr + c * OUT_COLS, *reinterpret_cast<uint32_t(*)[32]>(t));
          tmem_ld_32x32b_x32(taddr + c * OUT_COLS + 32, *reinterpret_cast<uint32_t(*)[32]>(t + 32));
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < OUT_COLS / 4; ++i)
            st_shared_f4(out_chunk(buf, lane, i), __uint_as_float(t[4 * i]), __uint_as_float(t[4 * i + 1]), __uint_as_float(t[4 * i + 2]), __uint_as_float(t[4 * i + 3]));
          const int col = col0 + c * OUT_COLS + q * 4;
          const bool in = col < N;
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(ep.C) + static_cast<long long>(row0 + r0) * ep.ldc + col;
          __syncwarp();
          if (!le.x) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int r = 4 * i + r0;
              float4 u = ld_shared_f4(out_chunk(buf, r, q)), v = ld_shared_f4(out_chunk(buf, r, q + 1));
              if (!in || row0 + r >= M) continue;
              if (col >= le.act_from) { u = square_relu4(u); v = square_relu4(v); }      // act_from is a multiple of 8
              *reinterpret_cast<uint4*>(dst + 4 * i * ep.ldc) = make_uint4(pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w), pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
            }
          } else {
            // The residual stream of four rows at a time is fetched before any of it is written; its new values go back into the
            // piece, and the norm follows in a loop that stays small.
            float step[8] = {}, nw[8] = {}, nb[8] = {};
            if (in) {
              if (le.step) unpack8(*reinterpret_cast<const uint4*>(le.step + col), step);
              unpack8(*reinterpret_cast<const uint4*>(le.nw + col), nw);
              unpack8(*reinterpret_cast<const uint4*>(le.nb + col), nb);
            }
            float* xp = le.x + static_cast<long long>(row0 + r0) * le.ldx + col;
            const float* e = le.e ? le.e + static_cast<long long>(row0 + r0) * le.ldx + col : nullptr;
#pragma unroll 1
            for (int h = 0; h < 8; h += 4) {
              float4 old[4][2], ev[4][2];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const long long off = 4 * (h + i) * le.ldx;
                const bool ok_x = in && row0 + 4 * (h + i) + r0 < M, ok_e = ok_x && e;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  old[i][k] = ok_x ? *reinterpret_cast<const float4*>(xp + off + 4 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
                  ev[i][k] = ok_e ? *reinterpret_cast<const float4*>(e + off + 4 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
              }
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int r = 4 * (h + i) + r0;
                const bool ok_x = in && row0 + r < M;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  float4 u = ld_shared_f4(out_chunk(buf, r, q + k));
                  u.x = u.x + old[i][k].x + ev[i][k].x + step[4 * k];
                  u.y = u.y + old[i][k].y + ev[i][k].y + step[4 * k + 1];
                  u.z = u.z + old[i][k].z + ev[i][k].z + step[4 * k + 2];
                  u.w = u.w + old[i][k].w + ev[i][k].w + step[4 * k + 3];
                  st_shared_f4(out_chunk(buf, r, q + k), u.x, u.y, u.z, u.w);      // (read again by this lane alone)
                  if (ok_x) *reinterpret_cast<float4*>(xp + 4 * (h + i) * le.ldx + 4 * k) = u;
                }
              }
            }
#pragma unroll 1
            for (int i = 0; i < 8; ++i) {
              const int r = 4 * i + r0;
              const float4 u = ld_shared_f4(out_chunk(buf, r, q)), v = ld_shared_f4(out_chunk(buf, r, q + 1));
              float t8[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
              for (int k = 0; k < 8; ++k) t8[k] = tanh_acc(alpha * t8[k]) * nw[k] + nb[k];
              if (in && row0 + r < M)
                *reinterpret_cast<uint4*>(dst + 4 * i * ep.ldc) = make_uint4(pack_bf16x2(t8[0], t8[1]), pack_bf16x2(t8[2], t8[3]), pack_bf16x2(t8[4], t8[5]), pack_bf16x2(t8[6], t8[7]));
            }
          }
          __syncwarp();      // the buffer may be written again
        }
      } else if (EPI == EPI_LINEAR) {
        const LinearEpi& le = ep.layer.lin;
        const __nv_bfloat16* table = nullptr;
        if (le.act == LIN_GELU_MUL && row_ok) table = static_cast<const __nv_bfloat16*>(le.table) + lin_token(le, row) * le.ld_table + le.table_off;
        const bool wide = le.act == LIN_GELU_MUL && ((le.ld_table | le.table_off) & 3) == 0;      // table pieces of four columns are aligned
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + c * 32, r);
          tmem_ld_wait();
          const int col = col0 + c * 32;
          if (!row_ok || col >= N) continue;
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
          if (le.bias) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (col + q * 8 < N) {
                const uint4 b = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(le.bias) + col + q * 8);
                const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y), b2 = unpack_bf16x2(b.z), b3 = unpack_bf16x2(b.w);
                v[q * 8 + 0] += b0.x; v[q * 8 + 1] += b0.y; v[q * 8 + 2] += b1.x; v[q * 8 + 3] += b1.y;
                v[q * 8 + 4] += b2.x; v[q * 8 + 5] += b2.y; v[q * 8 + 6] += b3.x; v[q * 8 + 7] += b3.y;
              }
          }
          if (lin_gated(le.act)) {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(ep.C) + static_cast<long long>(row) * ep.ldc + col / 2;
            uint32_t o[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
              o[i] = pack_bf16x2(gated_unit(le.act, v[4 * i], v[4 * i + 1], le.limit), gated_unit(le.act, v[4 * i + 2], v[4 * i + 3], le.limit));
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (col + q * 8 < N) *reinterpret_cast<uint2*>(dst + q * 4) = make_uint2(o[2 * q], o[2 * q + 1]);
            continue;
          }
          if (le.act == LIN_GELU_MUL) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              float t[4] = {0.f, 0.f, 0.f, 0.f};
              const int x = col + q * 4;
              if (wide && x + 4 <= le.table_cols) {
                const uint2 raw = *reinterpret_cast<const uint2*>(table + x);
                const float2 a = unpack_bf16x2(raw.x), b = unpack_bf16x2(raw.y);
                t[0] = a.x; t[1] = a.y; t[2] = b.x; t[3] = b.y;
              } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                  if (x + k < le.table_cols) t[k] = __bfloat162float(table[x + k]);
              }
#pragma unroll
              for (int k = 0; k < 4; ++k) {      // 0.5 z (1 + tanh y) = z / (1 + exp(-2 y))
                const float z = v[q * 4 + k];
                v[q * 4 + k] = x + k < le.table_cols ? z / (1.f + __expf(-1.5957691216057308f * (z + 0.044715f * z * z * z))) * t[k] : 0.f;
              }
            }
          }
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(ep.C) + static_cast<long long>(row) * ep.ldc + col;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (col + q * 8 < N)
              *reinterpret_cast<uint4*>(dst + q * 8) = make_uint4(pack_bf16x2(v[q * 8], v[q * 8 + 1]), pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]),
                                                                  pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]), pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]));
        }
      } else if (EPI == EPI_LOGPROB || EPI == EPI_LOGPROB_KEEP) {
        // Online softmax statistics of this row over the tile's columns.
        float mx = -INFINITY, sum = 0.f, zsum = 0.f;
        const int tgt = row_ok ? ep.targets[row] : -1;
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + c * 32, r);
          tmem_ld_wait();
          const int col = col0 + c * 32;
          if (col >= N) continue;
          // Whole pieces go without a test of each column, whose branches cost more than the exponentials: the epilogue of a 256 x 256 tile was as
          // long as a product of 2048, and longer with the logits' stores behind it (4096 x 128256 x 2048 with stores 2.39 ms, now 1.55).
          float cmax[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
          if (col + 32 <= N) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float z = __uint_as_float(r[i]) * ep.inv_temp;
              r[i] = __float_as_uint(z);
              cmax[i & 3] = fmaxf(cmax[i & 3], z);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              r[i] = col + i < N ? __float_as_uint(__uint_as_float(r[i]) * ep.inv_temp) : __float_as_uint(-INFINITY);
              cmax[i & 3] = fmaxf(cmax[i & 3], __uint_as_float(r[i]));
            }
          }
          if (EPI == EPI_LOGPROB_KEEP) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
              st_shared_f4(out_chunk(buf, lane, (c & 1) * 8 + q), __uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]),
                           __uint_as_float(r[4 * q + 3]));
            if ((c & 1) || col + 32 >= N) stream_piece(static_cast<float*>(ep.C), ep.ldc, buf, row0, col - (c & 1) * 32, M, N, lane);
          }
          const float nmx = fmaxf(mx, fmaxf(fmaxf(cmax[0], cmax[1]), fmaxf(cmax[2], cmax[3])));
          const float scale = __expf(mx - nmx);  // exp(-inf) = 0 on the first chunk
          float s4[4] = {sum * scale, 0.f, 0.f, 0.f}, z4[4] = {zsum * scale, 0.f, 0.f, 0.f};
          if (col + 32 <= N) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float z = __uint_as_float(r[i]), e = __expf(z - nmx);
              s4[i & 3] += e;
              z4[i & 3] += z * e;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (col + i < N) {
                const float z = __uint_as_float(r[i]), e = __expf(z - nmx);
                s4[i & 3] += e;
                z4[i & 3] += z * e;
              }
            }
          }
          sum = (s4[0] + s4[1]) + (s4[2] + s4[3]);
          zsum = (z4[0] + z4[1]) + (z4[2] + z4[3]);
          if (static_cast<unsigned>(tgt - col) < 32u && tgt < N) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (col + i == tgt) ep.target_logit[row] = __uint_as_float(r[i]);
          }
          mx = nmx;
        }
        if (row_ok) {
          const long long idx = static_cast<long long>(n_blk) * M + row;
          ep.part_max[idx] = mx;
          ep.part_sum[idx] = sum;
          ep.part_zsum[idx] = zsum;
        }
      } else {  // EPI_DLOGITS
        const int tgt = row_ok ? ep.targets[row] : -1;
        const float lse = row_ok ? ep.lse[row] : 0.f;
        const float g = row_ok ? ep.coef[row] : 0.f;
        const float ge = (row_ok && ep.ent_coef) ? ep.ent_coef[row] : 0.f;
        const float ent = (row_ok && ep.ent_coef) ? ep.entropy[row] : 0.f;
        for (int c = 0; c < BN / OUT_COLS && col0 + c * OUT_COLS < N; ++c) {
          uint32_t r[64];
          tmem_ld_32x32b_x32(taddr + c * OUT_COLS, *reinterpret_cast<uint32_t(*)[32]>(r));
          tmem_ld_32x32b_x32(taddr + c * OUT_COLS + 32, *reinterpret_cast<uint32_t(*)[32]>(r + 32));
          tmem_ld_wait();
          const int col = col0 + c * OUT_COLS;
          float v[64];
#pragma unroll
          for (int i = 0; i < OUT_COLS; ++i) {
            v[i] = dlogit(__uint_as_float(r[i]) * ep.inv_temp, col + i == tgt, lse, g, ge, ent, ep.inv_temp);
          }
#pragma unroll
          for (int q = 0; q < OUT_COLS / 4; ++q) st_shared_f4(out_chunk(buf, lane, q), v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          store_piece(ep, buf, row0, col, M, N, lane);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[acc]), 0));
        else mbar_arrive(smem_u32(&tempty_bar[acc]));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();      // nothing of the pair signals or writes the other CTA any more
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// EPI_DLOGITS without the product, from the logits that EPI_LOGPROB_KEEP wrote: 6 bytes a logit, bound by memory. A thread requests its 64 bytes
// before it computes.
constexpr int KEPT_COLS = 256 * 16;
__global__ void __launch_bounds__(256) dlogits_kept_kernel(const float* __restrict__ z, __nv_bfloat16* __restrict__ dz, int N, long long ldz, long long lddz,
                                                           const int* __restrict__ targets, float inv_temp, const float* __restrict__ lse_,
                                                           const float* __restrict__ coef, const float* __restrict__ ent_coef,
                                                           const float* __restrict__ entropy) {
  const long long row = blockIdx.y;
  const int col = blockIdx.x * KEPT_COLS + threadIdx.x * 8;      // and 2048 further on
  const float* src = z + row * ldz + col;
  float4 v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (col + (j >> 1) * 2048 < N) v[j] = __ldcs(reinterpret_cast<const float4*>(src + (j >> 1) * 2048) + (j & 1));
  const int tgt = targets[row];
  const float lse = lse_[row], g = coef[row];
  const float ge = ent_coef ? ent_coef[row] : 0.f, ent = ent_coef ? entropy[row] : 0.f;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int c = col + j * 2048;
    if (c >= N) continue;      // N is a multiple of 8
    const float e[8] = {v[2 * j].x, v[2 * j].y, v[2 * j].z, v[2 * j].w, v[2 * j + 1].x, v[2 * j + 1].y, v[2 * j + 1].z, v[2 * j + 1].w};
    float d[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) d[i] = dlogit(e[i], c + i == tgt, lse, g, ge, ent, inv_temp);
    *reinterpret_cast<uint4*>(dz + row * lddz + c) =
        make_uint4(pack_bf16x2(d[0], d[1]), pack_bf16x2(d[2], d[3]), pack_bf16x2(d[4], d[5]), pack_bf16x2(d[6], d[7]));
  }
}

// Folds the per-n-tile partials of EPI_LOGPROB into per-row results: 32 rows per CTA, the parts dealt out to its warps (one thread per row
// walked 501 parts twice, 126 us at 240 rows; eight warps
// take 37 us for 32 to 4000 rows, 32 warps 15 to 17; from 20000 rows on, where the CTAs fill the SMs several times, eight: 52 and 61).
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) logprob_combine_kernel(const float* __restrict__ part_max, const float* __restrict__ part_sum,
                                                              const float* __restrict__ part_zsum, const float* __restrict__ target_logit, int M, int num_parts,
                                                              float* __restrict__ logprob, float* __restrict__ entropy, float* __restrict__ lse_out) {
  __shared__ float s_max[WARPS][32], s_sum[WARPS][32], s_zsum[WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + lane;
  float mx = -INFINITY, sum = 0.f, zsum = 0.f;
  if (row < M) {
#pragma unroll 4
    for (int p = warp; p < num_parts; p += WARPS) mx = fmaxf(mx, part_max[static_cast<long long>(p) * M + row]);
#pragma unroll 4
    for (int p = warp; p < num_parts; p += WARPS) {
      const long long i = static_cast<long long>(p) * M + row;
      const float s = part_max[i] == -INFINITY ? 0.f : __expf(part_max[i] - mx);      // (a part without columns, or all of this warp's)
      sum += part_sum[i] * s;
      zsum += part_zsum[i] * s;
    }
  }
  s_max[warp][lane] = mx;
  s_sum[warp][lane] = sum;
  s_zsum[warp][lane] = zsum;
  __syncthreads();
  if (warp != 0 || row >= M) return;
  for (int w = 1; w < WARPS; ++w) mx = fmaxf(mx, s_max[w][lane]);
  sum = zsum = 0.f;
  for (int w = 0; w < WARPS; ++w) {
    const float s = s_max[w][lane] == -INFINITY ? 0.f : __expf(s_max[w][lane] - mx);
    sum += s_sum[w][lane] * s;
    zsum += s_zsum[w][lane] * s;
  }
  const float lse = mx + logf(sum);
  if (lse_out) lse_out[row] = lse;
  if (logprob) logprob[row] = target_logit[row] - lse;
  if (entropy) entropy[row] = lse - zsum / sum;  // H = lse - E[z]
}

int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

template <typename... Args>
void launch_combine(cudaStream_t s, const float* part_max, const float* part_sum, const float* part_zsum, const float* target_logit, int M, Args... args) {
  const int blocks = (M + 31) / 32;
  if (blocks <= 2 * sm_count()) logprob_combine_kernel<32><<<blocks, 1024, 0, s>>>(part_max, part_sum, part_zsum, target_logit, M, args...);
  else logprob_combine_kernel<8><<<blocks, 256, 0, s>>>(part_max, part_sum, part_zsum, target_logit, M, args...);
}

// Tiles of this size, and the waves of them on at most `max_ctas` CTAs (0: as many as there are SMs).
template <bool PAIR>
int num_tiles(int M, int N) { return ((M + Tile<PAIR>::BM - 1) / Tile<PAIR>::BM) * ((N + BN - 1) / BN); }
template <bool PAIR>
int slots(int max_ctas) {
  const int ctas = max_ctas > 0 && max_ctas < sm_count() ? max_ctas : sm_count();
  return ctas / Tile<PAIR>::CTAS;
}

// Pairs unless single CTAs need so many waves fewer that these, each some 10 to 15 % longer, are sooner done. Timed both ways over 250 products
// (64 to 9000 rows; forward, input and weight gradients, vocabulary): at equal waves pairs took 0.90 of single CTAs' time (0.84 to 1.05), at
// 1.11 to 1.14 times as many waves 0.98 to 0.99, at 1.17 1.00 to 1.05, at 1.25 to 1.33 1.02 to 1.17, at 1.5 to 2 1.05 to 1.6. So 640 x 14336 x 4096
// runs in 91 us (pairs 116), 1100 x 4096 x 14336 in 163 (267), 257 rows of a vocabulary of 128256 x 2048 in 228 (257).
constexpr int TILE_RATIO = 115;      // percent
bool takes_pairs(int M, int N, int max_ctas) {
  const int p = slots<true>(max_ctas), c = slots<false>(max_ctas);
  if (p == 0) return false;
  const int waves_p = (num_tiles<true>(M, N) + p - 1) / p, waves_c = (num_tiles<false>(M, N) + c - 1) / c;
  return 100 * waves_p <= TILE_RATIO * waves_c;
}

template <bool PAIR, bool A_MN, bool B_MN, int EPI>
int launch_tiles(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, const EpiParams& ep,
                 int* status, int max_ctas, cudaStream_t stream) {
  auto kern = gemm_bf16_kernel<PAIR, A_MN, B_MN, EPI>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<PAIR>::SMEM_BYTES);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  const int tiles = num_tiles<PAIR>(M, N), most = slots<PAIR>(max_ctas);
  kern<<<Tile<PAIR>::CTAS * (tiles < most ? tiles : most), NUM_THREADS, Tile<PAIR>::SMEM_BYTES, stream>>>(ta, tb, M, N, K, ep, status);
  return static_cast<int>(cudaGetLastError());
}

template <bool A_MN, bool B_MN, int EPI>
int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, const EpiParams& ep,
                int* status, int max_ctas, cudaStream_t stream) {
  return takes_pairs(M, N, max_ctas) ? launch_tiles<true, A_MN, B_MN, EPI>(ta, tb, M, N, K, ep, status, max_ctas, stream)
                                     : launch_tiles<false, A_MN, B_MN, EPI>(ta, tb, M, N, K, ep, status, max_ctas, stream);
}

template <int EPI>
int dispatch_layout(bool a_mn, bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K,
                    const EpiParams& ep, int* status, int max_ctas, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_gemm<false, false, EPI>(ta, tb, M, N, K, ep, status, max_ctas, stream);
  if (!a_mn && b_mn) return launch_gemm<false, true, EPI>(ta, tb, M, N, K, ep, status, max_ctas, stream);
  if (a_mn && b_mn) return launch_gemm<true, true, EPI>(ta, tb, M, N, K, ep, status, max_ctas, stream);
  return launch_gemm<true, false, EPI>(ta, tb, M, N, K, ep, status, max_ctas, stream);
}

int make_operand_maps(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb,
                      bool a_mn, bool b_mn, CUtensorMap* ta, CUtensorMap* tb, int max_ctas = 0) {
  const int b_rows = takes_pairs(M, N, max_ctas) ? Tile<true>::CTA_N : Tile<false>::CTA_N;
  int rc;
  if (!a_mn)
    rc = rlb_make_tmap_2d(ta, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, M, lda * 2, BK, CTA_M,
                          CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = rlb_make_tmap_2d(ta, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, K, lda * 2, 64, BK,
                          CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  if (!b_mn)
    rc = rlb_make_tmap_2d(tb, B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, N, ldb * 2, BK, b_rows,
                          CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = rlb_make_tmap_2d(tb, B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, N, K, ldb * 2, 64, BK,
                          CU_TENSOR_MAP_SWIZZLE_128B);
  return rc;
}

}  // namespace

// ---------------------------------------------------------------- host helpers (shared by all .cu files)
bool rlb_pdl_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("RLB_PDL");
    on = (e && e[0] == '0') ? 0 : 1;
  }
  return on == 1;
}

RlbEncodeTiledFn rlb_get_encode_tiled() {
  static RlbEncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<RlbEncodeTiledFn>(p);
  }
  return fn;
}

int rlb_make_tmap_2d(CUtensorMap* map, const void* base, CUtensorMapDataType dtype, int elem_bytes,
                     uint64_t inner, uint64_t outer, uint64_t pitch_bytes, uint32_t box_inner,
                     uint32_t box_outer, CUtensorMapSwizzle swizzle) {
  RlbEncodeTiledFn enc = rlb_get_encode_tiled();
  if (!enc) return -1;
  (void)elem_bytes;
  // The driver call needs the primary context current on the calling thread. Threads that have made
  // no runtime call yet (autograd's backward threads) get it bound by a no-op runtime call.
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    cudaFree(nullptr);
    ctx_bound = true;
  }
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {pitch_bytes};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, dtype, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return static_cast<int>(r);
}

// ---------------------------------------------------------------- C API
// C = op(A) op(B)^T (+bias) (+C). lda/ldb/ldc in elements; all of them, and the base pointers, must
// keep 16-byte alignment (multiples of 8 elements for bf16). Returns 0, a CUDA error, or a negative
// code for bad arguments.
RLB_API int rlb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                          long long ldb, long long ldc, int a_mn_major, int b_mn_major, int out_fp32,
                          int accumulate, const float* bias, const void* residual, long long ldr, int* status,
                          int max_ctas, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (ldc % (out_fp32 ? 4 : 8)) || (N % 8)) return -2;
  if (residual && ((ldr % 8) || (reinterpret_cast<uintptr_t>(residual) & 15))) return -2;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15)
    return -3;
  CUtensorMap ta, tb;
  int rc = make_operand_maps(A, B, M, N, K, lda, ldb, a_mn_major != 0, b_mn_major != 0, &ta, &tb, max_ctas);
  if (rc) return -100 - rc;
  EpiParams ep{};
  ep.C = C;
  ep.ldc = ldc;
  ep.bias = bias;
  ep.residual = residual;
  ep.ldr = ldr;
  ep.out_fp32 = out_fp32;
  ep.accumulate = accumulate;
  return dispatch_layout<EPI_STORE>(a_mn_major != 0, b_mn_major != 0, ta, tb, M, N, K, ep, status, max_ctas,
                                    static_cast<cudaStream_t>(stream));
}

// out[M, N] (bf16) = epilogue(A W^T) with LayerEpilogue's fields; N, K and all row strides multiples of 8, ldx of 4.
RLB_API int rlb_gemm_layer(const void* A, const void* W, void* out, int M, int N, int K, long long lda, long long ldw, long long ldo,
                           int act_from, float* x, long long ldx, const float* e, const void* step, const void* alpha, const void* nw,
                           const void* nb, int* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldw % 8) || (ldo % 8) || (N % 8) || (K % 8) || (act_from % 8) || (ldx % 4)) return -2;
  if (x && (!alpha || !nw || !nb)) return -2;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(x) |
       reinterpret_cast<uintptr_t>(e) | reinterpret_cast<uintptr_t>(step) | reinterpret_cast<uintptr_t>(nw) | reinterpret_cast<uintptr_t>(nb)) & 15)
    return -3;
  CUtensorMap ta, tb;
  int rc = make_operand_maps(A, W, M, N, K, lda, ldw, false, false, &ta, &tb);
  if (rc) return -100 - rc;
  EpiParams ep{};
  ep.C = out;
  ep.ldc = ldo;
  ep.layer = LayerEpilogue{x, ldx, e, static_cast<const __nv_bfloat16*>(step), static_cast<const __nv_bfloat16*>(alpha),
                           static_cast<const __nv_bfloat16*>(nw), static_cast<const __nv_bfloat16*>(nb), act_from, LinearEpi{}};
  return launch_gemm<false, false, EPI_LAYER>(ta, tb, M, N, K, ep, status, 0, static_cast<cudaStream_t>(stream));
}

// out (bf16) = epilogue(a w^T); N, K and the row strides multiples of 8.
RLB_API int rlb_linear_tiled(const RlbLinear* l, void* stream) {
  if (l->M <= 0 || l->N <= 0 || l->K <= 0) return 0;
  if ((l->lda % 8) || (l->ldw % 8) || (l->ldo % 8) || (l->N % 8) || (l->K % 8) || l->in_f32 || l->out_f32 || l->tile_expert || l->row_scale || l->act == LIN_CAP) return -2;
  if ((reinterpret_cast<uintptr_t>(l->a) | reinterpret_cast<uintptr_t>(l->w) | reinterpret_cast<uintptr_t>(l->out) | reinterpret_cast<uintptr_t>(l->bias)) & 15) return -3;
  if (l->act == LIN_GELU_MUL && (reinterpret_cast<uintptr_t>(l->table) & 7)) return -3;
  CUtensorMap ta, tb;
  int rc = make_operand_maps(l->a, l->w, l->M, l->N, l->K, l->lda, l->ldw, false, false, &ta, &tb);
  if (rc) return -100 - rc;
  EpiParams ep{};
  ep.C = l->out;
  ep.ldc = l->ldo;
  ep.layer.lin = rlb_linear_epi(*l);
  return launch_gemm<false, false, EPI_LINEAR>(ta, tb, l->M, l->N, l->K, ep, l->status, 0, static_cast<cudaStream_t>(stream));
}

// Number of n-tiles the vocab-projection epilogues split N into (size of the partial buffers).
RLB_API int rlb_gemm_num_n_tiles(int N) { return (N + BN - 1) / BN; }

// Fused vocab projection + log-softmax statistics: H[M,K] x W[N,K]^T, logits never stored.
// part_* are scratch of num_n_tiles*M floats each; target_logit is scratch of M floats.
// Outputs (any may be null): logprob[M], entropy[M], lse[M].
RLB_API int rlb_lm_head_logprob(const void* H, const void* W, int M, int N, int K, long long ldh, long long ldw,
                                const int* targets, float inv_temp, float* part_max, float* part_sum,
                                float* part_zsum, float* target_logit, float* logprob, float* entropy,
                                float* lse, float* logits, long long ldz, int* status, void* stream) {
  if (M <= 0) return 0;
  if ((ldh % 8) || (ldw % 8)) return -2;
  if (logits && ((N % 8) || (ldz % 4) || (reinterpret_cast<uintptr_t>(logits) & 15))) return -2;
  CUtensorMap ta, tb;
  int rc = make_operand_maps(H, W, M, N, K, ldh, ldw, false, false, &ta, &tb);
  if (rc) return -100 - rc;
  EpiParams ep{};
  ep.targets = targets;
  ep.inv_temp = inv_temp;
  ep.part_max = part_max;
  ep.part_sum = part_sum;
  ep.part_zsum = part_zsum;
  ep.target_logit = target_logit;
  ep.C = logits;
  ep.ldc = ldz;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rc = logits ? launch_gemm<false, false, EPI_LOGPROB_KEEP>(ta, tb, M, N, K, ep, status, 0, s)
              : launch_gemm<false, false, EPI_LOGPROB>(ta, tb, M, N, K, ep, status, 0, s);
  if (rc) return rc;
  const int parts = (N + BN - 1) / BN;
  launch_combine(s, part_max, part_sum, part_zsum, target_logit, M, parts, logprob, entropy, lse);
  return static_cast<int>(cudaGetLastError());
}

// Folds partials only (used by the vocab-parallel path after the cross-rank exchange).
RLB_API int rlb_logprob_combine(const float* part_max, const float* part_sum, const float* part_zsum,
                                const float* target_logit, int M, int parts, float* logprob, float* entropy,
                                float* lse, void* stream) {
  if (M <= 0) return 0;
  launch_combine(static_cast<cudaStream_t>(stream), part_max, part_sum, part_zsum, target_logit, M, parts, logprob, entropy, lse);
  return static_cast<int>(cudaGetLastError());
}

// Statistics pass only: writes the partials and the target logit, no combine. For a vocab-parallel
// lm_head each rank runs this on its shard; the partials are then exchanged and folded.
RLB_API int rlb_lm_head_partials(const void* H, const void* W, int M, int N, int K, long long ldh,
                                 long long ldw, const int* targets, float inv_temp, float* part_max,
                                 float* part_sum, float* part_zsum, float* target_logit, int* status,
                                 void* stream) {
  if (M <= 0) return 0;
  if ((ldh % 8) || (ldw % 8)) return -2;
  CUtensorMap ta, tb;
  int rc = make_operand_maps(H, W, M, N, K, ldh, ldw, false, false, &ta, &tb);
  if (rc) return -100 - rc;
  EpiParams ep{};
  ep.targets = targets;
  ep.inv_temp = inv_temp;
  ep.part_max = part_max;
  ep.part_sum = part_sum;
  ep.part_zsum = part_zsum;
  ep.target_logit = target_logit;
  return launch_gemm<false, false, EPI_LOGPROB>(ta, tb, M, N, K, ep, status, 0, static_cast<cudaStream_t>(stream));
}

// Backward of the fused projection: recomputes logits tile by tile and writes
// dZ[M,N] = (coef*(onehot - p) - ent_coef * p * (logp + H)) * inv_temp in bf16.
RLB_API int rlb_lm_head_dlogits(const void* H, const void* W, void* dZ, int M, int N, int K, long long ldh,
                                long long ldw, long long lddz, const int* targets, float inv_temp,
                                const float* lse, const float* coef, const float* ent_coef,
                                const float* entropy, int* status, void* stream) {
  if (M <= 0) return 0;
  if ((ldh % 8) || (ldw % 8) || (lddz % 8) || (N % 8)) return -2;
  CUtensorMap ta, tb;
  int rc = make_operand_maps(H, W, M, N, K, ldh, ldw, false, false, &ta, &tb);
  if (rc) return -100 - rc;
  EpiParams ep{};
  ep.C = dZ;
  ep.ldc = lddz;
  ep.targets = targets;
  ep.inv_temp = inv_temp;
  ep.lse = lse;
  ep.coef = coef;
  ep.ent_coef = ent_coef;
  ep.entropy = entropy;
  return launch_gemm<false, false, EPI_DLOGITS>(ta, tb, M, N, K, ep, status, 0, static_cast<cudaStream_t>(stream));
}

// The same gradient from kept logits (rlb_lm_head_logprob). N and lddz multiples of 8, ldz of 4, both starting on 16 bytes.
RLB_API int rlb_lm_head_dlogits_kept(const float* z, void* dZ, int M, int N, long long ldz, long long lddz, const int* targets, float inv_temp,
                                     const float* lse, const float* coef, const float* ent_coef, const float* entropy, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if ((ldz % 4) || (lddz % 8) || (N % 8) || M > 65535) return -2;
  if ((reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(dZ)) & 15) return -3;
  dlogits_kept_kernel<<<dim3((N + KEPT_COLS - 1) / KEPT_COLS, M), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      z, static_cast<__nv_bfloat16*>(dZ), N, ldz, lddz, targets, inv_temp, lse, coef, ent_coef, entropy);
  return static_cast<int>(cudaGetLastError());
}
