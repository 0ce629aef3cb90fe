// Expert products for few tokens (decode steps): every live expert's weights are a stream that is read once, its tokens a handful of columns.
//
// As in gemm_skinny.cu the operands are swapped: 128 rows of an expert's weight form the M side of the tcgen05 MMA, its tokens, padded to NT = 32 or
// 64 rows, the N side. Persistent CTAs, one per SM, take (tile of tokens, 128 weight rows) in turn; the producer runs ahead over the tiles, so that
// 160 KB per SM are in flight also between tiles. With GLU a tile is 64 gate rows on the 64 matching up rows and the epilogue writes
// silu(gate) * up, which saves the unit's own pass. Rows of padding are computed from whatever stands there and written, and never read.
// Bound by the weights' stream. The 128-row tiles of the grouped GEMM before it read 128 rows of tokens, nearly all padding, beside every 256 weight rows:
// 32 tokens, 8 of 128 experts each, width 2048, 768 per expert: both products 290 us, and 15 us for the unit, now 190 us where 160 us of weights are read.
#include "common.cuh"

namespace {
using namespace rlb;
constexpr int MS_BK = 64;
constexpr int MS_STAGES = 8;
constexpr int MS_THREADS = 192;

template <int NT>
struct MsCfg {
  static constexpr int W_BYTES = 128 * MS_BK * 2;
  static constexpr int X_BYTES = NT * MS_BK * 2;
  static constexpr int STAGE = W_BYTES + X_BYTES;
  static constexpr int LD = 132;      // floats of a staged token: 128 weight rows, offset against bank conflicts
  static constexpr int SMEM = MS_STAGES * STAGE + NT * LD * 4 + 256 + 1024;
};

struct MsArgs {
  const int* tile_expert;   // [max_tiles] expert of every NT rows; live tiles come first, then -1
  int max_tiles, w_tiles;   // w_tiles: tiles of an expert's output columns
  int n, K;                 // output columns, reduction
  __nv_bfloat16* out;
  long long ldo;
  int* status;
};

template <int NT, bool GLU>
__global__ void __launch_bounds__(MS_THREADS, 1)
moe_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, MsArgs g) {
  using Cfg = MsCfg<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* staged = reinterpret_cast<float*>(smem + MS_STAGES * Cfg::STAGE);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(staged + NT * Cfg::LD);
  uint64_t* empty_bar = full_bar + MS_STAGES;
  uint64_t* tfull_bar = empty_bar + MS_STAGES;   // [2]
  uint64_t* tempty_bar = tfull_bar + 2;          // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < MS_STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&tfull_bar[a]), 1);
      mbar_init(smem_u32(&tempty_bar[a]), 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
    prefetch_tmap(&tmap_w);
    prefetch_tmap(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 2 * NT);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_sync();
  const int num_k = g.K / MS_BK, work = g.max_tiles * g.w_tiles;

  if (warp == 0) {
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < work && ok; w += gridDim.x) {
        const int tile = w / g.w_tiles, wt = w - tile * g.w_tiles, e = g.tile_expert[tile];
        if (e < 0) break;
        const int row0 = GLU ? e * 2 * g.n + wt * 64 : e * g.n + wt * 128;
        for (int kb = 0; kb < num_k; ++kb) {
          if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, abort_flag, g.status, RLB_ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          const uint32_t bar = smem_u32(&full_bar[stage]), dst = smem_u32(smem + stage * Cfg::STAGE);
          mbar_arrive_expect_tx(bar, Cfg::STAGE);
          tma_load_2d(dst, &tmap_w, bar, kb * MS_BK, row0);
          if (GLU) tma_load_2d(dst + Cfg::W_BYTES / 2, &tmap_w, bar, kb * MS_BK, row0 + g.n);
          tma_load_2d(dst + Cfg::W_BYTES, &tmap_x, bar, kb * MS_BK, tile * NT);
          if (++stage == MS_STAGES) {
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
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(128, NT, false, false);
      uint32_t stage = 0, phase = 0, local = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < work && ok; w += gridDim.x, ++local) {
        if (g.tile_expert[w / g.w_tiles] < 0) break;
        const uint32_t acc = local & 1;
        if (!mbar_wait(smem_u32(&tempty_bar[acc]), ((local >> 1) & 1) ^ 1, abort_flag, g.status, RLB_ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        for (int kb = 0; kb < num_k; ++kb) {
          if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag, g.status, RLB_ERR_WAIT_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t addr = smem_u32(smem + stage * Cfg::STAGE);
          const uint64_t a = make_smem_desc_sw128(addr, 16, 1024), b = make_smem_desc_sw128(addr + Cfg::W_BYTES, 16, 1024);
#pragma unroll
          for (int kk = 0; kk < MS_BK / 16; ++kk) umma_f16(tmem_base + acc * NT, a + kk * 2, b + kk * 2, idesc, (kb | kk) != 0 ? 1u : 0u);
          umma_commit(smem_u32(&empty_bar[stage]));
          if (++stage == MS_STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit(smem_u32(&tfull_bar[acc]));
      }
    }
  } else {
    const int quarter = warp & 3, r = quarter * 32 + lane, t = threadIdx.x - 64;
    uint32_t local = 0;
    bool ok = true;
    for (int w = blockIdx.x; w < work; w += gridDim.x, ++local) {
      const int tile = w / g.w_tiles, wt = w - tile * g.w_tiles;
      if (g.tile_expert[tile] < 0) break;
      const uint32_t acc = local & 1;
      ok = ok && mbar_wait(smem_u32(&tfull_bar[acc]), (local >> 1) & 1, abort_flag, g.status, RLB_ERR_WAIT_TMEM_FULL);
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < NT; c += 32) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * NT + c, v);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) staged[(c + i) * Cfg::LD + r] = __uint_as_float(v[i]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ok) {      // two output columns per thread, rows one after the other
        constexpr int COLS = GLU ? 64 : 128, PAIRS = COLS / 2;
        const int n = (t % PAIRS) * 2;
        if (wt * COLS + n < g.n) {
          __nv_bfloat16* dst = g.out + static_cast<long long>(tile) * NT * g.ldo + wt * COLS + n;
#pragma unroll 4
          for (int c = t / PAIRS; c < NT; c += 128 / PAIRS) {
            float2 v = *reinterpret_cast<const float2*>(staged + c * Cfg::LD + n);
            if (GLU) {
              const float2 u = *reinterpret_cast<const float2*>(staged + c * Cfg::LD + 64 + n);
              // the products are rounded as a row of them in memory would be
              const float2 a = unpack_bf16x2(pack_bf16x2(v.x, v.y)), b = unpack_bf16x2(pack_bf16x2(u.x, u.y));
              v = make_float2(a.x / (1.f + __expf(-a.x)) * b.x, a.y / (1.f + __expf(-a.y)) * b.y);
            }
            *reinterpret_cast<uint32_t*>(dst + c * g.ldo) = pack_bf16x2(v.x, v.y);
          }
        }
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * NT);
  }
}

template <int NT, bool GLU>
int launch_ms(const CUtensorMap& tw, const CUtensorMap& tx, const MsArgs& g, cudaStream_t s) {
  auto kern = moe_skinny_kernel<NT, GLU>;
  static bool configured = false;
  static int sms = 0;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MsCfg<NT>::SMEM);
    if (e != cudaSuccess) return static_cast<int>(e);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    configured = true;
  }
  const int work = g.max_tiles * g.w_tiles;
  rlb_launch_pdl(kern, dim3(work < sms ? work : sms), dim3(MS_THREADS), MsCfg<NT>::SMEM, s, tw, tx, g);
  return static_cast<int>(cudaGetLastError());
}
}  // namespace

// out [mpad, n] = x [mpad, K] W[e]^T per tile of `rows` (32 or 64) rows, e = tile_expert[tile]; live tiles first, then -1 (left untouched).
// glu: W [E, 2n, K] = [gate | up] and out = silu(gate) * up, n a multiple of 64; else W [E, n, K]. K a multiple of 64, n of 8. Every row of a live
// tile is written; those of padding hold nothing of meaning.
RLB_API int rlb_moe_skinny(const void* x, long long ldx, const void* w, void* out, long long ldo, int mpad, int rows, int n, int K, int num_experts, const int* tile_expert, int glu,
                           int* status, void* stream) {
  if (mpad <= 0 || n <= 0 || K <= 0) return 0;
  if ((rows != 32 && rows != 64) || (mpad % rows) || (K % 64) || (n % 8) || (glu && (n % 64)) || (ldx % 8) || (ldo % 2)) return -2;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) return -3;
  CUtensorMap tw, tx;
  int rc = rlb_make_tmap_2d(&tw, w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, static_cast<uint64_t>(num_experts) * n * (glu ? 2 : 1), static_cast<uint64_t>(K) * 2, MS_BK, glu ? 64 : 128,
                            CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return -100 - rc;
  rc = rlb_make_tmap_2d(&tx, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, mpad, ldx * 2, MS_BK, rows, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return -100 - rc;
  MsArgs g{tile_expert, mpad / rows, glu ? n / 64 : (n + 127) / 128, n, K, static_cast<__nv_bfloat16*>(out), ldo, status};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (rows == 32) return glu ? launch_ms<32, true>(tw, tx, g, s) : launch_ms<32, false>(tw, tx, g, s);
  return glu ? launch_ms<64, true>(tw, tx, g, s) : launch_ms<64, false>(tw, tx, g, s);
}
