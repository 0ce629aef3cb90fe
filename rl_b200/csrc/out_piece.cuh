// Output of a 32-row x 64-column piece of an accumulator through shared memory, shared by the GEMM kernels' epilogues.
#pragma once

#include "common.cuh"

namespace rlb {
constexpr int OUT_COLS = 64;                                  // columns that an epilogue warp passes through shared memory at a time
constexpr int OUT_WARP_BYTES = 32 * OUT_COLS * 4;

struct OutPiece {
  void* C;              // bf16 or fp32
  long long ldc;
  const float* bias;    // [N] or null
  const void* residual; // bf16 [M, ldr] or null
  long long ldr;
  int out_fp32;
  int accumulate;       // C += result
};

// One 32-row x 64-column piece of fp32 values on its way out: lanes put their rows down, then the warp reads whole rows, so that every
// access to global memory covers full 32-byte sectors (rows written by single lanes made the weight gradient's fp32 read-add-write
// as long as its main loop). 16-byte chunks are permuted within the row so that both directions are free of bank conflicts.
__device__ __forceinline__ uint32_t out_chunk(uint32_t base, int r, int q) { return base + r * (OUT_COLS * 4) + ((q ^ (r & 7)) << 4); }
__device__ __forceinline__ void st_shared_f4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void add_bf16x4(float4& v, uint32_t lo, uint32_t hi) {
  const float2 a = unpack_bf16x2(lo), b = unpack_bf16x2(hi);
  v.x += a.x; v.y += a.y; v.z += b.x; v.w += b.y;
}

// Writes the staged piece: rows row0.., columns col.. of C, with bias, residual and the old values where `ep` (an OutPiece or a struct with its
// fields) has them. Old values (accumulation), and the residual of a bf16 output, are requested in the same layout before the warp has met, so
// that they arrive while it stages the piece; the residual of an fp32 output is read row by row.
template <typename Out>
__device__ __forceinline__ void store_piece(const Out& ep, uint32_t buf, int row0, int col, int M, int N, int lane) {
  if (ep.out_fp32) {
    const int q = lane & 15, c = col + q * 4;
    const bool in = c < N;                 // N is a multiple of 8
    float4 old[16];
    float* dst = reinterpret_cast<float*>(ep.C) + static_cast<long long>(row0 + (lane >> 4)) * ep.ldc + c;
    if (ep.accumulate) {
#pragma unroll
      for (int i = 0; i < 16; ++i)
        old[i] = in && row0 + 2 * i + (lane >> 4) < M ? *reinterpret_cast<const float4*>(dst + 2 * i * ep.ldc) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ep.bias && in) bias = make_float4(ep.bias[c], ep.bias[c + 1], ep.bias[c + 2], ep.bias[c + 3]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int r = 2 * i + (lane >> 4);
      float4 v = ld_shared_f4(out_chunk(buf, r, q));
      if (!in || row0 + r >= M) continue;
      v.x += bias.x; v.y += bias.y; v.z += bias.z; v.w += bias.w;
      if (ep.residual) {
        const uint2 o = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(ep.residual) + static_cast<long long>(row0 + r) * ep.ldr + c);
        add_bf16x4(v, o.x, o.y);
      }
      if (ep.accumulate) { v.x += old[i].x; v.y += old[i].y; v.z += old[i].z; v.w += old[i].w; }
      *reinterpret_cast<float4*>(dst + 2 * i * ep.ldc) = v;
    }
  } else {
    const int q = (lane & 7) * 2, c = col + q * 4;
    const bool in = c < N;
    uint4 res[8], old[8];
    const __nv_bfloat16* rsd = reinterpret_cast<const __nv_bfloat16*>(ep.residual) + static_cast<long long>(row0 + (lane >> 3)) * ep.ldr + c;
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(ep.C) + static_cast<long long>(row0 + (lane >> 3)) * ep.ldc + c;
    if (ep.residual) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        res[i] = in && row0 + 4 * i + (lane >> 3) < M ? *reinterpret_cast<const uint4*>(rsd + 4 * i * ep.ldr) : make_uint4(0, 0, 0, 0);
    }
    if (ep.accumulate) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        old[i] = in && row0 + 4 * i + (lane >> 3) < M ? *reinterpret_cast<const uint4*>(dst + 4 * i * ep.ldc) : make_uint4(0, 0, 0, 0);
    }
    float4 b0 = make_float4(0.f, 0.f, 0.f, 0.f), b1 = b0;
    if (ep.bias && in) {
      b0 = make_float4(ep.bias[c], ep.bias[c + 1], ep.bias[c + 2], ep.bias[c + 3]);
      b1 = make_float4(ep.bias[c + 4], ep.bias[c + 5], ep.bias[c + 6], ep.bias[c + 7]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 4 * i + (lane >> 3);
      float4 u = ld_shared_f4(out_chunk(buf, r, q)), v = ld_shared_f4(out_chunk(buf, r, q + 1));
      if (!in || row0 + r >= M) continue;
      u.x += b0.x; u.y += b0.y; u.z += b0.z; u.w += b0.w;
      v.x += b1.x; v.y += b1.y; v.z += b1.z; v.w += b1.w;
      if (ep.residual) { add_bf16x4(u, res[i].x, res[i].y); add_bf16x4(v, res[i].z, res[i].w); }
      if (ep.accumulate) { add_bf16x4(u, old[i].x, old[i].y); add_bf16x4(v, old[i].z, old[i].w); }
      *reinterpret_cast<uint4*>(dst + 4 * i * ep.ldc) = make_uint4(pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w), pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
    }
  }
  __syncwarp();      // the buffer may be written again
}

// The same for fp32 values that are stored as they are and not read again soon: eight chunks a lane are read from the buffer before the first is
// stored (with store_piece's tests and single chunks the kept logits of 4096 x 128256 x 2048 took 1.70 ms, now 1.55).
__device__ __forceinline__ void stream_piece(float* C, long long ldc, uint32_t buf, int row0, int col, int M, int N, int lane) {
  const int q = lane & 15, c = col + q * 4, half = lane >> 4;
  float* dst = C + static_cast<long long>(row0 + half) * ldc + c;
  const int live = c < N ? M - row0 - half : 0;      // rows below M
  __syncwarp();
#pragma unroll
  for (int b = 0; b < 16; b += 8) {
    float4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = ld_shared_f4(out_chunk(buf, 2 * (b + i) + half, q));
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (2 * (b + i) < live) __stcs(reinterpret_cast<float4*>(dst + 2 * (b + i) * ldc), v[i]);
  }
  __syncwarp();
}
}  // namespace rlb
