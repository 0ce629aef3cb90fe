// Memory-bound transformer kernels for sm_100a: RMSNorm, RoPE, SwiGLU, embedding, fused AdamW with a
// split fp32 master (bf16 + 16 low bits), gradient-norm partials, and the ClippedPG loss.
// All of them move 16 bytes per thread per access and keep the arithmetic in fp32.
//
// They stand in for the HF-eager / Transformer-Engine fused modules of the reference
// (nemo_rl/models/megatron/setup.py:1103-1110), torch.optim.AdamW
// (examples/configs/grpo_math_1B.yaml:344-350) and the torch-eager ClippedPGLossFn
// (nemo_rl/algorithms/loss/loss_functions.py:374-788).
#include "common.cuh"

#include <climits>

#include <math.h>

namespace {
using namespace rlb;

struct alignas(16) BF8 {
  uint32_t w[4];
};
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const BF8 v = *reinterpret_cast<const BF8*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = unpack_bf16x2(v.w[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  BF8 v;
#pragma unroll
  for (int i = 0; i < 4; ++i) v.w[i] = pack_bf16x2(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<BF8*>(p) = v;
}

// ------------------------------------------------------------------ RMSNorm
// y = x * rsqrt(mean(x^2) + eps) * w ; optional residual: h = x + res is normalised and written back
// to `res_out` (the new residual stream). One CTA per row; d must be a multiple of 8.
__global__ void rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                   __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out,
                                   int d, long long x_stride, long long y_stride, float eps) {
  pdl_sync();
  __shared__ float red[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * x_stride;
  const __nv_bfloat16* rr = res ? res + row * static_cast<long long>(d) : nullptr;
  __nv_bfloat16* ro = res_out ? res_out + row * static_cast<long long>(d) : nullptr;
  float ss = 0.f;
  for (int i = threadIdx.x * 8; i < d; i += blockDim.x * 8) {
    float f[8];
    load8(xr + i, f);
    if (rr) {
      float g[8];
      load8(rr + i, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
      // the normalised value must be the bf16-rounded residual stream, as a separate add would give
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16(f[j]));
      store8(ro + i, f);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / d + eps);
  if (rstd_out && threadIdx.x == 0) rstd_out[row] = rstd;
  const __nv_bfloat16* src = rr ? ro : xr;
  __nv_bfloat16* yr = y + row * y_stride;
  for (int i = threadIdx.x * 8; i < d; i += blockDim.x * 8) {
    float f[8], g[8];
    load8(src + i, f);
    load8(w + i, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * rstd * g[j];
    store8(yr + i, f);
  }
}

// The same for rows that fit the registers of one CTA, NV pieces of 8 elements a thread: all loads in flight at once, the row stays between the two
// passes, and small CTAs, many to an SM, hide one another's barrier. Timed with a flushed cache against the kernel above / a warp per row, us:
// d 2048: 600 rows 8.1 -> 8.0, 4000 14.6 -> 12.1, 20000 35.7 -> 30.7; d 4096: 600 10.1 -> 8.3, 4000 22.9 -> 16.6, 20000 70.4 -> 54.3 (6.0 TB/s);
// d 5120: 4000 28.6 -> 20.2, 20000 98.2 -> 68.1. Two and eight pieces were slower above d 1024; with a
// residual, which waits for two rows and stores one more, two are sooner done up to 4096 (one row of 2048, four / two / the kernel above: 2.2, 1.8, 2.0; 4000
// of 4096 21.6, 19.3, 22.8).
template <int NV, bool RES>
__global__ void __launch_bounds__(256) rmsnorm_regs_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res, const __nv_bfloat16* __restrict__ w,
                                                           __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out,
                                                           int d, long long x_stride, long long y_stride, float eps) {
  pdl_sync();
  __shared__ float red[8];
  const long long row = blockIdx.x;
  const int threads = blockDim.x;
  const __nv_bfloat16* xr = x + row * x_stride;
  BF8 v[NV], r[NV], g[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * threads) * 8;
    v[j].w[0] = v[j].w[1] = v[j].w[2] = v[j].w[3] = 0u;
    if (i < d) {
      v[j] = *reinterpret_cast<const BF8*>(xr + i);
      if (RES) r[j] = *reinterpret_cast<const BF8*>(res + row * d + i);
    }
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * threads) * 8;
    if (i < d) g[j] = *reinterpret_cast<const BF8*>(w + i);
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * threads) * 8;
    if (RES && i < d) {      // the normalised value is the bf16-rounded residual stream, as a separate add would give
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(v[j].w[k]), e = unpack_bf16x2(r[j].w[k]);
        v[j].w[k] = pack_bf16x2(f.x + e.x, f.y + e.y);
      }
      *reinterpret_cast<BF8*>(res_out + row * d + i) = v[j];
    }
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = unpack_bf16x2(v[j].w[k]);
      t += f.x * f.x + f.y * f.y;
    }
    ss += t;
  }
  ss = warp_sum(ss);
  if (threads > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.f;
    for (int i = 0; i < (threads >> 5); ++i) ss += red[i];
  }
  const float rstd = rsqrtf(ss / d + eps);
  if (rstd_out && threadIdx.x == 0) rstd_out[row] = rstd;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * threads) * 8;
    if (i < d) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(v[j].w[k]), u = unpack_bf16x2(g[j].w[k]);
        v[j].w[k] = pack_bf16x2(f.x * rstd * u.x, f.y * rstd * u.y);
      }
      *reinterpret_cast<BF8*>(y + row * y_stride + i) = v[j];
    }
  }
}

// The same without a residual for many short rows: one warp per row, which stays in registers between the two passes, all its loads in flight and no
// barrier. NV: pieces of 8 elements per lane. d 1024, 20000 rows: 20.9 us (a CTA per row 26.4), 2400 rows 8.8 either way.
template <int NV>
__global__ void __launch_bounds__(256, 2) rmsnorm_rows_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                                                           float* __restrict__ rstd_out, long long rows, int d, long long x_stride, long long y_stride, float eps) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const __nv_bfloat16* xr = x + row * x_stride;
  __nv_bfloat16* yr = y + row * y_stride;
  BF8 v[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (lane + 32 * j) * 8;
    if (i < d) v[j] = *reinterpret_cast<const BF8*>(xr + i);
    else v[j].w[0] = v[j].w[1] = v[j].w[2] = v[j].w[3] = 0u;
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = unpack_bf16x2(v[j].w[k]);
      t += f.x * f.x + f.y * f.y;
    }
    ss += t;
  }
  ss = warp_sum(ss);
  const float rstd = rsqrtf(ss / d + eps);
  if (rstd_out && lane == 0) rstd_out[row] = rstd;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (lane + 32 * j) * 8;
    if (i < d) {
      float g[8];
      load8(w + i, g);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 f = unpack_bf16x2(v[j].w[k]);
        v[j].w[k] = pack_bf16x2(f.x * rstd * g[2 * k], f.y * rstd * g[2 * k + 1]);
      }
      *reinterpret_cast<BF8*>(yr + i) = v[j];
    }
  }
}

// Gradient for d up to 4096: a CTA takes ROWS rows at a time, so that a barrier serves all of them, keeps them in registers, NV pieces of 8 columns a
// thread, and has requested the next ones before it works on these. As many rows as the registers hold: a requested value that is spilled is waited for
// at once. With a row more (256 threads of 128 registers, 56 to 100 bytes of them spilled) rows of 2048 were no sooner done than without requests ahead.
// 20000 rows, one launch after the other, the sums of the weight gradient included, one row at a time or four without requests / with spills / now, us: of 512
// 41 / 47 / 29, of 1024 64 / 64 / 37, of 2048 82 / 82 / 60, of 4096 170 / 128 / 113; 4000 of 2048 29 / 25 / 21, of 4096 51 / 35 / 31; 16 of 1024
// 8.3 / 10.3 / 8.3.
template <int NV, int ROWS, int THREADS>
__global__ void __launch_bounds__(THREADS, 2) rmsnorm_bwd_rows_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                                                  const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx,
                                                                  float* __restrict__ dw_partial, int rows, int d, long long x_stride, long long dy_stride, int add_to_dx) {
  __shared__ float red[2][ROWS][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, threads = blockDim.x;
  BF8 fw[NV];
  float acc[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int i = (threadIdx.x + v * threads) * 8;
#pragma unroll
    for (int k = 0; k < 4; ++k) fw[v].w[k] = 0u;
    if (i < d) fw[v] = *reinterpret_cast<const BF8*>(w + i);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[v][k] = 0.f;
  }
  BF8 nx[ROWS][NV], nd[ROWS][NV];
  float nr[ROWS];
  auto request = [&](long long row0) {
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const long long row = row0 + static_cast<long long>(q) * gridDim.x;
      nr[q] = row < rows ? rstd[row] : 0.f;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int i = (threadIdx.x + v * threads) * 8;
#pragma unroll
        for (int k = 0; k < 4; ++k) nx[q][v].w[k] = nd[q][v].w[k] = 0u;
        if (row < rows && i < d) {
          nx[q][v] = *reinterpret_cast<const BF8*>(x + row * x_stride + i);
          nd[q][v] = *reinterpret_cast<const BF8*>(dy + row * dy_stride + i);
        }
      }
    }
  };
  const long long step = static_cast<long long>(gridDim.x) * ROWS;
  request(blockIdx.x);
  int turn = 0;
  for (long long row0 = blockIdx.x; row0 < rows; row0 += step, turn ^= 1) {
    BF8 vx[ROWS][NV], vd[ROWS][NV];
    float rs[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      rs[q] = nr[q];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        vx[q][v] = nx[q][v];
        vd[q][v] = nd[q][v];
      }
    }
    request(row0 + step);
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      float dot = 0.f;
#pragma unroll
      for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 a = unpack_bf16x2(vx[q][v].w[k]), b = unpack_bf16x2(vd[q][v].w[k]), g = unpack_bf16x2(fw[v].w[k]);
          dot += b.x * g.x * a.x + b.y * g.y * a.y;
          acc[v][2 * k] += b.x * a.x * rs[q];
          acc[v][2 * k + 1] += b.y * a.y * rs[q];
        }
      dot = warp_sum(dot);
      if (lane == 0) red[turn][q][warp] = dot;
    }
    __syncthreads();      // (the other half of `red` is written next: everyone has read it by the next barrier but one)
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const long long row = row0 + static_cast<long long>(q) * gridDim.x;
      float dot = 0.f;
      for (int t = 0; t < warps; ++t) dot += red[turn][q][t];
      const float c = dot * rs[q] * rs[q] / d;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int i = (threadIdx.x + v * threads) * 8;
        if (i >= d || row >= rows) continue;
        __nv_bfloat16* dst = dx + row * static_cast<long long>(d) + i;
        float o[8];
        if (add_to_dx) load8(dst, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 a = unpack_bf16x2(vx[q][v].w[k]), b = unpack_bf16x2(vd[q][v].w[k]), g = unpack_bf16x2(fw[v].w[k]);
          const float v0 = rs[q] * (b.x * g.x - a.x * c), v1 = rs[q] * (b.y * g.y - a.y * c);
          o[2 * k] = add_to_dx ? o[2 * k] + v0 : v0;
          o[2 * k + 1] = add_to_dx ? o[2 * k + 1] + v1 : v1;
        }
        store8(dst, o);
      }
    }
  }
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int i = (threadIdx.x + v * threads) * 8;
    if (i >= d) continue;
    float* p = dw_partial + static_cast<long long>(blockIdx.x) * d + i;
    *reinterpret_cast<float4*>(p) = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(acc[v][4], acc[v][5], acc[v][6], acc[v][7]);
  }
}

// dx = rstd * (dy*w - x * rstd^2 * mean(dy*w*x)); dw partial per CTA (rows strided over the grid).
__global__ void rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                                   __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_partial, int rows,
                                   int d, long long x_stride, long long dy_stride, int add_to_dx) {
  __shared__ float red[32];
  // Each thread owns fixed column groups, so the dw partial lives in registers (d <= 8 * 8 * blockDim).
  constexpr int MAXV = 8;
  float dwacc[MAXV][8];
#pragma unroll
  for (int a = 0; a < MAXV; ++a)
#pragma unroll
    for (int j = 0; j < 8; ++j) dwacc[a][j] = 0.f;

  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16* xr = x + row * x_stride;
    const __nv_bfloat16* dyr = dy + row * dy_stride;
    const float rs = rstd[row];
    float dot = 0.f;
    {
      int a = 0;
      for (int i = threadIdx.x * 8; i < d; i += blockDim.x * 8, ++a) {
        float fx[8], fd[8], fw[8];
        load8(xr + i, fx);
        load8(dyr + i, fd);
        load8(w + i, fw);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dot += fd[j] * fw[j] * fx[j];
          if (a < MAXV) dwacc[a][j] += fd[j] * fx[j] * rs;
        }
      }
    }
    dot = block_sum(dot, red);
    const float c = dot * rs * rs / d;
    __nv_bfloat16* dxr = dx + row * static_cast<long long>(d);
    for (int i = threadIdx.x * 8; i < d; i += blockDim.x * 8) {
      float fx[8], fd[8], fw[8], o[8];
      load8(xr + i, fx);
      load8(dyr + i, fd);
      load8(w + i, fw);
      if (add_to_dx) load8(dxr + i, o);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float v = rs * (fd[j] * fw[j] - fx[j] * c);
        o[j] = add_to_dx ? o[j] + v : v;
      }
      store8(dxr + i, o);
    }
  }
  int a = 0;
  for (int i = threadIdx.x * 8; i < d; i += blockDim.x * 8, ++a) {
    if (a < MAXV) {
      float* p = dw_partial + static_cast<long long>(blockIdx.x) * d + i;
      *reinterpret_cast<float4*>(p) = make_float4(dwacc[a][0], dwacc[a][1], dwacc[a][2], dwacc[a][3]);
      *reinterpret_cast<float4*>(p + 4) = make_float4(dwacc[a][4], dwacc[a][5], dwacc[a][6], dwacc[a][7]);
    }
  }
}

// Column sums of a [parts, d] fp32 matrix, added into (or written to) a gradient buffer: 32 columns a block, the parts dealt out to its eight warps
// (a thread walked all of them, 17 us for 296 parts of 4096; now 8).
__global__ void __launch_bounds__(256) colsum_kernel(const float* __restrict__ partial, int parts, int d, float* __restrict__ out_f32,
                                                     __nv_bfloat16* __restrict__ out_bf16, int accumulate) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < d) {
#pragma unroll 8
    for (int p = warp; p < parts; p += 8) s += partial[static_cast<long long>(p) * d + c];
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || c >= d) return;
  for (int w = 1; w < 8; ++w) s += red[w][lane];
  if (out_f32) out_f32[c] = accumulate ? out_f32[c] + s : s;
  if (out_bf16) out_bf16[c] = __float2bfloat16(accumulate ? __bfloat162float(out_bf16[c]) + s : s);
}

// ------------------------------------------------------------------ RoPE (HF rotate_half convention)
// In place on `heads` consecutive heads of width D starting at `x` in each row. sign=+1 forward,
// -1 backward (the inverse rotation, which is the transpose). One warp per (row, head).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos,
                            const float* __restrict__ inv_freq, long long rows, int heads, int D,
                            long long row_stride, float sign) {
  pdl_sync();
  const long long wid = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= rows * heads) return;
  const long long row = wid / heads;
  const int head = static_cast<int>(wid - row * heads);
  __nv_bfloat16* p = x + row * row_stride + static_cast<long long>(head) * D;
  const float ps = static_cast<float>(pos[row]);
  const int half = D >> 1;
  for (int i = lane * 2; i < half; i += 64) {
    const float2 lo = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p + i));
    const float2 hi = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p + i + half));
    float s0, c0, s1, c1;
    sincosf(ps * inv_freq[i], &s0, &c0);
    sincosf(ps * inv_freq[i + 1], &s1, &c1);
    s0 *= sign;
    s1 *= sign;
    *reinterpret_cast<uint32_t*>(p + i) = pack_bf16x2(lo.x * c0 - hi.x * s0, lo.y * c1 - hi.y * s1);
    *reinterpret_cast<uint32_t*>(p + i + half) = pack_bf16x2(hi.x * c0 + lo.x * s0, hi.y * c1 + lo.y * s1);
  }
}

// The same for head dimensions that are multiples of 16 and 16-byte aligned rows: a block takes `block_rows` rows, computes their angles once
// and moves 16 bytes at a time (one warp per head recomputed 64 sines and cosines for each: 20480 rows of 40 heads of 128 took 169 us,
// now 85 us, 4.4 TB/s). From so many heads on that the SMs have several warps anyway: with fewer, a warp per head does not wait for a block's
// angles (us in a captured chain, warp per head / block: 40 heads of 128, 64 rows 1.9 / 2.4, 128 rows 2.5 / 2.2; heads of 64, 8 rows 1.6 / 1.7, 64 rows 1.9 / 1.8).
__global__ void __launch_bounds__(256) rope_rows_kernel(__nv_bfloat16* __restrict__ x, const int* __restrict__ pos, const float* __restrict__ inv_freq, long long rows, int heads, int D,
                                                        long long row_stride, float sign, int block_rows) {
  extern __shared__ __align__(16) float2 rope_cs[];
  pdl_sync();
  const int half = D >> 1, pieces = half >> 3, per_row = heads * pieces;
  const long long row0 = static_cast<long long>(blockIdx.x) * block_rows;
  const int n = static_cast<int>(rows - row0 < block_rows ? rows - row0 : block_rows);
  rope_table(rope_cs, pos + row0, inv_freq, n, half, sign);
  for (int i = threadIdx.x; i < n * per_row; i += blockDim.x) {
    const int r = i / per_row, w = i - r * per_row, h = w / pieces, c = w - h * pieces;
    uint4* lo = reinterpret_cast<uint4*>(x + (row0 + r) * row_stride + static_cast<long long>(h) * D + c * 8);
    uint4* hi = lo + pieces;
    uint4 a = *lo, b = *hi;
    rope_turn8(a, b, rope_cs + r * half + c * 8);
    *lo = a;
    *hi = b;
  }
}

// RMSNorms of the query and key heads of fused [q | k | v] rows in one pass; v is copied unless out is x. D a multiple of 64, at most 256:
// every lane has D / 32 elements of a head, in pairs 64 apart.
__global__ void __launch_bounds__(256) qk_rmsnorm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ wq, const __nv_bfloat16* __restrict__ wk, __nv_bfloat16* out,
                                                             float* __restrict__ rstd_out, long long rows, int Hq, int Hkv, int D, long long x_stride, long long out_stride, float eps) {
  pdl_sync();
  const int lane = threadIdx.x & 31, heads = Hq + 2 * Hkv;
  const long long item = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (item >= rows * heads) return;
  const long long row = item / heads;
  const int h = static_cast<int>(item - row * heads);
  const __nv_bfloat16* p = x + row * x_stride + static_cast<long long>(h) * D;
  __nv_bfloat16* q = out + row * out_stride + static_cast<long long>(h) * D;
  if (h >= Hq + Hkv) {
    if (p != q)
      for (int i = lane * 2; i < D; i += 64) *reinterpret_cast<uint32_t*>(q + i) = *reinterpret_cast<const uint32_t*>(p + i);
    return;
  }
  const __nv_bfloat16* w = h < Hq ? wq : wk;
  float2 v[4];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = j * 64 < D ? unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p + lane * 2 + j * 64)) : make_float2(0.f, 0.f);
    ss += v[j].x * v[j].x + v[j].y * v[j].y;
  }
  ss = warp_sum(ss);
  const float rs = rsqrtf(ss / D + eps);
  if (rstd_out && lane == 0) rstd_out[row * (Hq + Hkv) + h] = rs;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j * 64 < D) {
      const int i = lane * 2 + j * 64;
      const float2 g = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + i));
      *reinterpret_cast<uint32_t*>(q + i) = pack_bf16x2(v[j].x * rs * g.x, v[j].y * rs * g.y);
    }
}

// Gradients of the same: dx of the whole rows, per-block sums of the two weights' gradients [blocks][2][D]. Warps take heads in turn and keep their
// lanes' shares of both sums in registers (atomics on the D sums of a weight serialised the whole kernel: 8000 rows of 36 heads took
// 3.0 ms in two kernels and two copies, now 0.12 ms).
__global__ void __launch_bounds__(256) qk_rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ wq,
                                                             const __nv_bfloat16* __restrict__ wk, const float* __restrict__ rstd, __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part,
                                                             long long rows, int Hq, int Hkv, int D, long long x_stride, long long dy_stride, long long dx_stride) {
  __shared__ float s_dw[8][2 * 256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, heads = Hq + 2 * Hkv;
  float2 acc[2][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[0][j] = acc[1][j] = make_float2(0.f, 0.f);
  for (long long item = static_cast<long long>(blockIdx.x) * 8 + warp; item < rows * heads; item += static_cast<long long>(gridDim.x) * 8) {
    const long long row = item / heads;
    const int h = static_cast<int>(item - row * heads);
    const __nv_bfloat16* pd = dy + row * dy_stride + static_cast<long long>(h) * D;
    __nv_bfloat16* po = dx + row * dx_stride + static_cast<long long>(h) * D;
    if (h >= Hq + Hkv) {
      for (int i = lane * 2; i < D; i += 64) *reinterpret_cast<uint32_t*>(po + i) = *reinterpret_cast<const uint32_t*>(pd + i);
      continue;
    }
    const __nv_bfloat16* px = x + row * x_stride + static_cast<long long>(h) * D;
    const __nv_bfloat16* w = h < Hq ? wq : wk;
    const float rs = rstd[row * (Hq + Hkv) + h];
    float2 v[4], d[4];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[j] = d[j] = make_float2(0.f, 0.f);
      if (j * 64 < D) {
        const int i = lane * 2 + j * 64;
        v[j] = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(px + i));
        d[j] = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(pd + i));
        const float2 g = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + i));
        const float2 t = make_float2(d[j].x * v[j].x * rs, d[j].y * v[j].y * rs);
        if (h < Hq) { acc[0][j].x += t.x; acc[0][j].y += t.y; } else { acc[1][j].x += t.x; acc[1][j].y += t.y; }
        d[j].x *= g.x;
        d[j].y *= g.y;
        dot += d[j].x * v[j].x + d[j].y * v[j].y;
      }
    }
    dot = warp_sum(dot);
    const float c = dot * rs * rs / D;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j * 64 < D) *reinterpret_cast<uint32_t*>(po + lane * 2 + j * 64) = pack_bf16x2(rs * (d[j].x - v[j].x * c), rs * (d[j].y - v[j].y * c));
  }
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j * 64 < D) {
        s_dw[warp][k * D + lane * 2 + j * 64] = acc[k][j].x;
        s_dw[warp][k * D + lane * 2 + j * 64 + 1] = acc[k][j].y;
      }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) {
    float s = 0.f;
    for (int q = 0; q < 8; ++q) s += s_dw[q][i];
    dw_part[static_cast<long long>(blockIdx.x) * 2 * D + i] = s;
  }
}

// Per-head RMSNorm (Qwen3 q_norm / k_norm): rows x heads vectors of width D (<= 256, multiple of 8
// and of 64... one warp per vector, D/32 elements per lane handled as bf16x2 pairs).
__global__ void head_rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                        __nv_bfloat16* __restrict__ y, float* __restrict__ rstd_out,
                                        long long rows, int heads, int D, long long x_stride,
                                        long long y_stride, float eps) {
  pdl_sync();
  const long long wid = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= rows * heads) return;
  const long long row = wid / heads;
  const int head = static_cast<int>(wid - row * heads);
  const __nv_bfloat16* p = x + row * x_stride + static_cast<long long>(head) * D;
  __nv_bfloat16* q = y + row * y_stride + static_cast<long long>(head) * D;
  float ss = 0.f;
  for (int i = lane * 2; i < D; i += 64) {
    const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p + i));
    ss += v.x * v.x + v.y * v.y;
  }
  ss = warp_sum(ss);
  const float rs = rsqrtf(ss / D + eps);
  if (rstd_out && lane == 0) rstd_out[wid] = rs;
  for (int i = lane * 2; i < D; i += 64) {
    const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(p + i));
    const float2 g = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + i));
    *reinterpret_cast<uint32_t*>(q + i) = pack_bf16x2(v.x * rs * g.x, v.y * rs * g.y);
  }
}

__global__ void head_rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                                        const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                                        __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_accum,
                                        long long rows, int heads, int D, long long x_stride,
                                        long long dy_stride, long long dx_stride) {
  // dw is accumulated with atomics into a [D] fp32 buffer (D is tiny: 128).
  const long long wid = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= rows * heads) return;
  const long long row = wid / heads;
  const int head = static_cast<int>(wid - row * heads);
  const __nv_bfloat16* px = x + row * x_stride + static_cast<long long>(head) * D;
  const __nv_bfloat16* pd = dy + row * dy_stride + static_cast<long long>(head) * D;
  __nv_bfloat16* po = dx + row * dx_stride + static_cast<long long>(head) * D;
  const float rs = rstd[wid];
  float dot = 0.f;
  for (int i = lane * 2; i < D; i += 64) {
    const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(px + i));
    const float2 g = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + i));
    const float2 d = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(pd + i));
    dot += d.x * g.x * v.x + d.y * g.y * v.y;
    atomicAdd(dw_accum + i, d.x * v.x * rs);
    atomicAdd(dw_accum + i + 1, d.y * v.y * rs);
  }
  dot = warp_sum(dot);
  const float c = dot * rs * rs / D;
  for (int i = lane * 2; i < D; i += 64) {
    const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(px + i));
    const float2 g = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(w + i));
    const float2 d = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(pd + i));
    *reinterpret_cast<uint32_t*>(po + i) = pack_bf16x2(rs * (d.x * g.x - v.x * c), rs * (d.y * g.y - v.y * c));
  }
}

// ------------------------------------------------------------------ SwiGLU
// Row and vector of this thread where every vector has one of its own. Blocks start in order, so that those at work stay within some MB of one another:
// with a loop over a capped grid the streams drifted apart (20000 rows of 14336: SwiGLU 294 us, without 244; squares of 1.2e9 values 0.75 ms and 0.65).
__device__ __forceinline__ bool flat_vector(long long rows, int per_row, long long& row, int& v) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= rows * per_row) return false;
  row = i <= 0xffffffffll ? static_cast<uint32_t>(i) / static_cast<uint32_t>(per_row) : i / per_row;
  v = static_cast<int>(i - row * per_row);
  return true;
}
// gu: [rows, 2F] (gate | up). y[rows, F] = silu(gate) * up.
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ y,
                                  long long rows, int F) {
  pdl_sync();
  long long row;
  int c;
  if (flat_vector(rows, F / 8, row, c)) {
    c *= 8;
    float g[8], u[8], o[8];
    load8(gu + row * 2 * F + c, g);
    load8(gu + row * 2 * F + F + c, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.f + __expf(-g[j])) * u[j];
    store8(y + row * F + c, o);
  }
}
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ dgu, long long rows, int F) {
  long long row;
  int c;
  if (flat_vector(rows, F / 8, row, c)) {
    c *= 8;
    float g[8], u[8], d[8], dg[8], du[8];
    load8(gu + row * 2 * F + c, g);
    load8(gu + row * 2 * F + F + c, u);
    load8(dy + row * F + c, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = 1.f / (1.f + __expf(-g[j]));
      const float silu = g[j] * s;
      dg[j] = d[j] * u[j] * (s + silu * (1.f - s));
      du[j] = d[j] * silu;
    }
    store8(dgu + row * 2 * F + c, dg);
    store8(dgu + row * 2 * F + F + c, du);
  }
}

// ------------------------------------------------------------------ embedding
__global__ void embedding_fwd_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ table,
                                     __nv_bfloat16* __restrict__ out, long long rows, int d, int vocab) {
  pdl_sync();
  const long long vecs_per_row = d / 8;
  const long long total = rows * vecs_per_row;
  for (long long v = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; v < total;
       v += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long row = v / vecs_per_row;
    const int c = static_cast<int>(v - row * vecs_per_row) * 8;
    int id = ids[row];
    BF8 val;
    if (id < 0 || id >= vocab) {
      val.w[0] = val.w[1] = val.w[2] = val.w[3] = 0u;
    } else {
      val = *reinterpret_cast<const BF8*>(table + static_cast<long long>(id) * d + c);
    }
    *reinterpret_cast<BF8*>(out + row * d + c) = val;
  }
}
// Scatter-add of output gradients into an fp32 embedding gradient.
__global__ void embedding_bwd_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ dy,
                                     float* __restrict__ dtable, long long rows, int d, int vocab) {
  const long long vecs_per_row = d / 8;
  const long long total = rows * vecs_per_row;
  for (long long v = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; v < total;
       v += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long row = v / vecs_per_row;
    const int c = static_cast<int>(v - row * vecs_per_row) * 8;
    const int id = ids[row];
    if (id < 0 || id >= vocab) continue;
    float f[8];
    load8(dy + row * d + c, f);
    float* dst = dtable + static_cast<long long>(id) * d + c;
    if (reinterpret_cast<uintptr_t>(dtable) & 15) {
#pragma unroll
      for (int j = 0; j < 8; ++j) atomicAdd(dst + j, f[j]);
    } else {      // one request to memory for four sums (4000 rows of 4096: 101 us with single ones, now 43)
      atomicAdd(reinterpret_cast<float4*>(dst), make_float4(f[0], f[1], f[2], f[3]));
      atomicAdd(reinterpret_cast<float4*>(dst) + 1, make_float4(f[4], f[5], f[6], f[7]));
    }
  }
}

// ------------------------------------------------------------------ AdamW
// The fp32 master weight is stored as the bf16 parameter (the tensor the GEMMs read) plus a signed 16-bit
// remainder: master_bits = (bf16_bits << 16) + lo. The bf16 half is the master rounded to nearest with ties
// away from zero, which keeps the remainder inside [-32768, 32767] for every input, so the pair restores
// the fp32 value exactly at 4 bytes per parameter instead of 6.
__device__ __forceinline__ float master_join(__nv_bfloat16 hi, int16_t lo) {
  const uint32_t bits = (static_cast<uint32_t>(__bfloat16_as_ushort(hi)) << 16) + static_cast<uint32_t>(static_cast<int32_t>(lo));
  return __uint_as_float(bits);
}
__device__ __forceinline__ void master_split(float v, __nv_bfloat16& hi, int16_t& lo) {
  const uint32_t bits = __float_as_uint(v);
  const uint32_t hb = (bits + 0x8000u) & 0xFFFF0000u;
  hi = __ushort_as_bfloat16(static_cast<unsigned short>(hb >> 16));
  lo = static_cast<int16_t>(static_cast<int32_t>(bits - hb));
}

struct AdamArgs {
  float lr, beta1, beta2, eps, weight_decay, bc1, bc2;  // bc = 1 - beta^step
};

__device__ __forceinline__ float adamw_element(float w, float grad, float& m, float& v, const AdamArgs& a) {
  m = a.beta1 * m + (1.f - a.beta1) * grad;
  v = a.beta2 * v + (1.f - a.beta2) * grad * grad;
  w *= (1.f - a.lr * a.weight_decay);
  return w - a.lr * (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps);
}

// Split master weights, bound by memory (16 bytes read and 12 written an element with an fp32 gradient). A thread takes four neighbouring elements
// twice, a block's 2048 in whole 16-byte columns, all loads in flight before the first use. One block per 2048 elements and no loop: blocks start
// in order, so that those at work are within some MB of one another in each of the nine streams. With a loop over the grid, a warp's rows hundreds of
// MB apart, 1.2e9 parameters took 6.0 ms (eight elements a thread; 5.4 with four), through bulk copies and a ring in shared memory 5.0, now 4.86
// (6.9 TB/s).
template <typename GradT>
__global__ void __launch_bounds__(256) adamw_split_kernel(uint2* __restrict__ p, uint2* __restrict__ p_lo, const GradT* __restrict__ g, float4* __restrict__ m,
                                                          float4* __restrict__ v, long long n4, AdamArgs a, const float* __restrict__ grad_scale) {
  const float gs = grad_scale ? *grad_scale : 1.f;
  const long long first = static_cast<long long>(blockIdx.x) * 512 + threadIdx.x;
  uint2 hi[2], lo[2];
  float4 gr[2], mm[2], vv[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const long long i = first + j * 256;
    if (i >= n4) continue;
    hi[j] = p[i];
    lo[j] = p_lo[i];
    if constexpr (sizeof(GradT) == 4) {
      gr[j] = __ldcs(reinterpret_cast<const float4*>(g) + i);
    } else {
      const uint2 b = __ldcs(reinterpret_cast<const uint2*>(g) + i);
      const float2 x = unpack_bf16x2(b.x), y = unpack_bf16x2(b.y);
      gr[j] = make_float4(x.x, x.y, y.x, y.y);
    }
    mm[j] = m[i];
    vv[j] = v[i];
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const long long i = first + j * 256;
    if (i >= n4) continue;
    __nv_bfloat16* h4 = reinterpret_cast<__nv_bfloat16*>(&hi[j]);
    int16_t* l4 = reinterpret_cast<int16_t*>(&lo[j]);
    const float ge[4] = {gr[j].x, gr[j].y, gr[j].z, gr[j].w};
    float me[4] = {mm[j].x, mm[j].y, mm[j].z, mm[j].w}, ve[4] = {vv[j].x, vv[j].y, vv[j].z, vv[j].w};
#pragma unroll
    for (int k = 0; k < 4; ++k) master_split(adamw_element(master_join(h4[k], l4[k]), ge[k] * gs, me[k], ve[k], a), h4[k], l4[k]);
    p[i] = hi[j];
    p_lo[i] = lo[j];
    m[i] = make_float4(me[0], me[1], me[2], me[3]);
    v[i] = make_float4(ve[0], ve[1], ve[2], ve[3]);
  }
}

template <typename GradT>
__global__ void adamw_kernel(__nv_bfloat16* __restrict__ p, int16_t* __restrict__ p_lo, float* __restrict__ p32,
                             const GradT* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                             long long n, AdamArgs a, const float* __restrict__ grad_scale) {
  const float gs = grad_scale ? *grad_scale : 1.f;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float w = p32 ? p32[i] : master_join(p[i], p_lo[i]);
    float mi = m[i], vi = v[i];
    w = adamw_element(w, static_cast<float>(g[i]) * gs, mi, vi, a);
    m[i] = mi;
    v[i] = vi;
    if (p32) {
      p32[i] = w;
      if (p) p[i] = __float2bfloat16_rn(w);
    } else {
      __nv_bfloat16 hi;
      int16_t lo;
      master_split(w, hi, lo);
      p[i] = hi;
      p_lo[i] = lo;
    }
  }
}

// Sums of four or eight squares are taken in fp32, everything above in fp64: thousands of fp32 additions in a row lost part of the
// squares of small gradients beside large ones (2e-6 to 5e-6 of the norm at 1.2e9 to 1.9e9 parameters; now below 5e-7). Four 16-byte loads in flight: 2.28 -> 1.34 ms for 7.7 GB (5.7 TB/s). The blocks' sums are added up in fp64 as well, by a
// second kernel: as fp32 additions to `out`, a thousand sums that are nearly alike were all rounded the same way (5e-6 of the total).
// Runs of 64 KB a block, in order (flat_vector): 5.8 -> 6.9 TB/s; of 16 KB, one round of loads, where 64 would leave SMs without a block. A block on its own
// needs no second kernel, and that one is launched ahead of the first one's end (in a row, us, one kernel of fp32 additions / 64 KB and plain launches / now:
// 1000 values 4.2 / 6.3 / 4.1, 100000 4.2 / 6.5 / 4.7, 1048576 4.2 / 8.3 / 6.2, 1e7 10.4 / 14.5 / 12.1).
inline int sumsq_run(long long bytes) { return bytes < 4 * 148 * 65536ll ? 16384 : 65536; }
template <typename T>
__global__ void __launch_bounds__(256) sumsq_kernel(const T* __restrict__ x, long long n, int vecs, double* __restrict__ part, float* __restrict__ out) {
  __shared__ double red[8];
  double s = 0.0;
  constexpr int PER = 16 / sizeof(T);
  const long long nv = (reinterpret_cast<uintptr_t>(x) & 15) ? 0 : n / PER;
  const uint4* xv = reinterpret_cast<const uint4*>(x);
  const long long first = static_cast<long long>(blockIdx.x) * vecs + threadIdx.x;
#pragma unroll 1
  for (long long i = first; i < nv && i < first + vecs; i += 4 * 256) {
    uint4 q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = i + j * 256 < nv ? __ldcs(xv + i + j * 256) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const T* e = reinterpret_cast<const T*>(&q[j]);
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const float f = static_cast<float>(e[k]);
        t += f * f;
      }
      s += t;
    }
  }
  const long long step = static_cast<long long>(gridDim.x) * 256;
  for (long long i = nv * PER + static_cast<long long>(blockIdx.x) * 256 + threadIdx.x; i < n; i += step) {
    const float f = static_cast<float>(x[i]);
    s += f * f;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) s += red[w];
    if (gridDim.x == 1) atomicAdd(out, static_cast<float>(s));
    else part[blockIdx.x] = s;
  }
}

__global__ void __launch_bounds__(1024) sumsq_total_kernel(const double* __restrict__ part, int n, float* __restrict__ out) {
  pdl_sync();
  __shared__ double red[32];
  double s = 0.0;
#pragma unroll 8
  for (int i = threadIdx.x; i < n; i += 1024) s += part[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 32; ++w) s += red[w];
    atomicAdd(out, static_cast<float>(s));
  }
}

// scale = min(1, max_norm / (sqrt(sumsq) + 1e-6)) * extra ; also stores the norm.
__global__ void clip_scale_kernel(const float* __restrict__ sumsq, float max_norm, float extra,
                                  float* __restrict__ scale_out, float* __restrict__ norm_out) {
  const float norm = sqrtf(*sumsq);
  if (norm_out) *norm_out = norm;
  float s = 1.f;
  if (max_norm > 0.f) s = fminf(1.f, max_norm / (norm + 1e-6f));
  *scale_out = s * extra;
}

// ------------------------------------------------------------------ ClippedPG loss
// One pass over T tokens: per-token loss terms, their analytic gradient w.r.t. the current
// log-probability, and every metric partial sum. Slots of `sums`:
//  0 actor loss numerator (sum of w_is * clip_loss * mask)   1 kl numerator
//  2 sum ratio*mask   3 sum clamped ratio*mask   4 sum exp(|gen-prev|)*mask (token_mult_prob_error)
//  5 sum mask   6 gen_kl_error numerator   7 policy_kl_error numerator   8 sum w_is*mask
//  9 approx entropy numerator (-sum curr*mask... with IS weight)   10 ratio min  11 ratio max
//  12 clamped ratio min   13 clamped ratio max   14 js_divergence numerator  15 tokens whose IS weight left the truncation bounds
struct PGArgs {
  float eps_lo, eps_hi, dual_c;  // dual_c <= 0: no dual clip
  float kl_beta;
  int kl_type;  // 1,2,3
  float kl_in_clamp, kl_out_clamp;
  int use_is;        // importance-sampling correction
  int tis_type;      // 0 none, 1 tis (clamp max), 2 icepop (zero outside [min,max])
  float tis_max, tis_min;
  int force_on_policy;
  int use_cispo;
  int on_policy_kl_approx;
  float inv_norm;    // 1 / (global valid tokens + 1e-8)
};

// Sum over the block, in fp64: terms of either sign nearly cancel in the loss, and blocks add their sums in any order.
__device__ __forceinline__ double block_sum64(double v, double* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < nw; ++i) s += red[i];
  return s;      // (thread 0)
}

__global__ void clipped_pg_kernel(const float* __restrict__ curr, const float* __restrict__ prev,
                                  const float* __restrict__ gen, const float* __restrict__ ref,
                                  const float* __restrict__ adv, const float* __restrict__ mask, long long T,
                                  PGArgs a, double* __restrict__ sums, float* __restrict__ dcurr) {
  __shared__ float red[32];
  __shared__ double red64[32];
  float acc[10];
#pragma unroll
  for (int i = 0; i < 10; ++i) acc[i] = 0.f;
  float js = 0.f, nclip = 0.f, oob = 0.f;
  float rmin = INFINITY, rmax = -INFINITY, cmin = INFINITY, cmax = -INFINITY;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < T;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float mk = mask[i];
    const float c = curr[i];
    const float pv = a.force_on_policy ? c : prev[i];
    const float gn = gen ? gen[i] : pv;
    const float A = adv[i];
    float grad = 0.f;
    // KL penalty against the reference policy
    float kl = 0.f;
    if (a.kl_beta != 0.f && ref) {
      float logr = ref[i] - c;
      const bool inside = fabsf(logr) <= a.kl_in_clamp;  // same test as `logr == clamp(logr)`
      logr = fminf(fmaxf(logr, -a.kl_in_clamp), a.kl_in_clamp);
      float dkl_dc;  // d kl / d curr through logr (zero where the input clamp is active)
      if (a.kl_type == 1) {
        kl = -logr;
        dkl_dc = 1.f;
      } else if (a.kl_type == 2) {
        kl = 0.5f * logr * logr;
        dkl_dc = -logr;
      } else {
        const float e = __expf(logr);
        kl = e - 1.f - logr;
        dkl_dc = -(e - 1.f);
      }
      if (!inside) dkl_dc = 0.f;
      float wkl = 1.f;  // exp(curr - curr.detach()) = 1 in value, gradient kl * 1
      if (a.on_policy_kl_approx) wkl = __expf(c - gn);
      if (!isfinite(wkl)) wkl = 0.f;  // nan_to_num(nan = 0, +-inf = 0) on the weight
      // product rule; d wkl / d curr = wkl in both cases, except where the input clamp is active: there the weight is
      // detached, so the clamp suppresses the score-function term as well
      const float dw_dc = inside ? wkl : 0.f;
      float klw = kl * wkl;
      float dklw = dkl_dc * wkl + kl * dw_dc;
      if (isnan(klw)) {
        klw = 0.f;
        dklw = 0.f;
      }
      if (fabsf(klw) > a.kl_out_clamp) {
        klw = fminf(fmaxf(klw, -a.kl_out_clamp), a.kl_out_clamp);
        dklw = 0.f;
      }
      kl = klw;
      grad += a.kl_beta * dklw;
    }
    // ratio and clipped surrogate
    const float ratio = __expf(c - pv);
    const float rc = fminf(fmaxf(ratio, 1.f - a.eps_lo), 1.f + a.eps_hi);
    float loss, dloss;
    if (a.use_cispo) {
      loss = -A * rc * c;
      dloss = -A * rc;
    } else {
      const float l1 = -A * ratio, l2 = -A * rc;
      const bool clipped_active = l2 > l1;  // max picks the clamped branch: no gradient
      loss = clipped_active ? l2 : l1;
      dloss = clipped_active ? 0.f : -A * ratio;
      if (clipped_active) nclip += mk;
      if (a.dual_c > 0.f && A < 0.f) {
        const float l3 = -A * a.dual_c;
        if (l3 < loss) {
          loss = l3;
          dloss = 0.f;
        }
      }
    }
    // importance-sampling weight between trainer and generator probabilities (a constant w.r.t. curr)
    float wis = __expf(pv - gn);
    if (isnan(wis)) wis = 0.f;
    float wis_used = 1.f;
    if (a.use_is) {
      wis_used = wis;
      if (a.tis_type != 0 && (wis > a.tis_max || wis < a.tis_min)) oob += mk;
      if (a.tis_type == 1) wis_used = fminf(fmaxf(wis, a.tis_min), a.tis_max);
      else if (a.tis_type == 2) wis_used = (wis >= a.tis_min && wis <= a.tis_max) ? wis : 0.f;
    }
    grad += wis_used * dloss;
    if (dcurr) dcurr[i] = grad * mk * a.inv_norm;

    acc[0] += wis_used * loss * mk;
    acc[1] += kl * mk;
    acc[2] += ratio * mk;
    acc[3] += rc * mk;
    acc[4] += __expf(fabsf(gn - pv)) * mk;
    acc[5] += mk;
    {
      // gen_kl_error: KL(gen || train) estimated with logr = prev - gen; policy_kl_error: the reverse.
      const float d = pv - gn;
      float gk, pk;
      if (a.kl_type == 1) {
        gk = -d;
        pk = d;
      } else if (a.kl_type == 2) {
        gk = 0.5f * d * d;
        pk = gk;
      } else {
        gk = __expf(d) - 1.f - d;
        pk = __expf(-d) - 1.f + d;
      }
      acc[6] += gk * mk;
      acc[7] += pk * mk;
      // Jensen-Shannon: M = (P_train + P_gen) / 2, JSD = (KL(P_train||M) + KL(P_gen||M)) / 2, k3 estimates
      const float lm = __logf(0.5f * __expf(pv) + 0.5f * __expf(gn));
      const float a1 = pv - lm, a2 = gn - lm;
      js += 0.5f * ((__expf(a1) - 1.f - a1) + (__expf(a2) - 1.f - a2)) * mk;
    }
    acc[8] += wis * mk;
    acc[9] += -(__expf(c - gn) * c) * mk;
    if (mk > 0.f) {
      rmin = fminf(rmin, ratio);
      rmax = fmaxf(rmax, ratio);
      cmin = fminf(cmin, rc);
      cmax = fmaxf(cmax, rc);
    }
  }
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    const double s = block_sum64(acc[i], red64);
    if (threadIdx.x == 0) atomicAdd(sums + i, s);
  }
  {
    const double s = block_sum64(js, red64);
    if (threadIdx.x == 0) atomicAdd(sums + 14, s);
    (void)nclip;
    const double s2 = block_sum64(oob, red64);
    if (threadIdx.x == 0) atomicAdd(sums + 15, s2);
  }
  // min/max via integer atomics on non-negative values (ratios are > 0)
  rmin = -block_max(-rmin, red);
  rmax = block_max(rmax, red);
  cmin = -block_max(-cmin, red);
  cmax = block_max(cmax, red);
  if (threadIdx.x == 0) {
    long long* bits = reinterpret_cast<long long*>(sums);
    if (isfinite(rmin)) atomicMin(bits + 10, __double_as_longlong(rmin));
    if (isfinite(rmax)) atomicMax(bits + 11, __double_as_longlong(rmax));
    if (isfinite(cmin)) atomicMin(bits + 12, __double_as_longlong(cmin));
    if (isfinite(cmax)) atomicMax(bits + 13, __double_as_longlong(cmax));
  }
}

__global__ void pg_init_sums_kernel(double* sums) {
  const int i = threadIdx.x;
  if (i < 16) {
    double v = 0.0;
    if (i == 10 || i == 12) v = 3.0e38;  // running minima start high
    sums[i] = v;
  }
}

// ------------------------------------------------------------------ misc
__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, long long n) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    y[i] = __float2bfloat16_rn(x[i]);
}
// y = a + b (bf16), the residual add
__global__ void add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                __nv_bfloat16* __restrict__ y, long long n8) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n8;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float fa[8], fb[8];
    load8(a + i * 8, fa);
    load8(b + i * 8, fb);
#pragma unroll
    for (int j = 0; j < 8; ++j) fa[j] += fb[j];
    store8(y + i * 8, fa);
  }
}

inline int grid_for(long long work, int threads, int cap = 148 * 16) {
  long long g = (work + threads - 1) / threads;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return static_cast<int>(g);
}
inline int rms_threads(int d) {
  int t = d / 8;
  if (t > 512) t = 512;
  t = (t + 31) / 32 * 32;
  if (t < 32) t = 32;
  return t;
}

}  // namespace

#define S(stream) static_cast<cudaStream_t>(stream)
#define BF(p) reinterpret_cast<__nv_bfloat16*>(p)
#define CBF(p) reinterpret_cast<const __nv_bfloat16*>(p)

RLB_API int rlb_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* res_out, float* rstd,
                            long long rows, int d, long long x_stride, long long y_stride, float eps,
                            void* stream) {
  if (rows <= 0) return 0;
  if (d % 8 || x_stride % 8 || y_stride % 8) return -2;
  if (!res && d <= 1024 && rows >= 148 * 16) {
    rlb_launch_pdl(rmsnorm_rows_kernel<4>, dim3(static_cast<unsigned>((rows + 7) / 8)), dim3(256), 0, S(stream), CBF(x), CBF(w), BF(y), rstd, rows, d, x_stride, y_stride, eps);
    return static_cast<int>(cudaGetLastError());
  }
  if (d <= 8192) {
    const int pieces = d <= (res ? 4096 : 1024) ? 2 : 4, threads = (d / 8 + pieces * 32 - 1) / (pieces * 32) * 32;
    auto kern = res ? (pieces == 2 ? rmsnorm_regs_kernel<2, true> : rmsnorm_regs_kernel<4, true>) : (pieces == 2 ? rmsnorm_regs_kernel<2, false> : rmsnorm_regs_kernel<4, false>);
    rlb_launch_pdl(kern, dim3(static_cast<unsigned>(rows)), dim3(threads), 0, S(stream), CBF(x), CBF(res), CBF(w), BF(y), BF(res_out), rstd, d, x_stride, y_stride, eps);
    return static_cast<int>(cudaGetLastError());
  }
  rlb_launch_pdl(rmsnorm_fwd_kernel, dim3(static_cast<unsigned>(rows)), dim3(rms_threads(d)), 0, S(stream), 
      CBF(x), CBF(res), CBF(w), BF(y), BF(res_out), rstd, d, x_stride, y_stride, eps);
  return static_cast<int>(cudaGetLastError());
}

// Number of CTAs (= rows of the dw partial buffer) the backward uses.
RLB_API int rlb_rmsnorm_bwd_parts(long long rows) { return static_cast<int>(rows < 296 ? rows : 296); }

// dw_partial: scratch of rlb_rmsnorm_bwd_parts(rows) * d floats. The column sums are written (or
// added) to dw_f32 / dw_bf16, whichever is non-null.
RLB_API int rlb_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx,
                            float* dw_partial, float* dw_f32, void* dw_bf16, int dw_accumulate, long long rows,
                            int d, long long x_stride, long long dy_stride, int add_to_dx, void* stream) {
  if (rows <= 0) return 0;
  if (d % 8 || x_stride % 8 || dy_stride % 8) return -2;
  const int threads = rms_threads(d);
  if (d > threads * 8 * 8) return -4;
  const int parts = rlb_rmsnorm_bwd_parts(rows);
  if (d <= 4096) {
    const int pieces = d <= 2048 ? 1 : 2, width = (d / 8 + pieces * 32 - 1) / (pieces * 32) * 32;      // whole warps, the last of them cut
    auto kern = pieces == 2     ? rmsnorm_bwd_rows_kernel<2, 1, 256>
                : rows <= parts ? rmsnorm_bwd_rows_kernel<1, 1, 256>      // (a row a CTA)
                : width > 128   ? rmsnorm_bwd_rows_kernel<1, 3, 256>
                                : rmsnorm_bwd_rows_kernel<1, 4, 128>;
    kern<<<parts, width, 0, S(stream)>>>(CBF(dy), CBF(x), CBF(w), rstd, BF(dx), dw_partial, static_cast<int>(rows), d, x_stride, dy_stride, add_to_dx);
  } else {
    rmsnorm_bwd_kernel<<<parts, threads, 0, S(stream)>>>(CBF(dy), CBF(x), CBF(w), rstd, BF(dx), dw_partial,
                                                         static_cast<int>(rows), d, x_stride, dy_stride, add_to_dx);
  }
  colsum_kernel<<<(d + 31) / 32, 256, 0, S(stream)>>>(dw_partial, parts, d, dw_f32, BF(dw_bf16), dw_accumulate);
  return static_cast<int>(cudaGetLastError());
}

RLB_API int rlb_rope(void* x, const int* pos, const float* inv_freq, long long rows, int heads, int D,
                     long long row_stride, int backward, void* stream) {
  if (rows <= 0) return 0;
  if (D % 4) return -2;
  if (!(D % 16) && D <= 512 && !(row_stride % 8) && !(reinterpret_cast<uintptr_t>(x) & 15) && rows * heads > (D < 128 ? 512 : 4096)) {
    const int block_rows = rows >= 148 * 16 ? 4 : 1;      // enough blocks for every SM before a block takes several rows (2368: 16.4 us either way, 20480: 74 and 78)
    rlb_launch_pdl(rope_rows_kernel, dim3(static_cast<unsigned>((rows + block_rows - 1) / block_rows)), dim3(256), block_rows * D / 2 * sizeof(float2), S(stream), BF(x), pos, inv_freq,
                   rows, heads, D, row_stride, backward ? -1.f : 1.f, block_rows);
    return static_cast<int>(cudaGetLastError());
  }
  const long long warps = rows * heads;
  const int threads = 256;
  const long long blocks = (warps * 32 + threads - 1) / threads;
  rlb_launch_pdl(rope_kernel, dim3(static_cast<unsigned>(blocks)), dim3(threads), 0, S(stream), BF(x), pos, inv_freq, rows, heads, D,
                                                                         row_stride, backward ? -1.f : 1.f);
  return static_cast<int>(cudaGetLastError());
}

RLB_API int rlb_head_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, long long rows, int heads,
                                 int D, long long x_stride, long long y_stride, float eps, void* stream) {
  if (rows <= 0) return 0;
  if (D % 2) return -2;
  const long long blocks = (rows * heads * 32 + 255) / 256;
  rlb_launch_pdl(head_rmsnorm_fwd_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, S(stream), CBF(x), CBF(w), BF(y), rstd, rows,
                                                                                 heads, D, x_stride, y_stride, eps);
  return static_cast<int>(cudaGetLastError());
}
RLB_API int rlb_head_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, void* dx,
                                 float* dw_accum, long long rows, int heads, int D, long long x_stride,
                                 long long dy_stride, long long dx_stride, void* stream) {
  if (rows <= 0) return 0;
  const long long blocks = (rows * heads * 32 + 255) / 256;
  head_rmsnorm_bwd_kernel<<<static_cast<unsigned>(blocks), 256, 0, S(stream)>>>(
      CBF(dy), CBF(x), CBF(w), rstd, BF(dx), dw_accum, rows, heads, D, x_stride, dy_stride, dx_stride);
  return static_cast<int>(cudaGetLastError());
}

// RMSNorms of the q and k heads of fused [q | k | v] rows (v copied); out may be x; rstd [rows, Hq + Hkv] or null. D: a multiple of 64, at most 256.
RLB_API int rlb_qk_rmsnorm_fwd(const void* x, const void* wq, const void* wk, void* out, float* rstd, long long rows, int Hq, int Hkv, int D, long long x_stride, long long out_stride,
                               float eps, void* stream) {
  if (rows <= 0) return 0;
  if ((D % 64) || D > 256 || (x_stride % 2) || (out_stride % 2)) return -2;
  const long long blocks = (rows * (Hq + 2 * Hkv) * 32 + 255) / 256;
  rlb_launch_pdl(qk_rmsnorm_fwd_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, S(stream), CBF(x), CBF(wq), CBF(wk), BF(out), rstd, rows, Hq, Hkv, D, x_stride, out_stride, eps);
  return static_cast<int>(cudaGetLastError());
}
RLB_API int rlb_qk_rmsnorm_bwd_parts(long long rows) { return static_cast<int>(rows < 148 * 4 ? rows : 148 * 4); }
// dw_part: scratch of parts * 2 * D floats; dw [2, D] = the sums over rows and heads of both weights' gradients.
RLB_API int rlb_qk_rmsnorm_bwd(const void* dy, const void* x, const void* wq, const void* wk, const float* rstd, void* dx, float* dw_part, float* dw, long long rows, int Hq, int Hkv, int D,
                               long long x_stride, long long dy_stride, long long dx_stride, void* stream) {
  if (rows <= 0) return 0;
  if ((D % 64) || D > 256 || (x_stride % 2) || (dy_stride % 2) || (dx_stride % 2)) return -2;
  const int parts = rlb_qk_rmsnorm_bwd_parts(rows);
  qk_rmsnorm_bwd_kernel<<<parts, 256, 0, S(stream)>>>(CBF(dy), CBF(x), CBF(wq), CBF(wk), rstd, BF(dx), dw_part, rows, Hq, Hkv, D, x_stride, dy_stride, dx_stride);
  colsum_kernel<<<(2 * D + 31) / 32, 256, 0, S(stream)>>>(dw_part, parts, 2 * D, dw, nullptr, 0);
  return static_cast<int>(cudaGetLastError());
}

RLB_API int rlb_swiglu_fwd(const void* gu, void* y, long long rows, int F, void* stream) {
  if (rows <= 0) return 0;
  if (F % 8) return -2;
  rlb_launch_pdl(swiglu_fwd_kernel, dim3(grid_for(rows * (F / 8), 256, INT_MAX)), dim3(256), 0, S(stream), CBF(gu), BF(y), rows, F);
  return static_cast<int>(cudaGetLastError());
}
RLB_API int rlb_swiglu_bwd(const void* dy, const void* gu, void* dgu, long long rows, int F, void* stream) {
  if (rows <= 0) return 0;
  if (F % 8) return -2;
  swiglu_bwd_kernel<<<grid_for(rows * (F / 8), 256, INT_MAX), 256, 0, S(stream)>>>(CBF(dy), CBF(gu), BF(dgu), rows, F);
  return static_cast<int>(cudaGetLastError());
}

RLB_API int rlb_embedding_fwd(const int* ids, const void* table, void* out, long long rows, int d, int vocab,
                              void* stream) {
  if (rows <= 0) return 0;
  if (d % 8) return -2;
  rlb_launch_pdl(embedding_fwd_kernel, dim3(grid_for(rows * (d / 8), 256)), dim3(256), 0, S(stream), ids, CBF(table), BF(out), rows, d,
                                                                             vocab);
  return static_cast<int>(cudaGetLastError());
}
RLB_API int rlb_embedding_bwd(const int* ids, const void* dy, float* dtable, long long rows, int d, int vocab,
                              void* stream) {
  if (rows <= 0) return 0;
  if (d % 8) return -2;
  embedding_bwd_kernel<<<grid_for(rows * (d / 8), 256), 256, 0, S(stream)>>>(ids, CBF(dy), dtable, rows, d, vocab);
  return static_cast<int>(cudaGetLastError());
}

// AdamW over a flat shard. Master weight either fp32 (`p32`, with an optional bf16 copy `p`) or the
// split form (`p` bf16 + `p_lo` int16, p32 null). grad_is_bf16 selects the gradient type.
// grad_scale: device scalar multiplied into every gradient (clip coefficient / loss scale), or null.
RLB_API int rlb_adamw(void* p, void* p_lo, float* p32, const void* g, int grad_is_bf16, float* m, float* v,
                      long long n, float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                      const float* grad_scale, void* stream) {
  if (n <= 0) return 0;
  AdamArgs a{lr, beta1, beta2, eps, weight_decay, 1.f - powf(beta1, static_cast<float>(step)),
             1.f - powf(beta2, static_cast<float>(step))};
  const uintptr_t all = reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(p_lo) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v);
  const long long n4 = p && p_lo && !p32 && !(all & 15) ? n / 4 : 0;      // the rest, if any, goes element by element
  if (n4) {
    const unsigned blocks = static_cast<unsigned>((n4 + 511) / 512);
    if (grad_is_bf16)
      adamw_split_kernel<__nv_bfloat16><<<blocks, 256, 0, S(stream)>>>(reinterpret_cast<uint2*>(p), reinterpret_cast<uint2*>(p_lo), CBF(g), reinterpret_cast<float4*>(m),
                                                                       reinterpret_cast<float4*>(v), n4, a, grad_scale);
    else
      adamw_split_kernel<float><<<blocks, 256, 0, S(stream)>>>(reinterpret_cast<uint2*>(p), reinterpret_cast<uint2*>(p_lo), reinterpret_cast<const float*>(g),
                                                               reinterpret_cast<float4*>(m), reinterpret_cast<float4*>(v), n4, a, grad_scale);
    if (n4 * 4 == n) return static_cast<int>(cudaGetLastError());
    p = BF(p) + n4 * 4;
    p_lo = static_cast<int16_t*>(p_lo) + n4 * 4;
    g = static_cast<const char*>(g) + n4 * 4 * (grad_is_bf16 ? 2 : 4);
    m += n4 * 4;
    v += n4 * 4;
    n -= n4 * 4;
  }
  const int grid = grid_for(n, 256, 148 * 8);
  if (grad_is_bf16)
    adamw_kernel<__nv_bfloat16><<<grid, 256, 0, S(stream)>>>(BF(p), reinterpret_cast<int16_t*>(p_lo), p32, CBF(g), m,
                                                              v, n, a, grad_scale);
  else
    adamw_kernel<float><<<grid, 256, 0, S(stream)>>>(BF(p), reinterpret_cast<int16_t*>(p_lo), p32,
                                                      reinterpret_cast<const float*>(g), m, v, n, a, grad_scale);
  return static_cast<int>(cudaGetLastError());
}

// Doubles of scratch that rlb_sumsq needs: one a block.
RLB_API int rlb_sumsq_parts(long long n, int is_bf16) {
  const long long bytes = n * (is_bf16 ? 2 : 4);
  const int run = sumsq_run(bytes);
  return static_cast<int>((bytes + run - 1) / run);
}
// out += sum(x^2). `out` is a device float the caller zeroes.
RLB_API int rlb_sumsq(const void* x, int is_bf16, long long n, float* out, double* part, void* stream) {
  if (n <= 0) return 0;
  const int grid = rlb_sumsq_parts(n, is_bf16), vecs = sumsq_run(n * (is_bf16 ? 2 : 4)) / 16;
  if (is_bf16) sumsq_kernel<__nv_bfloat16><<<grid, 256, 0, S(stream)>>>(CBF(x), n, vecs, part, out);
  else sumsq_kernel<float><<<grid, 256, 0, S(stream)>>>(reinterpret_cast<const float*>(x), n, vecs, part, out);
  if (grid > 1) rlb_launch_pdl(sumsq_total_kernel, dim3(1), dim3(1024), 0, S(stream), part, grid, out);
  return static_cast<int>(cudaGetLastError());
}
RLB_API int rlb_clip_scale(const float* sumsq, float max_norm, float extra, float* scale_out, float* norm_out,
                           void* stream) {
  clip_scale_kernel<<<1, 1, 0, S(stream)>>>(sumsq, max_norm, extra, scale_out, norm_out);
  return static_cast<int>(cudaGetLastError());
}

RLB_API int rlb_clipped_pg(const float* curr, const float* prev, const float* gen, const float* ref,
                           const float* adv, const float* mask, long long T, float eps_lo, float eps_hi,
                           float dual_c, float kl_beta, int kl_type, float kl_in_clamp, float kl_out_clamp,
                           int use_is, int tis_type, float tis_max, float tis_min, int force_on_policy,
                           int use_cispo, int on_policy_kl_approx, float inv_norm, double* sums, float* dcurr,
                           void* stream) {
  PGArgs a{eps_lo, eps_hi, dual_c, kl_beta, kl_type, kl_in_clamp, kl_out_clamp, use_is, tis_type, tis_max,
           tis_min, force_on_policy, use_cispo, on_policy_kl_approx, inv_norm};
  pg_init_sums_kernel<<<1, 32, 0, S(stream)>>>(sums);
  if (T > 0)
    clipped_pg_kernel<<<grid_for(T, 256, 148 * 2), 256, 0, S(stream)>>>(curr, prev, gen, ref, adv, mask, T, a, sums,
                                                                        dcurr);
  return static_cast<int>(cudaGetLastError());
}

RLB_API int rlb_cast_f32_bf16(const float* x, void* y, long long n, void* stream) {
  if (n <= 0) return 0;
  cast_f32_to_bf16_kernel<<<grid_for(n, 256), 256, 0, S(stream)>>>(x, BF(y), n);
  return static_cast<int>(cudaGetLastError());
}
RLB_API int rlb_add_bf16(const void* a, const void* b, void* y, long long n, void* stream) {
  if (n <= 0) return 0;
  if (n % 8) return -2;
  add_bf16_kernel<<<grid_for(n / 8, 256), 256, 0, S(stream)>>>(CBF(a), CBF(b), BF(y), n / 8);
  return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------------ RMSNorm backward without device allocation
// See no_alloc.h for who this is for and what it costs. The scratch that rlb_rmsnorm_bwd takes from its caller is a
// fixed array in the library image here. In host code the array's name is only a host-side handle, not a device
// address, so the address the kernels receive is looked up once per device with cudaGetSymbolAddress.
#include "no_alloc.h"

namespace {
static __device__ __align__(256) float g_rmsnorm_static_scratch[RLB_RMSNORM_STATIC_MAX_PARTS * RLB_RMSNORM_STATIC_MAX_D];
constexpr int kMaxDevices = 64;
float* g_rmsnorm_static_ptr[kMaxDevices] = {nullptr};

// Device address of the scratch array on the current device, resolved on first use there.
int rmsnorm_static_scratch(float** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= kMaxDevices) return RLB_STATIC_ERR_NO_SYMBOL;
  if (!g_rmsnorm_static_ptr[dev]) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_rmsnorm_static_scratch);
    if (e != cudaSuccess || !p) return e != cudaSuccess ? static_cast<int>(e) : RLB_STATIC_ERR_NO_SYMBOL;
    g_rmsnorm_static_ptr[dev] = p;
  }
  *out = g_rmsnorm_static_ptr[dev];
  return 0;
}
}  // namespace

RLB_API int rlb_rmsnorm_bwd_static(const void* dy, const void* x, const void* w, const float* rstd, void* dx,
                                   float* dw_f32, int dw_accumulate, long long rows, int d, long long x_stride,
                                   long long dy_stride, void* stream) {
  if (rows <= 0) return 0;
  if (d <= 0 || d % 8 || x_stride % 8 || dy_stride % 8) return RLB_STATIC_ERR_BAD_SHAPE;
  if (d > RLB_RMSNORM_STATIC_MAX_D) return RLB_STATIC_ERR_TOO_LARGE;
  // The kernels use 16-byte vector loads and stores on every operand and index rows with int: refuse what would
  // otherwise reach the device as a misaligned address or a truncated row count.
  if (x_stride < d || dy_stride < d || rows > 2147483647ll) return RLB_STATIC_ERR_BAD_SHAPE;
  const void* vec_ptrs[4] = {dy, x, w, dx};  // bf16 operands: 16-byte vector access
  for (const void* q : vec_ptrs)
    if (q == nullptr || (reinterpret_cast<uintptr_t>(q) & 15u)) return RLB_STATIC_ERR_BAD_SHAPE;
  if (rstd == nullptr || dw_f32 == nullptr || (reinterpret_cast<uintptr_t>(rstd) & 3u) ||
      (reinterpret_cast<uintptr_t>(dw_f32) & 3u))
    return RLB_STATIC_ERR_BAD_SHAPE;
  float* scratch = nullptr;
  const int rc = rmsnorm_static_scratch(&scratch);
  if (rc) return rc;
  const int threads = rms_threads(d);
  const int parts = static_cast<int>(rows < RLB_RMSNORM_STATIC_MAX_PARTS ? rows : RLB_RMSNORM_STATIC_MAX_PARTS);
  // Every CTA writes its whole row of the partial matrix before the column-sum kernel reads it, so what an earlier
  // call left in the array is never read.
  rmsnorm_bwd_kernel<<<parts, threads, 0, S(stream)>>>(CBF(dy), CBF(x), CBF(w), rstd, BF(dx), scratch,
                                                       static_cast<int>(rows), d, x_stride, dy_stride, 0);
  colsum_kernel<<<(d + 31) / 32, 256, 0, S(stream)>>>(scratch, parts, d, dw_f32, nullptr, dw_accumulate);
  return static_cast<int>(cudaGetLastError());
}

RLB_API const char* rlb_rmsnorm_bwd_static_strerror(int code) {
  switch (code) {
    case 0: return "ok";
    case RLB_STATIC_ERR_BAD_SHAPE: return "d and the strides must be positive multiples of 8 elements (strides >= d, rows < 2^31), dy / x / w / dx non-null and 16-byte aligned, rstd / dw_f32 non-null";
    case RLB_STATIC_ERR_TOO_LARGE: return "d exceeds RLB_RMSNORM_STATIC_MAX_D (8192): use rlb_rmsnorm_bwd with caller scratch";
    case RLB_STATIC_ERR_NO_SYMBOL: return "the static scratch array's device address could not be resolved";
    default: return code > 0 ? "CUDA error (see cudaGetErrorString)" : "unknown code";
  }
}
