// Which tile of which packed sequence a CTA of the attention kernels takes.
#pragma once

#include "common.cuh"

namespace rlb {
constexpr int SORTED_SEQS = 128;      // four to a lane

// Finds the (sequence, tile-in-sequence) of a flat tile index; tiles of `rows` rows never straddle sequences. Called by a whole warp, 32
// sequences at a time (one thread walking them waited for memory at every one). Returns false when `tile` is past the last tile.
__device__ __forceinline__ bool locate_tile(const int* __restrict__ cu, int num_seqs, int rows, int tile, int& start, int& len, int& tile_in_seq) {
  const int lane = threadIdx.x & 31;
  int acc = 0;
  for (int s0 = 0; s0 < num_seqs; s0 += 32) {
    const int s = min(s0 + lane, num_seqs - 1);
    const int b = cu[s], e = cu[s + 1];
    const int n = s0 + lane < num_seqs ? (e - b + rows - 1) / rows : 0;
    int end = n;      // tiles of the sequences up to this lane's
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, tile < acc + end);
    if (hit) {
      const int src = __ffs(hit) - 1;
      start = __shfl_sync(0xffffffffu, b, src);
      len = __shfl_sync(0xffffffffu, e - b, src);
      tile_in_seq = tile - acc - __shfl_sync(0xffffffffu, end - n, src);
      return true;
    }
    acc += __shfl_sync(0xffffffffu, end, 31);
  }
  return false;
}

// The same in order of falling work, over all sequences: a causal tile sees as many others as it is from its sequence's start (`late`: query tiles) or end
// (key tiles), so all tiles that see d of them come before those that see d - 1. Block `index` of `most` (some past the last tile: false). More
// than 128 sequences go one after the other. With the CTAs of all heads side by side (the heads as the fast part of the block index) the last ones are the
// shortest of all; one head after the other, each with its own short and long tiles, left SMs without work for up to a quarter of the time (backward of
// 32 query and 8 KV heads of 128, us: 4 x 1000 383 -> 321, 8 x 500 277 -> 251, 7600 2755 -> 2371, 4 x 4096 3042 -> 2808). The place in the order comes from the grid's
// dimensions and the bounds stay in registers: with a division for head and tile each and the bounds read again, some 800 cycles, tiles of short sequences
// took a tenth longer (forward, 256 x 64 tokens 278 us, now 262; 1 x 64 8.3 and 7.2).
__device__ __forceinline__ bool locate_longest_first(const int* __restrict__ cu, int num_seqs, int rows, int index, int most, bool late, int& start, int& len,
                                                     int& tile_in_seq) {
  if (num_seqs > SORTED_SEQS) return locate_tile(cu, num_seqs, rows, late ? most - 1 - index : index, start, len, tile_in_seq);
  const int lane = threadIdx.x & 31;
  int tiles[SORTED_SEQS / 32], begin[SORTED_SEQS / 32], length[SORTED_SEQS / 32], top = 0;
#pragma unroll
  for (int k = 0; k < SORTED_SEQS / 32; ++k) {
    const int s = lane + 32 * k;
    begin[k] = s < num_seqs ? cu[s] : 0;
    length[k] = s < num_seqs ? cu[s + 1] - begin[k] : 0;
    tiles[k] = (length[k] + rows - 1) / rows;
    top = max(top, tiles[k]);
  }
  auto at_least = [&](int d) {      // tiles that see d others or more
    int n = 0;
#pragma unroll
    for (int k = 0; k < SORTED_SEQS / 32; ++k) n += max(0, tiles[k] - d + 1);
    return __reduce_add_sync(0xffffffffu, n);
  };
  if (index >= at_least(1)) return false;
  int lo = 1, hi = __reduce_max_sync(0xffffffffu, top);
  while (lo < hi) {      // the largest d with more than `index` tiles
    const int mid = (lo + hi + 1) >> 1;
    if (at_least(mid) > index) lo = mid;
    else hi = mid - 1;
  }
  int j = index - at_least(lo + 1);
#pragma unroll
  for (int k = 0; k < SORTED_SEQS / 32; ++k) {
    unsigned has = __ballot_sync(0xffffffffu, tiles[k] >= lo);
    const int n = __popc(has);
    if (j >= n) {
      j -= n;
      continue;
    }
    for (; j > 0; --j) has &= has - 1;
    const int src = __ffs(has) - 1;
    start = __shfl_sync(0xffffffffu, begin[k], src);
    len = __shfl_sync(0xffffffffu, length[k], src);
    tile_in_seq = late ? lo - 1 : __shfl_sync(0xffffffffu, tiles[k], src) - lo;
    return true;
  }
  return false;
}
}  // namespace rlb
