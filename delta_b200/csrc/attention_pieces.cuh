// The pieces (query tiles of the rows) of the tcgen05 attention kernels, listed from long to short.
//
// A block takes pieces in rounds, forwards and backwards in turn, which ends all blocks together when the pieces come from long to short
// and every number is a piece.  Numbered by (tile from a row's end, row) that holds for rows of one length only: with prompts of 1,301, 700
// and 47 tokens more than half of the numbers are no piece, and blocks that get two long ones end last.  So the pairs (row, tile) are sorted
// by their tiles of keys once at a block's start: 32 heads of attention_prefill_tc.cu 74 -> 49 us, 16 heads with shaped scores 109 -> 68 us.
// One row keeps the numbers (58 us for 2,048 tokens and 32 heads, 60 us with the list), and so do more than N pairs or 511 rows.
#pragma once
#include <stdint.h>

template <int N>
struct PieceList {
  uint32_t raw[N], sorted[N];      // tiles of keys (14 bits) | row (9) | query tile (9)
  int count;
};

// Called by the whole block.  tiles(row, query tile): its tiles of keys.  Returns the number of pairs, or -1 where they don't fit the list.
template <int N, typename Tiles>
__device__ __forceinline__ int list_pieces(PieceList<N>& list, const int* __restrict__ row_q_len, int rows, bool skip_singles, int query_tile, Tiles&& tiles) {
  if (rows == 1 || rows > 511) return -1;
  if (threadIdx.x == 0) list.count = 0;
  __syncthreads();
  for (int r = threadIdx.x; r < rows; r += blockDim.x) {
    const int q_len = row_q_len[r], n = skip_singles && q_len == 1 ? 0 : (q_len + query_tile - 1) / query_tile;
    if (n <= 0) continue;
    const int base = atomicAdd(&list.count, n);
    for (int q = 0; q < n && base + q < N; ++q) list.raw[base + q] = (uint32_t)min(tiles(r, q), 16383) << 18 | (uint32_t)r << 9 | (uint32_t)(q & 511);
  }
  __syncthreads();
  const int count = list.count;
  if (count > N) return -1;      // (N is below 512: no query tile is above 511 then)
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    const uint32_t key = list.raw[i];
    int rank = 0;
    for (int j = 0; j < count; ++j) rank += list.raw[j] > key;      // the keys differ
    list.sorted[rank] = key;
  }
  __syncthreads();
  return count;
}

// Rows [from, to) of boxes of 128-byte rows become zeros, by one warp, after their copy has arrived and before an MMA reads them: rows of a tile
// that no query of the piece sees.  Their weights are zero, but zero times what another request left in a page, or an earlier token that was
// not finite, need not be.
__device__ __forceinline__ void clear_rows(uint32_t boxes, int count, int box_bytes, int from, int to) {      // (an address in shared memory)
  if (from >= to) return;
#pragma unroll 1
  for (uint32_t at = boxes; count-- > 0; at += box_bytes)
#pragma unroll 1
    for (int i = from * 8 + (int)(threadIdx.x & 31); i < to * 8; i += 32)
      asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(at + i * 16), "r"(0) : "memory");
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");      // ordinary stores, read by the tensor cores
  __syncwarp();
}
