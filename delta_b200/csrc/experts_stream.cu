// The experts' products for a handful of tokens (decode steps), bfloat16: a stream over the chosen experts' weights.
//
// The rows of an expert are a tile of the sorted slots (experts.cu), nearly empty when a step brings few tokens.  As in gemm_small_m.cu a block owns
// 16 rows of an expert's matrix (and the 16 up rows that belong to its gate rows), its warps share K in chunks of 32 entries, and
// weights and activations go from memory into MMA fragments with sixteen-byte loads under a permutation of k that both share; the warps'
// sums are added in shared memory in a fixed order.  Bound by the memory: 8 tokens, 16 experts of 1,024, 4 chosen, width 2,048: 24.7
// and 13.4 us for the two products (188 MB); in tiles of 64 rows through shared memory (experts.cu) 38 and 21 us.
#include "common.cuh"
#include "mma_helpers.cuh"

namespace {
constexpr int TILE_M = 64;      // rows of a tile of the sorted slots

__device__ __forceinline__ uint4 ld_stream(const void* p) {      // weights: read once, do not keep in L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// MODE 1: gated, rows gathered from the tokens; 2: relu squared, gathered; 0: rows in sorted order, the result in 32 bit to the slots.
// Blocks that an SM shall have room for (0: as the compiler has it, 71 to 130 registers).  Up to eight rows: held to 64 registers (a few spilled), so that an SM
// has 32 warps and not 24 of these streams, and 1,024 blocks go in two rounds and not three: 16 experts of 2 x 1,024 x 2,048 and 2,048 x 1,024, 8 tokens:
// 28.1 -> 24.7 and 15.2 -> 13.4 us (5.4 and 5.0 TB/s); 48 registers with fewer loads under way 29.8 and 14.9.  But gated products of K <= 1,024 in blocks of four
// warps lose by it (the layer at width 1,024, 8 tokens: 34.6 -> 35.6 us), and so do results in 32 bit with K <= 512 behind them (SHORT: 34.8 -> 35.4; K = 1,024
// gains, 60.5 -> 58.4 at width 2,048).  The first product of relu squared gains for 17 and more rows by more loads under way,
// 106 registers and 16 warps: the layer with 24 tokens, width 2,048 and 1,024: 68.1 -> 61.2 and 32.1 -> 29.5.  The others of nine and more rows lose by more registers: relu
// squared, 16 tokens, 45.3 -> 51.4 and 26.6 -> 28.2; gated ones, whose 146 and 158 leave room for 12 warps and not 16, 74.1 -> 86.7 at 16 tokens and
// 92.4 -> 100.6 at 24, width 2,048; results in 32 bit for 17 and more rows, behind gated ones, 91.0 -> 95.5 at 24.
constexpr int least_blocks(int mode, int mt, int warps, bool shorter) {
  return mt == 1 && !shorter && !(mode == 1 && warps == 4) ? 32 / warps : mt == 4 && mode == 2 ? 16 / warps : 0;
}
template <int MODE, int MT, int WARPS, bool SHORT>
__global__ void __launch_bounds__(WARPS * 32, least_blocks(MODE, MT, WARPS, SHORT))
experts_stream_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ W, void* __restrict__ out, const int* __restrict__ sorted,
                      const int* __restrict__ tile_expert, int top, int N, int K, float limit, float alpha, float shift,
                      const float* __restrict__ row_scale) {
  constexpr int SETS = MODE == 1 ? 2 : 1, U = MT == 1 ? 4 : 2;
  const int e = tile_expert[blockIdx.y];
  if (e < 0) return;
  __shared__ float red[SETS][WARPS][16][8 * MT + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, n0 = blockIdx.x * 16;
  const int chunks = (K + 31) / 32;
  const __nv_bfloat16* wrow[SETS][2];
#pragma unroll
  for (int s = 0; s < SETS; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h) wrow[s][h] = W + ((size_t)e * SETS * N + (size_t)s * N + min(n0 + g + 8 * h, N - 1)) * K + t * 8;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  for (int m0 = 0; m0 < TILE_M; m0 += 8 * MT) {      // (an expert has as many rows as there are tokens at most: one round)
    const int p0 = blockIdx.y * TILE_M + m0;
    if (sorted[p0] < 0) break;      // a tile's rows come first
    const __nv_bfloat16* xrow[MT];
    int tiles = 1;
#pragma unroll
    for (int j = 0; j < MT; ++j) {
      const int s = sorted[p0 + 8 * j + g];
      xrow[j] = s < 0 ? nullptr : A + (size_t)(MODE != 0 ? s / top : p0 + 8 * j + g) * K + t * 8;
      if (__any_sync(0xffffffffu, s >= 0)) tiles = j + 1;
    }
    float acc[SETS][MT][4];
#pragma unroll
    for (int s = 0; s < SETS; ++s)
#pragma unroll
      for (int j = 0; j < MT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[s][j][q] = 0.f;
    for (int c0 = warp; c0 < chunks; c0 += U * WARPS) {
      uint4 wv[U][SETS][2], xv[U][MT];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = (c0 + u * WARPS) * 32;
        const bool in = k + t * 8 < K;
#pragma unroll
        for (int s = 0; s < SETS; ++s)
#pragma unroll
          for (int h = 0; h < 2; ++h) wv[u][s][h] = in ? ld_stream(wrow[s][h] + k) : zero;
#pragma unroll
        for (int j = 0; j < MT; ++j) xv[u][j] = in && j < tiles && xrow[j] != nullptr ? __ldg(reinterpret_cast<const uint4*>(xrow[j] + k)) : zero;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int s = 0; s < SETS; ++s) {
          const uint4 a = wv[u][s][0], b = wv[u][s][1];
          const uint32_t f0[4] = {a.x, b.x, a.y, b.y}, f1[4] = {a.z, b.z, a.w, b.w};
#pragma unroll
          for (int j = 0; j < MT; ++j)
            if (j < tiles) {
              mma_bf16(acc[s][j], f0, xv[u][j].x, xv[u][j].y);
              mma_bf16(acc[s][j], f1, xv[u][j].z, xv[u][j].w);
            }
        }
    }
    __syncthreads();      // the sums of the round before have been read
#pragma unroll
    for (int s = 0; s < SETS; ++s)
#pragma unroll
      for (int j = 0; j < MT; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) red[s][warp][g + 8 * (q >> 1)][8 * j + 2 * t + (q & 1)] = acc[s][j][q];
    __syncthreads();
    for (int i = threadIdx.x; i < 16 * 8 * MT; i += WARPS * 32) {
      const int n = n0 + (i & 15), m = i >> 4, s = sorted[p0 + m];
      if (s < 0 || n >= N) continue;
      float y = 0.f, u = 0.f;
#pragma unroll
      for (int q = 0; q < WARPS; ++q) {
        y += red[0][q][i & 15][m];
        if (MODE == 1) u += red[SETS - 1][q][i & 15][m];
      }
      const float rs = MODE != 0 && row_scale != nullptr ? row_scale[s] : 1.f;      // (w x) W^T = w (x W^T)
      if (MODE == 1)      // products rounded to bfloat16 first, as separate products would be
        ((__nv_bfloat16*)out)[(size_t)(p0 + m) * N + n] = __float2bfloat16_rn(dk_glu_value(
            __bfloat162float(__float2bfloat16_rn(y * rs)), __bfloat162float(__float2bfloat16_rn(u * rs)), limit, alpha, shift));
      else if (MODE == 2) {
        const float v = fmaxf(__bfloat162float(__float2bfloat16_rn(y * rs)), 0.f);
        ((__nv_bfloat16*)out)[(size_t)(p0 + m) * N + n] = __float2bfloat16_rn(v * v);
      } else {
        ((float*)out)[(size_t)s * N + n] = y;
      }
    }
  }
}
}  // namespace

extern "C" int dk_experts_stream_supported(int K) { return K > 0 && K % 8 == 0; }

// Arguments as for dk_experts_gemm (experts.cu) with bfloat16 operands.  `most`: an expert has about this many rows at most (more are taken in
// rounds).
extern "C" int dk_experts_stream(const void* A, const void* W, void* out, const int* sorted, const int* tile_expert, int max_tiles, int top, int N, int K,
                                 int act, float limit, float alpha, float shift, const float* row_scale, int most, cudaStream_t stream) {
  if (max_tiles == 0) return 0;
  DK_REQUIRE(max_tiles > 0 && max_tiles <= 65535 && N > 0 && top > 0 && most > 0 && dk_experts_stream_supported(K), "experts_stream: bad sizes tiles=%d N=%d K=%d top=%d",
             max_tiles, N, K, top);
  DK_REQUIRE(act >= 0 && act <= 2, "experts_stream: activation %d is not known (0 none, 1 gated, 2 relu squared)", act);
  DK_REQUIRE(((uintptr_t)A | (uintptr_t)W) % 16 == 0, "experts_stream: operands must start on 16-byte boundaries");
  const dim3 grid((N + 15) / 16, max_tiles);
  const auto *a = (const __nv_bfloat16*)A, *w = (const __nv_bfloat16*)W;
  // four warps a block where a warp of eight would have four chunks of K or fewer
#define RUN(MODE, MT, WARPS, SHORT) \
  experts_stream_kernel<MODE, MT, WARPS, SHORT><<<grid, WARPS * 32, 0, stream>>>(a, w, out, sorted, tile_expert, top, N, K, limit, alpha, shift, row_scale)
#define SIZE(MODE, MT)                                              \
  do {                                                              \
    if (MODE == 0 && MT == 1 && K <= 512) RUN(MODE, MT, 4, MODE == 0 && MT == 1); \
    else if (K <= 1024) RUN(MODE, MT, 4, false);                    \
    else RUN(MODE, MT, 8, false);                                   \
  } while (0)
#define PICK(MODE)                       \
  do {                                   \
    if (most <= 8) SIZE(MODE, 1);        \
    else if (most <= 16) SIZE(MODE, 2);  \
    else SIZE(MODE, 4);                  \
  } while (0)
  if (act == 1) PICK(1);
  else if (act == 2) PICK(2);
  else PICK(0);
#undef PICK
#undef SIZE
#undef RUN
  return dk_check_launch("experts_stream");
}
