// 32-bit product  C[M,N] = A[M,K] * W[N,K]^T  on the fifth-generation tensor cores, operands in three exact bfloat16 parts.
//
// A 32-bit number is three bfloat16 parts exactly (each what the parts before it leave, rounded to nearest), x = x1 + x2 + x3, and products of parts
// are exact in 32 bit.  Of the nine products of parts six are made; the three left out are at most 2^-24 of a term together, of either sign, 2^-26.5 in
// the mean square (a multiply-add's rounding: 2^-24.3).  A tensor core cuts off what it adds to its accumulator, so the high parts' products, of which a sum
// of 24 bits holds nearly all, have one of their own, which begins at zero every 64 entries of K; the other five, 2^-8 of those, are kept together for
// KEEP chunks.  Either is added to 32-bit sums in registers, rounded to nearest.  The order of a sum depends on nothing but W's sizes: a token's result
// has the same bits whatever shares its step.  Errors against 64 bits (2-norm), and those of chains of fused multiply-adds (gemm_plain.cu): normal operands,
// K of 1,024 to 11,008, 1.0e-7 to 1.5e-7 and 5.7e-7 to 18.8e-7; rows that one or four entries dominate 1.3e-7 to 1.7e-7 and 5.8e-7 to 18.5e-7; operands of one
// sign 0.5e-7 to 1.0e-7 and 4.4e-7 to 16.1e-7; rows of four entries 0.44e-7 to 0.47e-7 and 0.40e-7 to 0.41e-7; a single product is off by 2^-23 of it at most.
//   1. split_rows: the tokens' rows as three bfloat16 arrays, and which rows are out of the parts' reach;
//   2. the product: W's rows are the M side (128 lanes), tokens the N side of the tiles.  One persistent block per SM:
//      warp 0       fetches W (32 bit, TMA, 128-byte swizzle), warp 2 the tokens' parts (a box each, a ring of its own),
//      warps 4-11   turn W into parts: a thread holds half of a row, and its parts go straight into tensor memory as an MMA's first operand, so that the
//                   shared memory's bandwidth is left to the tokens' parts,
//      warp 1       issues 24 products a chunk, four of them the high parts',
//      warps 12-19  add finished chunks to the sums in registers and store them;
//   3. add_segments, where K is cut into segments (W of few tiles): their sums in order.
// Rows with infinite or NaN entries, or whose largest entry is outside 2^-40 .. 2^29, are found on the way, and their results are summed by FMA over k
// instead, a tile at a time, when nothing waits any more: by the product's own blocks behind their pieces, or by add_segments.
// A chunk takes about 1,650 cycles for few tokens, the converting warps' own time, and 2,500 for 160 of them: 24 products, and one chunk in four waits for
// sums that are being read.  Parts that are rounded cost half as much again as parts that are cut off, so eight warps make them and not four; a product's
// operands reach it from one elected thread in 50 to 80 cycles (in a branch for lane 0 in 100, which bound everything), and one wait stands for all that
// a chunk needs.  Everything cold, microseconds, against the tiles of gemm_plain.cu: 300 x 2,048 x 2,048 107 -> 40, 300 x 11,008 x 2,048 317 -> 97,
// 300 x 2,048 x 5,504 274 -> 63, 300 x 32,000 x 2,048 930 -> 212, 2,048 x 22,016 x 4,096 7,590 -> 1,690 (218 TFLOP/s); one row: 44 -> 24, 76 -> 46,
// 107 -> 34, 139 -> 83, and 203 -> 138 with 22,016 x 4,096.
//
// Every wait on an mbarrier is bounded: when one gives up, the kernel records it, stores nothing more, waits (bounded again) for the copies and
// products that it has under way, frees its tensor memory and returns.
#include "common.cuh"
#include "mma_helpers.cuh"
#include "tcgen05_helpers.cuh"
#include "ring.cuh"

namespace {
constexpr int BM = 128;                 // rows of W of a piece
constexpr int KC = 64;                  // entries of K of a chunk
constexpr int THREADS = 640, CONVERT = 4, STORE = 12;      // the first warp that turns W into parts, that adds up and stores
constexpr int W_STAGE = BM * KC * 4;
constexpr int MAX_W = 6, MAX_X = 12;
constexpr int SMEM_ROOM = 222 * 1024;
constexpr int TMEM_COLS = 512;
constexpr int KEEP = 4;                 // chunks for which the products of other parts than the high ones stay in tensor memory
constexpr int A_COLS = 3 * KC / 2;      // tensor memory of a chunk of W in parts
constexpr int MOST_ROWS = 16384;        // of A in a launch
constexpr long long MOST_PARTS = 48ll << 20, MOST_PARTIAL = 64ll << 20;      // bytes of the tokens' parts and of the segments' sums

// A row is in reach of the parts if its largest entry is zero or lies in 2^-40 .. 2^29.  Operands are multiplied by 2^24 first (the results by
// 2^-48): the last part of the smallest entry is still a normal bfloat16 number, and 2^20 products of two numbers in reach stay below the exponent's
// range.
constexpr float SCALE = 16777216.f, UNSCALE = 1.f / 16777216.f / 16777216.f;
__device__ __forceinline__ bool out_of_reach(uint32_t largest) { return largest != 0 && (largest < (127u - 40u) << 23 || largest >= (127u + 29u) << 23); }

// Two numbers' parts, each rounded to nearest: what a part leaves fits the two after it, and the products that are left out have either sign.
__device__ __forceinline__ uint32_t nearest(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void parts_of(float x, float y, uint32_t& high, uint32_t& middle, uint32_t& low) {
  x *= SCALE;
  y *= SCALE;
  high = nearest(x, y);
  x -= __uint_as_float(high << 16);
  y -= __uint_as_float(high & 0xffff0000u);
  middle = nearest(x, y);
  low = nearest(x - __uint_as_float(middle << 16), y - __uint_as_float(middle & 0xffff0000u));
}

// grid (rows): parts [3][M][K] and a row's flag; the flags of W's rows, and the one behind them, begin at zero.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ A, int lda, __nv_bfloat16* __restrict__ parts, int* __restrict__ flags,
                                                         int* __restrict__ w_flags, int M, int N, int K, int ldp, int vec) {
  for (int n = blockIdx.x * 256 + threadIdx.x; n <= N; n += gridDim.x * 256) w_flags[n] = 0;
  __shared__ uint32_t most[8];
  const int m = blockIdx.x, tid = threadIdx.x;
  const float* row = A + (size_t)m * lda;
  const size_t plane = (size_t)M * ldp;
  __nv_bfloat16* to = parts + (size_t)m * ldp;
  uint32_t largest = 0;
  for (int k = tid * 4; k < K; k += 1024) {      // K is a multiple of 4
    float4 v;
    if (vec) v = *reinterpret_cast<const float4*>(row + k);
    else v = make_float4(row[k], row[k + 1], row[k + 2], row[k + 3]);
    uint2 h, m2, l;
    parts_of(v.x, v.y, h.x, m2.x, l.x);
    parts_of(v.z, v.w, h.y, m2.y, l.y);
    *reinterpret_cast<uint2*>(to + k) = h;
    *reinterpret_cast<uint2*>(to + plane + k) = m2;
    *reinterpret_cast<uint2*>(to + 2 * plane + k) = l;
    const uint32_t a = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
    const uint32_t b = max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu);
    largest = max(largest, max(a, b));
  }
  largest = __reduce_max_sync(0xffffffffu, largest);
  if ((tid & 31) == 0) most[tid >> 5] = largest;
  __syncthreads();
  if (tid == 0) {
    for (int i = 1; i < 8; ++i) largest = max(largest, most[i]);
    flags[m] = out_of_reach(largest);
  }
}

template <int BN>
struct Sizes {
  static constexpr int X_STAGE = BN * KC * 2;
  static constexpr int WS = BN <= 32 ? 6 : BN <= 64 ? 4 : 3;
  static constexpr int XS = (SMEM_ROOM - WS * W_STAGE) / X_STAGE < MAX_X ? (SMEM_ROOM - WS * W_STAGE) / X_STAGE : MAX_X;
  static constexpr int SMEM = WS * W_STAGE + XS * X_STAGE + 1024;
  static_assert(XS >= 6, "two chunks of parts");
  static constexpr int D_COLS = (BN + 31) / 32 * 32;
  // Accumulators of the products of high parts, and of the others: two of either, as far as there is room beside two chunks of W.
  static constexpr int HIGH = 3 * D_COLS + 2 * A_COLS <= TMEM_COLS ? 2 : 1, REST = 4 * D_COLS + 2 * A_COLS <= TMEM_COLS ? 2 : 1;
  static_assert((HIGH + REST) * D_COLS + 2 * A_COLS <= TMEM_COLS, "accumulators beside two chunks of W");
};

struct F32Args {
  const float* A;
  const float* W;
  float* C;
  const int* flags;      // rows of A out of reach
  float* partial;        // [segments][M][N] where K is cut into segments, else null
  int* w_flags;          // [N + 1]: rows of W out of reach; the last, with segments: some row of A or W is
  int* err;
  int M, N, K, lda, ldw, ldc, tok_tiles, items;
  int vec;               // rows of A begin on 16-byte boundaries
  int segments, per;     // chunks of K of a segment
};

// Piece number `item`: token tiles fastest, so that a tile of W comes from memory once; then K's segments, then W's tiles.
struct Piece {
  int m0, n0, segment, first, chunks;
  __device__ __forceinline__ Piece(const F32Args& a, int item, int bn) {
    const int rest = item / a.tok_tiles;
    m0 = (item - rest * a.tok_tiles) * bn;
    segment = rest % a.segments;
    n0 = rest / a.segments * BM;
    first = segment * a.per;
    chunks = min(a.per, (a.K + KC - 1) / KC - first);
  }
};

// Results out of the parts' reach, for `most` tokens from m0 on and 128 rows of W from n0 on: the rows of A that need it, by the rows of W, every sum in the
// plain kernel's order over k.  A thread has EACH tokens by four rows of W; both come by cp.async, STAGES - 1 steps of K ahead.  Bound by the reads of
// shared memory (four cycles a sixteen-byte load, whatever its lanes share).
// 300 rows with a NaN each by 2,048 x 2,048 and 9,600 x 1,024: 227 and 323 us in all (gemm_plain.cu alone 105 and 186); one by 12,000 x 2,048 146 (75).
constexpr int FMA_K = 16, FMA_LD = FMA_K + 4;
template <int T, int EACH, int STAGES>
struct FmaTile {
  static constexpr int AT_ONCE = T / 32 * EACH;
  float w[STAGES][BM][FMA_LD], x[STAGES][AT_ONCE][FMA_LD];
  int rows[160], count;
};
template <int T, int EACH, int STAGES>
__device__ __forceinline__ void fma_tile(FmaTile<T, EACH, STAGES>& sm, const F32Args& a, int m0, int most, int n0) {
  constexpr int AT_ONCE = FmaTile<T, EACH, STAGES>::AT_ONCE, V = FMA_K / 4, LX = AT_ONCE * V;
  static_assert(LX <= T, "a vector a thread");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c = tid % V * 4;
  int w_odd = 0;      // of the thread's rows of W
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (n0 + lane + 32 * j < a.N) w_odd |= (*(volatile const int*)(a.w_flags + n0 + lane + 32 * j) != 0) << j;
  const bool all = __syncthreads_or(w_odd) != 0;
  if (warp == 0) {
    int count = 0;
    for (int j0 = 0; j0 < most; j0 += 32) {
      const int j = j0 + lane;
      const bool mine = j < most && m0 + j < a.M && (all || a.flags[m0 + j] != 0);
      const uint32_t them = __ballot_sync(0xffffffffu, mine);
      if (mine) sm.rows[count + __popc(them & ((1u << lane) - 1u))] = m0 + j;
      count += __popc(them);
    }
    if (lane == 0) sm.count = count;
  }
  __syncthreads();
  const int count = sm.count, steps = (a.K + FMA_K - 1) / FMA_K;
  for (int p0 = 0; p0 < count; p0 += AT_ONCE) {
    const bool has_x = tid < LX && p0 + tid / V < count;
    const float* xrow = a.A + (size_t)(has_x ? sm.rows[p0 + tid / V] : 0) * a.lda + c;
    auto fetch = [&](int s) {
      const int k0 = s * FMA_K;
      if (s < steps) {
        for (int v = tid; v < BM * V; v += T) {      // (T is a multiple of V)
          const int r = v / V;
          const bool in = n0 + r < a.N && k0 + c < a.K;
          cp_async_16(s2u(&sm.w[s % STAGES][r][c]), in ? a.W + (size_t)(n0 + r) * a.ldw + k0 + c : a.W, in);
        }
        if (tid < LX) {
          const bool in = has_x && k0 + c < a.K;
          float* to = &sm.x[s % STAGES][tid / V][c];
          if (a.vec) cp_async_16(s2u(to), in ? xrow + k0 : a.W, in);
          else
            for (int i = 0; i < 4; ++i) to[i] = in ? xrow[k0 + i] : 0.f;
        }
      }
      cp_async_commit();
    };
    float acc[EACH][4];
#pragma unroll
    for (int i = 0; i < EACH; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    const bool some = p0 + warp * EACH < count;
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    for (int s = 0; s < steps; ++s) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();      // step s is in, and everybody has left the one whose place is taken next
      fetch(s + STAGES - 1);
      if (!some) continue;
      const float *w = sm.w[s % STAGES][lane], *x = sm.x[s % STAGES][warp * EACH];
#pragma unroll
      for (int k = 0; k < FMA_K; k += 4) {
        float4 b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(w + j * 32 * FMA_LD + k);
#pragma unroll
        for (int i = 0; i < EACH; ++i) {
          const float4 v = *reinterpret_cast<const float4*>(x + i * FMA_LD + k);
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(v.w, b[j].w, fmaf(v.z, b[j].z, fmaf(v.y, b[j].y, fmaf(v.x, b[j].x, acc[i][j]))));
        }
      }
    }
    cp_async_wait<0>();
    __syncthreads();      // (the stages are the next tokens')
#pragma unroll
    for (int i = 0; i < EACH; ++i) {
      const int r = p0 + warp * EACH + i;
      if (r >= count) continue;
      const int m = sm.rows[r], x_odd = a.flags[m];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n0 + lane + 32 * j < a.N && (x_odd != 0 || (w_odd >> j & 1) != 0)) a.C[(size_t)m * a.ldc + n0 + lane + 32 * j] = acc[i][j];
    }
  }
  __syncthreads();      // (the list is another tile's next)
}
using OwnTile = FmaTile<THREADS, 7, 4>;

template <int BN>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                 const F32Args a) {
  constexpr int WS = Sizes<BN>::WS, XS = Sizes<BN>::XS, X_STAGE = Sizes<BN>::X_STAGE, D_COLS = Sizes<BN>::D_COLS, NC = BN / 2;
  constexpr int HIGH = Sizes<BN>::HIGH, REST = Sizes<BN>::REST;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* xs = smem + WS * W_STAGE;
  __shared__ __align__(8) unsigned long long bars[2 * MAX_W + 2 * MAX_X + 10];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int failed, odd;      // odd: some row of the block's pieces is out of reach
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t wfull = s2u(&bars[0]), wempty = s2u(&bars[MAX_W]), xfull = s2u(&bars[2 * MAX_W]), xempty = s2u(&bars[2 * MAX_W + MAX_X]);
  const uint32_t afull = s2u(&bars[2 * MAX_W + 2 * MAX_X]), done = afull + 16, dempty = afull + 32;
  const uint32_t rdone = afull + 48, rempty = afull + 64;      // the rest's sums are complete; have been read
  if (tid == 0) {
    for (int s = 0; s < WS; ++s) {
      mbar_init(wfull + 8 * s, 1);
      mbar_init(wempty + 8 * s, STORE - CONVERT);
    }
    for (int s = 0; s < XS; ++s) {
      mbar_init(xfull + 8 * s, 1);
      mbar_init(xempty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(afull + 8 * b, STORE - CONVERT);
      mbar_init(done + 8 * b, 1);
      mbar_init(dempty + 8 * b, 8);
      mbar_init(rdone + 8 * b, 1);
      mbar_init(rempty + 8 * b, 8);
    }
    failed = odd = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) tmem_alloc(s2u(&tmem_base_slot), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot, tmem_rest = tmem_base + HIGH * D_COLS, tmem_a = tmem_rest + REST * D_COLS;
  volatile int* gave_up = &failed;

  if (warp == 0) {
    if (lane == 0) {
      int c = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
        const Piece p(a, item, BN);
        for (int k = p.first; k < p.first + p.chunks; ++k, ++c) {
          const int s = ring_slot(c, WS);
          if (c >= WS && !mbar_wait(wempty + 8 * s, ring_parity(c - WS, WS))) {
            *gave_up = 1;
            ok = false;
            break;
          }
          const uint32_t to = s2u(smem + (size_t)s * W_STAGE), bar = wfull + 8 * s;
          mbar_expect_tx(bar, W_STAGE);
          tma_load_2d(to, &map_w, k * KC, p.n0, bar);      // rows past N and entries past K are zeros
          tma_load_2d(to + W_STAGE / 2, &map_w, k * KC + KC / 2, p.n0, bar);
        }
      }
      ring_drain(c, WS, [&](int s, uint32_t parity) { return mbar_wait(wfull + 8 * s, parity); });
    }
  } else if (warp == 2) {
    if (lane == 0) {
      int c = 0;      // parts asked for: the third, the second, the first of every chunk
      bool ok = true;
      for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
        const Piece piece(a, item, BN);
        for (int k = piece.first; k < piece.first + piece.chunks && ok; ++k)
          for (int p = 2; p >= 0; --p, ++c) {
            const int s = ring_slot(c, XS);
            if (c >= XS && !mbar_wait(xempty + 8 * s, ring_parity(c - XS, XS))) {
              *gave_up = 1;
              ok = false;
              break;
            }
            const uint32_t bar = xfull + 8 * s;
            mbar_expect_tx(bar, X_STAGE);
            tma_load_2d(s2u(xs + (size_t)s * X_STAGE), &map_x, k * KC, p * a.M + piece.m0, bar);      // (rows past M: another part's, of no token's column)
          }
      }
      ring_drain(c, XS, [&](int s, uint32_t parity) { return mbar_wait(xfull + 8 * s, parity); });
    }
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(BM, BN);
    int c = 0, rest = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const Piece p(a, item, BN);
      for (int k = 0; k < p.chunks; ++k, ++c) {
        const int b = c & 1, x = 3 * c, first = k % KEEP == 0;
        // a lane waits for each of what a chunk needs, all at once: in a branch of its own for each the waits took 870 cycles
        const int part = x + min(max(lane - 2, 0), 2);
        uint32_t bar = xfull + 8 * ring_slot(part, XS), parity = ring_parity(part, XS);
        if (lane == 0 && first && rest >= REST) bar = rempty + 8 * ((rest - REST) & 1), parity = ring_parity(rest - REST, 2);
        if (lane == 1) bar = afull + 8 * b, parity = ring_parity(c, 2);
        bool there = mbar_wait(bar, parity);
        if (__any_sync(0xffffffffu, !there)) {
          *gave_up = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t wa = tmem_a + b * A_COLS, xlast = xempty + 8 * ring_slot(x + 2, XS);
        const auto multiply = [&](uint32_t d, int q, int r, bool add) {      // the tokens' part q with W's part r
          const uint64_t db = smem_desc_k_major(s2u(xs + (size_t)ring_slot(x + 2 - q, XS) * X_STAGE));
#pragma unroll
          for (int i = 0; i < KC / 16; ++i) umma_a_tmem(d, wa + r * (KC / 2) + i * 8, db + (uint64_t)(i * 2), idesc, (add || i > 0) ? 1u : 0u);
        };
        if (elect_one()) {      // the smallest products first
          const uint32_t d = tmem_rest + rest % REST * D_COLS;
          multiply(d, 2, 0, !first);
          umma_commit(xempty + 8 * ring_slot(x, XS));
          multiply(d, 1, 1, true);
          multiply(d, 1, 0, true);
          umma_commit(xempty + 8 * ring_slot(x + 1, XS));
          multiply(d, 0, 2, true);
          multiply(d, 0, 1, true);
        }
        __syncwarp();
        if (k % KEEP == KEEP - 1 || k + 1 == p.chunks) {
          if (elect_one()) umma_commit(rdone + 8 * (rest & 1));
          ++rest;
        }
        there = c < HIGH || mbar_wait(dempty + 8 * ((c - HIGH) & 1), ring_parity(c - HIGH, 2));
        const bool go = !__any_sync(0xffffffffu, !there);
        tc_fence_after();
        if (elect_one()) {
          if (go) multiply(tmem_base + c % HIGH * D_COLS, 0, 0, false);
          umma_commit(xlast);
          if (go) umma_commit(done + 8 * b);
        }
        __syncwarp();
        if (!go) {
          *gave_up = 1;
          ok = false;
          ++c;
          break;
        }
      }
    }
    if (lane == 0) ring_drain(3 * c, XS, [&](int s, uint32_t parity) { return mbar_wait(xempty + 8 * s, parity); });      // its products are complete
  } else if (warp >= CONVERT && warp < STORE) {
    const int row = tid & 127, half = (warp - CONVERT) >> 2;      // 32 of a row's 64 entries
    int c = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const Piece p(a, item, BN);
      uint32_t largest = 0;
      for (int k = 0; k < p.chunks; ++k, ++c) {
        const int s = ring_slot(c, WS), b = c & 1;
        const bool there = mbar_wait(wfull + 8 * s, ring_parity(c, WS)) && (c < 2 || mbar_wait(done + 8 * b, ring_parity(c - 2, 2))) && *gave_up == 0;
        if (__any_sync(0xffffffffu, !there)) {      // the whole warp leaves, or none of it
          *gave_up = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        const unsigned char* from = smem + (size_t)s * W_STAGE + row * 128;
        const uint32_t to = tmem_a + b * A_COLS + ((uint32_t)((warp & 3) * 32) << 16);
        uint32_t h[16], m[16], l[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(from + half * (W_STAGE / 2) + ((j ^ (row & 7)) << 4));
          parts_of(v.x, v.y, h[2 * j], m[2 * j], l[2 * j]);
          parts_of(v.z, v.w, h[2 * j + 1], m[2 * j + 1], l[2 * j + 1]);
          largest = max(largest, max(max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu),
                                     max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu)));
        }
        tmem_st16(to + half * 16, h);
        tmem_st16(to + KC / 2 + half * 16, m);
        tmem_st16(to + KC + half * 16, l);
        if (k + 1 == p.chunks && out_of_reach(largest) && p.n0 + row < a.N) {      // (what the thread saw of the row: half of the piece's K)
          a.w_flags[p.n0 + row] = 1;
          odd = 1;
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(wempty + 8 * s);
          mbar_arrive(afull + 8 * b);
        }
      }
    }
  } else if (warp >= STORE) {
    const int quarter = warp & 3, half = (warp - STORE) >> 2;
    const int row = quarter * 32 + lane;
    int c = 0, rest = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < a.items && ok; item += gridDim.x) {
      const Piece p(a, item, BN);
      const int n = p.n0 + row, m0 = p.m0 + half * NC;
      float sum[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) sum[j] = 0.f;
      for (int k = 0; k < p.chunks; ++k, ++c) {
        const bool all = k % KEEP == KEEP - 1 || k + 1 == p.chunks;      // the rest is complete, too
#pragma unroll 1
        for (int high = all ? 0 : 1; high < 2; ++high) {
          const int use = high ? c : rest++;
          const bool there = mbar_wait((high ? done : rdone) + 8 * (use & 1), ring_parity(use, 2)) && *gave_up == 0;
          if (__any_sync(0xffffffffu, !there)) {
            *gave_up = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t at = (high ? tmem_base + use % HIGH * D_COLS : tmem_rest + use % REST * D_COLS) + half * NC + ((uint32_t)(quarter * 32) << 16);
          constexpr int G = NC > 64 ? 8 : NC > 48 ? 16 : 32;      // columns on their way at a time: as many as there are registers for
#pragma unroll
          for (int g = 0; g < NC; g += G) {
            float v[G];
#pragma unroll
            for (int j = 0; j < G; j += 8)
              if (g + j < NC) tmem_ld8_nowait(at + g + j, v + j);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < G; ++j)
              if (g + j < NC) sum[g + j] += v[j];
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive((high ? dempty : rempty) + 8 * (use & 1));
        }
        if (!ok) break;
      }
      if (!ok) break;
      float* to = a.partial != nullptr ? a.partial + (size_t)p.segment * a.M * a.N : a.C;
      const int ld = a.partial != nullptr ? a.N : a.ldc;
      const float unscale = a.partial != nullptr ? 1.f : UNSCALE;
#pragma unroll
      for (int j = 0; j < NC; ++j)
        if (n < a.N && m0 + j < a.M) to[(size_t)(m0 + j) * ld + n] = sum[j] * unscale;
    }
  } else if (warp == 3) {      // looks for tokens out of reach meanwhile
    bool mine = false;
    for (int item = blockIdx.x; item < a.items; item += gridDim.x) {
      const Piece p(a, item, BN);
      for (int j = lane; j < BN; j += 32) mine |= p.m0 + j < a.M && a.flags[p.m0 + j] != 0;
    }
    if (mine) odd = 1;
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (failed && tid == 0) dk_report(a.err, DK_DEV_TIMEOUT, blockIdx.x, 0, a.per);
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
  if (!odd || failed) return;
  if (a.partial != nullptr) {
    if (tid == 0) a.w_flags[a.N] = 1;
    return;
  }
  for (int item = blockIdx.x; item < a.items; item += gridDim.x) {      // (with no copy and no product under way, and nobody waiting)
    const Piece p(a, item, BN);
    fma_tile(*reinterpret_cast<OwnTile*>(smem), a, p.m0, BN, p.n0);
  }
}

// The segments' sums, added in their order.
__global__ void __launch_bounds__(256, 8) add_segments_kernel(const F32Args a) {      // (32 registers: the sums wait for memory)
  using Tile = FmaTile<256, 2, 2>;
  __shared__ __align__(16) Tile sm;
  const long long total = (long long)a.M * a.N;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
    const int m = (int)(i / a.N), n = (int)(i - (long long)m * a.N);
    float v = a.partial[i];
#pragma unroll 4
    for (int s = 1; s < a.segments; ++s) v += a.partial[i + s * total];
    if (a.w_flags[n] == 0 && a.flags[m] == 0) a.C[(size_t)m * a.ldc + n] = v * UNSCALE;
  }
  if (a.w_flags[a.N] == 0) return;
  const int across = (a.N + BM - 1) / BM, down = (a.M + Tile::AT_ONCE - 1) / Tile::AT_ONCE;
  for (int t = blockIdx.x; t < across * down; t += gridDim.x) fma_tile(sm, a, t / across * Tile::AT_ONCE, Tile::AT_ONCE, t % across * BM);
}

// 2-D tensor [rows, cols] of floats, boxes of [box_rows x 32], 128-byte swizzle, zeros where a box reaches past the tensor
bool make_tensor_map_f32(CUtensorMap* m, const void* base, long long rows, int cols, long long ld, int box_rows) {
  TensorMapEncodeFn fn = tensor_map_encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {32u, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN>
int launch(F32Args a, const __nv_bfloat16* parts, int ldp, const CUtensorMap& map_w, cudaStream_t stream) {
  static bool granted[DK_MAX_DEVICES] = {false};
  bool& ok = granted[dk_current_device()];
  if (!ok) {
    DK_REQUIRE(cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sizes<BN>::SMEM) == cudaSuccess,
               "gemm_f32_tc: %d bytes of shared memory were refused", Sizes<BN>::SMEM);
    ok = true;
  }
  CUtensorMap map_x;
  DK_REQUIRE(make_tensor_map_bf16(&map_x, parts, 3ll * a.M, a.K, ldp, BN), "gemm_f32_tc: cannot encode the tensor map of the parts");
  a.tok_tiles = (a.M + BN - 1) / BN;
  const long long items = (long long)a.tok_tiles * a.segments * ((a.N + BM - 1) / BM);
  DK_REQUIRE(items < (1ll << 30), "gemm_f32_tc: too many pieces");
  static_assert(sizeof(OwnTile) <= Sizes<BN>::SMEM - 1024 && BN <= 160, "the rows out of reach take the stages' place");
  a.items = (int)items;
  gemm_f32_tc_kernel<BN><<<min(a.items, dk_sm_count()), THREADS, Sizes<BN>::SMEM, stream>>>(map_w, map_x, a);
  return 0;
}
// How K is cut: by W's sizes alone, so that a token's sum has one order whatever the step.  A matrix of few tiles would leave most SMs idle
// (2,048 rows are 16 tiles); with segments of four chunks and more its tiles fill SPREAD of them, and their sums are added by a kernel of their own.
constexpr int SPREAD = 148, LEAST_CHUNKS = 4;
struct Cut {
  int segments, per;
  Cut(int N, int K) {
    const int chunks = (K + KC - 1) / KC;
    const long long tiles = (N + BM - 1) / BM;
    per = chunks;
    if (tiles <= SPREAD / 2) per = (int)max((long long)LEAST_CHUNKS, (chunks * tiles + SPREAD - 1) / SPREAD);
    segments = (chunks + per - 1) / per;
  }
};
// Rows of A that one launch takes: they bound the working memory to 113 MB and 4 bytes a row of W.  Every launch reads W
// anew: 2,048 rows by 2,048 x 5,504 are three, 345 us in all, of which W's 45 MB take 7 each.
int slab_rows(int N, int K, int segments) {
  long long rows = min((long long)MOST_ROWS, MOST_PARTS / (6ll * ((K + 7) / 8 * 8)));
  if (segments > 1) rows = min(rows, MOST_PARTIAL / (4ll * segments * N));
  return (int)max(32ll, rows / 32 * 32);
}
}  // namespace

// Whether a product with W [N, K] takes this way: a rule on W alone, so that a token's sums are made in one order whatever the step.
extern "C" int dk_gemm_f32_tc_supported(const void* W, int N, int K) {
  // Shorter sums are as fast or faster by FMA: 1,024 x 1,024 25.6 against 24.6 us for one row and 27.6 against 43 for 300; 256 x 512 23.6 against 16.4.
  return K >= (N >= 4096 ? 512 : 1024) && K <= (1 << 20) && K % 4 == 0 && N > 0 && N <= (1 << 24) && (uintptr_t)W % 16 == 0;
}

// Kilobytes of working memory for M rows, and the launches that they take.
extern "C" int dk_gemm_f32_tc_plan(int M, int N, int K, int* kilobytes, int* launches) {
  DK_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32_tc: bad sizes M=%d N=%d K=%d", M, N, K);
  const Cut cut(N, K);
  const int slab = slab_rows(N, K, cut.segments);
  const long long rows = min(M, slab), ldp = (K + 7) / 8 * 8;
  long long bytes = 6 * rows * ldp + 4 * rows + 16 + 4ll * N + 32;
  if (cut.segments > 1) bytes += 4ll * cut.segments * rows * N;
  *kilobytes = (int)((bytes + 1023) / 1024);
  *launches = (M + slab - 1) / slab * (cut.segments > 1 ? 3 : 2);
  return 0;
}

extern "C" int dk_gemm_f32_tc(const void* A, const void* W, void* C, void* work, int M, int N, int K, int lda, int ldw, int ldc, int* err,
                              cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  DK_REQUIRE(M > 0 && dk_gemm_f32_tc_supported(W, N, K), "gemm_f32_tc: sizes not taken: M=%d N=%d K=%d", M, N, K);
  DK_REQUIRE(lda >= K && ldw >= K && ldc >= N && ldw % 4 == 0, "gemm_f32_tc: leading sizes %d %d %d are not taken", lda, ldw, ldc);
  DK_REQUIRE(work != nullptr && (uintptr_t)work % 16 == 0, "gemm_f32_tc: working memory must start on a 16-byte boundary");
  const int ldp = (K + 7) / 8 * 8, sms = dk_sm_count();
  const Cut cut(N, K);
  const int slab = slab_rows(N, K, cut.segments);
  CUtensorMap map_w;
  DK_REQUIRE(make_tensor_map_f32(&map_w, W, N, K, ldw, BM), "gemm_f32_tc: cannot encode the tensor map of W");
  for (int m = 0; m < M; m += slab) {
    F32Args a = {};
    a.M = min(slab, M - m);
    a.A = (const float*)A + (size_t)m * lda;
    a.W = (const float*)W;
    a.C = (float*)C + (size_t)m * ldc;
    a.N = N; a.K = K; a.lda = lda; a.ldw = ldw; a.ldc = ldc;
    a.segments = cut.segments; a.per = cut.per;
    a.err = err;
    auto* parts = (__nv_bfloat16*)work;
    int* flags = (int*)(parts + 3ll * a.M * ldp);
    a.flags = flags;
    a.w_flags = flags + (a.M + 3) / 4 * 4;
    if (cut.segments > 1) a.partial = (float*)(a.w_flags + N / 4 * 4 + 4);
    a.vec = (uintptr_t)a.A % 16 == 0 && lda % 4 == 0;
    split_rows_kernel<<<a.M, 256, 0, stream>>>(a.A, lda, parts, flags, a.w_flags, a.M, N, K, ldp, a.vec);
    // Tokens of a piece: a chunk takes 12 cycles a token on the tensor cores, and about 2,000 whatever their number (W's way into parts, 24 products'
    // issue).  Least rounds of pieces times that, and the fewest tokens that give it: more stages of W beside them.
    const int sizes[] = {160, 144, 128, 112, 96, 80, 64, 48, 32, 16};
    int best = 0;
    long long least = 0;
    for (int bn : sizes) {
      const long long items = (long long)((a.M + bn - 1) / bn) * cut.segments * ((N + BM - 1) / BM), cost = (items + sms - 1) / sms * max(12 * bn, 2000);
      if (best == 0 || cost <= least) { best = bn; least = cost; }
    }
    int rc = 0;
    switch (best) {
      case 160: rc = launch<160>(a, parts, ldp, map_w, stream); break;
      case 144: rc = launch<144>(a, parts, ldp, map_w, stream); break;
      case 128: rc = launch<128>(a, parts, ldp, map_w, stream); break;
      case 112: rc = launch<112>(a, parts, ldp, map_w, stream); break;
      case 96: rc = launch<96>(a, parts, ldp, map_w, stream); break;
      case 80: rc = launch<80>(a, parts, ldp, map_w, stream); break;
      case 64: rc = launch<64>(a, parts, ldp, map_w, stream); break;
      case 48: rc = launch<48>(a, parts, ldp, map_w, stream); break;
      case 32: rc = launch<32>(a, parts, ldp, map_w, stream); break;
      default: rc = launch<16>(a, parts, ldp, map_w, stream);
    }
    if (rc) return rc;
    if (cut.segments > 1) {
      const long long blocks = ((long long)a.M * N + 255) / 256;
      add_segments_kernel<<<(int)min(blocks, 16ll * sms), 256, 0, stream>>>(a);
    }
  }
  return dk_check_launch("gemm_f32_tc");
}
