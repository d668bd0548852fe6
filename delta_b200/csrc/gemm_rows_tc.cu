// y[M,N] = x[M,K] W[N,K]^T on the fifth-generation tensor cores for many rows: prompt portions, and the products of a mixture of experts
// over rows sorted by expert.
//
// One persistent block per SM takes pieces of 128 rows of x (the M side of a tcgen05.mma tile) by 256 or 128 rows of W (its N side),
// numbered so that the pieces of one expert run at the same time.  x and W come by TMA into a ring of stages (64 entries of K,
// 128-byte swizzle); two accumulators in tensor memory take turns, so that a piece's epilogue runs under the next one's products:
//   warp 0      asks for the boxes,
//   warp 1      issues the products and owns the tensor memory,
//   warps 2-9   epilogue: a warp takes 32 rows and half of the columns, 16 at a time; a thread holds one row of the tile, and 16 x 32 values
//               are turned in shared memory, so that a store reaches four or eight rows in whole sectors and not 32; gated activations find gate and
//               up columns in one accumulator (half of the tile each).
// Bound by the shared memory's bandwidth: 48 KB a step are written and read once more by the tensor core, 96 bytes a cycle each.
// 2,048 x 22,016 x 4,096: 250 us = 1,480 TFLOP/s with or without the silu gate (one block a tile, its epilogue uncovered, took 404 and 456;
// the library 218 without the gate); an expert's products of a 2,048-token prompt (16 experts of 1,024, 4 chosen, width 2,048) 157 -> 62 us, and
// 64 -> 52 (two of them on average, the second with 67 MB of 32-bit results) since eight warps write instead of four, in rows that lanes share.
// (Rows gathered by the copies themselves, tile::gather4, in place of a kernel of 13 us before the first product: that product 55 -> 170 us.)
//
// Every wait on an mbarrier is bounded: when one gives up, the kernel records it, stores nothing more, waits (bounded again) for the copies and
// products that it has under way, frees its tensor memory and returns.
#include "common.cuh"
#include "tcgen05_helpers.cuh"
#include "ring.cuh"

namespace {
constexpr int BM = 128;            // rows of x of a piece
constexpr int KSTEP = 64;          // entries of K of a box: one 128-byte swizzle row
constexpr int EPI_WARPS = 8;
constexpr int THREADS = (2 + EPI_WARPS) * 32;
constexpr int EPI_COLS = 16;       // columns that a warp turns at a time
constexpr int EPI_LD = EPI_COLS + 4;
constexpr int EPI_BYTES = 32 * EPI_LD * 4;      // of shared memory a warp
constexpr int MAX_STAGES = 7;

enum Epilogue { PLAIN = 0, GLU = 1, RELU_SQUARED = 2, SILU = 3 };

struct RowsArgs {
  void* out;                // [rows, ldc] bfloat16 or float
  int* err;
  int M, N, K, ldc;         // N: columns of the output
  int out_f32, epilogue;
  int up_row;               // gated: first up row of a matrix
  const int* tile_expert;   // expert of every `per_expert_tile` row tiles (negative: no rows); null: one matrix
  int per_expert_tile, expert_rows;
  const int* row_map;       // output row of every row of x (negative: not stored); null: the same
  float limit, alpha, shift;
  int row_tiles, col_tiles;
};

template <int BN>
struct Sizes {
  static constexpr int STAGE = (BM + BN) * KSTEP * 2;
  static constexpr int ROOM = 224 * 1024 - EPI_WARPS * EPI_BYTES;
  static constexpr int STAGES = ROOM / STAGE < MAX_STAGES ? ROOM / STAGE : MAX_STAGES;
  static constexpr int SMEM = STAGES * STAGE + EPI_WARPS * EPI_BYTES + 1024;
};

template <int BN>
__global__ void __launch_bounds__(THREADS, 1) gemm_rows_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                                                                  const RowsArgs a) {
  constexpr int STAGE = Sizes<BN>::STAGE, STAGES = Sizes<BN>::STAGES;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long bars[2 * MAX_STAGES + 4];      // full, empty, accumulator full, accumulator empty
  __shared__ uint32_t tmem_base_slot;
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t full0 = s2u(&bars[0]), empty0 = s2u(&bars[MAX_STAGES]), tfull0 = s2u(&bars[2 * MAX_STAGES]), tempty0 = s2u(&bars[2 * MAX_STAGES + 2]);
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull0 + 8 * b, 1);
      mbar_init(tempty0 + 8 * b, EPI_WARPS);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) tmem_alloc(s2u(&tmem_base_slot), 2 * BN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  const bool gated = a.epilogue == GLU || a.epilogue == SILU;
  const int cols = gated ? BN / 2 : BN;      // output columns of a piece
  const int steps = (a.K + KSTEP - 1) / KSTEP, items = a.row_tiles * a.col_tiles;
  // Experts: column tiles fastest, so that an expert's row tiles meet its matrix together.  One matrix: row tiles fastest, so that a tile
  // of W comes from memory once.
  auto place = [&](int item, int& row_tile, int& col_tile, int& w_row) {
    w_row = 0;
    if (a.tile_expert != nullptr) {
      row_tile = item / a.col_tiles;
      col_tile = item - row_tile * a.col_tiles;
      const int expert = a.tile_expert[row_tile / a.per_expert_tile];
      w_row = expert * a.expert_rows;
      return expert >= 0;
    }
    col_tile = item / a.row_tiles;
    row_tile = item - col_tile * a.row_tiles;
    return true;
  };
  volatile int* gave_up = &failed;

  if (warp == 0) {
    if (lane == 0) {
      int step = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int rt, ct, w_row;
        if (!place(item, rt, ct, w_row)) continue;
        for (int k = 0; k < steps; ++k, ++step) {
          const int s = step % STAGES;
          if (step >= STAGES && !mbar_wait(empty0 + 8 * s, ((step / STAGES) - 1) & 1)) {
            *gave_up = 1;
            ok = false;
            break;
          }
          const uint32_t dst = s2u(smem + (size_t)s * STAGE), bar = full0 + 8 * s;
          mbar_expect_tx(bar, STAGE);
          tma_load_2d(dst, &map_x, k * KSTEP, rt * BM, bar);      // rows past M and entries past K are zeros
          if (gated) {
            tma_load_2d(dst + BM * KSTEP * 2, &map_w, k * KSTEP, w_row + ct * cols, bar);
            tma_load_2d(dst + (BM + BN / 2) * KSTEP * 2, &map_w, k * KSTEP, w_row + a.up_row + ct * cols, bar);
          } else {
            tma_load_2d(dst + BM * KSTEP * 2, &map_w, k * KSTEP, w_row + ct * cols, bar);
          }
        }
      }
      ring_drain(step, STAGES, [&](int s, uint32_t parity) { return mbar_wait(full0 + 8 * s, parity); });      // its copies have arrived
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = instr_desc_bf16(BM, BN);
      int step = 0, piece = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
        int rt, ct, w_row;
        if (!place(item, rt, ct, w_row)) continue;
        const int b = piece & 1;
        if (piece >= 2 && !mbar_wait(tempty0 + 8 * b, ((piece >> 1) - 1) & 1)) {
          *gave_up = 1;
          break;
        }
        tc_fence_after();
        for (int k = 0; k < steps; ++k, ++step) {
          const int s = step % STAGES;
          if (!mbar_wait(full0 + 8 * s, (step / STAGES) & 1)) {
            *gave_up = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t at = s2u(smem + (size_t)s * STAGE);
          const uint64_t da = smem_desc_k_major(at), db = smem_desc_k_major(at + BM * KSTEP * 2);
#pragma unroll
          for (int i = 0; i < KSTEP / 16; ++i)
            umma(tmem_base + b * BN, da + (uint64_t)(i * 2), db + (uint64_t)(i * 2), idesc, (k > 0 || i > 0) ? 1u : 0u);
          umma_commit(empty0 + 8 * s);      // the stage is free once these have read it
        }
        umma_commit(tfull0 + 8 * b);
        ++piece;
      }
      // its products are complete (a commit covers all before it, so the last one would do)
      ring_drain(step, STAGES, [&](int s, uint32_t parity) { return mbar_wait(empty0 + 8 * s, parity); });
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;      // the lanes of tensor memory that a warp may read, and its half of the columns
    float* turn = reinterpret_cast<float*>(smem + (size_t)STAGES * STAGE + (size_t)(warp - 2) * EPI_BYTES);
    int piece = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      int rt, ct, w_row;
      if (!place(item, rt, ct, w_row)) continue;
      const int b = piece & 1;
      const int r = rt * BM + quarter * 32 + lane;
      const int out_row = r < a.M ? (a.row_map != nullptr ? a.row_map[r] : r) : -1;
      const bool there = mbar_wait(tfull0 + 8 * b, (piece >> 1) & 1) && *gave_up == 0;
      if (__any_sync(0xffffffffu, !there)) {      // the whole warp leaves, or none of it
        *gave_up = 1;
        break;
      }
      tc_fence_after();
      const uint32_t acc = tmem_base + b * BN + ((uint32_t)(quarter * 32) << 16);
      const int n0 = ct * cols;
      for (int c = half * (cols / 2); c < (half + 1) * (cols / 2); c += EPI_COLS) {
        if (n0 + c >= a.N) break;
        float y[EPI_COLS], u[EPI_COLS];
        tmem_ld16(acc + c, y);
        if (gated) tmem_ld16(acc + BN / 2 + c, u);
        if (a.epilogue == GLU) {      // both products rounded to bfloat16 first, as separate products would be
#pragma unroll
          for (int i = 0; i < EPI_COLS; ++i)
            y[i] = dk_glu_value(__bfloat162float(__float2bfloat16_rn(y[i])), __bfloat162float(__float2bfloat16_rn(u[i])), a.limit, a.alpha, a.shift);
        } else if (a.epilogue == SILU) {
#pragma unroll
          for (int i = 0; i < EPI_COLS; ++i) y[i] = y[i] / (1.f + expf(-y[i])) * u[i];
        } else if (a.epilogue == RELU_SQUARED) {
#pragma unroll
          for (int i = 0; i < EPI_COLS; ++i) {
            const float v = fmaxf(__bfloat162float(__float2bfloat16_rn(y[i])), 0.f);
            y[i] = v * v;
          }
        }
        // a thread holds a row; through shared memory, so that neighbouring lanes store neighbouring pieces of a row
        __syncwarp();
#pragma unroll
        for (int g = 0; g < EPI_COLS / 4; ++g)
          *reinterpret_cast<float4*>(turn + lane * EPI_LD + 4 * g) = make_float4(y[4 * g], y[4 * g + 1], y[4 * g + 2], y[4 * g + 3]);
        __syncwarp();
        if (a.out_f32) {      // four lanes a row, eight rows at a time
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = i * 8 + (lane >> 2), n = n0 + c + (lane & 3) * 4;
            const int to = __shfl_sync(0xffffffffu, out_row, row);
            const float4 v = *reinterpret_cast<const float4*>(turn + row * EPI_LD + (lane & 3) * 4);
            if (to >= 0 && n < a.N) *reinterpret_cast<float4*>((float*)a.out + (size_t)to * a.ldc + n) = v;      // N is a multiple of 8
          }
        } else {      // two lanes a row
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int row = i * 16 + (lane >> 1), n = n0 + c + (lane & 1) * 8;
            const int to = __shfl_sync(0xffffffffu, out_row, row);
            const float4 p = *reinterpret_cast<const float4*>(turn + row * EPI_LD + (lane & 1) * 8);
            const float4 q = *reinterpret_cast<const float4*>(turn + row * EPI_LD + (lane & 1) * 8 + 4);
            const float v[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
            if (to >= 0 && n < a.N) store8<__nv_bfloat16>((__nv_bfloat16*)a.out + (size_t)to * a.ldc + n, v);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty0 + 8 * b);
      ++piece;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (failed && tid == 0) dk_report(a.err, DK_DEV_TIMEOUT, blockIdx.x, 0, steps);
  if (warp == 1) tmem_dealloc(tmem_base, 2 * BN);
}

template <int BN>
int launch(const RowsArgs& a, const CUtensorMap& map_w, const CUtensorMap& map_x, cudaStream_t stream) {
  static bool granted[DK_MAX_DEVICES] = {false};
  bool& ok = granted[dk_current_device()];
  if (!ok) {
    DK_REQUIRE(cudaFuncSetAttribute(gemm_rows_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sizes<BN>::SMEM) == cudaSuccess,
               "gemm_rows_tc: %d bytes of shared memory were refused", Sizes<BN>::SMEM);
    ok = true;
  }
  const long long items = (long long)a.row_tiles * a.col_tiles;
  DK_REQUIRE(items < (1ll << 30), "gemm_rows_tc: too many pieces");
  gemm_rows_tc_kernel<BN><<<(int)(items < dk_sm_count() ? items : dk_sm_count()), THREADS, Sizes<BN>::SMEM, stream>>>(map_w, map_x, a);
  return dk_check_launch("gemm_rows_tc");
}

// w_rows: rows of W in all; lda, ldw: leading sizes.
int run(RowsArgs a, const void* x, const void* W, long long w_rows, int lda, int ldw, cudaStream_t stream) {
  const bool gated = a.epilogue == GLU || a.epilogue == SILU;
  a.row_tiles = (a.M + BM - 1) / BM;
  // 256 rows of W a piece load least for what they multiply: a piece takes 1.22 times as long as one of 128 (25.0 and 20.5 us at
  // K = 4,096).  128 where that makes up for the SMs that the last round of wide pieces leaves idle.
  const int sms = dk_sm_count();
  auto tiles = [&](int bn) { return (a.N + (gated ? bn / 2 : bn) - 1) / (gated ? bn / 2 : bn); };
  const long long wide = (long long)a.row_tiles * tiles(256), narrow = (long long)a.row_tiles * tiles(128);
  const bool is_wide = (wide + sms - 1) / sms * 122 <= (narrow + sms - 1) / sms * 100;
  const int bn = is_wide ? 256 : 128;
  a.col_tiles = tiles(bn);
  CUtensorMap map_w, map_x;
  DK_REQUIRE(make_tensor_map_bf16(&map_w, W, w_rows, a.K, ldw, gated ? bn / 2 : bn), "gemm_rows_tc: cannot encode the tensor map of W");
  DK_REQUIRE(make_tensor_map_bf16(&map_x, x, a.M, a.K, lda, BM), "gemm_rows_tc: cannot encode the tensor map of x");
  return is_wide ? launch<256>(a, map_w, map_x, stream) : launch<128>(a, map_w, map_x, stream);
}
}  // namespace

// N: rows of W (gate and up rows together with `swiglu`).
extern "C" int dk_gemm_rows_tc_supported(int M, int N, int K, int swiglu) {
  if (M < 1 || M > (1 << 20) || K < 64 || K % 8 != 0) return 0;
  return swiglu ? N % 2 == 0 && (N / 2) % 64 == 0 : N > 0 && N % 8 == 0;
}

extern "C" int dk_gemm_rows_tc(const void* x, const void* W, void* out, int M, int N, int K, int lda, int ldw, int ldc, int out_dtype, int swiglu,
                               int* err, cudaStream_t stream) {
  DK_REQUIRE(dk_gemm_rows_tc_supported(M, N, K, swiglu), "gemm_rows_tc: sizes not taken: M=%d N=%d K=%d swiglu=%d", M, N, K, swiglu);
  DK_REQUIRE(lda % 8 == 0 && ldw % 8 == 0 && ((uintptr_t)x | (uintptr_t)W) % 16 == 0,
             "gemm_rows_tc: operands must start on 16-byte boundaries with leading sizes that are multiples of 8");
  DK_REQUIRE(out_dtype == DK_BF16 || out_dtype == DK_F32, "gemm_rows_tc: unknown output dtype %d", out_dtype);
  DK_REQUIRE(ldc % 8 == 0 && (uintptr_t)out % 16 == 0, "gemm_rows_tc: the output must start on a 16-byte boundary with a leading size that is a multiple of 8");
  RowsArgs a = {};
  a.out = out;
  a.err = err;
  a.M = M; a.N = swiglu ? N / 2 : N; a.K = K; a.ldc = ldc;
  a.out_f32 = out_dtype == DK_F32;
  a.epilogue = swiglu ? SILU : PLAIN;
  a.up_row = N / 2;
  return run(a, x, W, N, lda, ldw, stream);
}

// Grouped products for a mixture of experts: x [M, K] holds the rows of all experts in tiles of `tile_m` (128 or 256) rows, tile c belonging
// to expert chunk_expert[c] (negative: no rows); W [E * expert rows, K] holds the experts' matrices one after the other, [gate (n) | up (n)]
// rows each when `glu` is 1, else n rows.  out[row_map ? row_map[r] : r][0..n) for every row r of x (rows mapped to a negative number are not
// stored).  `glu` 1: the gated activation with clamped branches; 2: relu(y)^2.
extern "C" int dk_experts_gemm_tc_supported(int n, int K, int glu) { return dk_gemm_rows_tc_supported(128, glu == 1 ? 2 * n : n, K, glu == 1); }

extern "C" int dk_experts_gemm_tc(const void* x, const void* W, void* out, const int* chunk_expert, const int* row_map, int M, int tile_m, int n,
                                  int K, int E, int ldc, int out_dtype, int glu, float limit, float alpha, float shift, int* err,
                                  cudaStream_t stream) {
  if (M == 0) return 0;
  DK_REQUIRE(tile_m == 128 || tile_m == 256, "experts_gemm_tc: tiles of 128 or 256 rows, got %d", tile_m);
  DK_REQUIRE(M > 0 && M % tile_m == 0 && E > 0, "experts_gemm_tc: %d rows are no whole tiles of %d", M, tile_m);
  DK_REQUIRE(dk_experts_gemm_tc_supported(n, K, glu), "experts_gemm_tc: sizes not taken: n=%d K=%d glu=%d", n, K, glu);
  DK_REQUIRE(((uintptr_t)x | (uintptr_t)W | (uintptr_t)out) % 16 == 0 && ldc % 8 == 0,
             "experts_gemm_tc: operands must start on 16-byte boundaries with leading sizes that are multiples of 8");
  DK_REQUIRE(out_dtype == DK_BF16 || out_dtype == DK_F32, "experts_gemm_tc: unknown output dtype %d", out_dtype);
  DK_REQUIRE(chunk_expert != nullptr, "experts_gemm_tc: no tile map");
  RowsArgs a = {};
  a.out = out;
  a.err = err;
  a.M = M; a.N = n; a.K = K; a.ldc = ldc;
  a.out_f32 = out_dtype == DK_F32;
  a.epilogue = glu == 1 ? GLU : glu == 2 ? RELU_SQUARED : PLAIN;
  a.up_row = n;
  a.tile_expert = chunk_expert;
  a.per_expert_tile = tile_m / BM;
  a.expert_rows = glu == 1 ? 2 * n : n;
  a.row_map = row_map;
  a.limit = limit; a.alpha = alpha; a.shift = shift;
  return run(a, x, W, (long long)E * a.expert_rows, K, K, stream);
}
