// The linear attention with a constant decay per head of decay_attention.cu over long bfloat16 portions, in chunks of 128 tokens on the
// fifth-generation tensor cores, for heads of 128 x 128.  With a chunk's tokens 0..n-1 and S [dk, dv] the state before it,
//     o_t = lambda^(t+1) S^T q_t + sum_{s<=t} A_ts v_s ,   A_ts = lambda^(t-s) (q_t . k_s)
//     S  <- lambda^n S + sum_s (lambda^(n-1-s) k_s) v_s^T .
//   1. chunk:  every chunk in parallel: A, sum A v into the outputs, and the contribution U to the state;
//   2. scan:   S_c = lambda^n S_(c-1) + U_c along a row, element by element; the state BEFORE chunk c takes the place of U_c, the last one
//              goes to the request's slot;
//   3. out:    every chunk in parallel: what the state before it adds to its outputs.
// Activated queries, keys and values, A and S are 32 bit.  They enter the products times 2^24 as three bfloat16 parts each, which give the number
// exactly, and six of the nine products of parts are made; those left out are at most 2^-24 of a term together, of either sign.  A tensor core cuts off what
// it adds to its accumulator: a sum stays there for 64 of its 128 terms (32 in U), the small products before the large, and halves (quarters) are
// added in 32 bit.  Powers come from the 64-bit decay, never divided by.  A chunk with infinite, NaN or very large numbers is summed by FMA instead.
//
// A block has 16 warps that turn numbers into parts and one that issues products.  Queries and A go to tensor memory as the first operand: with both
// operands in shared memory, 192 KB of it here, a product takes twice as long (its reads come at 64 bytes a cycle), as U's does.  Every wait is bounded; one that gives up is reported, the rest runs through.
// Bound by turning numbers into parts (and activating them) between three products that wait for one another, one block an SM.  One row of 2,048
// tokens, 16 heads: chunk 53 (two rounds of 128 blocks and more), scan 8, out 24 us; the FMA kernels in chunks of 64 63, 12 and 75.  Against 64 bits
// (2-norm, 389 tokens): outputs 1.3e-7, states 0.6e-7 off, 2.0e-7 and 1.3e-7 there; rows that one entry dominates 1.8e-7 and 0.9e-7 (2.7e-7, 1.7e-7), operands
// of one sign 1.1e-7 and 0.5e-7 (2.0e-7, 1.1e-7), queries and keys of 2^-57 1.4e-7 and 0.9e-7 (2.7e-7, 1.8e-7); with parts cut off instead of rounded, normal
// operands, 2.2e-7 and 1.3e-7.
#include "common.cuh"
#include "tcgen05_helpers.cuh"
#include "ring.cuh"

namespace {
constexpr int TC = 128, D = 128;
constexpr int WARPS = 16, THREADS = (WARPS + 1) * 32;
constexpr int BOX = TC * 128, PART = 2 * BOX;      // bytes: 128 rows of 64 entries; an operand's part
constexpr int TURN_LD = 36;
constexpr int PRODUCTS = 3;      // of a block, at most
constexpr int TMEM_COLS = 512, COL_A = 0, COL_D = 192;      // the first operand's parts, and two accumulators; or four accumulators

__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }

// x^n for n up to TC, by squaring: 64 bit, off by less than 2^-45 of it before it is rounded to 32.
__device__ __forceinline__ float power(double x, int n) {
  double r = 1.0;
#pragma unroll
  for (int b = 1; b <= TC; b *= 2) {
    if (n & b) r *= x;
    x *= x;
  }
  return (float)r;
}

// Operands are in reach of the parts below 2^20 (queries, keys, values) and 2^50 (the state).  They are multiplied by 2^24 first, and so is A = q . k
// before it is an operand: the last part of the smallest number is still a normal bfloat16 number, and no product leaves the exponent's range.
constexpr float SCALE = 16777216.f, UNSCALE = 1.f / 16777216.f / 16777216.f;
constexpr int REACH = 20, STATE_REACH = 50;
template <int EXPONENT>
__device__ __forceinline__ bool out_of_reach(const float (&x)[32]) {      // infinities and NaNs too
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 32; ++i) m = max(m, __float_as_uint(x[i]) & 0x7fffffffu);
  return m >= (127u + EXPONENT) << 23;
}

// Two numbers' parts, each rounded to nearest: what is left behind a part fits the two after it, so the three give the number, and the products
// that are left out have either sign (with parts cut off they would all add to the error).
__device__ __forceinline__ uint32_t nearest(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void parts_of(float x, float y, uint32_t& high, uint32_t& middle, uint32_t& low) {
  high = nearest(x, y);
  x -= __uint_as_float(high << 16);
  y -= __uint_as_float(high & 0xffff0000u);
  middle = nearest(x, y);
  low = nearest(x - __uint_as_float(middle << 16), y - __uint_as_float(middle & 0xffff0000u));
}

// How 512 threads share an operand of 128 rows of 128 entries: a thread takes eight neighbouring entries of four rows, so that sixteen lanes read
// and write a row.
__device__ __forceinline__ int row_of(int tid, int i) { return (tid >> 4) + 32 * i; }
__device__ __forceinline__ void fetch_rows(uint4 (&raw)[4], const __nv_bfloat16* src, int stride, int n, int tid) {      // zeros behind the last row
#pragma unroll
  for (int i = 0; i < 4; ++i)
    raw[i] = row_of(tid, i) < n ? *reinterpret_cast<const uint4*>(src + (size_t)row_of(tid, i) * stride + (tid & 15) * 8) : make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void activate(float (&x)[32], const uint4 (&raw)[4], int act) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float a = __uint_as_float(w[e] << 16), b = __uint_as_float(w[e] & 0xffff0000u);
      x[8 * i + 2 * e] = act ? silu(a) : a;
      x[8 * i + 2 * e + 1] = act ? silu(b) : b;
    }
  }
}
// Rows times factor(row) times 2^24 as parts in shared memory: [row][entry], boxes of 64 entries with the 128-byte swizzle.
template <typename F>
__device__ __forceinline__ void parts_to_shared(unsigned char* to, int row, int piece, const float* x, F&& f) {
  unsigned char* at = to + (piece >> 3) * BOX + row * 128 + (((piece & 7) ^ (row & 7)) << 4);
  const float w = f(row) * SCALE;
  uint4 p[3];
  parts_of(x[0] * w, x[1] * w, p[0].x, p[1].x, p[2].x);
  parts_of(x[2] * w, x[3] * w, p[0].y, p[1].y, p[2].y);
  parts_of(x[4] * w, x[5] * w, p[0].z, p[1].z, p[2].z);
  parts_of(x[6] * w, x[7] * w, p[0].w, p[1].w, p[2].w);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(at + i * PART) = p[i];
}
template <typename F>
__device__ __forceinline__ void rows_to_shared(unsigned char* to, const float (&x)[32], int tid, F&& f) {
#pragma unroll
  for (int i = 0; i < 4; ++i) parts_to_shared(to, row_of(tid, i), tid & 15, x + 8 * i, f);
}
__device__ __forceinline__ float as_it_is(int) { return 1.f; }
// 32 entries of a row times `scale` as an MMA's first operand in tensor memory: a row a lane
__device__ __forceinline__ void parts_to_tmem(uint32_t lanes, int group, const float (&x)[32], float scale) {
#pragma unroll
  for (int g = 0; g < 32; g += 16) {
    uint32_t h[8], m[8], l[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) parts_of(x[g + 2 * i] * scale, x[g + 2 * i + 1] * scale, h[i], m[i], l[i]);
    tmem_st8(lanes + COL_A + group * 16 + g / 2, h);
    tmem_st8(lanes + COL_A + 64 + group * 16 + g / 2, m);
    tmem_st8(lanes + COL_A + 128 + group * 16 + g / 2, l);
  }
}
// 32 columns of a product: the sums of its SPLIT accumulators, 128 columns apart, added, times `unscale`
template <int SPLIT>
__device__ __forceinline__ void read_product(uint32_t at, int group, float (&x)[32], float unscale) {
#pragma unroll
  for (int c = 0; c < 32; c += 8) {
    float y[SPLIT][8];
#pragma unroll
    for (int q = 0; q < SPLIT; ++q) tmem_ld8_nowait(at + q * D + group * 32 + c, y[q]);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (SPLIT == 2) x[c + i] = (y[0][i] + y[1][i]) * unscale;
      else x[c + i] = ((y[0][i] + y[1][i]) + (y[2][i] + y[3][i])) * unscale;
    }
  }
}

// A product of 128 x 128 x 128 by one thread: six products of parts, the small ones first, SPLIT equal stretches of K in accumulators of their own.
// multiply(accumulator's number, part of either operand, step of 16 of K, whether to add)
template <int SPLIT, typename Multiply>
__device__ __forceinline__ void issue(Multiply&& multiply) {
  constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0}, STEPS = D / 16 / SPLIT;
#pragma unroll
  for (int q = 0; q < SPLIT; ++q)
#pragma unroll
    for (int c = 0; c < 6; ++c)
#pragma unroll
      for (int k = 0; k < STEPS; ++k) multiply(q, PA[c], PB[c], q * STEPS + k, (c > 0 || k > 0) ? 1u : 0u);
}
// rows are those of the result, K runs along them; K runs over the rows
__device__ __forceinline__ uint64_t along(uint32_t parts, int p, int s) { return smem_desc_k_major(parts + p * PART + (s >> 2) * BOX) + (uint64_t)((s & 3) * 2); }
__device__ __forceinline__ uint64_t across(uint32_t parts, int p, int s) { return smem_desc_mn_major(parts + p * PART + s * 2048, BOX); }

struct Shared {
  float pw[TC + 4];
  unsigned long long done[PRODUCTS];      // a product's operands have been read and its sums are there
  uint32_t tmem_base_slot;
  int failed;
};
__device__ __forceinline__ void begin(Shared& sh, int warp, int tid, double decay) {
  if (tid == 0) {
    for (int p = 0; p < PRODUCTS; ++p) mbar_init(s2u(&sh.done[p]), 1);
    sh.failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (tid <= TC) sh.pw[tid] = power(decay, tid);
  if (warp == WARPS) tmem_alloc(s2u(&sh.tmem_base_slot), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}
// `issued`: products that the caller's warp has issued; each is complete before the block leaves, whatever became of the waits for it
__device__ __forceinline__ void end(Shared& sh, int warp, int lane, int issued, int* err) {
  if (warp == WARPS && lane == 0) ring_drain(issued, PRODUCTS, [&](int p, uint32_t parity) { return mbar_wait(s2u(&sh.done[p]), parity); });
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (sh.failed && threadIdx.x == 0) dk_report(err, DK_DEV_TIMEOUT, blockIdx.x, blockIdx.y, 0);
  if (warp == WARPS) tmem_dealloc(sh.tmem_base_slot, TMEM_COLS);
}
// The next product, unless a wait has given up (what it would read may not be there, and nobody waits for it).  By an elected thread: in a branch for lane 0
// an MMA took 100 cycles to issue.
template <typename Issue>
__device__ __forceinline__ void issue_next(Shared& sh, int& issued, Issue&& product) {
  if (__all_sync(0xffffffffu, *(volatile int*)&sh.failed == 0)) {
    if (elect_one()) {
      product();
      umma_commit(s2u(&sh.done[issued]));
    }
    ++issued;
  }
  __syncwarp();
}
// Number `p` (0, 1, ..) of a block's products is complete.
__device__ __forceinline__ void wait_product(Shared& sh, int p) {
  volatile int* gave_up = &sh.failed;
  if (*gave_up == 0 && !mbar_wait(s2u(&sh.done[p]), 0)) *gave_up = 1;
  tc_fence_after();
}
// A warp's 32 rows of 32 floats as they lie in memory, neighbouring lanes at neighbouring places: f(row, column, float4)
template <typename F>
__device__ __forceinline__ void turned(float* turn, const float (&x)[32], int lane, F&& f) {
  __syncwarp();
#pragma unroll
  for (int g = 0; g < 8; ++g) *reinterpret_cast<float4*>(turn + lane * TURN_LD + 4 * g) = make_float4(x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) f(i * 4 + (lane >> 3), (lane & 7) * 4, *reinterpret_cast<const float4*>(turn + (i * 4 + (lane >> 3)) * TURN_LD + (lane & 7) * 4));
}

// The chunk's work by FMA, for numbers that the parts do not reach.
__device__ __noinline__ void chunk_by_fma(float* sm, const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, int stride, int act, int n,
                                          const float* pw, float* U, float* out, int out_stride) {
  float *K = sm, *V = K + TC * D, *A = V + TC * D;
  for (int i = threadIdx.x; i < TC * D; i += THREADS) {
    const int t = i / D, c = i % D;
    const float a = t < n ? __bfloat162float(k[(size_t)t * stride + c]) : 0.f, b = t < n ? __bfloat162float(v[(size_t)t * stride + c]) : 0.f;
    K[i] = act ? silu(a) : a;
    V[i] = act ? silu(b) : b;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < TC * TC; i += THREADS) {
    const int t = i / TC, s = i % TC;
    float sum = 0.f;
    if (s <= t && t < n)
      for (int c = 0; c < D; ++c) {
        const float a = __bfloat162float(q[(size_t)t * stride + c]);
        sum = fmaf(act ? silu(a) : a, K[s * D + c], sum);
      }
    A[i] = sum * (s <= t ? pw[t - s] : 0.f);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < D * D; i += THREADS) {
    const int r = i / D, c = i % D;
    float sum = 0.f;
    for (int s = 0; s < n; ++s) sum = fmaf(K[s * D + r], V[s * D + c] * pw[n - 1 - s], sum);
    U[i] = sum;
  }
  for (int i = threadIdx.x; i < n * D; i += THREADS) {
    const int t = i / D, c = i % D;
    float sum = 0.f;
    for (int s = 0; s <= t; ++s) sum = fmaf(A[t * TC + s], V[s * D + c], sum);
    out[(size_t)t * out_stride + c] = sum;
  }
}

// grid (most chunks of a row, rows * H)
__global__ void __launch_bounds__(THREADS, 1)
decay_tc_chunk_kernel(const __nv_bfloat16* __restrict__ src, int stride, int q_off, int k_off, int v_off, int act, const double* __restrict__ decays,
                      float* __restrict__ U, float* __restrict__ out, const int* __restrict__ row_q_start, const int* __restrict__ row_q_len,
                      const int* __restrict__ chunk_base, int H, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) Shared sh;
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char *R0 = smem, *R1 = smem + 3 * PART;      // values; keys, then decayed keys
  const int row = blockIdx.y / H, h = blockIdx.y % H, c0 = blockIdx.x * TC, n_new = row_q_len[row];
  if (c0 >= n_new) return;
  const int n = min(TC, n_new - c0), t0 = row_q_start[row] + c0, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  begin(sh, warp, tid, decays[h]);
  const uint32_t tmem = sh.tmem_base_slot;
  const __nv_bfloat16* at = src + (size_t)t0 * stride + (size_t)h * D;
  float* Uc = U + (((size_t)chunk_base[row] + blockIdx.x) * H + h) * D * D;
  float* oc = out + ((size_t)t0 * H + h) * D;
  // of a thread that reads a product: a row and 32 of its columns
  const int r = (warp & 3) * 32 + lane, group = (warp >> 2) & 3;
  const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const bool converts = warp < WARPS;
  const uint32_t r0 = s2u(R0), r1 = s2u(R1);
  float x[32], k[32];
  uint4 raw[4];
  bool odd = false;
  if (converts) {
    const __nv_bfloat16* mine = at + q_off + (size_t)(r < n ? r : 0) * stride + group * 32;      // 32 entries of a row
    uint4 first[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) first[i] = r < n ? *reinterpret_cast<const uint4*>(mine + 8 * i) : make_uint4(0, 0, 0, 0);
    fetch_rows(raw, at + k_off, stride, n, tid);
    activate(x, first, act);
    odd = out_of_reach<REACH>(x);
    parts_to_tmem(lanes, group, x, SCALE);
    activate(k, raw, act);
    fetch_rows(raw, at + v_off, stride, n, tid);
    odd |= out_of_reach<REACH>(k);
    rows_to_shared(R1, k, tid, as_it_is);
    tmem_wait_st();
    fence_async_smem();
    tc_fence_before();
  }
  odd = __syncthreads_or(odd) != 0;
  tc_fence_after();
  int issued = 0;
  const bool scored = !odd;
  if (scored && warp == WARPS)
    issue_next(sh, issued, [&]() {      // q . k
      const uint32_t idesc = instr_desc_bf16(TC, TC);
      issue<2>([&](int q, int a, int b, int s, uint32_t add) { umma_a_tmem(tmem + COL_D + q * D, tmem + COL_A + a * 64 + s * 8, along(r1, b, s), idesc, add); });
    });
  bool odd_v = false;
  if (converts) {      // meanwhile
    activate(x, raw, act);
    odd_v = out_of_reach<REACH>(x);
    rows_to_shared(R0, x, tid, as_it_is);
  }
  odd |= __syncthreads_or(odd_v) != 0;
  if (odd) {
    if (scored) wait_product(sh, 0);      // before its operands are overwritten
    __syncthreads();
    chunk_by_fma(reinterpret_cast<float*>(smem), at + q_off, at + k_off, at + v_off, stride, act, n, sh.pw, Uc, oc, H * D);
    end(sh, warp, lane, issued, err);
    return;
  }
  if (converts) {
    wait_product(sh, 0);
    rows_to_shared(R1, k, tid, [&](int s) { return s < n ? sh.pw[n - 1 - s] : 0.f; });
    read_product<2>(lanes + COL_D, group, x, 1.f / SCALE);      // (A is an operand: times 2^24)
    fence_async_smem();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  if (warp == WARPS) {
    issue_next(sh, issued, [&]() {      // the contribution to the state: keys' entries by values' entries, both operands read transposed
      const uint32_t idesc = instr_desc_bf16(TC, D, true) | 1u << 15;
      issue<4>([&](int q, int a, int b, int s, uint32_t add) { umma(tmem + q * D, across(r1, a, s), across(r0, b, s), idesc, add); });
    });
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int s = group * 32 + j;
      x[j] = s <= r ? x[j] * sh.pw[r - s] : 0.f;
    }
    wait_product(sh, 1);
    read_product<4>(lanes, group, k, UNSCALE);
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(WARPS * 32) : "memory");      // A takes columns of what was read
    tc_fence_after();
    parts_to_tmem(lanes, group, x, 1.f);
    tmem_wait_st();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  if (warp == WARPS) {
    issue_next(sh, issued, [&]() {      // A v
      const uint32_t idesc = instr_desc_bf16(TC, D, true);
      issue<2>([&](int q, int a, int b, int s, uint32_t add) { umma_a_tmem(tmem + COL_D + q * D, tmem + COL_A + a * 64 + s * 8, across(r0, b, s), idesc, add); });
    });
  } else {
    float* turn = reinterpret_cast<float*>(R1) + warp * 32 * TURN_LD;      // (the keys have been read)
    float* to = Uc + (size_t)((warp & 3) * 32) * D + group * 32;
    turned(turn, k, lane, [&](int i, int c, float4 v) { *reinterpret_cast<float4*>(to + (size_t)i * D + c) = v; });
    wait_product(sh, 2);
    read_product<2>(lanes + COL_D, group, x, UNSCALE);
    float* o = oc + group * 32;
    turned(turn, x, lane, [&](int i, int c, float4 v) {
      const int t = (warp & 3) * 32 + i;
      if (t < n) *reinterpret_cast<float4*>(o + (size_t)t * H * D + c) = v;
    });
  }
  end(sh, warp, lane, issued, err);
}

// grid (dk dv / 4 / 128, rows * H): four neighbouring entries a thread, four chunks' under way
__global__ void __launch_bounds__(128)
decay_tc_scan_kernel(float* __restrict__ U, float* __restrict__ state, const double* __restrict__ decays, const int* __restrict__ row_slot,
                     const int* __restrict__ row_q_len, const int* __restrict__ chunk_base, int H) {
  constexpr int AHEAD = 4;
  const int row = blockIdx.y / H, h = blockIdx.y % H, e = (blockIdx.x * blockDim.x + threadIdx.x) * 4, n_new = row_q_len[row];
  if (n_new <= 0) return;
  const int chunks = (n_new + TC - 1) / TC;
  const float full = power(decays[h], TC), last = power(decays[h], n_new - (chunks - 1) * TC);
  float4* st = reinterpret_cast<float4*>(state + ((size_t)row_slot[row] * H + h) * D * D + e);
  float* u = U + ((size_t)chunk_base[row] * H + h) * D * D + e;
  const size_t step = (size_t)H * D * D;
  float4 next[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < chunks) next[i] = *reinterpret_cast<const float4*>(u + (size_t)i * step);
  float4 S = *st;
  for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int c = c0 + i;
      if (c < chunks) {
        const float4 cur = next[i];
        if (c + AHEAD < chunks) next[i] = *reinterpret_cast<const float4*>(u + (size_t)(c + AHEAD) * step);
        *reinterpret_cast<float4*>(u + (size_t)c * step) = S;
        const float w = c + 1 < chunks ? full : last;
        S.x = fmaf(w, S.x, cur.x); S.y = fmaf(w, S.y, cur.y); S.z = fmaf(w, S.z, cur.z); S.w = fmaf(w, S.w, cur.w);
      }
    }
  }
  *st = S;
}

// grid (most chunks of a row, rows * H)
__global__ void __launch_bounds__(THREADS, 1)
decay_tc_out_kernel(const __nv_bfloat16* __restrict__ src, int stride, int q_off, int act, const double* __restrict__ decays, const float* __restrict__ U,
                    float* __restrict__ out, const int* __restrict__ row_q_start, const int* __restrict__ row_q_len, const int* __restrict__ chunk_base,
                    int H, int* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) Shared sh;
  unsigned char* Sp = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int row = blockIdx.y / H, h = blockIdx.y % H, c0 = blockIdx.x * TC, n_new = row_q_len[row];
  if (c0 >= n_new) return;
  const int n = min(TC, n_new - c0), t0 = row_q_start[row] + c0, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  begin(sh, warp, tid, decays[h]);
  const uint32_t tmem = sh.tmem_base_slot;
  const __nv_bfloat16* q = src + (size_t)t0 * stride + (size_t)h * D + q_off;
  const float* S = U + (((size_t)chunk_base[row] + blockIdx.x) * H + h) * D * D;
  float* oc = out + ((size_t)t0 * H + h) * D;
  const int r = (warp & 3) * 32 + lane, group = (warp >> 2) & 3;
  const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint32_t sp = s2u(Sp);
  int issued = 0;
  float x[32];
  bool odd = false;
  if (warp < WARPS) {
    uint4 raw[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      raw[i] = r < n ? *reinterpret_cast<const uint4*>(q + (size_t)r * stride + group * 32 + 8 * i) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float v[8];
      load8<float>(S + (size_t)row_of(tid, i) * D + (tid & 15) * 8, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) x[8 * i + e] = v[e];
    }
    odd = out_of_reach<STATE_REACH>(x);
    rows_to_shared(Sp, x, tid, as_it_is);
    activate(x, raw, act);
    odd |= out_of_reach<REACH>(x);
    parts_to_tmem(lanes, group, x, SCALE);
    tmem_wait_st();
    fence_async_smem();
    tc_fence_before();
  }
  if (__syncthreads_or(odd)) {
    for (int i = tid; i < n * D; i += THREADS) {
      const int t = i / D, c = i % D;
      float sum = 0.f;
      for (int e = 0; e < D; ++e) {
        const float a = __bfloat162float(q[(size_t)t * stride + e]);
        sum = fmaf(act ? silu(a) : a, S[e * D + c], sum);
      }
      oc[(size_t)t * H * D + c] = fmaf(sum, sh.pw[t + 1], oc[(size_t)t * H * D + c]);
    }
    end(sh, warp, lane, issued, err);
    return;
  }
  tc_fence_after();
  if (warp == WARPS) {
    issue_next(sh, issued, [&]() {
      const uint32_t idesc = instr_desc_bf16(TC, D, true);
      issue<2>([&](int q, int a, int b, int s, uint32_t add) { umma_a_tmem(tmem + COL_D + q * D, tmem + COL_A + a * 64 + s * 8, across(sp, b, s), idesc, add); });
    });
  } else {
    wait_product(sh, 0);
    read_product<2>(lanes + COL_D, group, x, UNSCALE);
    const float w = sh.pw[r + 1];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] *= w;
    float* o = oc + group * 32;
    turned(reinterpret_cast<float*>(Sp) + warp * 32 * TURN_LD, x, lane, [&](int i, int c, float4 v) {      // (the state has been read)
      const int t = (warp & 3) * 32 + i;
      if (t < n) {
        float4* to = reinterpret_cast<float4*>(o + (size_t)t * H * D + c);
        const float4 y = *to;
        *to = make_float4(y.x + v.x, y.y + v.y, y.z + v.z, y.w + v.w);
      }
    });
  }
  end(sh, warp, lane, issued, err);
}
constexpr int CHUNK_SMEM = 6 * PART + 1024, OUT_SMEM = 3 * PART + 1024;
static_assert(3 * TC * D * 4 <= 6 * PART && WARPS * 32 * TURN_LD * 4 <= 3 * PART, "what else the parts' memory is used for");
}  // namespace

extern "C" int dk_decay_attention_tc_chunk() { return TC; }

// Heads of 128 x 128 whose columns begin on 16-byte boundaries (bfloat16).
extern "C" int dk_decay_attention_tc_supported(int dk, int dv, int stride, int q_off, int k_off, int v_off) {
  return dk == D && dv == D && stride % 8 == 0 && q_off % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0;
}

// Arguments as for dk_decay_attention_tiles, with chunks of dk_decay_attention_tc_chunk() tokens; `work`: total_chunks x H x 128 x 128 floats.
extern "C" int dk_decay_attention_tc(const void* src, int stride, int q_off, int k_off, int v_off, int act, const double* decays, float* state, float* out,
                                     float* work, const int* row_slot, const int* row_q_start, const int* row_q_len, const int* chunk_base, int rows,
                                     int max_chunks, int H, int* err, cudaStream_t stream) {
  if (rows == 0 || max_chunks == 0) return 0;
  DK_REQUIRE(rows > 0 && max_chunks > 0 && H > 0 && dk_decay_attention_tc_supported(D, D, stride, q_off, k_off, v_off),
             "decay_attention_tc: rows of %d and offsets %d %d %d are not taken", stride, q_off, k_off, v_off);
  DK_REQUIRE((long long)rows * H <= 65535, "decay_attention_tc: %d rows of %d heads are above the grid's limit", rows, H);
  DK_REQUIRE(((uintptr_t)src | (uintptr_t)work | (uintptr_t)state | (uintptr_t)out) % 16 == 0, "decay_attention_tc: a tensor begins off its boundary");
  static bool granted[DK_MAX_DEVICES] = {false};
  bool& ok = granted[dk_current_device()];
  if (!ok) {
    DK_REQUIRE(cudaFuncSetAttribute(decay_tc_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CHUNK_SMEM) == cudaSuccess &&
                   cudaFuncSetAttribute(decay_tc_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_SMEM) == cudaSuccess,
               "decay_attention_tc: shared memory was refused");
    ok = true;
  }
  const auto* s = (const __nv_bfloat16*)src;
  const dim3 grid(max_chunks, rows * H);
  decay_tc_chunk_kernel<<<grid, THREADS, CHUNK_SMEM, stream>>>(s, stride, q_off, k_off, v_off, act, decays, work, out, row_q_start, row_q_len, chunk_base, H, err);
  decay_tc_scan_kernel<<<dim3(D * D / 4 / 128, rows * H), 128, 0, stream>>>(work, state, decays, row_slot, row_q_len, chunk_base, H);
  decay_tc_out_kernel<<<grid, THREADS, OUT_SMEM, stream>>>(s, stride, q_off, act, decays, work, out, row_q_start, row_q_len, chunk_base, H, err);
  return dk_check_launch("decay_attention_tc");
}
