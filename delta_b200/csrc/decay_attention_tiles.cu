// The linear attention with a constant decay per head of decay_attention.cu over long portions, in chunks of 64 tokens, for heads of 64 or
// 128 entries.  With a chunk's tokens 0..n-1 and S [dk, dv] the state before it,
//     o_t = lambda^(t+1) S^T q_t + sum_{s<=t} A_ts v_s ,   A_ts = lambda^(t-s) (q_t . k_s)
//     S  <- lambda^n S + sum_s k_s (lambda^(n-1-s) v_s)^T .
//   1. chunk:  every chunk in parallel: its contribution U to the state, and A;
//   2. scan:   S_c = lambda^n S_(c-1) + U_c along a row, element by element; the state BEFORE chunk c takes the place of U_c, the last one
//              goes to the request's slot;
//   3. out:    every chunk in parallel: one product [q | A] [S ; v] of 64 rows, the first part's sums multiplied by lambda^(t+1) in between.
// 32-bit FMA throughout, powers from the 64-bit decay, never divided by.  Bound by the FMA units and shared memory: a thread holds
// 8 x 8 sums of U, or 8 x 4 of an output, in registers and reads shared memory sixteen bytes at a time; S comes by cp.async, 16 rows a
// stage.  At 128 x 128 the output kernel's 118 KB leave an SM one block of eight warps (its registers would allow two).  One row of 2,048 tokens, 16 heads of 128 x 128: chunk 63, scan 12, out 75 us
// (outputs of 8 x 8 sums in blocks of 128 threads: the layer 283 instead of 236 us); the kernels with chunks of 32 and 4 x 4 sums a
// thread 50, 27 and 160 us.  Against 64 bits: outputs 2.0e-7 off as before, states 1.0e-7 (1.5e-7).
#include "common.cuh"
#include "mma_helpers.cuh"

namespace {
constexpr int TC = 64;
constexpr int THREADS = 256;
constexpr int ALD = TC + 4;
constexpr int KS = 16;              // rows of S of a stage
constexpr int STAGES = 4;

__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }

// x^n for n up to TC, by squaring: 64 bit, off by less than 2^-46 of it before it is rounded to 32.  (pow() takes several times as long,
// and a block's first products wait for the table.)
__device__ __forceinline__ float power(double x, int n) {
  double r = 1.0;
#pragma unroll
  for (int b = 1; b <= TC; b *= 2) {
    if (n & b) r *= x;
    x *= x;
  }
  return (float)r;
}

// 64 tokens' entries of a head, activated, into rows of D + 4; zeros behind the last token.
template <typename T, int D>
__device__ __forceinline__ void load_rows(float* to, const T* src, int stride, int n, int act, const float* pw, int tid) {
  for (int v = tid; v < TC * (D / 8); v += THREADS) {
    const int t = v / (D / 8), c = v % (D / 8) * 8;
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (t < n) {
      load8<T>(src + (size_t)t * stride + c, x);
      const float f = pw != nullptr ? pw[n - 1 - t] : 1.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = (act ? silu(x[e]) : x[e]) * f;
    }
    *reinterpret_cast<float4*>(to + t * (D + 4) + c) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(to + t * (D + 4) + c + 4) = make_float4(x[4], x[5], x[6], x[7]);
  }
}

template <int I>
struct Number {
  static constexpr int value = I;
};
// Four tokens s.. of the chunk after four, each for the rows that see some of them: number I on for s in TI I .. TI (I + 1) - 1.
template <int I, int RT, int TI, typename F>
__device__ __forceinline__ void near_rows(int n, int ti, F&& step) {
  if constexpr (I < RT) {
#pragma unroll
    for (int s = TI * I; s < TI * (I + 1); s += 4)
      if (s < n) step(Number<I>(), s);
    near_rows<I + 1, RT, TI>(n, ti, step);
  }
}

template <int DK, int DV>
constexpr int chunk_smem() { return (TC * (DK + 4) * 2 + TC * (DV + 4) + TC + 4) * (int)sizeof(float); }
template <int DK, int DV>
constexpr int out_smem() { return (TC * (DK + 4) + TC * (DV + 4) + TC * ALD + STAGES * KS * DV + TC + 4) * (int)sizeof(float); }

// grid (most chunks of a row, rows * H)
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
decay_tiles_chunk_kernel(const T* __restrict__ src, int stride, int q_off, int k_off, int v_off, int act, const double* __restrict__ decays,
                         float* __restrict__ U, float* __restrict__ A, const int* __restrict__ row_q_start, const int* __restrict__ row_q_len,
                         const int* __restrict__ chunk_base, int H) {
  constexpr int RI = DK / 16, RJ = DV / 16;      // a thread's sums of U: RI x RJ, four neighbours at a time
  extern __shared__ __align__(16) float sm[];
  const int row = blockIdx.y / H, h = blockIdx.y % H, c0 = blockIdx.x * TC, n_new = row_q_len[row], tid = threadIdx.x;
  if (c0 >= n_new) return;
  const int n = min(TC, n_new - c0);
  float* Q = sm;
  float* K = Q + TC * (DK + 4);
  float* V = K + TC * (DK + 4);      // times lambda^(n-1-s)
  float* pw = V + TC * (DV + 4);
  if (tid <= TC) pw[tid] = power(decays[h], tid);
  __syncthreads();
  const T* at = src + (size_t)(row_q_start[row] + c0) * stride;
  load_rows<T, DK>(Q, at + q_off + (size_t)h * DK, stride, n, act, nullptr, tid);
  load_rows<T, DK>(K, at + k_off + (size_t)h * DK, stride, n, act, nullptr, tid);
  load_rows<T, DV>(V, at + v_off + (size_t)h * DV, stride, n, act, pw, tid);
  __syncthreads();
  const int tx = tid & 15, ty = tid >> 4;
  const size_t chunk = ((size_t)chunk_base[row] + blockIdx.x) * H + h;
  {      // A: rows ty + 16 i, columns tx + 16 j, j <= i
    float acc[4][4] = {};
#pragma unroll 2
    for (int k = 0; k < DK; k += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(K + (tx + 16 * j) * (DK + 4) + k);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(Q + (ty + 16 * i) * (DK + 4) + k);
#pragma unroll
        for (int j = 0; j <= i; ++j) {
          acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
          acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
          acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
          acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
        }
      }
    }
    float* to = A + chunk * TC * TC;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = ty + 16 * i, s = tx + 16 * j;
        to[t * TC + s] = s <= t ? acc[i][j] * pw[t - s] : 0.f;
      }
  }
  float acc[RI][RJ] = {};
#pragma unroll 4
  for (int s = 0; s < n; ++s) {
    float4 a[RI / 4], b[RJ / 4];
#pragma unroll
    for (int i = 0; i < RI / 4; ++i) a[i] = *reinterpret_cast<const float4*>(K + s * (DK + 4) + i * 64 + ty * 4);
#pragma unroll
    for (int j = 0; j < RJ / 4; ++j) b[j] = *reinterpret_cast<const float4*>(V + s * (DV + 4) + j * 64 + tx * 4);
#pragma unroll
    for (int i = 0; i < RI / 4; ++i)
#pragma unroll
      for (int j = 0; j < RJ / 4; ++j) {
        const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, bv[4] = {b[j].x, b[j].y, b[j].z, b[j].w};
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < 4; ++y) acc[4 * i + x][4 * j + y] = fmaf(av[x], bv[y], acc[4 * i + x][4 * j + y]);
      }
  }
  float* to = U + chunk * DK * DV;
#pragma unroll
  for (int i = 0; i < RI; ++i)
#pragma unroll
    for (int j = 0; j < RJ / 4; ++j)
      *reinterpret_cast<float4*>(to + (size_t)(i / 4 * 64 + ty * 4 + i % 4) * DV + j * 64 + tx * 4) =
          make_float4(acc[i][4 * j], acc[i][4 * j + 1], acc[i][4 * j + 2], acc[i][4 * j + 3]);
}

// grid (dk dv / 4 / 128, rows * H): four neighbouring entries a thread, four chunks' under way
__global__ void __launch_bounds__(128)
decay_tiles_scan_kernel(float* __restrict__ U, float* __restrict__ state, const double* __restrict__ decays, const int* __restrict__ row_slot,
                        const int* __restrict__ row_q_len, const int* __restrict__ chunk_base, int H, int per_head) {
  constexpr int AHEAD = 4;
  const int row = blockIdx.y / H, h = blockIdx.y % H, e = (blockIdx.x * blockDim.x + threadIdx.x) * 4, n_new = row_q_len[row];
  if (e >= per_head || n_new <= 0) return;
  const int chunks = (n_new + TC - 1) / TC;
  const float full = power(decays[h], TC), last = power(decays[h], n_new - (chunks - 1) * TC);
  float4* st = reinterpret_cast<float4*>(state + ((size_t)row_slot[row] * H + h) * per_head + e);
  float* u = U + ((size_t)chunk_base[row] * H + h) * per_head + e;
  const size_t step = (size_t)H * per_head;
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
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
decay_tiles_out_kernel(const T* __restrict__ src, int stride, int q_off, int v_off, int act, const double* __restrict__ decays,
                       const float* __restrict__ U, const float* __restrict__ A, float* __restrict__ out, const int* __restrict__ row_q_start,
                       const int* __restrict__ row_q_len, const int* __restrict__ chunk_base, int H) {
  constexpr int JT = DV / 4, RT = TC * JT / THREADS, TI = TC / RT;      // a thread: RT tokens TI apart, four neighbouring entries
  extern __shared__ __align__(16) float sm[];
  const int row = blockIdx.y / H, h = blockIdx.y % H, c0 = blockIdx.x * TC, n_new = row_q_len[row], tid = threadIdx.x;
  if (c0 >= n_new) return;
  const int n = min(TC, n_new - c0), t0 = row_q_start[row] + c0;
  float* Q = sm;
  float* V = Q + TC * (DK + 4);
  float* At = V + TC * (DV + 4);      // [TC][ALD]
  float* Ss = At + TC * ALD;          // [STAGES][KS][DV]
  float* pw = Ss + STAGES * KS * DV;
  const size_t chunk = ((size_t)chunk_base[row] + blockIdx.x) * H + h;
  const float* Sc = U + chunk * DK * DV;
  auto fetch = [&](int s) {
    if (s < DK / KS)
      for (int v = tid; v < KS * DV / 4; v += THREADS) cp_async_16(smem_u32(Ss + (s % STAGES) * KS * DV + v * 4), Sc + (size_t)s * KS * DV + v * 4, true);
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  if (tid <= TC) pw[tid] = power(decays[h], tid);
  const T* at = src + (size_t)t0 * stride;
  load_rows<T, DK>(Q, at + q_off + (size_t)h * DK, stride, n, act, nullptr, tid);
  load_rows<T, DV>(V, at + v_off + (size_t)h * DV, stride, n, act, nullptr, tid);
  for (int v = tid; v < TC * TC / 4; v += THREADS)
    *reinterpret_cast<float4*>(At + v / (TC / 4) * ALD + v % (TC / 4) * 4) = *reinterpret_cast<const float4*>(A + chunk * TC * TC + v * 4);
  const int tj = tid % JT, ti = tid / JT;
  float4 acc[RT];
#pragma unroll
  for (int i = 0; i < RT; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  // four steps of the sums of the rows from number FIRST on (the first of them only where `with_first`)
  auto add = [&](auto FIRST, bool with_first, const float* left, int ld, const float* right, int rd) {
    float4 b[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) b[e] = *reinterpret_cast<const float4*>(right + e * rd + 4 * tj);
#pragma unroll
    for (int i = FIRST.value; i < RT; ++i) {
      if (i == FIRST.value && !with_first) continue;
      const float4 a = *reinterpret_cast<const float4*>(left + (ti + TI * i) * ld);
      const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc[i].x = fmaf(av[e], b[e].x, acc[i].x);
        acc[i].y = fmaf(av[e], b[e].y, acc[i].y);
        acc[i].z = fmaf(av[e], b[e].z, acc[i].z);
        acc[i].w = fmaf(av[e], b[e].w, acc[i].w);
      }
    }
  };
  for (int s = 0; s < DK / KS; ++s) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();      // stage s is in, and everybody has left the one that is fetched into next
    fetch(s + STAGES - 1);
#pragma unroll
    for (int k = 0; k < KS; k += 4) add(Number<0>(), true, Q + s * KS + k, DK + 4, Ss + ((s % STAGES) * KS + k) * DV, DV);
  }
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    const float w = pw[ti + TI * i + 1];
    acc[i].x *= w; acc[i].y *= w; acc[i].z *= w; acc[i].w *= w;
  }
  near_rows<0, RT, TI>(n, ti, [&](auto FIRST, int s) { add(FIRST, ti + TI * FIRST.value >= s, At + s, ALD, V + s * (DV + 4), DV + 4); });
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    const int t = ti + TI * i;
    if (t < n) *reinterpret_cast<float4*>(out + ((size_t)(t0 + t) * H + h) * DV + 4 * tj) = acc[i];
  }
}

template <typename T, int DK, int DV>
int launch(const T* src, int stride, int q_off, int k_off, int v_off, int act, const double* decays, float* state, float* out, float* U, float* A,
           const int* row_slot, const int* row_q_start, const int* row_q_len, const int* chunk_base, int rows, int max_chunks, int H,
           cudaStream_t stream) {
  static bool granted[DK_MAX_DEVICES] = {false};
  bool& ok = granted[dk_current_device()];
  if (!ok) {
    DK_REQUIRE(cudaFuncSetAttribute(decay_tiles_chunk_kernel<T, DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, chunk_smem<DK, DV>()) == cudaSuccess &&
                   cudaFuncSetAttribute(decay_tiles_out_kernel<T, DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, out_smem<DK, DV>()) == cudaSuccess,
               "decay_attention_tiles: shared memory was refused");
    ok = true;
  }
  const dim3 grid(max_chunks, rows * H);
  decay_tiles_chunk_kernel<T, DK, DV><<<grid, THREADS, chunk_smem<DK, DV>(), stream>>>(src, stride, q_off, k_off, v_off, act, decays, U, A, row_q_start,
                                                                                      row_q_len, chunk_base, H);
  decay_tiles_scan_kernel<<<dim3((DK * DV / 4 + 127) / 128, rows * H), 128, 0, stream>>>(U, state, decays, row_slot, row_q_len, chunk_base, H, DK * DV);
  decay_tiles_out_kernel<T, DK, DV><<<grid, THREADS, out_smem<DK, DV>(), stream>>>(src, stride, q_off, v_off, act, decays, U, A, out, row_q_start,
                                                                                  row_q_len, chunk_base, H);
  return dk_check_launch("decay_attention_tiles");
}
}  // namespace

extern "C" int dk_decay_attention_tiles_chunk() { return TC; }

// Heads of 64 or 128 entries whose columns begin on 16-byte boundaries.
extern "C" int dk_decay_attention_tiles_supported(int dk, int dv, int stride, int q_off, int k_off, int v_off) {
  return (dk == 64 || dk == 128) && (dv == 64 || dv == 128) && stride % 8 == 0 && q_off % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0;
}

// Floats of working memory per (chunk, head).
extern "C" int dk_decay_attention_tiles_floats(int dk, int dv) { return dk * dv + TC * TC; }

// Arguments as for dk_decay_attention_chunked, with chunks of dk_decay_attention_tiles_chunk() tokens; `work`: total_chunks x H x
// dk_decay_attention_tiles_floats floats.
extern "C" int dk_decay_attention_tiles(const void* src, int stride, int q_off, int k_off, int v_off, int act, const double* decays, float* state,
                                        float* out, float* work, const int* row_slot, const int* row_q_start, const int* row_q_len,
                                        const int* chunk_base, int rows, int total_chunks, int max_chunks, int H, int dk, int dv, int dtype,
                                        cudaStream_t stream) {
  if (rows == 0 || max_chunks == 0) return 0;
  DK_REQUIRE(rows > 0 && H > 0 && dk_decay_attention_tiles_supported(dk, dv, stride, q_off, k_off, v_off),
             "decay_attention_tiles: heads of %d x %d, rows of %d and offsets %d %d %d are not taken", dk, dv, stride, q_off, k_off, v_off);
  DK_REQUIRE((long long)rows * H <= 65535, "decay_attention_tiles: %d rows of %d heads are above the grid's limit", rows, H);
  DK_REQUIRE(max_chunks > 0 && total_chunks >= max_chunks, "decay_attention_tiles: %d chunks in all, %d in a row", total_chunks, max_chunks);
  DK_REQUIRE(((uintptr_t)src | (uintptr_t)work | (uintptr_t)state | (uintptr_t)out) % 16 == 0, "decay_attention_tiles: a tensor begins off its boundary");
  float* A = work + (size_t)total_chunks * H * dk * dv;
#define RUN(T, K, V) \
  return launch<T, K, V>((const T*)src, stride, q_off, k_off, v_off, act, decays, state, out, work, A, row_slot, row_q_start, row_q_len, chunk_base, rows, \
                         max_chunks, H, stream)
#define PICK(T)                            \
  do {                                     \
    if (dk == 128 && dv == 128) RUN(T, 128, 128); \
    if (dk == 128) RUN(T, 128, 64);        \
    if (dv == 128) RUN(T, 64, 128);        \
    RUN(T, 64, 64);                        \
  } while (0)
  if (dtype == DK_BF16) PICK(__nv_bfloat16);
  if (dtype == DK_F32) PICK(float);
#undef PICK
#undef RUN
  DK_REQUIRE(false, "decay_attention_tiles: unknown dtype %d", dtype);
  return 0;
}
