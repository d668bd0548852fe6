// Plain matrix product  C[M,N] = A[M,K] * W[N,K]^T  on the FMA units, float
// accumulation, no reduced-precision matrix mode and no split over K: the sum of
// one output element runs over k in the same order whatever M is, so a token's
// result does not depend on what shares its batch.  This is the plain twin of the
// tensor-core products, and the 32-bit path's product where sums are short (long
// ones: gemm_f32_tc.cu).
//
// Two kernels.  32-bit operands whose rows begin on 16-byte boundaries: tiles come by cp.async, three to four stages ahead, and stay as
// they lie (rows of 16 entries, 20 apart, so that eight neighbouring rows' 16-byte reads meet no bank twice); a thread keeps TM x TN
// sums in registers and reads four k of a row at a time.  Bound by the FMA units.  At 300 rows 32,000 x 2,048 takes 932 us = 42 TFLOP/s, 2,048 x 2,048 107 us
// (tiles of 64 x 64 with one step of K fetched between barriers, as it was: 16 TFLOP/s over a small Yi model's products).
// Other operands (bfloat16, odd rows): one tile size through registers, 16 sums a thread.
#include "common.cuh"

namespace {
constexpr int BK = 16;

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pair_of(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpair(unsigned long long v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}

// Four neighbouring entries of a row from column k on; VEC: they exist and begin on a vector's boundary, or the row has none.
template <typename T, bool VEC>
__device__ __forceinline__ float4 load4(const T* row, int k, int K, bool in) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!in) return v;
  if constexpr (VEC) {
    if (k >= K) return v;
    if constexpr (sizeof(T) == 4) {
      v = *reinterpret_cast<const float4*>(row + k);
    } else {
      const uint2 raw = *reinterpret_cast<const uint2*>(row + k);
      const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
      v = make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
    }
  } else {
    if (k < K) v.x = to_f32<T>(row[k]);
    if (k + 1 < K) v.y = to_f32<T>(row[k + 1]);
    if (k + 2 < K) v.z = to_f32<T>(row[k + 2]);
    if (k + 3 < K) v.w = to_f32<T>(row[k + 3]);
  }
  return v;
}

template <typename TI, typename TO, int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN)) gemm_nt_kernel(const TI* __restrict__ A, const TI* __restrict__ W, TO* __restrict__ C,
                                                                        int M, int N, int K, int lda, int ldw, int ldc,
                                                                        long long sa, long long sw, long long sc) {
  constexpr int NT = (BM / TM) * (BN / TN), LA = BM * BK / 4 / NT, LW = BN * BK / 4 / NT, GM = TM / 4, GN = TN / 4;
  static_assert(LA * NT * 4 == BM * BK && LW * NT * 4 == BN * BK, "a tile is a whole number of vectors a thread");
  A += (size_t)blockIdx.z * sa;      // one product per blockIdx.z: the operands of the next lie sa, sw, sc elements on
  W += (size_t)blockIdx.z * sw;
  C += (size_t)blockIdx.z * sc;
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Ws[2][BK][BN + 4];
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

  float4 ra[LA], rw[LW];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int v = tid + i * NT, r = m0 + v / (BK / 4);
      ra[i] = load4<TI, VEC>(A + (size_t)r * lda, k0 + v % (BK / 4) * 4, K, r < M);
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int v = tid + i * NT, r = n0 + v / (BK / 4);
      rw[i] = load4<TI, VEC>(W + (size_t)r * ldw, k0 + v % (BK / 4) * 4, K, r < N);
    }
  };
  auto keep = [&](int b) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int v = tid + i * NT, r = v / (BK / 4), c = v % (BK / 4) * 4;
      As[b][c][r] = ra[i].x; As[b][c + 1][r] = ra[i].y; As[b][c + 2][r] = ra[i].z; As[b][c + 3][r] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int v = tid + i * NT, r = v / (BK / 4), c = v % (BK / 4) * 4;
      Ws[b][c][r] = rw[i].x; Ws[b][c + 1][r] = rw[i].y; Ws[b][c + 2][r] = rw[i].z; Ws[b][c + 3][r] = rw[i].w;
    }
  };
  const int steps = (K + BK - 1) / BK;
  fetch(0);
  keep(0);
  __syncthreads();
  for (int s = 0; s < steps; ++s) {
    const int b = s & 1;
    if (s + 1 < steps) fetch((s + 1) * BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float4 a[GM];
      ulonglong2 w[GN];
#pragma unroll
      for (int g = 0; g < GM; ++g) a[g] = *reinterpret_cast<const float4*>(&As[b][kk][g * (BM / GM) + ty * 4]);
#pragma unroll
      for (int g = 0; g < GN; ++g) w[g] = *reinterpret_cast<const ulonglong2*>(&Ws[b][kk][g * (BN / GN) + tx * 4]);
#pragma unroll
      for (int g = 0; g < GM; ++g) {
        const unsigned long long d[4] = {pair_of(a[g].x, a[g].x), pair_of(a[g].y, a[g].y), pair_of(a[g].z, a[g].z), pair_of(a[g].w, a[g].w)};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int h = 0; h < GN; ++h) {
            fma2(acc[g * 4 + i][h * 2], d[i], w[h].x);
            fma2(acc[g * 4 + i][h * 2 + 1], d[i], w[h].y);
          }
      }
    }
    if (s + 1 < steps) {
      keep(b ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + (i / 4) * (BM / GM) + ty * 4 + i % 4;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) {
      const int n = n0 + (j / 2) * (BN / GN) + tx * 4 + (j % 2) * 2;
      float x, y;
      unpair(acc[i][j], x, y);
      if (n < N) C[(size_t)m * ldc + n] = from_f32<TO>(x);
      if (n + 1 < N) C[(size_t)m * ldc + n + 1] = from_f32<TO>(y);
    }
  }
}

__device__ __forceinline__ void copy16(float* to, const float* from, bool in) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(to);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(from), "r"(in ? 16 : 0));
}

// Rows of A and W begin on 16-byte boundaries and K is a multiple of 4.
template <int BM, int BN, int TM, int TN, int STAGES, int PER_SM>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), PER_SM) gemm_nt_f32_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                                    float* __restrict__ C, int M, int N, int K, int lda, int ldw,
                                                                                    int ldc, long long sa, long long sw, long long sc) {
  constexpr int NT = (BM / TM) * (BN / TN), LD = BK + 4, LA = BM * BK / 4 / NT, LW = BN * BK / 4 / NT, RM = BM / TM, RN = BN / TN;
  static_assert(LA * NT * 4 == BM * BK && LW * NT * 4 == BN * BK, "a tile is a whole number of vectors a thread");
  extern __shared__ __align__(16) float smem[];
  A += (size_t)blockIdx.z * sa;
  W += (size_t)blockIdx.z * sw;
  C += (size_t)blockIdx.z * sc;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, tid = threadIdx.x;
  const int tx = tid % RN, ty = tid / RN;
  const int steps = (K + BK - 1) / BK;
  auto fetch = [&](int s) {
    if (s < steps) {
      float* to = smem + (s % STAGES) * (BM + BN) * LD;
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        const int v = tid + i * NT, r = v / (BK / 4), k = s * BK + v % (BK / 4) * 4;
        const bool in = m0 + r < M && k < K;
        copy16(to + r * LD + v % (BK / 4) * 4, in ? A + (size_t)(m0 + r) * lda + k : A, in);
      }
#pragma unroll
      for (int i = 0; i < LW; ++i) {
        const int v = tid + i * NT, r = v / (BK / 4), k = s * BK + v % (BK / 4) * 4;
        const bool in = n0 + r < N && k < K;
        copy16(to + (BM + r) * LD + v % (BK / 4) * 4, in ? W + (size_t)(n0 + r) * ldw + k : W, in);
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) fetch(s);
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2));
    __syncthreads();      // stage s is in, and everybody has left the one that is fetched into next
    fetch(s + STAGES - 1);
    const float* as = smem + (s % STAGES) * (BM + BN) * LD + ty * LD;
    const float* ws = smem + (s % STAGES) * (BM + BN) * LD + (BM + tx) * LD;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * RM * LD + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 w = *reinterpret_cast<const float4*>(ws + j * RN * LD + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, w.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, w.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, w.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, w.w, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * RM;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * RN;
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}

template <int BM, int BN, int TM, int TN, int STAGES, int PER_SM>
int launch_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch, long long sa, long long sw,
               long long sc, cudaStream_t stream) {
  constexpr int SMEM = STAGES * (BM + BN) * (BK + 4) * (int)sizeof(float);
  auto* kernel = gemm_nt_f32_kernel<BM, BN, TM, TN, STAGES, PER_SM>;
  if constexpr (SMEM > 48 * 1024) {
    static bool granted[DK_MAX_DEVICES] = {false};
    bool& g = granted[dk_current_device()];
    if (!g) {
      DK_REQUIRE(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess, "gemm: %d bytes of shared memory were refused", SMEM);
      g = true;
    }
  }
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
  kernel<<<grid, (BM / TM) * (BN / TN), SMEM, stream>>>(A, W, C, M, N, K, lda, ldw, ldc, sa, sw, sc);
  return 0;
}

template <typename TI, typename TO>
int launch(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int batch, long long sa, long long sw,
           long long sc, cudaStream_t stream) {
  const dim3 grid((N + 63) / 64, (M + 31) / 32, batch);
  const uintptr_t vec = 4 * sizeof(TI);      // rows of four entries as one vector, where every row and product begins on one's boundary
  const bool aligned = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && sa % 4 == 0 && sw % 4 == 0 && (uintptr_t)A % vec == 0 && (uintptr_t)W % vec == 0;
  if constexpr (sizeof(TI) == 4) {
    if (aligned) {
      const float *a = (const float*)A, *w = (const float*)W;
      const long long sms = dk_sm_count();
      auto blocks = [&](int bm, int bn) { return ((long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn) * batch + sms - 1) / sms; };
      // An SM's share of the sums, times what a sum costs in that tile (measured), and a fifth more where the SM gets so few
      // warps that its loads show.  Whatever the tile, a sum runs over k in order.
      const long long b0 = blocks(64, 128), b1 = blocks(32, 64), b2 = blocks(32, 32);
      const long long c0 = b0 * 64 * 128 * (b0 < 2 ? 120 : 100), c1 = b1 * 32 * 64 * (b1 < 4 ? 132 : 110), c2 = b2 * 32 * 32 * 112;
      if (c0 <= c1 && c0 <= c2) return launch_f32<64, 128, 8, 8, 4, 3>(a, w, (float*)C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
      if (c1 <= c2) return launch_f32<32, 64, 4, 8, 4, 6>(a, w, (float*)C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
      return launch_f32<32, 32, 4, 4, 4, 8>(a, w, (float*)C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
    }
  }
#define RUN(V) gemm_nt_kernel<TI, TO, 32, 64, 4, 4, V><<<grid, 128, 0, stream>>>((const TI*)A, (const TI*)W, (TO*)C, M, N, K, lda, ldw, ldc, sa, sw, sc)
  if (aligned) RUN(true);
  else RUN(false);
#undef RUN
  return 0;
}

int launch_any(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int batch, long long sa, long long sw,
               long long sc, int in_dtype, int out_dtype, cudaStream_t stream) {
  DK_REQUIRE((M + 63LL) / 64 <= 65535, "gemm: M=%d is too large for this kernel", M);
  DK_REQUIRE(in_dtype == DK_F32 ? out_dtype == DK_F32 : in_dtype == DK_BF16 && (out_dtype == DK_BF16 || out_dtype == DK_F32),
             "gemm: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
  constexpr int MOST = 65535 * 32;      // rows that tiles of 32 can number: more of them go in two launches
  for (int m = 0; m < M; m += MOST) {
    const int rows = min(M - m, MOST);
#define LAUNCH(TI, TO) \
  launch<TI, TO>((const TI*)A + (size_t)m * lda, W, (TO*)C + (size_t)m * ldc, rows, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream)
    int rc;
    if (in_dtype == DK_F32) rc = LAUNCH(float, float);
    else if (out_dtype == DK_BF16) rc = LAUNCH(__nv_bfloat16, __nv_bfloat16);
    else rc = LAUNCH(__nv_bfloat16, float);
#undef LAUNCH
    if (rc) return rc;
  }
  return 0;
}
}  // namespace

// in_dtype: type of A and W; out_dtype: type of C (float output from bfloat16
// operands is how logits are made).
extern "C" int dk_gemm_nt_plain(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc,
                                int in_dtype, int out_dtype, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  DK_REQUIRE(M > 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  DK_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm: leading sizes %d %d %d too small", lda, ldw, ldc);
  const int rc = launch_any(A, W, C, M, N, K, lda, ldw, ldc, 1, 0, 0, 0, in_dtype, out_dtype, stream);
  return rc ? rc : dk_check_launch("gemm_nt_plain");
}

// `batch` products of the same sizes in one launch (one per head of an attention layer, say): product b reads
// A + b*sa, W + b*sw and writes C + b*sc (strides in elements; the operands may interleave, as heads do in a row).
extern "C" int dk_gemm_nt_plain_batched(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc,
                                        int batch, long long sa, long long sw, long long sc, int in_dtype, int out_dtype,
                                        cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  DK_REQUIRE(M > 0 && N > 0 && K > 0 && batch > 0, "gemm: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
  DK_REQUIRE(batch <= 65535, "gemm: %d products in one launch are too many", batch);
  const int rc = launch_any(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, in_dtype, out_dtype, stream);
  return rc ? rc : dk_check_launch("gemm_nt_plain_batched");
}
