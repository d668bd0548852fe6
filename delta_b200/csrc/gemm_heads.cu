// Up to 16 rows through one small matrix per head,  C_b[M, N] = A_b[M, K] W_b[N, K]^T  for bfloat16, in one launch: a decode step's
// way into the latent space and out of it (latent attention).
//
// Bound by latency: W is a megabyte or two.  A warp takes 16 rows of one W_b and all of K; lane (g, t) of the MMA layout loads 16
// bytes of rows g and g + 8 of W and of row g of A at the same k, which are two fragments of 16 k each (in an order of k that both
// operands share), so every load of four k blocks is under way before the first product.  Every MMA starts from zero and its sum of 16 exact
// products is added by an FADD: an MMA that adds to its accumulator cuts the sum off instead of rounding it.  8 rows, 16 heads of 256 x 128: 15.2 -> 3.1 us
// (the FMA product in tiles of 64 x 64).
#include "common.cuh"
#include "mma_helpers.cuh"

namespace {
constexpr int WARPS = 4;

template <int MT>      // tiles of 8 rows of A
__global__ void __launch_bounds__(WARPS * 32) gemm_heads_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ W,
                                                                __nv_bfloat16* __restrict__ C, int M, int N, int K, int lda, int ldc,
                                                                long long sa, long long sw, long long sc) {
  const int lane = threadIdx.x & 31, g = lane / 4, t = lane % 4;
  const int n0 = (blockIdx.x * WARPS + threadIdx.x / 32) * 16;
  if (n0 >= N) return;
  A += (size_t)blockIdx.y * sa;
  W += (size_t)blockIdx.y * sw;
  C += (size_t)blockIdx.y * sc;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const __nv_bfloat16* w0 = W + (size_t)min(n0 + g, N - 1) * K + t * 8;
  const __nv_bfloat16* w1 = W + (size_t)min(n0 + g + 8, N - 1) * K + t * 8;
  float acc[MT][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += 128) {
    uint4 a[4], b[4], x[MT][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int k = k0 + s * 32;
      const bool in = k < K;
      a[s] = in ? *reinterpret_cast<const uint4*>(w0 + k) : zero;
      b[s] = in ? *reinterpret_cast<const uint4*>(w1 + k) : zero;
#pragma unroll
      for (int i = 0; i < MT; ++i)
        x[i][s] = in && i * 8 + g < M ? *reinterpret_cast<const uint4*>(A + (size_t)(i * 8 + g) * lda + k + t * 8) : zero;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const uint32_t f0[4] = {a[s].x, b[s].x, a[s].y, b[s].y}, f1[4] = {a[s].z, b[s].z, a[s].w, b[s].w};
        mma_add(acc[i], f0, x[i][s].x, x[i][s].y);
        mma_add(acc[i], f1, x[i][s].z, x[i][s].w);
      }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = i * 8 + t * 2 + (j & 1), n = n0 + g + (j >> 1) * 8;
      if (m < M && n < N) C[(size_t)m * ldc + n] = __float2bfloat16_rn(acc[i][j]);
    }
}
}  // namespace

// Rows of A lie lda, rows of C ldc elements apart; the operands of the next head lie sa, sw, sc elements on.
extern "C" int dk_gemm_heads(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldc, int batch, long long sa, long long sw,
                             long long sc, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  DK_REQUIRE(M > 0 && M <= 16 && N > 0 && K > 0 && batch > 0 && batch <= 65535, "gemm_heads: %d products of M=%d N=%d K=%d are not taken", batch, M, N, K);
  DK_REQUIRE(K % 32 == 0 && lda % 8 == 0 && sa % 8 == 0 && sw % 8 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0,
             "gemm_heads: K=%d must be a multiple of 32 and every row of A and W begin on a 16-byte boundary", K);
  const dim3 grid((N + 16 * WARPS - 1) / (16 * WARPS), batch);
  const auto *a = (const __nv_bfloat16*)A, *w = (const __nv_bfloat16*)W;
  if (M <= 8) gemm_heads_kernel<1><<<grid, WARPS * 32, 0, stream>>>(a, w, (__nv_bfloat16*)C, M, N, K, lda, ldc, sa, sw, sc);
  else gemm_heads_kernel<2><<<grid, WARPS * 32, 0, stream>>>(a, w, (__nv_bfloat16*)C, M, N, K, lda, ldc, sa, sw, sc);
  return dk_check_launch("gemm_heads");
}
