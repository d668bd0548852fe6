// Paged attention in 32 bit for rows that bring several tokens: 32 queries of a head and 32 keys a tile, products, softmax
// and sums on the FMA units, the running maximum and denominator of a query with four neighbouring threads.  Key tiles begin at
// multiples of 32 of the request's positions and a query's sums run over them in order, so a token's result does not depend on how
// its prompt was cut or on what shares its batch.
//
// Bound by shared memory reads of the two products' register tiles.  The plain kernel (one block a token and head) fetches every key
// for every query anew, 4 bytes a thread and 512 apart: a tile shares them between 32 queries.  300 tokens, 16 heads
// of 128: 449 -> 99 us a layer.
#include "common.cuh"
#include "attention_params.h"

namespace {
constexpr int TQ = 32, TK = 32, THREADS = 128;

template <int HD>
__global__ void __launch_bounds__(THREADS) attention_f32_kernel(const DkAttnParams p) {
  constexpr int LD = HD + 4, VECS = HD / 4, MINE = HD / 16;      // MINE: a thread's vectors of an output row
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                 // [TQ][LD]
  float* ks = qs + TQ * LD;         // [TK][LD]
  float* vs = ks + TK * LD;         // [TK][LD]
  float* sc = vs + TK * LD;         // [TQ][TK + 1]
  const int row = blockIdx.z, h = blockIdx.y, tid = threadIdx.x;
  const int q_len = p.row_q_len[row], first = blockIdx.x * TQ;
  if (first >= q_len || (p.row_filter == 2 && q_len == 1)) return;
  const int t0 = p.row_q_start[row] + first, n = min(TQ, q_len - first), pos0 = p.row_pos_start[row] + first;
  const int g = h / (p.H / p.KV);
  const float* kv = (const float*)p.kv;
  for (int v = tid; v < TQ * VECS; v += THREADS) {
    const int r = v / VECS, c = v % VECS * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n) x = *reinterpret_cast<const float4*>((const float*)p.q + (size_t)(t0 + r) * p.q_stride + (size_t)h * HD + c);
    *reinterpret_cast<float4*>(qs + r * LD + c) = x;
  }
  const int last = pos0 + n - 1;
  const int lowest = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;      // the first key that some query of the tile sees
  // scores: rows sr, sr + 16, keys sk + 8 j;   softmax and output: row tid / 4, its part tid % 4
  const int sr = tid / 8, sk = tid % 8, orow = tid / 4, part = tid % 4;
  const int opos = pos0 + orow, olow = p.window > 0 ? max(0, opos - p.window + 1) : 0;
  float m = -INFINITY, l = 0.f;
  float4 o[MINE];
#pragma unroll
  for (int i = 0; i < MINE; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);

  for (int k0 = lowest / TK * TK; k0 <= last; k0 += TK) {
    __syncthreads();      // the tile before has been read
    for (int v = tid; v < TK * VECS; v += THREADS) {
      const int r = v / VECS, c = v % VECS * 4, key = k0 + r, lp = key / p.ps;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
      if (key >= lowest && key <= last && lp < p.max_pages) {
        const int page = p.block_table[(size_t)row * p.max_pages + lp];
        if (page >= 0 && page < p.num_pages) {
          const float* at = kv + (((size_t)page * 2 * p.KV + g) * p.ps + key % p.ps) * HD + c;
          a = *reinterpret_cast<const float4*>(at);
          b = *reinterpret_cast<const float4*>(at + (size_t)p.KV * p.ps * HD);
        } else {
          dk_report(p.err, DK_DEV_BAD_PAGE, t0, lp, page);      // (its score is left out below)
        }
      }
      *reinterpret_cast<float4*>(ks + r * LD + c) = a;
      *reinterpret_cast<float4*>(vs + r * LD + c) = b;
    }
    __syncthreads();
    float s[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
    for (int c = 0; c < HD; c += 4) {
      const float4 a = *reinterpret_cast<const float4*>(qs + sr * LD + c), b = *reinterpret_cast<const float4*>(qs + (sr + 16) * LD + c);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 k = *reinterpret_cast<const float4*>(ks + (sk + 8 * j) * LD + c);
        s[0][j] = fmaf(a.w, k.w, fmaf(a.z, k.z, fmaf(a.y, k.y, fmaf(a.x, k.x, s[0][j]))));
        s[1][j] = fmaf(b.w, k.w, fmaf(b.z, k.z, fmaf(b.y, k.y, fmaf(b.x, k.x, s[1][j]))));
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[(sr + 16 * i) * (TK + 1) + sk + 8 * j] = s[i][j];
    __syncthreads();
    // four threads a query: eight keys each
    float x[8], big = -INFINITY;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int key = k0 + part * 8 + j, lp = key / p.ps;
      bool sees = orow < n && key >= olow && key <= opos && lp < p.max_pages;
      if (sees) {
        const int page = p.block_table[(size_t)row * p.max_pages + lp];
        sees = page >= 0 && page < p.num_pages;
      }
      x[j] = sees ? sc[orow * (TK + 1) + part * 8 + j] * p.scale : -INFINITY;
      big = fmaxf(big, x[j]);
    }
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
    const float m_new = fmaxf(m, big);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      x[j] = x[j] == -INFINITY ? 0.f : expf(x[j] - m_new);
      sum += x[j];
      sc[orow * (TK + 1) + part * 8 + j] = x[j];
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const float corr = m == -INFINITY ? 0.f : expf(m - m_new);
    l = l * corr + sum;
    m = m_new;
    __syncwarp();      // a query's four threads share a warp
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      o[i].x *= corr; o[i].y *= corr; o[i].z *= corr; o[i].w *= corr;
    }
    const int k_end = min(TK, opos - k0 + 1);      // (keys a query does not see stay out of its sums, whatever their values hold)
#pragma unroll 4
    for (int k = max(0, olow - k0); k < k_end; ++k) {
      const float w = sc[orow * (TK + 1) + k];
#pragma unroll
      for (int i = 0; i < MINE; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(vs + k * LD + (i * 4 + part) * 4);
        o[i].x = fmaf(w, v.x, o[i].x); o[i].y = fmaf(w, v.y, o[i].y); o[i].z = fmaf(w, v.z, o[i].z); o[i].w = fmaf(w, v.w, o[i].w);
      }
    }
  }
  if (orow >= n) return;
  const float inv = l > 0.f ? 1.f / l : 0.f;
  float* out = (float*)p.out + ((size_t)(t0 + orow) * p.H + h) * HD;
#pragma unroll
  for (int i = 0; i < MINE; ++i)
    *reinterpret_cast<float4*>(out + (i * 4 + part) * 4) = make_float4(o[i].x * inv, o[i].y * inv, o[i].z * inv, o[i].w * inv);
  if (p.lse != nullptr && part == 0) p.lse[(size_t)(t0 + orow) * p.H + h] = l > 0.f ? m + logf(l) : -INFINITY;
}

template <int HD>
int launch(const DkAttnParams& p, int max_q_len, cudaStream_t stream) {
  constexpr int SMEM = (3 * TQ * (HD + 4) + TQ * (TK + 1)) * (int)sizeof(float);
  if constexpr (SMEM > 48 * 1024) {
    static bool granted[DK_MAX_DEVICES] = {false};
    bool& ok = granted[dk_current_device()];
    if (!ok) {
      DK_REQUIRE(cudaFuncSetAttribute(attention_f32_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess,
                 "attention_f32: %d bytes of shared memory were refused", SMEM);
      ok = true;
    }
  }
  attention_f32_kernel<HD><<<dim3((max_q_len + TQ - 1) / TQ, p.H, p.rows), THREADS, SMEM, stream>>>(p);
  return dk_check_launch("attention_f32");
}
}  // namespace

extern "C" int dk_attention_f32_supported(int dtype, int H, int KV, int hd, int q_stride) {
  return dtype == DK_F32 && KV > 0 && H % KV == 0 && H <= 65535 && (hd == 32 || hd == 64 || hd == 128) && q_stride % 4 == 0;
}

// max_q_len: the most tokens a row brings.  Chosen pages and score dumps are the plain kernel's.
extern "C" int dk_attention_f32(const DkAttnParams* pp, int max_q_len, cudaStream_t stream) {
  const DkAttnParams& p = *pp;
  if (p.T == 0 || p.rows == 0) return 0;
  DK_REQUIRE(dk_attention_f32_supported(p.dtype, p.H, p.KV, p.hd, p.q_stride), "attention_f32: dtype %d, %d / %d heads of %d, stride %d are not taken",
             p.dtype, p.H, p.KV, p.hd, p.q_stride);
  DK_REQUIRE(p.T > 0 && max_q_len > 0 && p.rows <= 65535, "attention_f32: bad sizes T=%d, %d rows of up to %d", p.T, p.rows, max_q_len);
  DK_REQUIRE(p.ps >= 1 && p.max_pages > 0, "attention_f32: bad page size %d or table width %d", p.ps, p.max_pages);
  DK_REQUIRE(p.sel_pages == nullptr && p.dump == nullptr, "attention_f32: chosen pages and score dumps are not taken");
  DK_REQUIRE(p.row_q_len != nullptr && p.row_q_start != nullptr && p.row_pos_start != nullptr, "attention_f32: the rows' starts and lengths are missing");
  DK_REQUIRE(((uintptr_t)p.q | (uintptr_t)p.kv | (uintptr_t)p.out) % 16 == 0, "attention_f32: q, cache and output begin on 16-byte boundaries");
  if (p.hd == 128) return launch<128>(p, max_q_len, stream);
  if (p.hd == 64) return launch<64>(p, max_q_len, stream);
  return launch<32>(p, max_q_len, stream);
}
