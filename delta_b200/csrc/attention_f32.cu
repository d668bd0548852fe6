// Paged attention in 32 bit for rows that bring several tokens: 32 queries of a head a block, products, softmax and sums on the FMA units,
// the running maximum and denominator of a query with four neighbouring threads.
//
// Every rounding is the one that attention_plain.cu makes: a query takes its keys in passes of 128 from the request's first one, a score is
// one chain of FMAs over the head, a pass' weights are added as a block of 128 threads adds them there, an output's sum runs over the keys in
// order.  So, without a window that cuts keys off, a token has the same bits whichever of the two kernels takes it, and neither how a prompt
// is cut nor what shares its batch changes them.  (Under a window a pass begins at multiples of 128 here and at the window's first page there.)
//
// Bound by shared memory reads of the two products' register tiles and, with less than two blocks an SM, by their latency.  The plain kernel
// (one block a token and head) fetches every key for every query anew, 4 bytes a thread and 512 apart: a tile shares them between 32
// queries.  Keys and values come by cp.async in tiles of 32, two ahead.  300 tokens, 16 heads of 128: 449 -> 94 us a layer (99 with a running
// maximum for every 32 keys, which had other roundings); what pays when stands at attention_kernels.tiles_pay.
#include "common.cuh"
#include "attention_params.h"
#include "mma_helpers.cuh"

namespace {
constexpr int TQ = 32, TK = 32, PASS = 128, SUBS = PASS / TK, THREADS = 128, STAGES = 3;
constexpr int SLD = PASS + 4;

template <int HD>
__global__ void __launch_bounds__(THREADS) attention_f32_kernel(const DkAttnParams p) {
  constexpr int LD = HD + 4, VECS = HD / 4, MINE = HD / 16;      // MINE: a thread's vectors of an output row
  extern __shared__ __align__(16) float smem[];
  __shared__ unsigned char there[2][PASS];      // by the passes' parity: the key lies in a page of the pool
  float* qs = smem;                     // [TQ][LD]
  float* ring = qs + TQ * LD;           // [STAGES][TK][LD]
  float* sc = ring + STAGES * TK * LD;  // [TQ][SLD]
  const int row = blockIdx.z, h = blockIdx.y, tid = threadIdx.x;
  const int q_len = p.row_q_len[row], first = blockIdx.x * TQ;
  if (first >= q_len || (p.row_filter == 2 && q_len == 1)) return;
  const int t0 = p.row_q_start[row] + first, n = min(TQ, q_len - first), pos0 = p.row_pos_start[row] + first;
  const int g = h / (p.H / p.KV);
  const float* kv = (const float*)p.kv;
  const int last = pos0 + n - 1;
  const int lowest = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;      // the first key that some query of the tile sees
  const int begin = lowest / PASS * PASS;
  auto subs_of = [&](int c0) { return min(SUBS, (last - c0) / TK + 1); };
  // Tile i of the pass from c0 on: its keys' tiles, then its values'.
  auto fetch = [&](int c0, int i, int stage) {
    const int subs = subs_of(c0), sub = i < subs ? i : i - subs;
    float* to = ring + stage * TK * LD;
    if (c0 <= last) {
#pragma unroll
      for (int v = tid; v < TK * VECS; v += THREADS) {
        const int r = v / VECS, c = v % VECS * 4, key = c0 + sub * TK + r, lp = key / p.ps;
        bool in = key >= lowest && key <= last && lp < p.max_pages;
        const float* at = kv;
        if (in) {
          const int page = p.block_table[(size_t)row * p.max_pages + lp];
          in = page >= 0 && page < p.num_pages;
          if (in) at = kv + ((((size_t)page * 2 + (i < subs ? 0 : 1)) * p.KV + g) * p.ps + key % p.ps) * HD + c;
          else if (i < subs && c == 0) dk_report(p.err, DK_DEV_BAD_PAGE, t0, lp, page);      // (its score is left out below)
        }
        if (i < subs && c == 0) there[(c0 / PASS) & 1][sub * TK + r] = in;
        cp_async_16(smem_u32(to + r * LD + c), at, in);
      }
    }
    cp_async_commit();
  };
  int fetch_c = begin, fetch_i = 0, fetched = 0;
  auto fetch_next = [&]() {
    fetch(fetch_c, fetch_i, fetched % STAGES);
    ++fetched;
    if (fetch_c <= last && ++fetch_i == 2 * subs_of(fetch_c)) {
      fetch_i = 0;
      fetch_c += PASS;
    }
  };
  fetch_next();
  fetch_next();
  for (int v = tid; v < TQ * VECS; v += THREADS) {
    const int r = v / VECS, c = v % VECS * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n) x = *reinterpret_cast<const float4*>((const float*)p.q + (size_t)(t0 + r) * p.q_stride + (size_t)h * HD + c);
    *reinterpret_cast<float4*>(qs + r * LD + c) = x;
  }
  // scores: rows sr, sr + 16, keys sk + 8 j;   softmax and output: row tid / 4, its part tid % 4
  const int sr = tid / 8, sk = tid % 8, orow = tid / 4, part = tid % 4;
  const int opos = pos0 + orow, olow = p.window > 0 ? max(0, opos - p.window + 1) : 0;
  float m = -INFINITY, l = 0.f;
  float4 o[MINE];
#pragma unroll
  for (int i = 0; i < MINE; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);

  int used = 0;
  auto next_tile = [&]() {      // the next tile is in, everybody has left the one before it, whose stage is fetched into
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    fetch_next();
    return ring + used++ % STAGES * TK * LD;
  };
  for (int c0 = begin; c0 <= last; c0 += PASS) {
    const int subs = subs_of(c0);
    for (int i = 0; i < subs; ++i) {
      const float* ks = next_tile();
      float s[2][4] = {};
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
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) sc[(sr + 16 * r) * SLD + i * TK + sk + 8 * j] = s[r][j];
    }
    __syncthreads();
    // four threads a query, every fourth key each
    float x[SUBS][8], big = -INFINITY;
#pragma unroll
    for (int i = 0; i < SUBS; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int at = i * TK + part + 4 * j, key = c0 + at;
        const bool sees = orow < n && key >= olow && key <= opos && there[(c0 / PASS) & 1][at];
        x[i][j] = sees ? __fmul_rn(sc[orow * SLD + at], p.scale) : -INFINITY;
        big = fmaxf(big, x[i][j]);
      }
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
    const bool none = big == -INFINITY;      // nothing of this pass is seen, or nothing that weighs
    if (!none) {
      const float m_new = fmaxf(m, big), corr = m == -INFINITY ? 0.f : expf(m - m_new);
      float sum[SUBS];
#pragma unroll
      for (int i = 0; i < SUBS; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          x[i][j] = x[i][j] == -INFINITY ? 0.f : expf(x[i][j] - m_new);
          sc[orow * SLD + i * TK + part + 4 * j] = x[i][j];
        }
        // as a warp adds a tile's 32 weights: lanes 16, 8 and 4 apart, then (below) 2 and 1
        sum[i] = ((x[i][0] + x[i][4]) + (x[i][2] + x[i][6])) + ((x[i][1] + x[i][5]) + (x[i][3] + x[i][7]));
      }
#pragma unroll
      for (int i = 0; i < SUBS; ++i) {
        // (all four threads of a query are here, or none of them)
        const uint32_t mates = 0xfu << (threadIdx.x & 28);
        sum[i] += __shfl_xor_sync(mates, sum[i], 2);
        sum[i] += __shfl_xor_sync(mates, sum[i], 1);
      }
      l = fmaf(l, corr, (sum[0] + sum[2]) + (sum[1] + sum[3]));
      m = m_new;
#pragma unroll
      for (int i = 0; i < MINE; ++i) {
        o[i].x *= corr; o[i].y *= corr; o[i].z *= corr; o[i].w *= corr;
      }
    }
    __syncwarp();      // a query's four threads share a warp
    for (int i = 0; i < subs; ++i) {
      const float* vs = next_tile();
      const int k0 = c0 + i * TK;
      const int k_end = none ? 0 : min(TK, opos - k0 + 1);      // (keys a query does not see stay out of its sums, whatever their values hold)
#pragma unroll 4
      for (int k = max(0, olow - k0); k < k_end; ++k) {
        const float w = sc[orow * SLD + i * TK + k];
#pragma unroll
        for (int e = 0; e < MINE; ++e) {
          const float4 v = *reinterpret_cast<const float4*>(vs + k * LD + (e * 4 + part) * 4);
          o[e].x = fmaf(w, v.x, o[e].x); o[e].y = fmaf(w, v.y, o[e].y); o[e].z = fmaf(w, v.z, o[e].z); o[e].w = fmaf(w, v.w, o[e].w);
        }
      }
    }
  }
  cp_async_wait<0>();
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
  constexpr int SMEM = ((TQ + STAGES * TK) * (HD + 4) + TQ * SLD) * (int)sizeof(float);
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
