// Paged attention in 32 bit for rows that bring several tokens: 16 queries of a head a block, products, softmax and sums on the FMA units,
// the running maximum and denominator of a query with eight neighbouring threads.
//
// Every rounding is the one that attention_plain.cu makes: a query takes its keys in passes of 128 from the request's first one, a score is
// one chain of FMAs over the head, a pass' weights are added as a block of 128 threads adds them there, an output's sum runs over the keys in
// order.  So, without a window that cuts keys off, a token has the same bits whichever of the two kernels takes it, and neither how a prompt
// is cut nor what shares its batch changes them.  (Under a window a pass begins at multiples of 128 here and at the window's first page there.)
//
// Bound by shared memory reads of the two products' register tiles: 1.1 MB a block for every 32 keys, and the serial sums over them.  The plain
// kernel (one block a token and head) fetches every key for every query anew, 4 bytes a thread and 512 apart: a tile shares them between its
// queries.  A fifth warp fetches keys and values by bulk copies, a lane a row, three tiles of 32 ahead: the pages' lookups and the asking are
// no longer in the products' way.  Sixteen queries a tile, not 32, so that 300 tokens of 16 heads are 304 blocks for the 148 SMs, and the tiles
// with most keys go first.  300 tokens, 16 heads of 128, a layer: plain 449 us; tiles of 32 queries and cp.async by all threads 88; bulk copies
// asked for by the first warp between the products 81 (eight threads a query 83); tiles of 16 67; the warp of its own 47.  A running maximum
// for every 32 keys would cost 5 % and other roundings.  What pays when stands at attention_kernels.tiles_pay.
#include "common.cuh"
#include "attention_params.h"
#include "tcgen05_helpers.cuh"
#include "ring.cuh"

namespace {
constexpr int TQ = 16, TK = 32, PASS = 128, SUBS = PASS / TK, STAGES = 3;
constexpr int PARTS = 8, THREADS = TQ * PARTS, PER = TK / PARTS;      // threads a query; a thread's weights of a tile
constexpr int SLD = PASS + 4;

template <int HD>
__global__ void __launch_bounds__(THREADS + 32) attention_f32_kernel(const DkAttnParams p) {
  constexpr int LD = HD + 4, VECS = HD / 4, MINE = VECS / PARTS;      // MINE: a thread's vectors of an output row
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(8) unsigned long long bars[2 * STAGES];
  __shared__ int failed;
  const uint32_t full0 = s2u(&bars[0]), empty0 = full0 + 8 * STAGES;
  volatile int* gave_up = &failed;
  __shared__ unsigned char there[2][PASS];      // by the passes' parity: the key lies in a page of the pool
  float* qs = smem;                     // [TQ][LD]
  float* ring = qs + TQ * LD;           // [STAGES][TK][LD]
  float* sc = ring + STAGES * TK * LD;  // [TQ][SLD]
  const int row = blockIdx.y, h = blockIdx.x % p.H, tid = threadIdx.x;
  const int q_len = p.row_q_len[row], first = (gridDim.x - 1 - blockIdx.x) / p.H * TQ;      // (the tiles that see most keys go first)
  if (first >= q_len || (p.row_filter == 2 && q_len == 1)) return;
  const int t0 = p.row_q_start[row] + first, n = min(TQ, q_len - first), pos0 = p.row_pos_start[row] + first;
  const int g = h / (p.H / p.KV);
  const float* kv = (const float*)p.kv;
  const int last = pos0 + n - 1;
  const int lowest = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;      // the first key that some query of the tile sees
  const int begin = lowest / PASS * PASS;
  auto subs_of = [&](int c0) { return min(SUBS, (last - c0) / TK + 1); };
  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(empty0 + 8 * i, THREADS / 32);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (tid >= THREADS) {
    // the last warp fetches: of every pass the keys' tiles, then the values', a lane a row, whose page it looks up
    const int lane = tid - THREADS;
    int asked = 0;
    bool fine = true;
    for (int c0 = begin; c0 <= last && fine; c0 += PASS) {
      const int subs = subs_of(c0);
      for (int i = 0; i < 2 * subs && fine; ++i) {
        const int sub = i < subs ? i : i - subs, key = c0 + sub * TK + lane, lp = key / p.ps, stage = ring_slot(asked, STAGES);
        float* to = ring + (stage * TK + lane) * LD;
        bool in = key >= lowest && key <= last && lp < p.max_pages;
        const float* at = kv;
        if (in) {
          const int page = p.block_table[(size_t)row * p.max_pages + lp];
          in = page >= 0 && page < p.num_pages;
          if (in) at = kv + ((((size_t)page * 2 + (i < subs ? 0 : 1)) * p.KV + g) * p.ps + key % p.ps) * HD;
          else if (i < subs) dk_report(p.err, DK_DEV_BAD_PAGE, t0, lp, page);      // (its score is left out below)
        }
        if (asked >= STAGES) fine = __all_sync(0xffffffffu, *gave_up == 0 && mbar_wait(empty0 + 8 * stage, ring_parity(asked, STAGES) ^ 1u));
        if (!fine) break;
        if (i < subs) there[(c0 / PASS) & 1][sub * TK + lane] = in;
        if (!in) {
          for (int c = 0; c < HD; c += 4) *reinterpret_cast<float4*>(to + c) = make_float4(0.f, 0.f, 0.f, 0.f);
          fence_async_smem();      // (before a copy that takes the row's place later)
        }
        const uint32_t rows = __popc(__ballot_sync(0xffffffffu, in));
        __syncwarp();
        if (lane == 0) mbar_expect_tx(full0 + 8 * stage, rows * HD * 4);
        __syncwarp();
        if (in) bulk_load(s2u(to), at, HD * 4, full0 + 8 * stage);
        ++asked;
      }
    }
    // (the block stays until its copies are in, whatever became of the other warps)
    const bool in = ring_drain(asked, STAGES, [&](int i, uint32_t parity) { return mbar_wait(full0 + 8 * i, parity); });
    if (lane == 0 && !(fine && in)) dk_report(p.err, DK_DEV_TIMEOUT, row, h, first);
    return;
  }
  for (int v = tid; v < TQ * VECS; v += THREADS) {
    const int r = v / VECS, c = v % VECS * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n) x = *reinterpret_cast<const float4*>((const float*)p.q + (size_t)(t0 + r) * p.q_stride + (size_t)h * HD + c);
    *reinterpret_cast<float4*>(qs + r * LD + c) = x;
  }
  // scores: rows sr, sr + 8, keys sk, sk + 16;   softmax and output: row tid / 8, its part tid % 8
  const int sr = tid / 16, sk = tid % 16, orow = tid / PARTS, part = tid % PARTS;
  const int opos = pos0 + orow, olow = p.window > 0 ? max(0, opos - p.window + 1) : 0;
  float m = -INFINITY, l = 0.f;
  float4 o[MINE];
#pragma unroll
  for (int i = 0; i < MINE; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);

  int used = 0;
  auto next_tile = [&]() {      // the next tile is in
    // (a wait that gives up lets the rest run through, on whatever is there)
    if (!mbar_try_wait(full0 + 8 * ring_slot(used, STAGES), ring_parity(used, STAGES)) && *gave_up == 0 &&
        !mbar_wait(full0 + 8 * ring_slot(used, STAGES), ring_parity(used, STAGES)))
      *gave_up = 1;
    return ring + ring_slot(used, STAGES) * TK * LD;
  };
  auto leave_tile = [&]() {
    __syncwarp();
    if (tid % 32 == 0) mbar_arrive(empty0 + 8 * ring_slot(used, STAGES));
    ++used;
  };
  auto all_sync = []() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); };      // (but the warp that fetches)
  all_sync();
  for (int c0 = begin; c0 <= last; c0 += PASS) {
    const int subs = subs_of(c0);
    for (int i = 0; i < subs; ++i) {
      const float* ks = next_tile();
      float s[2][2] = {};
#pragma unroll 4
      for (int c = 0; c < HD; c += 4) {
        const float4 a = *reinterpret_cast<const float4*>(qs + sr * LD + c), b = *reinterpret_cast<const float4*>(qs + (sr + TQ / 2) * LD + c);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float4 k = *reinterpret_cast<const float4*>(ks + (sk + 16 * j) * LD + c);
          s[0][j] = fmaf(a.w, k.w, fmaf(a.z, k.z, fmaf(a.y, k.y, fmaf(a.x, k.x, s[0][j]))));
          s[1][j] = fmaf(b.w, k.w, fmaf(b.z, k.z, fmaf(b.y, k.y, fmaf(b.x, k.x, s[1][j]))));
        }
      }
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < 2; ++j) sc[(sr + TQ / 2 * r) * SLD + i * TK + sk + 16 * j] = s[r][j];
      leave_tile();
    }
    all_sync();
    // eight threads a query, every eighth key each
    float x[SUBS][PER], big = -INFINITY;
#pragma unroll
    for (int i = 0; i < SUBS; ++i)
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int at = i * TK + part + PARTS * j, key = c0 + at;
        const bool sees = orow < n && key >= olow && key <= opos && there[(c0 / PASS) & 1][at];
        x[i][j] = sees ? __fmul_rn(sc[orow * SLD + at], p.scale) : -INFINITY;
        big = fmaxf(big, x[i][j]);
      }
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
    big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 4));
    const bool none = big == -INFINITY;      // nothing of this pass is seen, or nothing that weighs
    if (!none) {
      const float m_new = fmaxf(m, big), corr = m == -INFINITY ? 0.f : expf(m - m_new);
      float sum[SUBS];
#pragma unroll
      for (int i = 0; i < SUBS; ++i) {
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          x[i][j] = x[i][j] == -INFINITY ? 0.f : expf(x[i][j] - m_new);
          sc[orow * SLD + i * TK + part + PARTS * j] = x[i][j];
        }
        // as a warp adds a tile's 32 weights: lanes 16 and 8 apart, then (below) 4, 2 and 1
        sum[i] = (x[i][0] + x[i][2]) + (x[i][1] + x[i][3]);
      }
#pragma unroll
      for (int i = 0; i < SUBS; ++i) {
        // (all eight threads of a query are here, or none of them)
        const uint32_t mates = 0xffu << (threadIdx.x & 24);
        sum[i] += __shfl_xor_sync(mates, sum[i], 4);
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
    __syncwarp();      // a query's eight threads share a warp
    for (int i = 0; i < subs; ++i) {
      const float* vs = next_tile();
      const int k0 = c0 + i * TK;
      const int k_end = none ? 0 : min(TK, opos - k0 + 1);      // (keys a query does not see stay out of its sums, whatever their values hold)
#pragma unroll 4
      for (int k = max(0, olow - k0); k < k_end; ++k) {
        const float w = sc[orow * SLD + i * TK + k];
#pragma unroll
        for (int e = 0; e < MINE; ++e) {
          const float4 v = *reinterpret_cast<const float4*>(vs + k * LD + (e * PARTS + part) * 4);
          o[e].x = fmaf(w, v.x, o[e].x); o[e].y = fmaf(w, v.y, o[e].y); o[e].z = fmaf(w, v.z, o[e].z); o[e].w = fmaf(w, v.w, o[e].w);
        }
      }
      leave_tile();
    }
    all_sync();      // (the weights are read: the next pass' scores take their place)
  }
  if (failed && tid == 0) dk_report(p.err, DK_DEV_TIMEOUT, row, h, first);
  if (orow >= n) return;
  const float inv = l > 0.f ? 1.f / l : 0.f;
  float* out = (float*)p.out + ((size_t)(t0 + orow) * p.H + h) * HD;
#pragma unroll
  for (int i = 0; i < MINE; ++i)
    *reinterpret_cast<float4*>(out + (i * PARTS + part) * 4) = make_float4(o[i].x * inv, o[i].y * inv, o[i].z * inv, o[i].w * inv);
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
  attention_f32_kernel<HD><<<dim3((max_q_len + TQ - 1) / TQ * p.H, p.rows), THREADS + 32, SMEM, stream>>>(p);
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
