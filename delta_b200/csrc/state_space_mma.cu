// The state-space recurrence of state_space.cu over long bfloat16 portions, in chunks of 64 tokens with warp-level MMA.
//
// With L_t the sum of the log decays of a chunk's tokens 0..t, S [N, P] the state before it and w_s = e^(L_last - L_s) dt_s,
//     y_t = e^(L_t) S^T C_t + sum_{s<=t} M_ts x_s + D x_t ,     M_ts = (C_t . B_s) e^(L_t - L_s) dt_s
//     S  <- e^(L_last) S + sum_s B_s (w_s x_s)^T .
// C, B and x are bfloat16 as they come; S, M and w x are 32 bit and enter the MMAs as three bfloat16 parts each, whose products with
// the other operand are exact.  The parts' sums are kept in two accumulators (the high parts', the others'), a chunk's contribution to
// the state begins at zero, and everything is put together in 32-bit FMA: no operand, sum or result has fewer bits than before.
//   1. ssd_chunk_mma: every chunk in parallel: the products C_t . B_s of a group, dt and L of its heads;
//   2. ssd_intra_mma: every chunk in parallel: what it adds to its own outputs, M x + D x;
//   3. ssd_walk_mma:  along a row, chunk after chunk, a block holds 32 channels of a head: the state, and its share of the outputs.
// An MMA rounds the sum it adds to towards zero: the high parts' products therefore start from zero and are added by FMA units, which
// round to nearest; decays and step sizes come from 64-bit functions.  The walk is bound by the chain along a row (64 heads fill 128 blocks, one an SM):
// 4,100 cycles a chunk, two or three warps a scheduler waiting for one another's MMAs and splits.  One row of 2,048 tokens, 64 heads of 64 x 128: chunks 16 us,
// their own outputs 22, walk 71 (with the own outputs made in the walk and tiles fetched by cp.async, of whose issue a step waited 3,500 cycles, 137);
// the 32-bit kernels, in chunks of 32, 27 and 310 us.  Errors against 64 bits (2-norm, 200 to 1,500 tokens) of
// outputs and states, in units of 1e-8: decays near one 10 to 13 and 9 to 13 here, 25 to 62 and 25 to 74 in the 32-bit kernels; mixed decays 9.4
// to 10.1 and 6.0 to 7.6 here, 7.8 to 10.0 and 4.8 to 11.6 there; strong ones 6.7 to 8.2 and 3.7 to 4.9 here, 6.6 to 8.3 and 4.4 to 4.7 there.
// An infinite state entry stays in its channel; an infinite C, B or x meets zero parts of the other operand and may give a NaN.
#include "common.cuh"
#include "mma_helpers.cuh"
#include "split_bf16.cuh"
#include "tcgen05_helpers.cuh"
#include "ring.cuh"

namespace {
constexpr int TC = 64;                  // tokens of a chunk
constexpr int PS = 32;                  // channels of a block of the walk
constexpr int THREADS = 128;
constexpr int STATE_WARPS = 8, OUT_WARPS = 8;      // of the walk
constexpr int WALK_THREADS = (STATE_WARPS + OUT_WARPS) * 32;
constexpr double LOG2E = 1.4426950408889634;
constexpr double LEAST_LOG2 = -1000.0;   // 2^-1000 is zero in 32 bit: a token's log decay is no smaller, so that sums stay finite
constexpr int HEAD_FLOATS = 5 * TC;     // per (chunk, head): dt, the sums of log2 decays as two floats, e^(L_last - L_s) dt_s and e^(L_t)
constexpr int GROUP_FLOATS = TC * TC;   // per (chunk, group): C_t . B_s

__device__ __forceinline__ double softplus_ss(double x) { return x > 40.0 ? x : log1p(exp(x)); }

// grid (most chunks of a row, rows * G)
template <int N>
__global__ void __launch_bounds__(THREADS)
ssd_chunk_mma_kernel(const __nv_bfloat16* __restrict__ xbc, int stride, const __nv_bfloat16* __restrict__ dtraw, int dt_stride,
                     const float* __restrict__ A_log, const float* __restrict__ dt_bias, float* __restrict__ scores, float* __restrict__ heads,
                     const int* __restrict__ row_q_start, const int* __restrict__ row_q_len, const int* __restrict__ chunk_base, int H, int G, int P) {
  constexpr int LD = N + 8;
  __shared__ __align__(16) __nv_bfloat16 tiles[2][TC][LD];      // C, B
  __shared__ float raw[TC][33];
  const int row = blockIdx.y / G, g = blockIdx.y % G, c0 = blockIdx.x * TC, n_new = row_q_len[row];
  if (c0 >= n_new) return;
  const int n = min(TC, n_new - c0), t0 = row_q_start[row] + c0, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t chunk = (size_t)chunk_base[row] + blockIdx.x;
  for (int v = tid; v < 2 * TC * (N / 8); v += THREADS) {
    const int r = v / (N / 8), i = v % (N / 8) * 8, t = r % TC, which = r / TC;
    cp_async_16(smem_u32(&tiles[which][t][i]), xbc + (size_t)(t0 + (t < n ? t : 0)) * stride + (size_t)H * P + (size_t)(which ? g : G + g) * N + i, t < n);
  }
  cp_async_commit();
  const int per = H / G;
  for (int h0 = 0; h0 < per; h0 += 32) {      // 32 heads at a time: a token's steps lie side by side
    const int hs = min(32, per - h0);
    __syncthreads();
    for (int v = tid; v < n * 32; v += THREADS)
      if (v % 32 < hs) raw[v / 32][v % 32] = __bfloat162float(dtraw[(size_t)(t0 + v / 32) * dt_stride + g * per + h0 + v % 32]);
    __syncthreads();
    for (int j = warp; j < hs; j += THREADS / 32) {      // a lane takes two neighbouring tokens
      const int h = g * per + h0 + j;
      // 64-bit functions, a few thousand a chunk: what decays and step sizes are made of is rounded once
      const double rate = -exp((double)A_log[h]) * LOG2E, bias = dt_bias[h];
      double dt[2], L[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = 2 * lane + e;
        dt[e] = t < n ? softplus_ss((double)raw[t][j] + bias) : 0.0;
        L[e] = t < n ? fmax(rate * dt[e], LEAST_LOG2) : 0.0;      // behind a short chunk's end the sums stay the same
      }
      L[1] += L[0];
      double sum = L[1];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += up;
      }
      const double before = sum - L[1], total = __shfl_sync(0xffffffffu, sum, 31);
      float* out = heads + (chunk * H + h) * HEAD_FLOATS;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double at = e ? sum : before + L[0];
        const float hi = (float)at;
        out[2 * lane + e] = (float)dt[e];
        out[TC + 2 * lane + e] = hi;
        out[2 * TC + 2 * lane + e] = (float)(at - (double)hi);
        out[3 * TC + 2 * lane + e] = (float)(exp2(fmin(total - at, 0.0)) * dt[e]);
        out[4 * TC + 2 * lane + e] = (float)exp2(at);
      }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  // a warp takes 16 rows t and the columns s that any of them reads
  float acc[TC / 8][4];
#pragma unroll
  for (int j = 0; j < TC / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
  for (int k = 0; k < N / 16; ++k) {
    uint32_t a[4];
    ldmatrix_x4(a[0], a[1], a[2], a[3], smem_u32(&tiles[0][warp * 16 + (lane & 15)][k * 16 + (lane >> 4) * 8]));
#pragma unroll
    for (int j = 0; j < TC / 16; ++j) {
      if (j > warp) continue;
      uint32_t b[4];
      ldmatrix_x4(b[0], b[1], b[2], b[3], smem_u32(&tiles[1][j * 16 + (lane >> 4) * 8 + (lane & 7)][k * 16 + ((lane >> 3) & 1) * 8]));
      mma_add(acc[2 * j], a, b[0], b[1]);
      mma_add(acc[2 * j + 1], a, b[2], b[3]);
    }
  }
  float* out = scores + (chunk * G + g) * GROUP_FLOATS;
#pragma unroll
  for (int j = 0; j < TC / 8; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = warp * 16 + (lane >> 2) + 8 * e, s = j * 8 + (lane & 3) * 2;
      *reinterpret_cast<float2*>(out + t * TC + s) = make_float2(s <= t ? acc[j][2 * e] : 0.f, s + 1 <= t ? acc[j][2 * e + 1] : 0.f);
    }
}

// What a chunk adds to itself: out = M x + D x.  grid (most chunks of a row, rows * H); a warp takes 16 tokens and PW channels at a time.
template <int PW>
__global__ void __launch_bounds__(THREADS, 4)
ssd_intra_mma_kernel(const __nv_bfloat16* __restrict__ xbc, int stride, const float* __restrict__ scores, const float* __restrict__ heads,
                     const float* __restrict__ D, float* __restrict__ out, const int* __restrict__ row_q_start, const int* __restrict__ row_q_len,
                     const int* __restrict__ chunk_base, int H, int G, int P) {
  constexpr int LD = PW + 8;
  __shared__ __align__(16) __nv_bfloat16 X[TC][LD];
  __shared__ __align__(16) float hd[3 * TC];      // dt, the sums of log2 decays as two floats
  const int row = blockIdx.y / H, h = blockIdx.y % H, c0 = blockIdx.x * TC, n_new = row_q_len[row];
  if (c0 >= n_new) return;
  const int n = min(TC, n_new - c0), t0 = row_q_start[row] + c0, tid = threadIdx.x, lane = tid & 31, m = tid >> 5, g = h / (H / G);
  const int lg = lane >> 2, lt = lane & 3;
  const size_t chunk = (size_t)chunk_base[row] + blockIdx.x;
  const float* fs = scores + (chunk * G + g) * GROUP_FLOATS;
  const float* hs = heads + (chunk * H + h) * HEAD_FLOATS;
  const float Dh = D[h];
  for (int v = tid; v < 3 * TC / 4; v += THREADS) cp_async_16(smem_u32(hd + v * 4), hs + v * 4, true);
  for (int p0 = 0; p0 < P; p0 += PW) {
    __syncthreads();
    for (int v = tid; v < TC * (PW / 8); v += THREADS) {
      const int t = v / (PW / 8), i = v % (PW / 8) * 8;
      cp_async_16(smem_u32(&X[t][i]), xbc + (size_t)(t0 + (t < n ? t : 0)) * stride + (size_t)h * P + p0 + i, t < n);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const float *dt = hd, *hi = dt + TC, *lo = hi + TC;
    // rows m 16 .. of M, in the layout of an MMA's first operand, times x
    float zh[PW / 8][4], zl[PW / 8][4];
#pragma unroll
    for (int p = 0; p < PW / 8; ++p)
#pragma unroll
      for (int e = 0; e < 4; ++e) zh[p][e] = zl[p][e] = 0.f;
    const int ta = m * 16 + lg, tb = ta + 8;
    const float ha = hi[ta], hb = hi[tb], la = lo[ta], lb = lo[tb];
    for (int k = 0; k <= m; ++k) {
      uint32_t a[3][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int s = k * 16 + lt * 2 + (q >> 1) * 8, t = (q & 1) ? tb : ta;
        const float2 sh = *reinterpret_cast<const float2*>(hi + s), sl = *reinterpret_cast<const float2*>(lo + s), sd = *reinterpret_cast<const float2*>(dt + s);
        const float th = (q & 1) ? hb : ha, tl = (q & 1) ? lb : la;
        const float2 f = *reinterpret_cast<const float2*>(fs + t * TC + s);
        const float m0 = s <= t ? f.x * exp2f((th - sh.x) + (tl - sl.x)) * sd.x : 0.f;
        const float m1 = s + 1 <= t ? f.y * exp2f((th - sh.y) + (tl - sl.y)) * sd.y : 0.f;
        split3(m0, m1, a[0][q], a[1][q], a[2][q]);
      }
#pragma unroll
      for (int p = 0; p < PW / 16; ++p) {
        uint32_t b[4];
        ldmatrix_x4_trans(b[0], b[1], b[2], b[3], smem_u32(&X[k * 16 + (lane & 15)][p * 16 + (lane >> 4) * 8]));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          mma_bf16(zl[2 * p + e], a[2], b[2 * e], b[2 * e + 1]);
          mma_bf16(zl[2 * p + e], a[1], b[2 * e], b[2 * e + 1]);
          mma_add(zh[2 * p + e], a[0], b[2 * e], b[2 * e + 1]);
        }
      }
    }
#pragma unroll
    for (int p = 0; p < PW / 8; ++p)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = e ? tb : ta;
        if (t >= n) continue;
        const uint32_t x = *reinterpret_cast<const uint32_t*>(&X[t][p * 8 + lt * 2]);
        *reinterpret_cast<float2*>(out + (size_t)(t0 + t) * H * P + (size_t)h * P + p0 + p * 8 + lt * 2) =
            make_float2(fmaf(Dh, bf16_low(x), zh[p][2 * e] + zl[p][2 * e]), fmaf(Dh, bf16_high(x), zh[p][2 * e + 1] + zl[p][2 * e + 1]));
      }
  }
}

// Shared memory of the walk: tiles of 64 tokens x 64 entries as TMA leaves them (rows of 128 bytes, 16-byte pieces exchanged by the row's
// number in its group of eight): C, B and x of four chunks, and the heads' numbers; the state before two chunks in parts.
template <int N>
struct Walk {
  static constexpr int TILE = TC * 128, LD = N + 8, DEEP = 4, PARTS = 3 * PS * LD * 2;
  static constexpr int STEP = 2 * (N / 64) * TILE + TILE;      // C, B, x
  static constexpr int HEADS_AT = DEEP * STEP, PARTS_AT = HEADS_AT + DEEP * 2 * TC * 4;
  static constexpr int SMEM = PARTS_AT + 2 * PARTS + 1024;
};
// entries 8 piece .. of a tile's row
__device__ __forceinline__ uint32_t tile_at(uint32_t tile, int row, int piece) { return tile + row * 128 + ((piece ^ (row & 7)) << 4); }

// grid (P / 32, rows * H).  Eight warps hold the state, each 16 channels and a quarter of the state entries, in the accumulators of an MMA whose
// rows are channels.  In a step they leave the state in parts for the eight output warps, which work a chunk behind them, and go on to the
// next; one of the latter fetches three chunks ahead.
template <int N>
__global__ void __launch_bounds__(WALK_THREADS, 1)
ssd_walk_mma_kernel(const __grid_constant__ CUtensorMap map, const float* __restrict__ heads, float* __restrict__ state, float* __restrict__ out,
                    const int* __restrict__ row_slot, const int* __restrict__ row_q_start, const int* __restrict__ row_q_len,
                    const int* __restrict__ chunk_base, int H, int G, int P, int* __restrict__ err) {
  using L = Walk<N>;
  constexpr int LD = L::LD, NQ = N / 4, NT = NQ / 8, TILES = N / 64;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long bars[L::DEEP];
  __shared__ int failed;
  const int row = blockIdx.y / H, h = blockIdx.y % H, p0 = blockIdx.x * PS, n_new = row_q_len[row];
  if (n_new <= 0) return;
  const int g = h / (H / G), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q0 = row_q_start[row];
  const int lg = lane >> 2, lt = lane & 3;
  const int chunks = (n_new + TC - 1) / TC;
  const size_t first = chunk_base[row];
  auto c_of = [&](int c) { return s2u(smem + c % L::DEEP * L::STEP); };
  auto b_of = [&](int c) { return s2u(smem + c % L::DEEP * L::STEP + TILES * L::TILE); };
  auto x_of = [&](int c) { return s2u(smem + c % L::DEEP * L::STEP + 2 * TILES * L::TILE); };
  auto heads_of = [&](int c) { return reinterpret_cast<float*>(smem + L::HEADS_AT + c % L::DEEP * 2 * TC * 4); };
  auto parts_of = [&](int c) { return reinterpret_cast<__nv_bfloat16*>(smem + L::PARTS_AT + (c & 1) * L::PARTS); };
  const uint32_t full0 = s2u(&bars[0]);
  volatile int* gave_up = &failed;
  if (tid == 0) {
    for (int s = 0; s < L::DEEP; ++s) mbar_init(full0 + 8 * s, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  auto arrived = [&](int c) {      // chunk c is in; a wait that gives up lets the rest run through, on whatever is there
    if (mbar_try_wait(full0 + 8 * ring_slot(c, L::DEEP), ring_parity(c, L::DEEP))) return;
    if (*gave_up == 0 && !mbar_wait(full0 + 8 * ring_slot(c, L::DEEP), ring_parity(c, L::DEEP))) *gave_up = 1;
  };

  auto fetch = [&](int c) {
    if (c >= chunks) return;
    const uint32_t bar = full0 + 8 * ring_slot(c, L::DEEP);
    const int t = q0 + c * TC;
    mbar_expect_tx(bar, L::STEP + 2 * TC * 4);
#pragma unroll
    for (int i = 0; i < TILES; ++i) {
      tma_load_2d(c_of(c) + i * L::TILE, &map, H * P + (G + g) * N + i * 64, t, bar);
      tma_load_2d(b_of(c) + i * L::TILE, &map, H * P + g * N + i * 64, t, bar);
    }
    tma_load_2d(x_of(c), &map, h * P + p0, t, bar);
    bulk_load(s2u(heads_of(c)), heads + ((first + c) * H + h) * HEAD_FLOATS + 3 * TC, 2 * TC * 4, bar);      // e^(L_last - L_s) dt_s, e^(L_t)
  };

  if (warp >= STATE_WARPS) {      // the outputs of the chunk before: 32 tokens and eight channels a warp
    const int w = warp - STATE_WARPS, m0 = (w & 1) * 32, ch = (w >> 1) * 8;
    const bool fetches = w == 0 && lane == 0;
    if (fetches) {
      for (int c = 0; c < L::DEEP - 1; ++c) fetch(c);
    }
    for (int c = -1; c < chunks; ++c) {
      __syncthreads();      // everybody has left chunk c - 1, whose tiles chunk c + 3 takes
      if (c < 0) continue;
      if (fetches) fetch(c + L::DEEP - 1);
      const int n = min(TC, n_new - c * TC);
      float* o = out + (size_t)(q0 + c * TC) * H * P + (size_t)h * P + p0 + ch + lt * 2;
      float2 y[2][2];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int t = m0 + m * 16 + lg + 8 * e;
          y[m][e] = t < n ? *reinterpret_cast<const float2*>(o + (size_t)t * H * P) : make_float2(0.f, 0.f);
        }
      arrived(c);
      const uint32_t Cs = c_of(c), Sp = s2u(parts_of(c));
      const float* wo = heads_of(c) + TC;
      float yh[2][4], yl[2][4];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) yh[m][e] = yl[m][e] = 0.f;
#pragma unroll
      for (int k = 0; k < N / 32; ++k) {      // 32 of the state entries
        uint32_t b[3][4];
#pragma unroll
        for (int i = 0; i < 3; ++i)
          ldmatrix_x4(b[i][0], b[i][1], b[i][2], b[i][3], Sp + 2 * ((i * PS + ch + (lane & 7)) * LD + k * 32 + (lane >> 3) * 8));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t a[2][4];
#pragma unroll
          for (int m = 0; m < 2; ++m)
            ldmatrix_x4(a[m][0], a[m][1], a[m][2], a[m][3], tile_at(Cs + k / 2 * L::TILE, m0 + m * 16 + (lane & 15), k % 2 * 4 + e * 2 + (lane >> 4)));
#pragma unroll
          for (int m = 0; m < 2; ++m) mma_bf16(yl[m], a[m], b[2][2 * e], b[2][2 * e + 1]);
#pragma unroll
          for (int m = 0; m < 2; ++m) mma_add(yh[m], a[m], b[0][2 * e], b[0][2 * e + 1]);
#pragma unroll
          for (int m = 0; m < 2; ++m) mma_bf16(yl[m], a[m], b[1][2 * e], b[1][2 * e + 1]);
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int t = m0 + m * 16 + lg + 8 * e;
          const float f = wo[t];
          if (t < n)
            *reinterpret_cast<float2*>(o + (size_t)t * H * P) =
                make_float2(fmaf(f, yh[m][2 * e] + yl[m][2 * e], y[m][e].x), fmaf(f, yh[m][2 * e + 1] + yl[m][2 * e + 1], y[m][e].y));
        }
    }
    if (fetches) ring_drain(chunks, L::DEEP, [&](int s, uint32_t parity) { return mbar_wait(full0 + 8 * s, parity); });
  } else {
    const int quarter = warp & 3, ph = warp >> 2;      // a quarter of the state entries, 16 of the channels
    float* st = state + (((size_t)row_slot[row] * H + h) * P + p0 + ph * 16) * N + quarter * NQ;
    float S[NT][4];      // rows: channels lg and lg + 8, columns: two state entries of each eight
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float2 v = *reinterpret_cast<const float2*>(st + (size_t)(lg + 8 * e) * N + j * 8 + lt * 2);
        S[j][2 * e] = v.x;
        S[j][2 * e + 1] = v.y;
      }
    for (int c = 0; c <= chunks; ++c) {
      __syncthreads();
      if (c == chunks) break;
      __nv_bfloat16* Sp = parts_of(c) + (ph * 16 + lg) * LD + quarter * NQ + lt * 2;
      arrived(c);
      const uint32_t Bs = b_of(c), X = x_of(c);
      const int n = n_new - c * TC;
      if (n < TC) {      // the tokens behind a row's end are another request's: zeros for them
        for (int v = tid; v < (TC - n) * 8 * (TILES + 1); v += STATE_WARPS * 32) {
          const int t = n + v / (8 * (TILES + 1)), i = v % (8 * (TILES + 1));
          const uint32_t at = i < 8 * TILES ? Bs + i / 8 * L::TILE + t * 128 + i % 8 * 16 : X + t * 128 + i % 8 * 16;
          asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(at), "r"(0) : "memory");
        }
        asm volatile("bar.sync 1, %0;" ::"n"(STATE_WARPS * 32) : "memory");
      }
      const float *wi = heads_of(c), *wo = wi + TC;
      // the state behind the chunk
      float uh[NT][4], ul[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) uh[j][e] = ul[j][e] = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t x[4], a[3][4], b[NT / 2][4];      // x: (tokens 0-7, channels 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15); rows of the operand: channels
        ldmatrix_x4_trans(x[0], x[1], x[2], x[3], tile_at(X, k * 16 + (lane & 15), ph * 2 + (lane >> 4)));
        const float2 w0 = *reinterpret_cast<const float2*>(wi + k * 16 + lt * 2), w1 = *reinterpret_cast<const float2*>(wi + k * 16 + lt * 2 + 8);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 w = q < 2 ? w0 : w1;
          const uint32_t xx = x[(q & 1) * 2 + (q >> 1)];
          split3(bf16_low(xx) * w.x, bf16_high(xx) * w.y, a[0][q], a[1][q], a[2][q]);
        }
#pragma unroll
        for (int j = 0; j < NT / 2; ++j) {
          const int col = quarter * NQ + j * 16;
          ldmatrix_x4_trans(b[j][0], b[j][1], b[j][2], b[j][3], tile_at(Bs + col / 64 * L::TILE, k * 16 + (lane & 15), col % 64 / 8 + (lane >> 4)));
        }
        // (one accumulator after the other, so that no MMA waits for the one before it)
#pragma unroll
        for (int j = 0; j < NT; ++j) mma_bf16(ul[j], a[2], b[j / 2][2 * (j & 1)], b[j / 2][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < NT; ++j) mma_add(uh[j], a[0], b[j / 2][2 * (j & 1)], b[j / 2][2 * (j & 1) + 1]);
#pragma unroll
        for (int j = 0; j < NT; ++j) mma_bf16(ul[j], a[1], b[j / 2][2 * (j & 1)], b[j / 2][2 * (j & 1) + 1]);
        if (k < NT) {      // meanwhile a part of the state before the chunk, for its outputs
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            uint32_t s[3];
            split3(S[k][2 * e], S[k][2 * e + 1], s[0], s[1], s[2]);
#pragma unroll
            for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(Sp + (i * PS + 8 * e) * LD + k * 8) = s[i];
          }
        }
      }
      const float keep = wo[TC - 1];
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[j][e] = fmaf(keep, S[j][e], uh[j][e] + ul[j][e]);
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        *reinterpret_cast<float2*>(st + (size_t)(lg + 8 * e) * N + j * 8 + lt * 2) = make_float2(S[j][2 * e], S[j][2 * e + 1]);
  }
  __syncthreads();
  if (failed && tid == 0) dk_report(err, DK_DEV_TIMEOUT, blockIdx.x, blockIdx.y, chunks);
}
}  // namespace

extern "C" int dk_state_space_mma_chunk() { return TC; }

// States of 64 or 128 entries a channel, channels in slices of 32, rows that begin on 16-byte boundaries.
extern "C" int dk_state_space_mma_supported(int N, int P, int stride) { return (N == 64 || N == 128) && P > 0 && P % PS == 0 && stride % 8 == 0; }

// Floats of working memory per chunk.
extern "C" int dk_state_space_mma_floats(int H, int G) { return G * GROUP_FLOATS + H * HEAD_FLOATS; }

// Arguments as for dk_state_space_chunked, with chunks of dk_state_space_mma_chunk() tokens; xbc and dtraw are bfloat16.
extern "C" int dk_state_space_mma(const void* xbc, int stride, const void* dtraw, int dt_stride, const float* A_log, const float* dt_bias,
                                  const float* D, float* state, float* out, float* work, const int* row_slot, const int* row_q_start,
                                  const int* row_q_len, const int* chunk_base, int tokens, int rows, int total_chunks, int max_chunks, int H,
                                  int G, int N, int P, int* err, cudaStream_t stream) {
  if (rows == 0 || max_chunks == 0) return 0;
  DK_REQUIRE(rows > 0 && H > 0 && G > 0 && H % G == 0 && dk_state_space_mma_supported(N, P, stride), "state_space_mma: H=%d G=%d N=%d P=%d stride=%d are not taken",
             H, G, N, P, stride);
  DK_REQUIRE((long long)rows * H <= 65535, "state_space_mma: %d rows of %d heads are above the grid's limit", rows, H);
  DK_REQUIRE(max_chunks > 0 && total_chunks >= max_chunks, "state_space_mma: %d chunks in all, %d in a row", total_chunks, max_chunks);
  DK_REQUIRE(stride >= H * P + 2 * G * N, "state_space_mma: rows of %d elements do not hold x, B and C", stride);
  DK_REQUIRE(((uintptr_t)xbc | (uintptr_t)work) % 16 == 0 && ((uintptr_t)state | (uintptr_t)out) % 8 == 0, "state_space_mma: a tensor begins off its boundary");
  float* heads = work + (size_t)total_chunks * G * GROUP_FLOATS;
  const auto *x = (const __nv_bfloat16*)xbc, *d = (const __nv_bfloat16*)dtraw;
  CUtensorMap map;      // [tokens][x | B | C], boxes of 64 x 64
  DK_REQUIRE(tokens > 0 && make_tensor_map_bf16(&map, xbc, tokens, H * P + 2 * G * N, stride, TC), "state_space_mma: cannot encode the tensor map of %d tokens", tokens);
#define RUN(NN)                                                                                                                                \
  do {                                                                                                                                         \
    static bool granted[DK_MAX_DEVICES] = {false};                                                                                             \
    bool& ok = granted[dk_current_device()];                                                                                                   \
    if (!ok) {                                                                                                                                 \
      DK_REQUIRE(cudaFuncSetAttribute(ssd_walk_mma_kernel<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Walk<NN>::SMEM) == cudaSuccess,    \
                 "state_space_mma: %d bytes of shared memory were refused", Walk<NN>::SMEM);                                                   \
      ok = true;                                                                                                                               \
    }                                                                                                                                          \
    ssd_chunk_mma_kernel<NN><<<dim3(max_chunks, rows * G), THREADS, 0, stream>>>(x, stride, d, dt_stride, A_log, dt_bias, work, heads, row_q_start, \
                                                                                 row_q_len, chunk_base, H, G, P);                              \
    if (P % 64 == 0) INTRA(64);                                                                                                                \
    else INTRA(32);                                                                                                                            \
    ssd_walk_mma_kernel<NN><<<dim3(P / PS, rows * H), WALK_THREADS, Walk<NN>::SMEM, stream>>>(map, heads, state, out, row_slot, row_q_start,   \
                                                                                              row_q_len, chunk_base, H, G, P, err);            \
  } while (0)
#define INTRA(PW) \
  ssd_intra_mma_kernel<PW><<<dim3(max_chunks, rows * H), THREADS, 0, stream>>>(x, stride, work, heads, D, out, row_q_start, row_q_len, chunk_base, H, G, P)
  if (N == 128) RUN(128);
  else RUN(64);
#undef INTRA
#undef RUN
  return dk_check_launch("state_space_mma");
}
