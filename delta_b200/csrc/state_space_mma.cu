// The state-space recurrence of state_space.cu over long bfloat16 portions, in chunks of 64 tokens with warp-level MMA.
//
// With L_t the sum of the log decays of a chunk's tokens 0..t, S [N, P] the state before it and w_s = e^(L_last - L_s) dt_s,
//     y_t = e^(L_t) S^T C_t + sum_{s<=t} M_ts x_s + D x_t ,     M_ts = (C_t . B_s) e^(L_t - L_s) dt_s
//     S  <- e^(L_last) S + sum_s B_s (w_s x_s)^T .
// C, B and x are bfloat16 as they come; S, M and w x are 32 bit and enter the MMAs as three bfloat16 parts each, whose products with
// the other operand are exact.  The parts' sums are kept in two accumulators (the high parts', the others'), a chunk's contribution to
// the state begins at zero, and everything is put together in 32-bit FMA: no operand, sum or result has fewer bits than before.
//   1. ssd_chunk_mma: every chunk in parallel: the products C_t . B_s of a group, dt and L of its heads;
//   2. ssd_walk_mma:  along a row, chunk after chunk; a block holds 32 channels of a head.  Four warps hold the state, each 16 channels
//      and half of the state entries, in the accumulators of an MMA whose rows are channels: a state's accumulators are, as they lie,
//      the operand of the next chunk's first product, so the state never leaves the registers.  Four other warps work a chunk ahead:
//      they fetch (cp.async, three buffers) and make what does not depend on the state, M x + D x.
// An MMA rounds the sum it adds to towards zero: the high parts' products therefore start from zero and are added by FMA units, which
// round to nearest; decays and step sizes come from 64-bit functions.  Bound by the chain along a row (64 heads fill 128 blocks, one an SM).  One row of 2,048 tokens, 64 heads of 64 x 128:
// chunks 16 us and walk 137 us; the 32-bit kernels, in chunks of 32, 27 and 310 us.  Errors against 64 bits (2-norm, 200 to 1,500 tokens) of
// outputs and states, in units of 1e-8: decays near one 10 to 13 and 9 to 13 here, 25 to 62 and 25 to 74 in the 32-bit kernels; mixed decays 9.4
// to 10.1 and 6.0 to 7.6 here, 7.8 to 10.0 and 4.8 to 11.6 there; strong ones 6.7 to 8.2 and 3.7 to 4.9 here, 6.6 to 8.3 and 4.4 to 4.7 there.
// An infinite state entry stays in its channel; an infinite C, B or x meets zero parts of the other operand and may give a NaN.
#include "common.cuh"
#include "mma_helpers.cuh"
#include "split_bf16.cuh"

namespace {
constexpr int TC = 64;                  // tokens of a chunk
constexpr int PS = 32;                  // channels of a block of the walk
constexpr int THREADS = 128;
constexpr int XLD = PS + 8;             // padded rows: neighbours begin 16 bytes apart modulo a bank's round
constexpr int FLD = TC + 8;             // (of floats: eight rows' pairs meet no bank twice)
constexpr int YLD = PS + 8;
constexpr int WALK_THREADS = 256;
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

template <int N>
struct Walk {
  static constexpr int LD = N + 8;
  static constexpr int STAGE = (2 * TC * LD + TC * XLD) * 2 + (TC * FLD + HEAD_FLOATS) * 4;      // bytes: C, B, x, then floats
  static constexpr int SMEM = 3 * STAGE + 2 * TC * YLD * 4 + 4 * 2 * 2 * 32 * 16;
};

// grid (P / 32, rows * H)
template <int N>
__global__ void __launch_bounds__(WALK_THREADS)
ssd_walk_mma_kernel(const __nv_bfloat16* __restrict__ xbc, int stride, const float* __restrict__ scores, const float* __restrict__ heads,
                    const float* __restrict__ D, float* __restrict__ state, float* __restrict__ out, const int* __restrict__ row_slot,
                    const int* __restrict__ row_q_start, const int* __restrict__ row_q_len, const int* __restrict__ chunk_base, int H, int G, int P) {
  constexpr int LD = Walk<N>::LD, STAGE = Walk<N>::STAGE, NH = N / 2, NT = NH / 8;
  extern __shared__ __align__(16) unsigned char smem[];
  const int row = blockIdx.y / H, h = blockIdx.y % H, p0 = blockIdx.x * PS, n_new = row_q_len[row];
  if (n_new <= 0) return;
  const int g = h / (H / G), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q0 = row_q_start[row];
  const int lg = lane >> 2, lt = lane & 3;
  float* intra = reinterpret_cast<float*>(smem + 3 * STAGE);       // [2][TC][YLD]: M x + D x
  float4* swap = reinterpret_cast<float4*>(intra + 2 * TC * YLD);  // [4 warps][2 row tiles][2][32]
  const int chunks = (n_new + TC - 1) / TC;
  const size_t first = chunk_base[row];
  const float Dh = D[h];

  if (warp >= 4) {      // a chunk ahead of the others
    const int pt = tid - 128, m = warp - 4;
    auto fetch = [&](int c) {
      if (c < chunks) {
        const int n = min(TC, n_new - c * TC);
        __nv_bfloat16* to = reinterpret_cast<__nv_bfloat16*>(smem + (c % 3) * STAGE);
        const __nv_bfloat16* from = xbc + (size_t)(q0 + c * TC) * stride;
        for (int v = pt; v < 2 * TC * (N / 8); v += 128) {
          const int r = v / (N / 8), i = v % (N / 8) * 8, t = r % TC, which = r / TC;
          cp_async_16(smem_u32(to + r * LD + i), from + (size_t)(t < n ? t : 0) * stride + (size_t)H * P + (size_t)(which ? g : G + g) * N + i, t < n);
        }
        for (int v = pt; v < TC * (PS / 8); v += 128) {
          const int t = v / (PS / 8), i = v % (PS / 8) * 8;
          cp_async_16(smem_u32(to + 2 * TC * LD + t * XLD + i), from + (size_t)(t < n ? t : 0) * stride + (size_t)h * P + p0 + i, t < n);
        }
        float* fl = reinterpret_cast<float*>(to + 2 * TC * LD + TC * XLD);
        const float* sc = scores + ((first + c) * G + g) * GROUP_FLOATS;
        const float* hs = heads + ((first + c) * H + h) * HEAD_FLOATS;
        for (int v = pt; v < GROUP_FLOATS / 4; v += 128) {
          const int t = v / (TC / 4), i = v % (TC / 4) * 4;
          if (i <= t) cp_async_16(smem_u32(fl + t * FLD + i), sc + t * TC + i, true);      // (what lies above the diagonal is not read)
        }
        for (int v = pt; v < HEAD_FLOATS / 4; v += 128) cp_async_16(smem_u32(fl + TC * FLD + v * 4), hs + v * 4, true);
      }
      cp_async_commit();
    };
    auto prepare = [&](int c) {
      const __nv_bfloat16* X = reinterpret_cast<const __nv_bfloat16*>(smem + (c % 3) * STAGE) + 2 * TC * LD;
      const float* fs = reinterpret_cast<const float*>(X + TC * XLD);
      const float *dt = fs + TC * FLD, *hi = dt + TC, *lo = hi + TC;
      // rows m 16 .. of M, in the layout of an MMA's first operand, times x
      float zh[PS / 8][4], zl[PS / 8][4];
#pragma unroll
      for (int p = 0; p < PS / 8; ++p)
#pragma unroll
        for (int e = 0; e < 4; ++e) zh[p][e] = zl[p][e] = 0.f;
      const int ta = m * 16 + lg, tb = ta + 8;
      const float ha = hi[ta], hb = hi[tb], la = lo[ta], lb = lo[tb];
      for (int k = 0; k <= m; ++k) {
        uint32_t a[3][4], b[2][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int s = k * 16 + lt * 2 + (q >> 1) * 8, t = (q & 1) ? tb : ta;
          const float2 sh = *reinterpret_cast<const float2*>(hi + s), sl = *reinterpret_cast<const float2*>(lo + s), sd = *reinterpret_cast<const float2*>(dt + s);
          const float th = (q & 1) ? hb : ha, tl = (q & 1) ? lb : la;
          const float2 f = *reinterpret_cast<const float2*>(fs + t * FLD + s);
          const float m0 = s <= t ? f.x * exp2f((th - sh.x) + (tl - sl.x)) * sd.x : 0.f;
          const float m1 = s + 1 <= t ? f.y * exp2f((th - sh.y) + (tl - sl.y)) * sd.y : 0.f;
          split3(m0, m1, a[0][q], a[1][q], a[2][q]);
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
          ldmatrix_x4_trans(b[p][0], b[p][1], b[p][2], b[p][3], smem_u32(X + (k * 16 + (lane & 15)) * XLD + p * 16 + (lane >> 4) * 8));
#pragma unroll
        for (int p = 0; p < PS / 8; ++p) {
          const uint32_t b0 = b[p / 2][p % 2 * 2], b1 = b[p / 2][p % 2 * 2 + 1];
          mma_bf16(zl[p], a[2], b0, b1);
          mma_bf16(zl[p], a[1], b0, b1);
          mma_add(zh[p], a[0], b0, b1);
        }
      }
      float* y = intra + (c & 1) * TC * YLD;
#pragma unroll
      for (int p = 0; p < PS / 8; ++p)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int t = e ? tb : ta;
          const uint32_t x = *reinterpret_cast<const uint32_t*>(X + t * XLD + p * 8 + lt * 2);
          *reinterpret_cast<float2*>(y + t * YLD + p * 8 + lt * 2) =
              make_float2(fmaf(Dh, bf16_low(x), zh[p][2 * e] + zl[p][2 * e]), fmaf(Dh, bf16_high(x), zh[p][2 * e + 1] + zl[p][2 * e + 1]));
        }
    };
    fetch(0);
    fetch(1);
    cp_async_wait<1>();
    asm volatile("bar.sync 3, 128;" ::: "memory");
    prepare(0);
    for (int c = 0; c < chunks; ++c) {
      __syncthreads();      // chunk c is prepared; everybody has left chunk c - 1, whose buffer the next fetch takes
      fetch(c + 2);
      if (c + 1 < chunks) {
        cp_async_wait<1>();
        asm volatile("bar.sync 3, 128;" ::: "memory");
        prepare(c + 1);
      }
    }
    return;
  }

  const int half = warp & 1, ph = warp >> 1;      // half of the state entries, 16 of the channels
  float* st = state + (((size_t)row_slot[row] * H + h) * P + p0 + ph * 16) * N + half * NH;
  float S[NT][4];      // rows: channels lg and lg + 8, columns: two state entries of each eight
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float2 v = *reinterpret_cast<const float2*>(st + (size_t)(lg + 8 * e) * N + j * 8 + lt * 2);
      S[j][2 * e] = v.x;
      S[j][2 * e + 1] = v.y;
    }
  for (int c = 0; c < chunks; ++c) {
    const int n = min(TC, n_new - c * TC);
    const __nv_bfloat16* Cs = reinterpret_cast<const __nv_bfloat16*>(smem + (c % 3) * STAGE);
    const __nv_bfloat16* Bs = Cs + TC * LD;
    const __nv_bfloat16* X = Bs + TC * LD;
    const float *wi = reinterpret_cast<const float*>(X + TC * XLD) + TC * FLD + 3 * TC, *wo = wi + TC, *y0 = intra + (c & 1) * TC * YLD;
    __syncthreads();      // the chunk is prepared
    // C S over this warp's half of the state entries
    float yh[4][2][4], yl[4][2][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int e = 0; e < 4; ++e) yh[m][p][e] = yl[m][p][e] = 0.f;
#pragma unroll
    for (int k = 0; k < NT / 2; ++k) {
      uint32_t b[2][2][3];      // [eight channels][eight entries][part]
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int e = 0; e < 2; ++e) split3(S[2 * k + e][2 * p], S[2 * k + e][2 * p + 1], b[p][e][0], b[p][e][1], b[p][e][2]);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        uint32_t a[4];
        ldmatrix_x4(a[0], a[1], a[2], a[3], smem_u32(Cs + (m * 16 + (lane & 15)) * LD + half * NH + k * 16 + (lane >> 4) * 8));
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          mma_bf16(yl[m][p], a, b[p][0][2], b[p][1][2]);
          mma_bf16(yl[m][p], a, b[p][0][1], b[p][1][1]);
          mma_add(yh[m][p], a, b[p][0][0], b[p][1][0]);
        }
      }
    }
    // the warp that holds the other half of the entries finishes the other two row tiles
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if ((m >> 1) != half)
#pragma unroll
        for (int p = 0; p < 2; ++p)
          swap[((warp * 2 + (m & 1)) * 2 + p) * 32 + lane] = make_float4(yh[m][p][0] + yl[m][p][0], yh[m][p][1] + yl[m][p][1],
                                                                         yh[m][p][2] + yl[m][p][2], yh[m][p][3] + yl[m][p][3]);
    asm volatile("bar.sync %0, 64;" ::"r"(1 + ph) : "memory");
#pragma unroll
    for (int m = 0; m < 4; ++m)
      if ((m >> 1) == half)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const float4 v = swap[(((warp ^ 1) * 2 + (m & 1)) * 2 + p) * 32 + lane];
          const float o[4] = {(yh[m][p][0] + yl[m][p][0]) + v.x, (yh[m][p][1] + yl[m][p][1]) + v.y, (yh[m][p][2] + yl[m][p][2]) + v.z,
                              (yh[m][p][3] + yl[m][p][3]) + v.w};
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int t = m * 16 + lg + 8 * e, ch = ph * 16 + p * 8 + lt * 2;
            if (t < n) {
              const float2 y = *reinterpret_cast<const float2*>(y0 + t * YLD + ch);
              const float w = wo[t];
              *reinterpret_cast<float2*>(out + (size_t)(q0 + c * TC + t) * H * P + (size_t)h * P + p0 + ch) =
                  make_float2(fmaf(w, o[2 * e], y.x), fmaf(w, o[2 * e + 1], y.y));
            }
          }
        }
    // the state behind the chunk
    float uh[NT][4], ul[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) uh[j][e] = ul[j][e] = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t x[4], a[3][4];      // x: (tokens 0-7, channels 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15); rows of the operand: channels
      ldmatrix_x4_trans(x[0], x[1], x[2], x[3], smem_u32(X + (k * 16 + (lane & 15)) * XLD + ph * 16 + (lane >> 4) * 8));
      const float2 w0 = *reinterpret_cast<const float2*>(wi + k * 16 + lt * 2), w1 = *reinterpret_cast<const float2*>(wi + k * 16 + lt * 2 + 8);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 w = q < 2 ? w0 : w1;
        const uint32_t xx = x[(q & 1) * 2 + (q >> 1)];
        split3(bf16_low(xx) * w.x, bf16_high(xx) * w.y, a[0][q], a[1][q], a[2][q]);
      }
#pragma unroll
      for (int j = 0; j < NT / 2; ++j) {
        uint32_t b[4];
        ldmatrix_x4_trans(b[0], b[1], b[2], b[3], smem_u32(Bs + (k * 16 + (lane & 15)) * LD + half * NH + j * 16 + (lane >> 4) * 8));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          mma_bf16(ul[2 * j + e], a[2], b[2 * e], b[2 * e + 1]);
          mma_bf16(ul[2 * j + e], a[1], b[2 * e], b[2 * e + 1]);
          mma_add(uh[2 * j + e], a[0], b[2 * e], b[2 * e + 1]);
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
}  // namespace

extern "C" int dk_state_space_mma_chunk() { return TC; }

// States of 64 or 128 entries a channel, channels in slices of 32, rows that begin on 16-byte boundaries.
extern "C" int dk_state_space_mma_supported(int N, int P, int stride) { return (N == 64 || N == 128) && P > 0 && P % PS == 0 && stride % 8 == 0; }

// Floats of working memory per chunk.
extern "C" int dk_state_space_mma_floats(int H, int G) { return G * GROUP_FLOATS + H * HEAD_FLOATS; }

// Arguments as for dk_state_space_chunked, with chunks of dk_state_space_mma_chunk() tokens; xbc and dtraw are bfloat16.
extern "C" int dk_state_space_mma(const void* xbc, int stride, const void* dtraw, int dt_stride, const float* A_log, const float* dt_bias,
                                  const float* D, float* state, float* out, float* work, const int* row_slot, const int* row_q_start,
                                  const int* row_q_len, const int* chunk_base, int rows, int total_chunks, int max_chunks, int H, int G, int N,
                                  int P, cudaStream_t stream) {
  if (rows == 0 || max_chunks == 0) return 0;
  DK_REQUIRE(rows > 0 && H > 0 && G > 0 && H % G == 0 && dk_state_space_mma_supported(N, P, stride), "state_space_mma: H=%d G=%d N=%d P=%d stride=%d are not taken",
             H, G, N, P, stride);
  DK_REQUIRE((long long)rows * H <= 65535, "state_space_mma: %d rows of %d heads are above the grid's limit", rows, H);
  DK_REQUIRE(max_chunks > 0 && total_chunks >= max_chunks, "state_space_mma: %d chunks in all, %d in a row", total_chunks, max_chunks);
  DK_REQUIRE(stride >= H * P + 2 * G * N, "state_space_mma: rows of %d elements do not hold x, B and C", stride);
  DK_REQUIRE(((uintptr_t)xbc | (uintptr_t)work) % 16 == 0 && ((uintptr_t)state | (uintptr_t)out) % 8 == 0, "state_space_mma: a tensor begins off its boundary");
  float* heads = work + (size_t)total_chunks * G * GROUP_FLOATS;
  const auto *x = (const __nv_bfloat16*)xbc, *d = (const __nv_bfloat16*)dtraw;
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
    ssd_walk_mma_kernel<NN><<<dim3(P / PS, rows * H), WALK_THREADS, Walk<NN>::SMEM, stream>>>(x, stride, work, heads, D, state, out, row_slot, row_q_start, \
                                                                                         row_q_len, chunk_base, H, G, P);                      \
  } while (0)
  if (N == 128) RUN(128);
  else RUN(64);
#undef RUN
  return dk_check_launch("state_space_mma");
}
