// Paged attention over a cache of rows (row_attention_params.h) whose value is the front part of its key, with keys of up to 320 and
// values of up to 256 entries: latent attention over portions of prompts, on tcgen05, bfloat16, causal, optionally a window or chunks, a
// sink and a gate per head.
//
// A block owns 128 queries of one head.  Keys come by TMA in tiles of 64 cached rows, once: the value's columns of the same tile are
// the operand of the second product, read with the contracted dimension along the rows.  Tensor memory holds two tiles' scores
// (64 columns each) that take turns, and one accumulator of 256 columns.  The softmax weights keep 16 bits of mantissa, P = P_hi + P_lo,
// two products a tile; P takes the place of the scores it was made from and is the A operand from there.
//
//   warps 0-3   softmax: thread r owns query r, which is lane r of the tensor memory
//   warp 4      producer of queries and keys (three stages)
//   warp 5      issues the score products, warp 6 the products with the values
//
// While the softmax threads work on one tile, the tensor cores make the next one's scores and the products of the one before; a block
// takes pieces (128 queries of a head) forwards and backwards in turn, from long to short, so that all blocks end together.
// Bound by the tensor cores' reads of shared memory: a tile's scores take 20 products of 64 keys (6 KB read for 32 cycles of work), its values 8 of
// 256 columns.  One prompt of 2,048 tokens, 16 heads, keys of 320 and values of 256: 60 us; warp-level MMA (attention_rows_mma.cu)
// 275 us.
//
// Every wait is bounded; when one gives up the block records it, stores nothing more, waits (bounded again) for the copies and products that it
// has under way, frees its tensor memory and returns.
#include "common.cuh"
#include "row_attention_params.h"
#include "tcgen05_helpers.cuh"
#include "attention_pieces.cuh"
#include "ring.cuh"

namespace {
constexpr int QT = 128, KT = 64, DKP = 320, DVP = 256;
constexpr int BOXES = DKP / 64;
constexpr int THREADS = 256;
constexpr int STAGES = 3;
constexpr int Q_BOX = QT * 128, K_BOX = KT * 128;      // bytes of a box of 64 columns
constexpr int OFF_K = BOXES * Q_BOX, STAGE = BOXES * K_BOX, SMEM = OFF_K + STAGES * STAGE + 1024;
constexpr int COL_S = 0, COL_O = 2 * KT, TMEM_COLS = 512;
constexpr float RESCALE_STEP = 8.f;      // in powers of two
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

struct Piece {
  int row, h, nq, t0, pos0, first_key, last_key, kt_first, n_tiles, first_page, last_page;
};

constexpr int LISTED = 256;      // pairs of row and query tile that the list holds

// Pieces are numbered with the head fastest, then as the block's list has them (attention_pieces.cuh); without a list by the rows, then a row's
// query tiles from its latest (which has the most keys) on.
__device__ __forceinline__ bool piece_of(const DkRowAttnParams& p, int index, const uint32_t* list, int listed, Piece& w) {
  w.h = index % p.H;
  w.row = listed >= 0 ? (list[index / p.H] >> 9) & 511 : (index / p.H) % p.rows;
  const int q_len = p.row_q_len[w.row], qt = listed >= 0 ? (int)(list[index / p.H] & 511) : (q_len + QT - 1) / QT - 1 - index / (p.H * p.rows);
  if (qt < 0 || (p.row_filter == 2 && q_len == 1)) return false;
  w.nq = min(QT, q_len - qt * QT);
  w.t0 = p.row_q_start[w.row] + qt * QT;
  w.pos0 = p.row_pos_start[w.row] + qt * QT;
  w.first_key = row_first_key(p, w.pos0);
  w.last_key = w.pos0 + w.nq - 1;
  w.kt_first = w.first_key / KT;
  w.n_tiles = w.last_key / KT - w.kt_first + 1;
  w.first_page = w.first_key / p.ps;
  w.last_page = w.last_key / p.ps;
  return true;
}

// Barriers.  Tiles are numbered through all of a block's pieces; tile g has stage g % 3 and scores g % 2.
struct Bars {
  unsigned long long q_full, q_empty, k_edge, k_full[STAGES], k_empty[STAGES], s_full[2], p_full[2], o_done[2];
};

__global__ void __launch_bounds__(THREADS, 1)
attention_rows_wide_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           const __grid_constant__ CUtensorMap map_k_run, const DkRowAttnParams p, const int n_qt) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) Bars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int failed;
  __shared__ PieceList<LISTED> pieces;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t q_full = s2u(&bars.q_full), q_empty = s2u(&bars.q_empty), k_edge = s2u(&bars.k_edge), k_full = s2u(bars.k_full), k_empty = s2u(bars.k_empty),
                 s_full = s2u(bars.s_full), p_full = s2u(bars.p_full), o_done = s2u(bars.o_done);
  if (tid == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    mbar_init(k_edge, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(k_full + 8 * s, 1);
      mbar_init(k_empty + 8 * s, 1);
    }
    for (int c = 0; c < 2; ++c) {
      mbar_init(s_full + 8 * c, 1);
      mbar_init(p_full + 8 * c, QT);
      mbar_init(o_done + 8 * c, 1);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  const int listed = list_pieces<LISTED>(pieces, p.row_q_len, p.rows, p.row_filter == 2, QT, [&](int row, int qt) {
    const int pos0 = p.row_pos_start[row] + qt * QT, last = p.row_pos_start[row] + min(p.row_q_len[row], (qt + 1) * QT) - 1;
    return last / KT - row_first_key(p, pos0) / KT + 1;
  });
  const int n_pieces = p.H * (listed >= 0 ? listed : n_qt * p.rows);
  if (warp == 5) tmem_alloc(s2u(&tmem_slot), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot, sm_q = s2u(smem), sm_k = s2u(smem + OFF_K);
  auto piece_index = [&](int round) {
    const int b = (round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x;
    return round * (int)gridDim.x + b;
  };
  auto together = [&](bool ok) { return __all_sync(0xffffffffu, ok && failed == 0) != 0; };      // the same answer in every lane
  int g = 0, done = 0;      // tiles and pieces before the current ones
  Piece w;

  if (warp == 4) {
    const int ppt = KT / p.ps;      // pages of a tile
    int q_asked = 0, edges = 0;
    for (int round = 0; round * (int)gridDim.x < n_pieces; ++round) {
      const int index = piece_index(round);
      if (index >= n_pieces || !piece_of(p, index, pieces.sorted, listed, w)) continue;
      if (!together(done == 0 || mbar_wait(q_empty, (done - 1) & 1))) { failed = 1; break; }
      if (lane == 0) {
        mbar_expect_tx(q_full, BOXES * Q_BOX);
        for (int i = 0; i < BOXES; ++i)      // (columns behind the head's last one are zeros)
          tma_load_4d(sm_q + i * Q_BOX, &map_q, i * 64, w.h, 0, w.t0, q_full);
      }
      ++q_asked;
      const int kvh = w.h / (p.H / p.KV);
      for (int j = 0; j < w.n_tiles; ++j, ++g) {
        const int s = g % STAGES, lp = (w.kt_first + j) * ppt + lane;
        int page = -1;
        if (lane < ppt && lp >= w.first_page && lp <= w.last_page && lp < p.max_pages) {
          page = p.block_table[(size_t)w.row * p.max_pages + lp];
          if (page < 0 || page >= p.num_pages) {
            dk_report(p.err, DK_DEV_BAD_PAGE, w.row, lp, page);
            page = -1;
          }
        }
        const int first = __shfl_sync(0xffffffffu, page, 0);
        const bool run = __all_sync(0xffffffffu, lane >= ppt || (page >= 0 && page == first + lane));
        const uint32_t there = __ballot_sync(0xffffffffu, page >= 0);
        const int other = there != 0 ? __shfl_sync(0xffffffffu, page, __ffs(there) - 1) : 0;
        if (page < 0) page = other;      // what no query of the piece sees: cleared and masked below
        if (!together(g < STAGES || mbar_wait(k_empty + 8 * s, (g / STAGES - 1) & 1))) { failed = 1; break; }
        // a tile with keys at its ends that nobody sees is announced when they are cleared
        const int from = j == 0 ? w.first_key % KT : 0, to = j == w.n_tiles - 1 ? w.last_key % KT + 1 : KT;
        const bool edge = from > 0 || to < KT;
        const uint32_t bar = edge ? k_edge : k_full + 8 * s, dst = sm_k + s * STAGE;
        if (lane == 0) mbar_expect_tx(bar, STAGE);
        __syncwarp();
        if (run) {
          if (lane == 0)
            for (int i = 0; i < BOXES; ++i) tma_load_4d(dst + i * K_BOX, &map_k_run, i * 64, 0, kvh, first, bar);
        } else if (lane < ppt) {
          for (int i = 0; i < BOXES; ++i) tma_load_2d(dst + i * K_BOX + lane * p.ps * 128, &map_k, i * 64, (page * p.KV + kvh) * p.ps, bar);
        }
        if (edge) {
          if (!together(mbar_wait(k_edge, edges++ & 1))) { failed = 1; break; }
          clear_rows(dst, BOXES, K_BOX, 0, from);
          clear_rows(dst, BOXES, K_BOX, to, KT);
          if (lane == 0) mbar_arrive(k_full + 8 * s);
        }
      }
      if (failed) break;
      ++done;
    }
    if (lane == 0) {      // its copies have arrived
      ring_drain(q_asked, 1, [&](int, uint32_t parity) { return mbar_wait(q_full, parity); });
      ring_drain(edges, 1, [&](int, uint32_t parity) { return mbar_wait(k_edge, parity); });
      ring_drain(g, STAGES, [&](int s, uint32_t parity) { return mbar_wait(k_full + 8 * s, parity); });
    }
    __syncwarp();
  } else if (warp == 5) {
    const bool leader = elect_one();
    const uint32_t idesc = instr_desc_bf16(QT, KT);
    const uint64_t dq = smem_desc_k_major(sm_q);
    bool ok = true;
    for (int round = 0; ok && round * (int)gridDim.x < n_pieces; ++round) {
      const int index = piece_index(round);
      if (index >= n_pieces || !piece_of(p, index, pieces.sorted, listed, w)) continue;
      ok = together(mbar_wait(q_full, done & 1));
      for (int j = 0; ok && j < w.n_tiles; ++j, ++g) {
        const int s = g % STAGES, c = g & 1;
        ok = together((g < 2 || mbar_wait(o_done + 8 * c, ((g >> 1) - 1) & 1)) && mbar_wait(k_full + 8 * s, (g / STAGES) & 1));
        if (!ok) break;
        tc_fence_after();
        const uint64_t dk = smem_desc_k_major(sm_k + s * STAGE);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < DKP / 16; ++kk)
            umma(tmem + COL_S + c * KT, dq + (uint64_t)(((kk / 4) * Q_BOX + (kk % 4) * 32) >> 4), dk + (uint64_t)(((kk / 4) * K_BOX + (kk % 4) * 32) >> 4),
                 idesc, kk > 0 ? 1u : 0u);
          umma_commit(s_full + 8 * c);
          if (j == w.n_tiles - 1) umma_commit(q_empty);
        }
        __syncwarp();
      }
      ++done;
    }
    if (!ok) failed = 1;
    if (lane == 0) ring_drain(g, 2, [&](int c, uint32_t parity) { return mbar_wait(s_full + 8 * c, parity); });      // its products are complete
    __syncwarp();
  } else if (warp == 6) {
    const bool leader = elect_one();
    const uint32_t idesc = instr_desc_bf16(QT, DVP, true);
    bool ok = true;
    for (int round = 0; ok && round * (int)gridDim.x < n_pieces; ++round) {
      const int index = piece_index(round);
      if (index >= n_pieces || !piece_of(p, index, pieces.sorted, listed, w)) continue;
      for (int j = 0; j < w.n_tiles; ++j, ++g) {
        const int s = g % STAGES, c = g & 1;
        ok = together(mbar_wait(k_full + 8 * s, (g / STAGES) & 1) && mbar_wait(p_full + 8 * c, (g >> 1) & 1));
        if (!ok) break;
        tc_fence_after();
        const uint32_t tp = tmem + COL_S + c * KT;      // P_hi, then P_lo: 8 columns for 16 keys
        const uint64_t dv = smem_desc_mn_major(sm_k + s * STAGE, K_BOX);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < KT / 16; ++kk) {      // 16 keys further: two groups of 8 rows
            const uint64_t d = dv + (uint64_t)(kk * (2048 >> 4));
            umma_a_tmem(tmem + COL_O, tp + kk * 8, d, idesc, (j > 0 || kk > 0) ? 1u : 0u);
            umma_a_tmem(tmem + COL_O, tp + KT / 2 + kk * 8, d, idesc, 1u);
          }
          umma_commit(k_empty + 8 * s);
          umma_commit(o_done + 8 * c);
        }
        __syncwarp();
      }
    }
    if (!ok) failed = 1;
    if (lane == 0) ring_drain(g, 2, [&](int c, uint32_t parity) { return mbar_wait(o_done + 8 * c, parity); });
    __syncwarp();
  } else if (warp < 4) {
    const int r = tid;      // query = lane of the tensor memory
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16, t_o = tmem + lane_base + COL_O;
    const float sl2 = p.scale * LOG2E;
    bool good = true;
#pragma unroll 1
    for (int round = 0; good && round * (int)gridDim.x < n_pieces; ++round) {
      const int index = piece_index(round);
      if (index >= n_pieces || !piece_of(p, index, pieces.sorted, listed, w)) continue;
      const int qpos = w.pos0 + r, last_pos = w.pos0 + w.nq - 1;
      const int q_first = row_first_key(p, qpos), last_first = row_first_key(p, last_pos);      // the first keys this and the last query see
      float m_used = -INFINITY, l_sum = 0.f;
#pragma unroll 1
      for (int j = 0; j < w.n_tiles; ++j, ++g) {
        const int c = g & 1, kbase = (w.kt_first + j) * KT;
        const uint32_t t_s = tmem + lane_base + COL_S + c * KT;
        if (!together(mbar_wait(s_full + 8 * c, (g >> 1) & 1))) { failed = 1; good = false; break; }
        tc_fence_after();
        float v[KT];
        tmem_ld32_nowait(t_s, v);
        tmem_ld32_nowait(t_s + 32, v + 32);
        tmem_wait_ld();
        if (kbase + KT - 1 > w.pos0 || kbase < last_first) {
          const int hi = qpos - kbase, lo = q_first - kbase;
#pragma unroll
          for (int i = 0; i < KT; ++i)
            if (!(i <= hi && i >= lo)) v[i] = -INFINITY;
        }
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < KT; i += 4) {
          mx4[0] = fmaxf(mx4[0], v[i]);
          mx4[1] = fmaxf(mx4[1], v[i + 1]);
          mx4[2] = fmaxf(mx4[2], v[i + 2]);
          mx4[3] = fmaxf(mx4[3], v[i + 3]);
        }
        const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2);
        const bool grow = m_new > m_used + RESCALE_STEP;      // also the first finite maximum of a row
        float factor = 1.f;
        if (grow) {
          factor = m_used == -INFINITY ? 0.f : fast_exp2(m_used - m_new);
          m_used = m_new;
        }
        const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
        float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int b = 0; b < KT / 32; ++b) {
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float e0 = fast_exp2(fmaf(v[b * 32 + 2 * i], sl2, neg_m)), e1 = fast_exp2(fmaf(v[b * 32 + 2 * i + 1], sl2, neg_m));
            sum4[(2 * i) & 3] += e0;
            sum4[(2 * i + 1) & 3] += e1;
            const __nv_bfloat162 h2 = __floats2bfloat162_rn(e0, e1);
            hi[i] = *reinterpret_cast<const uint32_t*>(&h2);
            lo[i] = pack2(e0 - __low2float(h2), e1 - __high2float(h2));
          }
          tmem_st16(t_s + b * 16, hi);
          tmem_st16(t_s + KT / 2 + b * 16, lo);
        }
        l_sum = l_sum * factor + ((sum4[0] + sum4[1]) + (sum4[2] + sum4[3]));
        if (j > 0 && __any_sync(0xffffffffu, grow)) {      // the accumulator at rest: the tile before is in it, this one waits for P
          if (!together(mbar_wait(o_done + 8 * (c ^ 1), ((g - 1) >> 1) & 1))) { failed = 1; good = false; break; }
          tc_fence_after();
#pragma unroll 1
          for (int b = 0; b < DVP / 32; ++b) {
            float o[32];
            tmem_ld32_nowait(t_o + b * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= factor;
            tmem_st32(t_o + b * 32, o);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(p_full + 8 * c);
      }
      if (!good) break;
      // the last tile's products are in the accumulator
      if (!together(mbar_wait(o_done + 8 * ((g - 1) & 1), ((g - 1) >> 1) & 1))) { failed = 1; break; }
      tc_fence_after();
      const float sink2 = p.sink != nullptr ? p.sink[w.h] * LOG2E : -INFINITY;      // the sink: a key with this logit and no value
      const float m_all = fmaxf(m_used, sink2);
      const float f = m_used == -INFINITY ? 0.f : fast_exp2(m_used - m_all);
      float l_all = l_sum * f;
      if (p.sink != nullptr) l_all += fast_exp2(sink2 - m_all);
      const float scale = l_all > 0.f ? f * (r < w.nq ? row_head_gate<__nv_bfloat16>(p, w.t0 + r, w.h) : 1.f) / l_all : 0.f;
      __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.out) + ((size_t)(w.t0 + r) * p.H + w.h) * p.dv;
#pragma unroll 1
      for (int b = 0; b < DVP / 32; ++b) {
        float o[32];
        tmem_ld32_nowait(t_o + b * 32, o);
        tmem_wait_ld();
        if (r < w.nq) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 st;
            st.x = pack2(o[q * 8] * scale, o[q * 8 + 1] * scale);
            st.y = pack2(o[q * 8 + 2] * scale, o[q * 8 + 3] * scale);
            st.z = pack2(o[q * 8 + 4] * scale, o[q * 8 + 5] * scale);
            st.w = pack2(o[q * 8 + 6] * scale, o[q * 8 + 7] * scale);
            if (b * 32 + q * 8 < p.dv) *reinterpret_cast<uint4*>(orow + b * 32 + q * 8) = st;      // (value sizes are multiples of 8)
          }
        }
        __syncwarp();
      }
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (failed && tid == 0) dk_report(p.err, DK_DEV_TIMEOUT, (int)blockIdx.x, (int)gridDim.x, n_pieces);
  if (warp == 5) tmem_dealloc(tmem, TMEM_COLS);
}
}  // namespace

// Values that are the front part of their keys, sizes above what attention_rows_tc.cu takes.
extern "C" int dk_attention_rows_wide_supported(const DkRowAttnParams* pp) {
  const DkRowAttnParams& p = *pp;
  if (p.dtype != DK_BF16 || p.KV <= 0 || p.H % p.KV != 0) return 0;
  if (p.k_off != p.v_off || p.dv > p.dk || p.dk % 8 || p.dv % 8 || p.dk <= 128 || p.dk > DKP || p.dv < 64 || p.dv > DVP) return 0;
  if (p.row_width % 8 || p.k_off % 8 || p.q_stride % 8 || p.q_head_stride % 8) return 0;
  if (p.ps != 8 && p.ps != 16 && p.ps != 32 && p.ps != 64) return 0;
  if (p.softcap > 0.f || p.dist_bias != nullptr || !(p.scale > 0.f)) return 0;
  return (((uintptr_t)p.q | (uintptr_t)p.cache | (uintptr_t)p.out) % 16) == 0;
}

// max_q_len: the most tokens any row brings.
extern "C" int dk_attention_rows_wide(const DkRowAttnParams* pp, int max_q_len, cudaStream_t stream) {
  const DkRowAttnParams& p = *pp;
  if (p.T == 0 || p.rows == 0) return 0;
  DK_REQUIRE(dk_attention_rows_wide_supported(pp), "attention_rows_wide: sizes not taken: dk=%d dv=%d width=%d offsets %d %d ps=%d", p.dk, p.dv, p.row_width,
             p.k_off, p.v_off, p.ps);
  DK_REQUIRE(max_q_len >= 1 && p.window >= 0 && p.chunk >= 0, "attention_rows_wide: bad sizes max_q_len=%d window=%d chunk=%d", max_q_len, p.window, p.chunk);
  DK_REQUIRE(p.gate == nullptr || p.gate_stride >= p.H, "attention_rows_wide: rows of %d gates do not hold %d heads", p.gate_stride, p.H);
  DK_REQUIRE(p.row_q_start && p.row_q_len && p.row_pos_start && p.block_table, "attention_rows_wide: row tables are missing");
  const long long rows = (long long)p.num_pages * p.KV * p.ps, pieces = (long long)p.H * ((max_q_len + QT - 1) / QT) * p.rows;
  DK_REQUIRE(rows < (1ll << 31) && pieces < (1ll << 30), "attention_rows_wide: %lld cached rows or %lld pieces are too many", rows, pieces);
  CUtensorMap map_q, map_k, map_k_run;
  const unsigned long long strides[3] = {(unsigned long long)p.row_width * 2, (unsigned long long)p.ps * p.row_width * 2,
                                         (unsigned long long)p.KV * p.ps * p.row_width * 2};
  const unsigned long long dims[4] = {(unsigned long long)p.dk, (unsigned long long)p.ps, (unsigned long long)p.KV, (unsigned long long)p.num_pages};
  const __nv_bfloat16* base = reinterpret_cast<const __nv_bfloat16*>(p.cache) + p.k_off;
  DK_REQUIRE(make_tensor_map_of_heads(&map_q, p.q, p.T, p.H, p.dk, p.q_stride, p.q_head_stride, QT) &&
                 make_tensor_map_bf16(&map_k, base, rows, p.dk, p.row_width, p.ps) &&
                 make_tensor_map_bf16_4d(&map_k_run, base, dims, strides, p.ps, KT / p.ps),
             "attention_rows_wide: cannot encode a tensor map");
  static bool granted[DK_MAX_DEVICES] = {false};
  bool& ok = granted[dk_current_device()];
  if (!ok) {
    DK_REQUIRE(cudaFuncSetAttribute(attention_rows_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) == cudaSuccess,
               "attention_rows_wide: %d bytes of shared memory were refused", SMEM);
    ok = true;
  }
  const int sms = dk_sm_count();
  attention_rows_wide_kernel<<<(int)(pieces < sms ? pieces : sms), THREADS, SMEM, stream>>>(map_q, map_k, map_k_run, p, (max_q_len + QT - 1) / QT);
  return dk_check_launch("attention_rows_wide");
}
