// Causal attention of prompt portions over a latent cache with the latents expanded, on the 5th-generation tensor cores
// (tcgen05 + TMEM + TMA), bfloat16.  A portion of many tokens behind a history pays for making every key's per-head keys and
// values once ([keys, R] x [R, H (D + V)], one product) and then attends with keys of D + P and values of V elements,
// where the absorbed form (attention_latent.cu) scores R + P and sums R elements per pair: 320 against 1088 at D = V =
// 128, P = 64, R = 512.  Single tokens stay with the absorbed form, which reads nothing but the cache.
//
//   latent_rows        the latents of the portions' requests out of their pages: [key][c (R) | rotated part (P)], request
//                      after request, only those that bring more than one token, with a window from its first visible key
//                      on; every request filled up with zero rows to whole key tiles, so that no tile holds another request's
//                      rows (a masked key still meets 0 * V), and zeros behind the last up to the caller's bound
//   latent_q_turn      the last P elements of every head of q, rotated in place
//   attention_latent_umma
//       S = [q_h | q_rot] [k_h | k_rot]^T, softmax, O += P V with k_h, v_h from the expanded rows [key][h][k (D) | v (V)]
//       and k_rot from the gathered latents (the same for all heads).
//
// The attention kernel's scheme is that of attention_umma.cu at one query head per key head: a CTA owns 2 x 128 tokens of
// one (request, head), key tiles of 128, two threads per row in the softmax, P back into tensor memory over S, one
// MMA thread that serves the two row tiles in turn, lazy rescale of O.  What differs: the rows of a tile are contiguous, so
// a stage is three (two) boxes; the 64-wide rotated part is a third part of Q and K (a narrower one is filled up with
// zeros by TMA, beyond the row's end); shared memory holds Q (96 KB), two stages of K (96 KB) and one of V (32 KB) at
// D = 128, so its small arrays share a row.
// Bounded waits; status codes 31-36, and 37 for a step whose portions pass the bounds of its launch (rows, row-tile pairs).
#include <cuda.h>

#include "common.cuh"
#include "umma_attention.cuh"

using namespace dinfer;
using namespace dinfer_umma;

namespace {

constexpr int BM = 128, BN = 128, NTHREADS = 608;              // rows per row tile (two per CTA), keys per tile
constexpr int MIN_SHARED = 6, LONG_WALK = 16;                  // key tiles of a pair that two CTAs share; of a long one
constexpr int V_WARP = 18;
constexpr uint32_t PART = BM * 128;                            // bytes of a 128 x 64 part of a tile

struct Params {
  __nv_bfloat16* out; int64_t ldo;
  const int* cu_seqlens; const int* seq_lens;
  int B, window, rows;
  float scale_log2;
  const float* sinks;
  int* status;
};

// What request i of the batch contributes: its row-tile pairs, its rows in the gathered latents and the keys in front of them.
struct Share { int pairs, keys, rows, skip; };
__device__ __forceinline__ Share share_of(const int* cu, const int* seq, int i, int window) {
  const int q = cu[i + 1] - cu[i];
  if (q <= 1) return {0, 0, 0, 0};
  const int skip = window > 0 ? max(0, seq[i] - q - window + 1) : 0;
  const int keys = seq[i] - skip;
  return {(q + 2 * BM - 1) / (2 * BM), keys, (keys + BN - 1) / BN * BN, skip};
}
__device__ __forceinline__ int warp_inclusive(int v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}

template <int D> struct Shape {
  static constexpr int NH = D / 64;                            // 64-wide parts of a head
  static constexpr int K_STAGES = 2, V_STAGES = D == 128 ? 1 : 2;
  static constexpr uint32_t Q_BYTES = (NH + 1) * PART, K_BYTES = (NH + 1) * PART, V_BYTES = NH * PART;
  static constexpr uint32_t TILES = 2 * Q_BYTES + K_STAGES * K_BYTES + V_STAGES * V_BYTES;
  static constexpr uint32_t SMEM = TILES + 2 * 2 * BM * 4 + 256;   // + row maxima (later sums) by halves, barriers
  static_assert(SMEM <= 227 * 1024, "fits a CTA");
};

// SPLIT: a cluster of two CTAs to a row-tile pair, half of its keys each where it has MIN_SHARED key tiles or more (else the
// second has nothing to do).  Each then writes out one of the two row tiles and sends what it has of the other (unnormalised
// sums, reference maximum, sum of exponentials) through distributed shared memory, where Q lay, behind two cluster barriers.  A
// prompt's last pair walks all its key tiles, its first one two: 2048 tokens of 16 heads are 128 CTAs whose longest takes 16 tiles
// of 2.85 us where the mean is 8.5.
template <int D, bool SPLIT>
__global__ void __maxnreg__(96)
attention_latent_umma_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv,
                             const __grid_constant__ CUtensorMap map_r, const Params p) {
  using S = Shape<D>;
  constexpr int NH = S::NH, KS = S::K_STAGES, VS = S::V_STAGES;
  constexpr int TMEM_COLS = 512, O_COL = 256;
  extern __shared__ __align__(1024) unsigned char smem[];
  float (*s_max)[2][BM] = reinterpret_cast<float (*)[2][BM]>(smem + S::TILES);     // [row tile][half of the keys][row]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::TILES + 2 * 2 * BM * 4);
  uint64_t *q_full = bars, *k_full = bars + 1, *k_empty = k_full + 2, *v_full = k_empty + 2, *v_empty = v_full + 2,
           *s_full = v_empty + 2, *p_full = s_full + 2, *o_full = p_full + 2;      // 15 barriers
  volatile uint32_t* s_tmem_base = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* s_abort = reinterpret_cast<int*>(bars + 17);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = SPLIT ? blockIdx.x >> 1 : blockIdx.x, rank = SPLIT ? blockIdx.x & 1 : 0;
  pdl_wait();
  // which request's pair this is, and where its keys begin: every warp adds the requests up for itself (the last block's all of
  // them: a captured graph may be replayed on any lengths, and pairs beyond the grid would go unnoticed)
  int b = -1, pair = 0, pairs_b = 0, key0 = 0, key_end = 0;
  {
    const int y = blockIdx.y;
    const bool all = y == (int)gridDim.y - 1 && blockIdx.x == 0;
    int before = 0, keys_before = 0;
    for (int i0 = 0; i0 < p.B; i0 += 32) {
      const int i = i0 + lane;
      const Share sh = i < p.B ? share_of(p.cu_seqlens, p.seq_lens, i, p.window) : Share{0, 0, 0, 0};
      const int incl = warp_inclusive(sh.pairs, lane), kincl = warp_inclusive(sh.rows, lane);
      const int chunk = __shfl_sync(0xffffffffu, incl, 31);
      if (b < 0 && y < before + chunk) {
        const unsigned hit = __ballot_sync(0xffffffffu, y >= before + incl - sh.pairs && y < before + incl);
        const int src = __ffs(hit) - 1;
        b = i0 + src;
        pair = y - before - __shfl_sync(0xffffffffu, incl - sh.pairs, src);
        pairs_b = __shfl_sync(0xffffffffu, sh.pairs, src);
        key0 = keys_before + __shfl_sync(0xffffffffu, kincl - sh.rows, src);
        key_end = keys_before + __shfl_sync(0xffffffffu, kincl, src);
        if (!all) break;
      }
      before += chunk;
      keys_before += __shfl_sync(0xffffffffu, kincl, 31);
    }
    if (all && before > (int)gridDim.y && threadIdx.x == 0) atomicExch(p.status, 37);
  }
  if (b < 0) return;                                           // beyond the batch's pairs
  if (key_end > p.rows) {                                      // keys that were not gathered
    if (threadIdx.x == 0) atomicExch(p.status, 37);
    return;
  }
  const int t0 = p.cu_seqlens[b];
  const int rows_total = p.cu_seqlens[b + 1] - t0;
  const int row0 = (pairs_b - 1 - pair) * 2 * BM;              // the latest rows, which see the most keys, start first
  // positions count from the request's first gathered key on
  const int hist = p.seq_lens[b] - rows_total - share_of(p.cu_seqlens, p.seq_lens, b, p.window).skip;
  const bool b_on = row0 + BM < rows_total;                    // the second row tile exists
  const int last_a = min(row0 + BM, rows_total) - 1, last = min(row0 + 2 * BM, rows_total) - 1;
  const int hi = hist + last + 1, hi_a = hist + last_a + 1;
  const int tile0 = first_key(hist + row0, p.window, 0) / BN;
  const int n_all = (hi + BN - 1) / BN - tile0;                // tiles of B (or of A when B does not exist)
  const int n_all_a = (hi_a + BN - 1) / BN - tile0;
  const bool shared = SPLIT && n_all >= MIN_SHARED;
  if (SPLIT && rank == 1 && !shared) return;
  const int per = shared ? (n_all + 1) / 2 : n_all;            // this CTA's: the first ones, or the rest
  const int tile_first = tile0 + rank * per;
  const int n_tiles = min(per, n_all - rank * per);
  const int n_tiles_a = max(0, min(per, n_all_a - rank * per));

  const uint32_t base = smem_u32(smem);
  const uint32_t sQ = base, sK = sQ + 2 * S::Q_BYTES, sV = sK + KS * S::K_BYTES;
  if (base & 1023u) {                                          // the swizzled tiles' addresses: the same for every CTA
    if (threadIdx.x == 0) atomicExch(p.status, 31);
    return;
  }
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_kv) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_r) : "memory");
    mbar_init(smem_u32(q_full), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&k_full[s]), 1); mbar_init(smem_u32(&k_empty[s]), 1);
      mbar_init(smem_u32(&v_full[s]), 1); mbar_init(smem_u32(&v_empty[s]), 1);
      mbar_init(smem_u32(&s_full[s]), 1); mbar_init(smem_u32(&p_full[s]), 256); mbar_init(smem_u32(&o_full[s]), 1);
    }
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)s_tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();                                     // (now that the tensor memory is ours)
  const uint32_t tmem = *s_tmem_base;

  if (warp == 0 || warp == V_WARP) {
    // ---- TMA producers: warp 0 brings Q (once) and the K tiles, another warp the V tiles
    if (lane == 0) {
      const bool is_k = warp == 0;
      if (is_k) {
        const uint32_t qb = smem_u32(q_full);
        mbar_expect_tx(qb, (b_on ? 2 : 1) * S::Q_BYTES);
        for (int w = 0; w < (b_on ? 2 : 1); ++w)
          for (int h = 0; h <= NH; ++h)                        // (part NH: the rotated elements, from D on)
            tma_load_3d(sQ + w * S::Q_BYTES + h * PART, &map_q, h * 64, head, t0 + row0 + w * BM, qb);
      }
      const int stages = is_k ? KS : VS;
      uint64_t *full = is_k ? k_full : v_full, *empty = is_k ? k_empty : v_empty;
      for (int j = 0; j < n_tiles; ++j) {
        const int s = j % stages;
        if (!mbar_wait(smem_u32(&empty[s]), ((j / stages) & 1) ^ 1)) { *s_abort = 1; atomicExch(p.status, 31); break; }
        const int row = key0 + (tile_first + j) * BN;
        const uint32_t bar = smem_u32(&full[s]);
        mbar_expect_tx(bar, is_k ? S::K_BYTES : S::V_BYTES);
        const uint32_t dst = is_k ? sK + s * S::K_BYTES : sV + s * S::V_BYTES;
        for (int h = 0; h < NH; ++h) tma_load_2d(dst + h * PART, &map_kv, head * 2 * D + (is_k ? 0 : D) + h * 64, row, bar);
        if (is_k) tma_load_2d(dst + NH * PART, &map_r, 0, row, bar);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---- MMA issue: one thread, the two row tiles strictly in turn (see attention_umma.cu)
      constexpr uint32_t idesc_qk = idesc_bf16(BM, BN, 0), idesc_pv = idesc_bf16(BM, D, 1);
      const uint64_t dq = desc_k_major(sQ), dk = desc_k_major(sK);
      const uint64_t dv = desc_mn_major(sV, PART);
      const int n_of[2] = {n_tiles_a, b_on ? n_tiles : 0};
      // Every 16 elements of D + 64 are multiplied, zeros behind P included, in one straight run.  (With a run-time bound on the
      // run, k < (D + P + 15) / 16, sums came out with parts missing and memory outside the block was read.  Why is not known:
      // nothing documented asks for more than one issuing thread, and the conditions on the step around these runs, here and
      // in attention_umma.cu, are borne out by every test.  The zeros cost at most four products a tile.)
      auto issue_qk = [&](int w, int t) {
        const uint64_t dqs = dq + (uint64_t)(w * (S::Q_BYTES >> 4));
        const uint64_t dks = dk + (uint64_t)((t % KS) * (S::K_BYTES >> 4));
#pragma unroll
        for (int k = 0; k < (NH + 1) * 4; ++k)
          tc_mma(tmem + w * BN, dqs + (uint64_t)(((k / 4) * PART + (k % 4) * 32) >> 4),
                 dks + (uint64_t)(((k / 4) * PART + (k % 4) * 32) >> 4), idesc_qk, k > 0 ? 1u : 0u);
        tc_commit(smem_u32(&s_full[w]));
      };
      auto issue_pv = [&](int w, int j) {
        const uint64_t dvs = dv + (uint64_t)((j % VS) * (S::V_BYTES >> 4));
        const uint32_t s_tmem = tmem + w * BN, o_tmem = tmem + O_COL + w * 128;
#pragma unroll
        for (int k = 0; k < BN / 16; ++k)
          tc_mma_ts(o_tmem, s_tmem + (k / 4) * 64 + (k % 4) * 8, dvs + (uint64_t)((k * 16 * 128) >> 4), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
      };
      bool ok = mbar_wait(smem_u32(q_full), 0) && mbar_wait(smem_u32(&k_full[0]), 0);
      if (!ok) { *s_abort = 1; atomicExch(p.status, 32); }
      if (ok) {                                                // S of the first key tile, for both row tiles
        tc_fence_after();
        for (int w = 0; w < 2; ++w)
          if (n_of[w] > 0) issue_qk(w, 0);
        tc_commit(smem_u32(&k_empty[0]));
      }
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int sv = j % VS, s1 = (j + 1) % KS;
        if (!mbar_spin(smem_u32(&v_full[sv]), (j / VS) & 1) ||
            (j + 1 < n_tiles && !mbar_spin(smem_u32(&k_full[s1]), ((j + 1) / KS) & 1))) {
          *s_abort = 1; atomicExch(p.status, 34); break;
        }
        for (int w = 0; w < 2 && ok; ++w) {
          if (j < n_of[w]) {
            if (!mbar_spin(smem_u32(&p_full[w]), j & 1)) { *s_abort = 1; atomicExch(p.status, 33); ok = false; break; }
            tc_fence_after();
            issue_pv(w, j);
            if (j + 1 == n_of[w]) tc_commit(smem_u32(&o_full[w]));
          }
          if (j + 1 < n_of[w]) issue_qk(w, j + 1);
        }
        if (!ok) break;
        tc_commit(smem_u32(&v_empty[sv]));                     // the stages go back when the products issued so far have read them
        if (j + 1 < n_tiles) tc_commit(smem_u32(&k_empty[s1]));
      }
      // the last commits arrive on the stages' barriers: the block's memory has to be there still
      if (ok && !(mbar_wait(smem_u32(&v_empty[(n_tiles - 1) % VS]), ((n_tiles - 1) / VS) & 1) &&
                  mbar_wait(smem_u32(&k_empty[(n_tiles - 1) % KS]), ((n_tiles - 1) / KS) & 1))) {
        *s_abort = 1; atomicExch(p.status, 34);
      }
    }
  } else {
    // ---- softmax and output: two threads per row, 64 keys each (see attention_umma.cu)
    const int idx = (warp - 2) >> 2;
    const int w = idx >> 1, h = idx & 1;
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const int row = row0 + w * BM + r;
    const bool row_ok = row < rows_total;
    const int pos = row_ok ? hist + row : -1;
    const int n_w = w == 0 ? n_tiles_a : (b_on ? n_tiles : 0);
    const int row_lo = row_ok ? first_key(pos, p.window, 0) : 0;
    const int lo_all = first_key(hist + (w == 0 ? last_a : last), p.window, 0);
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + w * BN, o_addr = lane_addr + O_COL + w * 128 + h * (D / 2);
    const int pair_bar = 1 + w * 4 + quarter;                  // named barrier of the two warps on these 32 rows
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_w; ++j) {
      if (ok && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&s_full[w]), j & 1))) { *s_abort = 1; atomicExch(p.status, 35); ok = false; }
      __syncwarp();
      tc_fence_after();
      const int jbase = (tile_first + j) * BN;
      const bool need_mask = (jbase + BN - 1 > hist + row0 + w * BM) || jbase < lo_all;
      float v0[32], v1[32];
      float mx = -INFINITY;
      if (ok) {
        tmem_ld32(s_addr + h * 64, v0);
        tmem_ld32(s_addr + h * 64 + 32, v1);
        tmem_ld_wait();
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int ja = jbase + h * 64 + i, jc = ja + 32;
            if (!(ja <= pos && ja >= row_lo)) v0[i] = -INFINITY;
            if (!(jc <= pos && jc >= row_lo)) v1[i] = -INFINITY;
          }
        }
        float mq[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) mq[i] = fmaxf(v0[i], v1[i]);
#pragma unroll
        for (int i = 8; i < 32; ++i) mq[i & 7] = fmaxf(mq[i & 7], fmaxf(v0[i], v1[i]));
        mx = fmaxf(fmaxf(fmaxf(mq[0], mq[1]), fmaxf(mq[2], mq[3])), fmaxf(fmaxf(mq[4], mq[5]), fmaxf(mq[6], mq[7])));
      }
      // the row's maximum is the larger of its two halves'.  One slot is enough: the next tile's S, and with it the next
      // write here, comes only after every softmax thread of the row tile has handed this tile's P over.
      s_max[w][h][r] = mx;
      asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
      if (!ok) continue;
      mx = fmaxf(mx, s_max[w][1 - h][r]) * p.scale_log2;
      const bool raise = mx > m_run + 8.f;
      if (j > 0 && __any_sync(0xffffffffu, raise)) {
        const float alpha = raise ? fast_exp2(m_run - mx) : 1.f;
        l_run *= alpha;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[16];
          tmem_ld16(o_addr + c * 16, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st16(o_addr + c * 16, o);
        }
      }
      if (raise) m_run = mx;
      const float neg_m = m_run == -INFINITY ? 0.f : -m_run;
      float sq[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) sq[i] = 0.f;
      {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float e0 = fast_exp2(fmaf(v0[i], p.scale_log2, neg_m));
          const float e1 = fast_exp2(fmaf(v0[i + 1], p.scale_log2, neg_m));
          sq[(i >> 1) & 7] += e0 + e1;
          pk[i >> 1] = pack_bf16(e0, e1);
        }
        tmem_st16(s_addr + h * 64, pk);
      }
      {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float e0 = fast_exp2(fmaf(v1[i], p.scale_log2, neg_m));
          const float e1 = fast_exp2(fmaf(v1[i + 1], p.scale_log2, neg_m));
          sq[(i >> 1) & 7] += e0 + e1;
          pk[i >> 1] = pack_bf16(e0, e1);
        }
        tmem_st16(s_addr + h * 64 + 16, pk);
      }
      l_run += ((sq[0] + sq[1]) + (sq[2] + sq[3])) + ((sq[4] + sq[5]) + (sq[6] + sq[7]));
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(smem_u32(&p_full[w]));
    }
    if (ok && n_w > 0) {
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&o_full[w]), 0))) { *s_abort = 1; atomicExch(p.status, 36); ok = false; }
      tc_fence_after();
    }
    s_max[w][h][r] = l_run;                                    // (every thread of the row tile is past its last maximum)
    asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
    const bool have = ok && n_w > 0;                           // O holds something (the same for a whole warp)
    const float l_own = have ? s_max[w][0][r] + s_max[w][1][r] : 0.f;
    const float m_own = have ? m_run : -INFINITY;
    __nv_bfloat16* dst = p.out + (int64_t)(t0 + row) * p.ldo + (int64_t)head * D + h * (D / 2);
    if (!shared) {
      if (have) {
        float l = l_own;
        if (p.sinks) l += exp2f(sink_log2(p.sinks, head) - m_run);
        const float inv = l > 0.f ? 1.f / l : 0.f;
        // all of tensor memory is read ahead of the one branch on row_ok: tcgen05.ld is an instruction of the whole warp, and
        // between two branches on the same lanes' condition the compiler may let the lanes go their ways in between as well
        uint32_t y[D / 4];
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          float o[32];
          __syncwarp();
          tmem_ld32(o_addr + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) y[c * 16 + i] = pack_bf16(o[2 * i] * inv, o[2 * i + 1] * inv);
        }
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < D / 16; ++i)
            reinterpret_cast<uint4*>(dst)[i] = make_uint4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
        }
      }
    } else if constexpr (SPLIT) {
      // what a CTA receives: [4-column group][row] float4 where Q lay, and [row] maxima and sums where the row tiles' were
      float* x_max = &s_max[0][0][0];
      float* x_sum = &s_max[0][1][0];
      cluster_sync_all();                                      // both CTAs' products have completed, their maxima are read
      if (w != rank) {
        const uint32_t peer = 1 - rank;
        const uint32_t remote = map_to_rank(sQ, peer) + (uint32_t)((h * (D / 8) * BM + r) * 16);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          float o[32];
          __syncwarp();
          tmem_ld32(o_addr + c * 32, o);                       // (anything where this CTA has no keys for the tile: its sum says so)
          tmem_ld_wait();
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            st_cluster_f32x4(remote + (uint32_t)((c * 8 + q4) * BM * 16), o[q4 * 4], o[q4 * 4 + 1], o[q4 * 4 + 2], o[q4 * 4 + 3]);
        }
        if (h == 0) {
          st_cluster_f32(map_to_rank(smem_u32(&x_max[r]), peer), m_own);
          st_cluster_f32(map_to_rank(smem_u32(&x_sum[r]), peer), l_own);
        }
      }
      cluster_sync_all();
      if (w == rank && ok) {
        const float m_x = x_max[r], l_x = x_sum[r], m = fmaxf(m_own, m_x);
        const float a_own = l_own > 0.f ? fast_exp2(m_own - m) : 0.f, a_x = l_x > 0.f ? fast_exp2(m_x - m) : 0.f;
        float l = l_own * a_own + l_x * a_x;
        if (l_own != l_own || l_x != l_x) l = l_own + l_x;     // (not a number: stays one)
        if (p.sinks) l += exp2f(sink_log2(p.sinks, head) - m);
        const float inv = l > 0.f ? 1.f / l : (l != l ? l : 0.f);
        const float4* recv = reinterpret_cast<const float4*>(smem) + h * (D / 8) * BM + r;
        uint32_t y[D / 4];
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          float o[32];
          __syncwarp();
          tmem_ld32(o_addr + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4) {
            const float4 v = recv[(c * 8 + q4) * BM];
            const float x[4] = {v.x, v.y, v.z, v.w};
            float z[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {                      // (a side without keys holds anything)
              z[i] = a_own != 0.f ? o[q4 * 4 + i] * a_own : 0.f;
              if (a_x != 0.f) z[i] = fmaf(a_x, x[i], z[i]);
              z[i] *= inv;
            }
            y[c * 16 + q4 * 2] = pack_bf16(z[0], z[1]);
            y[c * 16 + q4 * 2 + 1] = pack_bf16(z[2], z[3]);
          }
        }
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < D / 16; ++i)
            reinterpret_cast<uint4*>(dst)[i] = make_uint4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
        }
      }
    }
  }
  if (SPLIT && shared && (warp < 2 || warp == V_WARP)) {       // the other warps pass the cluster's two barriers too
    cluster_sync_all();
    cluster_sync_all();
  }
  __syncwarp();                                                // (lanes that had no part in a warp's role wait for the one that did)
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*s_abort) {
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// One warp per row of the result: which request's key it is, its page, W / 8 16-byte pieces; rows without a key are zeros.
__global__ void __launch_bounds__(256)
latent_rows_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ cache, const int* __restrict__ table,
                   int max_blocks, const int* __restrict__ cu, const int* __restrict__ seq, int B, int rows, int W, int block_size,
                   int window) {
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= rows) return;
  int b = -1, j = 0, before = 0;
  for (int i0 = 0; i0 < B; i0 += 32) {
    const int i = i0 + lane;
    const Share sh = i < B ? share_of(cu, seq, i, window) : Share{0, 0, 0, 0};
    const int incl = warp_inclusive(sh.rows, lane);
    const int chunk = __shfl_sync(0xffffffffu, incl, 31);
    if (row < before + chunk) {
      const unsigned hit = __ballot_sync(0xffffffffu, row >= before + incl - sh.rows && row < before + incl);
      const int src = __ffs(hit) - 1;
      j = row - before - __shfl_sync(0xffffffffu, incl - sh.rows, src);
      if (j < __shfl_sync(0xffffffffu, sh.keys, src)) b = i0 + src;
      j += __shfl_sync(0xffffffffu, sh.skip, src);
      break;
    }
    before += chunk;
  }
  const int64_t blk = b >= 0 ? table[(int64_t)b * max_blocks + j / block_size] : -1;
  uint4* dst = reinterpret_cast<uint4*>(out + (int64_t)row * W);
  const uint4* src = reinterpret_cast<const uint4*>(cache + (blk >= 0 ? (blk * block_size + j % block_size) * W : 0));
  for (int c = lane; c < W / 8; c += 32) dst[c] = blk >= 0 ? src[c] : make_uint4(0, 0, 0, 0);
}

// A thread per pair: q [T, H, D + P], elements D + (2i, 2i + 1), or with `halves` D + (i, i + rot / 2), i < rot / 2
__global__ void __launch_bounds__(256)
latent_q_turn_kernel(__nv_bfloat16* __restrict__ q, int64_t ldq, const int* __restrict__ positions,
                     const float* __restrict__ cos_sin, int rot, int H, int D, int P, int halves) {
  pdl_enter();
  const int t = blockIdx.x, half = rot / 2;
  const float* cs = cos_sin + (int64_t)positions[t] * rot;
  for (int idx = threadIdx.x; idx < H * half; idx += blockDim.x) {
    const int h = idx / half, i = idx % half;
    __nv_bfloat16* x = q + (int64_t)t * ldq + (int64_t)h * (D + P) + D;
    const int ia = halves ? i : 2 * i, ib = halves ? i + half : 2 * i + 1;
    const float a = to_f32<__nv_bfloat16>(x[ia]), b = to_f32<__nv_bfloat16>(x[ib]);
    const float c = cs[i], s = cs[half + i];
    x[ia] = from_f32<__nv_bfloat16>(a * c - b * s);
    x[ib] = from_f32<__nv_bfloat16>(b * c + a * s);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}
// a map of `n` dimensions of bfloat16 whose boxes are 64 wide and 128 rows high (in the last dimension)
bool make_map(CUtensorMap* m, const void* base, int n, const cuuint64_t* dims, const cuuint64_t* strides) {
  const cuuint32_t box2[2] = {64, BN}, box3[3] = {64, 1, BM}, ones[3] = {1, 1, 1};
  EncodeTiledFn fn = encode_fn();
  return fn && fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, n, const_cast<void*>(base), dims, strides, n == 2 ? box2 : box3, ones,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int num_sms() {                                             // of the current device, asked once
  static const int n = [] {
    int dev = 0, v = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

template <int D, bool SPLIT>
int launch(const CUtensorMap& mq, const CUtensorMap& mkv, const CUtensorMap& mr, const Params& p, int H, int pairs, cudaStream_t stream) {
  auto k = attention_latent_umma_kernel<D, SPLIT>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<D>::SMEM);
  if (e != cudaSuccess) return refuse((int)e, "attention_latent_umma: shared memory opt-in failed: %s", cudaGetErrorString(e));
  e = launch_pdl_cluster(k, dim3(SPLIT ? 2 * H : H, pairs), dim3(NTHREADS), dim3(SPLIT ? 2 : 1, 1, 1), Shape<D>::SMEM, stream, mq, mkv, mr, p);
  if (e != cudaSuccess) return refuse((int)e, "attention_latent_umma: launch failed: %s", cudaGetErrorString(e));
  return cuda_status("attention_latent_umma");
}

bool aligned16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

DINFER_DEFINE_LAST_ERROR()

// out [rows, W] bf16, rows >= the sum over the requests that bring more than one token of their keys (those beyond the window
// left out), each rounded up to a multiple of 128;
// cache [pages, block_size, W] bf16; block_table [B, max_blocks]; cu_seqlens [B + 1]; seq_lens [B].
DINFER_API int dinfer_latent_rows(void* out, const void* cache, const int* block_table, int max_blocks, const int* cu_seqlens,
                                  const int* seq_lens, int B, int rows, int W, int block_size, int window, cudaStream_t stream) {
  if (B <= 0 || rows < 0 || W <= 0 || W % 8 || block_size <= 0 || max_blocks <= 0 || !aligned16(out) || !aligned16(cache))
    return refuse(DINFER_BAD_ARGUMENT, "latent_rows: bad sizes B=%d rows=%d W=%d block=%d (rows of whole 16-byte pieces)", B, rows, W,
                  block_size);
  if (rows == 0) return 0;
  launch_pdl(latent_rows_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, (__nv_bfloat16*)out, (const __nv_bfloat16*)cache,
             block_table, max_blocks, cu_seqlens, seq_lens, B, rows, W, block_size, window);
  return cuda_status("latent_rows");
}

// q [T, H * (D + P)] bf16 rows of stride ldq, turned in place; cos_sin [max_pos, rot] f32, rot <= P even.
DINFER_API int dinfer_latent_q_turn(void* q, int64_t ldq, const int* positions, const float* cos_sin, int rot, int T, int H, int D,
                                    int P, int halves, cudaStream_t stream) {
  if (T < 0 || H <= 0 || D < 0 || P < 0 || rot < 0 || rot % 2 || rot > P || ldq < (int64_t)H * (D + P))
    return refuse(DINFER_BAD_ARGUMENT, "latent_q_turn: bad sizes T=%d H=%d D=%d P=%d rot=%d", T, H, D, P, rot);
  if (T == 0 || rot == 0 || !cos_sin) return 0;
  launch_pdl(latent_q_turn_kernel, dim3(T), dim3(256), 0, stream, (__nv_bfloat16*)q, ldq, positions, cos_sin, rot, H, D, P, halves);
  return cuda_status("latent_q_turn");
}

DINFER_API int dinfer_attention_latent_umma_supports(int R, int P, int D, int V) {
  return (D == 64 || D == 128) && V == D && P >= 0 && P <= 64 && P % 8 == 0 && R > 0 && R % 8 == 0;
}

// Whether a launch takes two CTAs to a pair: where those of all pairs run at once, or where the longest pair's walk is what a single
// round of CTAs waits for (a cluster waits for two SMs, and a shared pair takes some 4 us more).  us alone and shared, 128 wide: 8
// heads, 2048 tokens 50 and 32; 16 heads, 1024 29 and 21; 16, 512 behind 4000 103 and 59; 32, 256 behind 8000 206 and 113; in a
// round of 128 pairs: 16, 2048 51 and 45; 16, 2048 behind 4000 146 and 132; but 32, 1024 30 and 39; 16, 500 + 700 + 900 29 and 37.
DINFER_API int dinfer_attention_latent_umma_shares(int H, int pair_bound, int window, int max_keys) {
  const int64_t n = (int64_t)H * pair_bound;
  const int longest = ((window > 0 && max_keys > window + 2 * BM ? window + 2 * BM : max_keys) + BN - 1) / BN;
  return longest >= MIN_SHARED && (2 * n <= num_sms() || (n <= num_sms() && longest >= LONG_WALK));
}

// Portions (more than one token) only.  q [T, H, D + P] rows of stride ldq (turned), out [T, H, D] rows of stride ldo;
// latents [rows, R + P] as dinfer_latent_rows leaves them, expanded [rows, H, 2 D] with a head's key, then its value.
// pair_bound >= the sum over the portions of ceil(tokens / 256); max_keys: about the keys of the longest request (0: not known).  sinks [H] f32 or null.  window <= 0: all keys.
DINFER_API int dinfer_attention_latent_umma(const void* q, int64_t ldq, void* out, int64_t ldo, const void* latents,
                                            const void* expanded, int rows, const int* cu_seqlens, const int* seq_lens, int T,
                                            int B, int H, int R, int P, int D, float scale, int window, const float* sinks,
                                            int pair_bound, int max_keys, int* status, cudaStream_t stream) {
  if (T <= 0 || B <= 0 || H <= 0 || rows <= 0 || pair_bound <= 0 || pair_bound > 65535)
    return refuse(DINFER_BAD_ARGUMENT, "attention_latent_umma: bad sizes T=%d B=%d H=%d rows=%d pairs=%d", T, B, H, rows, pair_bound);
  if (!dinfer_attention_latent_umma_supports(R, P, D, D))
    return refuse(DINFER_BAD_ARGUMENT, "attention_latent_umma: R=%d P=%d D=%d not supported", R, P, D);
  if (ldq % 8 || ldo % 8 || !aligned16(q) || !aligned16(out) || !aligned16(latents) || !aligned16(expanded) || !(scale > 0.f) || !status)
    return refuse(DINFER_BAD_ARGUMENT, "attention_latent_umma: 16-byte aligned rows, a positive scale and a status word");
  CUtensorMap mq, mkv, mr;
  const cuuint64_t dq[3] = {(cuuint64_t)(D + P), (cuuint64_t)H, (cuuint64_t)T}, sq[2] = {(cuuint64_t)(D + P) * 2, (cuuint64_t)ldq * 2};
  const cuuint64_t dkv[2] = {(cuuint64_t)H * 2 * D, (cuuint64_t)rows}, skv[1] = {(cuuint64_t)H * 2 * D * 2};
  // the rotated part as a tensor of its own, P wide: what a 64-wide box reaches beyond it is zeros.  (With P = 0 the box
  // begins where a row's latents do; Q's part is zeros then.)
  const cuuint64_t dr[2] = {(cuuint64_t)(P > 0 ? P : R), (cuuint64_t)rows}, sr[1] = {(cuuint64_t)(R + P) * 2};
  if (!make_map(&mq, q, 3, dq, sq) || !make_map(&mkv, expanded, 2, dkv, skv) ||
      !make_map(&mr, (const __nv_bfloat16*)latents + (P > 0 ? R : 0), 2, dr, sr))
    return refuse(DINFER_BAD_ARGUMENT, "attention_latent_umma: a tensor map could not be made");
  Params p{};
  p.out = (__nv_bfloat16*)out; p.ldo = ldo; p.cu_seqlens = cu_seqlens; p.seq_lens = seq_lens; p.B = B; p.window = window; p.rows = rows;
  p.scale_log2 = scale * 1.4426950408889634f; p.sinks = sinks; p.status = status;
  const bool split = dinfer_attention_latent_umma_shares(H, pair_bound, window, max_keys);
  if (D == 64) return split ? launch<64, true>(mq, mkv, mr, p, H, pair_bound, stream) : launch<64, false>(mq, mkv, mr, p, H, pair_bound, stream);
  return split ? launch<128, true>(mq, mkv, mr, p, H, pair_bound, stream) : launch<128, false>(mq, mkv, mr, p, H, pair_bound, stream);
}
