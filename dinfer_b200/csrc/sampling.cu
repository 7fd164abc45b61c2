// Sampling on f32 logits.  A row is shared by a thread-block cluster of ROW_CTAS CTAs (of 512 threads in the sampler, of 1024
// in argmax): every CTA keeps its contiguous slice of the row (scaled by 1/temperature) in shared memory, so the
// row is read from memory once, and the CTAs exchange their partial results through each other's
// shared memory (st.shared::cluster + one cluster barrier per exchange).
//
//   dinfer_argmax      greedy, ties to the lowest index
//   dinfer_sample      temperature -> min_p -> top-k -> top-p -> inverse CDF in vocabulary order,
//                      the uniform number from Philox4x32-10 keyed by the request's seed and
//                      counted by the number of tokens the request has produced, so a request's
//                      tokens do not depend on its place in the batch; rows whose temperature is
//                      <= 1e-5 are greedy
//   dinfer_penalties   repetition / frequency / presence penalties from the token history
//   dinfer_logit_bias  per-request additive biases on given tokens
//   dinfer_logprobs    log-probability and rank of the chosen token and the k most likely tokens
//
// Same contract as the reference (crates/kernels/cuda/sampling.cu:13-56,60-133,143-157,196-283,
// 322-349; order of operations models/qwen3/src/executor.rs:552-605).  Unlike it the logits are not
// rewritten: the three filters reduce to one keep-threshold on the scaled logits, the largest value t such that the kept entries
// >= t number at least k (have at least the share p of the mass).  A pass over the row in shared memory counts (and weighs)
// the entries above a few cuts below the maximum; further ones cut up the gap that holds the threshold, until at most
// CAND_MAX entries are left in it (the first pass, nearly always).  Those are collected in every CTA and sorted, and the
// threshold is read off; for a small k the whole top of the row is collected, so that top-p is read off it too.  Where more
// entries than that crowd the gap to the end, a radix-16 descent over the order-preserving 32-bit image of a float goes on
// inside it.  All sums are taken in a fixed order (segment, warp of segments, CTA rank), so the same logits, seed and count
// give the same token.
#include "common.cuh"

using namespace dinfer;

namespace {

constexpr int BLOCK = 1024;
// A CTA's slice is cut into SEGMENTS runs of neighbouring ids, and 32 neighbouring segments are a warp of segments: what a
// sum's order is made of, whatever the block's size.  The sampling kernel's blocks have 512 threads with VT = 2 segments each
// (t and t + 512): at 64 registers a thread two blocks share an SM, so that one works while the other waits at a cluster
// barrier, and a wave holds twice the rows.  us for 8 / 16 / 64 rows of 151936, temperature alone: 1024 threads 12.2 / 22.8 /
// 55, 512 threads 11.9 / 13.3 / 28.
constexpr int SEGMENTS = 1024;
constexpr int WARPS_OF_SEGMENTS = SEGMENTS / 32;
constexpr int VT = 2;
constexpr int NT = SEGMENTS / VT;           // threads of the sampling kernel
constexpr int ROW_CTAS = 8;                 // cluster size: CTAs that share a row
constexpr int MAX_SLICE = 48 * 1024;        // floats of a row slice that shared memory holds (192 KB)
// Dynamic shared memory that keeps a second CTA of the sampling kernel off an SM.  With as few rows as find an SM for every CTA
// two of them share one all the same otherwise: 8 rows without likely tokens, top-p 0.9 42 us on shared SMs and 37 apart, top-k
// 1000 35 and 31.
constexpr size_t LONE_SMEM = 110 * 1024;
constexpr int XCH = 16;                     // floats a CTA hands to the others per exchange
constexpr int ARGMAX_MANY_ROWS = 40;        // from so many rows on the argmax runs a CTA per row

// ---- cluster plumbing
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void st_cluster_f32(uint32_t local_addr, uint32_t rank, float v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local_addr), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

// What the CTAs of a row share: two exchange buffers used alternately (a CTA may write the next
// exchange while a slower one still reads the last) and the block-level scratch.
struct Shared {
  float xchg[2][ROW_CTAS][XCH];
  float warp_part[32][XCH];
  float blk[XCH];
  float warp_tot[32];
  int pick[4];
};

// Which exchange is next, the same in all threads; -1: the cluster's first barrier phase (every CTA runs, so that its memory may be
// written) is still to be waited for.
struct Turn { int next = -1; };
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// Every CTA contributes n <= XCH floats (valid in threads 0..n-1 as `mine`); afterwards
// sh.xchg[turn][r][j] holds the contribution j of CTA r, the same in every CTA.  Returns the buffer.  (The cluster's barrier is one of
// every CTA's threads too.)
__device__ float (*exchange(Shared& sh, Turn& turn, float mine, int n, uint32_t rank))[XCH] {
  if (turn.next < 0) { cluster_wait(); turn.next = 0; }
  const int t = turn.next;
  turn.next = t ^ 1;
  if ((int)threadIdx.x < n) {
#pragma unroll
    for (uint32_t r = 0; r < ROW_CTAS; ++r) st_cluster_f32(smem_u32(&sh.xchg[t][rank][threadIdx.x]), r, mine);
  }
  cluster_sync_all();
  return sh.xchg[t];
}

// Sum over the whole row of what every segment contributes: fill(segment, v) adds segment's share to v[0..N).  Warps of
// segments by a shuffle tree, then those in order, then the CTAs in rank order.  Returns the CTAs' shares.
template <int N, typename F>
__device__ __forceinline__ float (*row_sum(Shared& sh, Turn& turn, uint32_t rank, float (&out)[N], F fill))[XCH] {
  const int lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll 1
  for (int vt = 0; vt < VT; ++vt) {
    const int u = vt * NT + threadIdx.x;
    float v[N];
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = 0.f;
    fill(u, v);
#pragma unroll
    for (int j = 0; j < N; ++j) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
    }
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < N; ++j) sh.warp_part[u >> 5][j] = v[j];
    }
  }
  __syncthreads();
  float mine = 0.f;
  if ((int)threadIdx.x < N)
    for (int w = 0; w < WARPS_OF_SEGMENTS; ++w) mine += sh.warp_part[w][threadIdx.x];
  float (*x)[XCH] = exchange(sh, turn, mine, N, rank);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    float t = 0.f;
#pragma unroll
    for (int r = 0; r < ROW_CTAS; ++r) t += x[r][j];
    out[j] = t;
  }
  return x;
}

// order-preserving image of a float: a < b  <=>  key(a) < key(b)   (-0 is folded into +0 by the caller)
__device__ __forceinline__ uint32_t float_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct ArgMax { float v; int i; };
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}

// argmax over the row (ties to the lowest index), the same in every CTA of the cluster
template <int THREADS>
__device__ int row_argmax(Shared& sh, Turn& turn, const float* xs, int n_mine, int first, uint32_t rank) {
  ArgMax best{-INFINITY, 0x7fffffff};
  for (int i = threadIdx.x; i < n_mine; i += THREADS) best = better(best, ArgMax{xs[i], first + i});
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    best = better(best, ArgMax{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) { sh.warp_part[warp][0] = best.v; sh.warp_part[warp][1] = __int_as_float(best.i); }
  __syncthreads();
  if (warp == 0) {
    best = lane < THREADS / 32 ? ArgMax{sh.warp_part[lane][0], __float_as_int(sh.warp_part[lane][1])} : ArgMax{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      best = better(best, ArgMax{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
    if (lane == 0) { sh.blk[0] = best.v; sh.blk[1] = __int_as_float(best.i); }
  }
  __syncthreads();
  const float mine = threadIdx.x < 2 ? sh.blk[threadIdx.x] : 0.f;
  float (*x)[XCH] = exchange(sh, turn, mine, 2, rank);
  ArgMax all{-INFINITY, 0x7fffffff};
#pragma unroll
  for (int r = 0; r < ROW_CTAS; ++r) all = better(all, ArgMax{x[r][0], __float_as_int(x[r][1])});
  return all.i == 0x7fffffff ? 0 : all.i;
}

__device__ __forceinline__ uint32_t mulhilo(uint32_t a, uint32_t b, uint32_t* hi) {
  const uint64_t p = (uint64_t)a * b;
  *hi = (uint32_t)(p >> 32);
  return (uint32_t)p;
}

// counter (offset_lo, offset_hi, 0, 0), key (seed_lo, seed_hi), ten rounds, u = (c0 >> 8) / 2^24
__device__ float philox_uniform(uint64_t seed, uint64_t offset) {
  uint32_t c0 = (uint32_t)offset, c1 = (uint32_t)(offset >> 32), c2 = 0, c3 = 0;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int r = 0; r < 10; ++r) {
    uint32_t hi0, hi1;
    const uint32_t lo0 = mulhilo(0xD2511F53u, c0, &hi0);
    const uint32_t lo1 = mulhilo(0xCD9E8D57u, c2, &hi1);
    const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return (float)(c0 >> 8) * (1.f / 16777216.f);
}

// The slice of the row this CTA owns: ids [first, first + n_mine).  Segment u holds the contiguous
// ids [u*seg, (u+1)*seg) of the slice, so segment order, then CTA rank, is vocabulary order.
struct Slice {
  const float* xs;      // scaled values in shared memory, or null: read the row and scale on the fly
  const float* row;
  float inv_t;
  int first, n_mine, seg;
  __device__ __forceinline__ float at(int i) const { return xs ? xs[i] : row[first + i] * inv_t + 0.f; }
  __device__ __forceinline__ int begin(int u) const { return min(n_mine, u * seg); }
  __device__ __forceinline__ int end(int u) const { return min(n_mine, (u + 1) * seg); }
};

// Where a threshold is known to lie: the float_key from `base` on, `width` more at most, and the weight of the entries beyond.
struct Bracket {
  uint32_t base = 0, width = 0xffffffffu;
  float above = 0.f;
};

// The largest value t of the bracket such that the entries x >= max(t, floor_) weigh at least `target`, where an
// entry weighs 1 (MASS = false) or exp(x - m) (MASS = true).  Radix-16 descent over float_key - base: `above` is the
// weight of the entries beyond the digits fixed so far.  Eight passes over the row for all floats, fewer for a bracket.
template <bool MASS>
__device__ float radix_threshold(Shared& sh, Turn& turn, const Slice& sl, uint32_t rank, float m, float floor_, float target,
                                 const Bracket& where) {
  uint32_t prefix = 0;
  float above = where.above;
  const int first = where.width ? (31 - __clz(where.width)) & ~3 : 0;
#pragma unroll 1
  for (int shift = first; shift >= 0; shift -= 4) {
    float tot[16];
    row_sum<16>(sh, turn, rank, tot, [&](int u, float (&h)[16]) {
      const int i1 = sl.end(u);
      for (int i = sl.begin(u); i < i1; ++i) {
        const float x = sl.at(i);
        if (!(x >= floor_)) continue;
        const uint32_t k = float_key(x) - where.base;      // (a key below the base wraps beyond the width)
        if (k > where.width || (shift < first && (k >> (shift + 4)) != (prefix >> (shift + 4)))) continue;
        const float w = MASS ? expf(x - m) : 1.f;
        const int dgt = (k >> shift) & 15;
#pragma unroll
        for (int d = 0; d < 16; ++d) h[d] += dgt == d ? w : 0.f;
      }
    });
    int chosen = 0;
    float run = above;
    bool found = false;
#pragma unroll
    for (int d = 15; d >= 0; --d) {
      if (!found) {
        if (run + tot[d] >= target) { chosen = d; found = true; }
        else run += tot[d];
      }
    }
    if (!found) { chosen = 0; run -= tot[0]; }          // less than the target in all: keep everything
    above = run;
    prefix |= (uint32_t)chosen << shift;
  }
  return key_float(where.base + prefix);
}

// ---- the short way to the two thresholds: where at most CAND_MAX entries hold the k largest, or the share p of the mass
constexpr int CAND_MAX = 1024;
constexpr int CUTS = 8;                       // cuts a pass counts at, the last one the floor
constexpr int CUT_ROUNDS = 4;
static_assert(CAND_MAX <= SEGMENTS && 2 * CUTS <= XCH, "a candidate per segment; counts and masses in one exchange");

struct Candidates {
  float x[CAND_MAX];                  // the candidates, the same list in every CTA of the row, in vocabulary order
  float s[CAND_MAX];                  // and from the largest down
  int warp_tot[WARPS_OF_SEGMENTS];
  float warp_mass[WARPS_OF_SEGMENTS];
  int found;
};

// inclusive prefix sums of the segments' v, in segment order; `total` is the block's sum
__device__ __forceinline__ void segment_scan(int (&v)[VT], int* warp_tot, int& total) {
  const int lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll
  for (int vt = 0; vt < VT; ++vt) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v[vt], o);
      if (lane >= o) v[vt] += t;
    }
    if (lane == 31) warp_tot[(vt * NT + threadIdx.x) >> 5] = v[vt];
  }
  __syncthreads();
  int all = 0;
#pragma unroll 8
  for (int w = 0; w < WARPS_OF_SEGMENTS; ++w) {
    const int t = warp_tot[w];
#pragma unroll
    for (int vt = 0; vt < VT; ++vt)
      if (w < ((vt * NT + (int)threadIdx.x) >> 5)) v[vt] += t;
    all += t;
  }
  total = all;
}

// The highest of a few cuts c such that the kept entries (x >= floor_) with x >= c are enough: at least k of them (MASS
// false), or at least the share p of the mass of all kept ones (true; `denom` is then that mass).  The first pass cuts at
// fixed distances below the maximum (x is in units of the softmax's exponent), further ones inside the gap between the lowest
// cut that is not enough and the highest that is.  Returns whether at most CAND_MAX entries are left to look through: with
// `whole` those from the cut up, else those of the gap, from the cut up to `below` (gap.above is what lies beyond weighs), and `place` how many they are.
// Where there are more after CUT_ROUNDS passes, or equal ones crowd a gap of few floats, a descent inside the gap finds the
// threshold.
constexpr int UPPER = CUTS - 2;             // cuts that few entries reach
// candidates of the CTAs before this one, and of all
struct Place { int base, n; };
template <bool MASS>
__device__ bool find_cut(Shared& sh, Turn& turn, const Slice& sl, uint32_t rank, float m, float lo, float floor_, float need, bool whole,
                         float& cut, float& below, float& denom, Bracket& gap, Place& place) {
  float c[CUTS] = {m - 1.f, m - 2.f, m - 4.f, m - 6.f, m - 9.f, m - 13.f, m - 18.f, floor_};
#pragma unroll
  for (int j = 0; j < CUTS; ++j) c[j] = fmaxf(c[j], floor_);
  float target = need, hi = m, n_above = 0.f, before_above = 0.f;
  const auto before = [&](float (*x)[XCH], int j) {        // entries from cut j up in the CTAs before this one
    float t = 0.f;
#pragma unroll
    for (int r = 0; r < ROW_CTAS; ++r) t += r < (int)rank ? x[r][j] : 0.f;
    return t;
  };
  below = INFINITY;                                        // (no cut that is not enough was met yet)
#pragma unroll 1
  for (int round = 0; round < CUT_ROUNDS; ++round) {
    float tot[MASS ? 2 * CUTS : CUTS];
    float (*x)[XCH] = row_sum<MASS ? 2 * CUTS : CUTS>(sh, turn, rank, tot, [&](int u, float (&h)[MASS ? 2 * CUTS : CUTS]) {
      const int i1 = sl.end(u);
      for (int i = sl.begin(u); i < i1; ++i) {
        const float x = sl.at(i);
        const float w = MASS ? (x >= c[CUTS - 1] ? expf(x - m) : 0.f) : 0.f;
        // the cuts fall, and most entries of a row lie below all but the last ones
        const auto count = [&](int j) {
          h[j] += x >= c[j] ? 1.f : 0.f;
          if (MASS) h[CUTS + j] += x >= c[j] ? w : 0.f;
        };
        if (x >= c[UPPER - 1]) {
#pragma unroll
          for (int j = 0; j < UPPER; ++j) count(j);
        }
#pragma unroll
        for (int j = UPPER; j < CUTS; ++j) count(j);
      }
    });
    if (MASS && round == 0) { denom = tot[(MASS ? CUTS : 0) + CUTS - 1]; target = need * denom; }
    float n = tot[CUTS - 1], before_cut = 0.f;
    bool reached = false;
    cut = c[CUTS - 1];
#pragma unroll
    for (int j = 0; j < CUTS; ++j) {
      const float have = MASS ? tot[(MASS ? CUTS : 0) + j] : tot[j];
      if (!reached) {
        if (have >= target || j == CUTS - 1) { reached = true; cut = c[j]; n = tot[j]; before_cut = before(x, j); }
        else { hi = below = c[j]; n_above = tot[j]; before_above = before(x, j); gap.above = have; }
      }
    }
    if (whole && n <= (float)CAND_MAX) { below = INFINITY; place = Place{(int)before_cut, (int)n}; return true; }
    if (!whole && n - n_above <= (float)CAND_MAX) { place = Place{(int)(before_cut - before_above), (int)(n - n_above)}; return true; }
    const float low = fmaxf(cut, lo);                      // (the floor may be -inf, and masked entries with it)
    gap.base = float_key(MASS ? low : cut);                // (masked entries have no mass, but they count)
    gap.width = hi <= lo ? 0u : float_key(hi) - (below < INFINITY ? 1u : 0u) - gap.base;
    if (gap.width < 256u || (whole && n_above >= (float)CAND_MAX)) return false;
    const bool masked = low > cut;                         // then the lowest cut but one is the smallest finite entry
    const float step = (hi - low) * (masked ? 1.f / (CUTS - 1) : 1.f / CUTS);
#pragma unroll
    for (int j = 0; j < CUTS - 1; ++j) c[j] = hi - (float)(j + 1) * step;
    if (masked) c[CUTS - 2] = low;
    c[CUTS - 1] = cut;
  }
  return false;
}

// Fills cd.x with the entries from `cut` up and below `below` (at most CAND_MAX), in vocabulary order, and cd.s with the same
// from the largest down; returns their number.
template <bool GAP>
__device__ int gather_sorted(Candidates& cd, const Slice& sl, float cut, float below, const Place& place) {
  int cnt[VT], end[VT], cta_total;
#pragma unroll
  for (int vt = 0; vt < VT; ++vt) {
    const int u = vt * NT + threadIdx.x, i1 = sl.end(u);
    int n = 0;
    for (int i = sl.begin(u); i < i1; ++i) {
      const float xv = sl.at(i);
      n += xv >= cut && (!GAP || xv < below);
    }
    cnt[vt] = end[vt] = n;
  }
  segment_scan(end, cd.warp_tot, cta_total);
  const int base = place.base;
  int n = place.n;
#pragma unroll
  for (int vt = 0; vt < VT; ++vt) {
    const int u = vt * NT + threadIdx.x, i1 = sl.end(u);
    int at = base + end[vt] - cnt[vt];
    for (int i = sl.begin(u); i < i1 && cnt[vt] > 0; ++i) {
      const float xv = sl.at(i);
      if (xv >= cut && (!GAP || xv < below) && at < CAND_MAX) {
        const uint32_t dst = smem_u32(&cd.x[at]);
#pragma unroll
        for (uint32_t r = 0; r < ROW_CTAS; ++r) st_cluster_f32(dst, r, xv);
        ++at;
      }
    }
  }
  cluster_sync_all();
  __syncthreads();
  // ranks by counting (equal values in vocabulary order): NT / n2 threads to a candidate, n2 the next power of two
  n = min(n, CAND_MAX);
  int n2 = 32;
  while (n2 < n) n2 <<= 1;
  const int tpc = n2 >= NT ? 1 : min(32, NT / n2);
  const int per = NT / tpc;                                // candidates a round ranks
  for (int i0 = 0; i0 < n; i0 += per) {
    const int i = i0 + (int)threadIdx.x / tpc;
    const float v = i < n ? cd.x[i] : 0.f;
    int before = 0;
    if (i < n)
      for (int j = threadIdx.x % tpc; j < n; j += tpc) {
        const float xj = cd.x[j];
        before += xj > v || (xj == v && j < i);
      }
    for (int o = 1; o < tpc; o <<= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (i < n && threadIdx.x % tpc == 0) cd.s[before] = v;
  }
  __syncthreads();
  return n;
}

// The largest of the sorted candidates v >= floor_ such that those >= v and what weighs `above` beyond them hold at least the
// share p of `denom` (of the mass of the candidates >= floor_ where denom < 0).
__device__ float topp_of_sorted(Candidates& cd, int n, float m, float floor_, float p, float denom, float above) {
  const int lane = threadIdx.x & 31;
  float cum[VT];
  if (threadIdx.x == 0) cd.found = n;
#pragma unroll
  for (int vt = 0; vt < VT; ++vt) {
    const int u = vt * NT + threadIdx.x;
    cum[vt] = u < n && cd.s[u] >= floor_ ? expf(cd.s[u] - m) : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float t = __shfl_up_sync(0xffffffffu, cum[vt], o);
      if (lane >= o) cum[vt] += t;
    }
    if (lane == 31) cd.warp_mass[u >> 5] = cum[vt];
  }
  __syncthreads();
  float before[VT], all = 0.f;
#pragma unroll
  for (int vt = 0; vt < VT; ++vt) before[vt] = above;
#pragma unroll 8
  for (int w = 0; w < WARPS_OF_SEGMENTS; ++w) {
    const float t = cd.warp_mass[w];
#pragma unroll
    for (int vt = 0; vt < VT; ++vt)
      if (w < ((vt * NT + (int)threadIdx.x) >> 5)) before[vt] += t;
    all += t;
  }
  const float target = p * (denom < 0.f ? all : denom);
#pragma unroll
  for (int vt = 0; vt < VT; ++vt) {
    const int u = vt * NT + threadIdx.x;
    if (u < n && cd.s[u] >= floor_ && before[vt] + cum[vt] >= target) atomicMin(&cd.found, u);
  }
  __syncthreads();
  if (cd.found < n) return cd.s[cd.found];
  return n > 0 ? fmaxf(floor_, cd.s[n - 1]) : floor_;      // not reached by a rounding: all of them
}

__global__ void __launch_bounds__(BLOCK)
argmax_kernel(const float* __restrict__ logits, int64_t ld, int* __restrict__ out, int vocab) {
  extern __shared__ __align__(16) float xs_dyn[];
  __shared__ Shared sh;
  pdl_enter();
  const uint32_t rank = cluster_ctarank();
  const int b = blockIdx.x / ROW_CTAS;
  const float* row = logits + (int64_t)b * ld;
  const int per = (vocab + ROW_CTAS - 1) / ROW_CTAS;
  const int first = min(vocab, (int)rank * per), n_mine = min(vocab, first + per) - first;
  Turn turn;
  cluster_arrive();                                      // (waited for ahead of the first write into another CTA's memory)
  const int r = row_argmax<BLOCK>(sh, turn, row + first, n_mine, first, rank);
  if (rank == 0 && threadIdx.x == 0) out[b] = r;         // (behind the last barrier nobody writes to another any more)
}

// Many rows: a CTA per row (no cluster: with 8 CTAs a row, 64 rows are two waves of CTAs that mostly wait for each
// other), four floats a load where the row allows.
__global__ void __launch_bounds__(BLOCK)
argmax_many_kernel(const float* __restrict__ logits, int64_t ld, int* __restrict__ out, int vocab) {
  __shared__ float part_v[BLOCK / 32];
  __shared__ int part_i[BLOCK / 32];
  pdl_enter();
  const int b = blockIdx.x;
  const float* row = logits + (int64_t)b * ld;
  ArgMax best{-INFINITY, 0x7fffffff};
  if (!(reinterpret_cast<uintptr_t>(row) & 15)) {
    const int n4 = vocab >> 2;
    const float4* row4 = reinterpret_cast<const float4*>(row);
    for (int i = threadIdx.x; i < n4; i += BLOCK) {
      const float4 v = row4[i];
      best = better(best, ArgMax{v.x, 4 * i});
      best = better(best, ArgMax{v.y, 4 * i + 1});
      best = better(best, ArgMax{v.z, 4 * i + 2});
      best = better(best, ArgMax{v.w, 4 * i + 3});
    }
    for (int i = 4 * n4 + threadIdx.x; i < vocab; i += BLOCK) best = better(best, ArgMax{row[i], i});
  } else {
    for (int i = threadIdx.x; i < vocab; i += BLOCK) best = better(best, ArgMax{row[i], i});
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    best = better(best, ArgMax{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { part_v[warp] = best.v; part_i[warp] = best.i; }
  __syncthreads();
  if (warp == 0) {
    best = ArgMax{part_v[lane], part_i[lane]};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      best = better(best, ArgMax{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
    if (lane == 0) out[b] = best.i == 0x7fffffff ? 0 : best.i;
  }
}

// What bounds it: the instructions of its passes over the row in shared memory and the cluster barriers between them, not
// the one read of the row (39 MB for 64 rows of 151936: 6 us).  64 rows, greedy / temperature / top-k 20 + top-p 0.95 /
// top-p 0.9 in turn, took 165 us with eight radix rounds for the top-p threshold, a shared-memory histogram for the top-k
// one and one block of 1024 threads to an SM; 53 us now (59 with the block's barriers in every exchange).  Alone, at 8 and 64 rows: top-k 20 + top-p 24 and 118 -> 22 and
// 57 us, top-p 0.9 72 and 359 -> 26 and 68 us.  Rows without likely tokens (normal, sigma 1.4 and 4.3), top-p 0.95: 80 and 397,
// 77 and 381 -> 60 and 204, 46 to 62 and 164 us (90 and 298, 101 and 318 where only whole rows' candidates and a descent over
// all floats were known); top-k 1000 70 and 344 -> 31 to 45 and 115 to 136.
__global__ void __launch_bounds__(NT, 2)
sample_kernel(const float* __restrict__ logits, int64_t ld, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ min_p,
              const uint64_t* __restrict__ seeds, const uint64_t* __restrict__ offsets,
              int* __restrict__ out, int vocab, int cache_slice) {
  extern __shared__ __align__(16) float xs_dyn[];
  __shared__ Shared sh;
  __shared__ Candidates cand;
  pdl_enter();
  const uint32_t rank = cluster_ctarank();
  const int b = blockIdx.x / ROW_CTAS;
  const float* row = logits + (int64_t)b * ld;
  const int per = (vocab + ROW_CTAS - 1) / ROW_CTAS;
  const int first = min(vocab, (int)rank * per), n_mine = min(vocab, first + per) - first;
  Turn turn;
  cluster_arrive();                                      // (waited for ahead of the first write into another CTA's memory)
  const float temp = temperature[b];
  if (temp <= 1e-5f) {
    const int r = row_argmax<NT>(sh, turn, row + first, n_mine, first, rank);
    if (rank == 0 && threadIdx.x == 0) out[b] = r;
    return;
  }
  const float inv_t = 1.f / temp;
  Slice sl;
  sl.row = row; sl.inv_t = inv_t; sl.first = first; sl.n_mine = n_mine;
  sl.seg = (per + SEGMENTS - 1) / SEGMENTS;
  sl.xs = cache_slice ? xs_dyn : nullptr;

  // one pass over the row: scaled values into shared memory, maximum and smallest finite value
  float m = -INFINITY, lo = INFINITY;
  for (int i = threadIdx.x; i < n_mine; i += NT) {
    const float x = row[first + i] * inv_t + 0.f;        // + 0: -0 becomes +0 (one image per value)
    if (cache_slice) xs_dyn[i] = x;
    m = fmaxf(m, x);
    if (x > -INFINITY) lo = fminf(lo, x);
  }
  {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { sh.warp_part[warp][0] = m; sh.warp_part[warp][1] = lo; }
    __syncthreads();
    if (threadIdx.x < 2) {
      float v = sh.warp_part[0][threadIdx.x];
      for (int w = 1; w < NT / 32; ++w) v = threadIdx.x == 0 ? fmaxf(v, sh.warp_part[w][0]) : fminf(v, sh.warp_part[w][1]);
      sh.blk[threadIdx.x] = v;
    }
    __syncthreads();
    const float mine = threadIdx.x < 2 ? sh.blk[threadIdx.x] : 0.f;
    float (*x)[XCH] = exchange(sh, turn, mine, 2, rank);
    m = -INFINITY; lo = INFINITY;
#pragma unroll
    for (int r = 0; r < ROW_CTAS; ++r) { m = fmaxf(m, x[r][0]); lo = fminf(lo, x[r][1]); }
  }

  // keep-threshold on x: min_p, then top-k, then top-p on what top-k and min_p left
  float thr = -INFINITY;
  const float mp = min_p ? min_p[b] : 0.f;
  if (mp > 0.f) thr = m + logf(mp);                      // p_i >= min_p * p_max
  const int k = top_k ? top_k[b] : -1;
  const bool finite = m < INFINITY && m > -INFINITY;      // else nothing is kept, whatever the thresholds
  int n_cand = -1;                                       // >= 0: cand holds every entry from the top-k threshold up
  float cut, below, denom = -1.f;
  Bracket gap;                                           // (all floats where no cut is looked for)
  Place place{0, 0};
  if (k > 0 && k < vocab) {
    const bool whole = k <= CAND_MAX / 2;                // a small k leaves the candidates to top-p
    if (finite && find_cut<false>(sh, turn, sl, rank, m, lo, thr, (float)k, whole, cut, below, denom, gap, place)) {
      const int n = whole ? gather_sorted<false>(cand, sl, cut, below, place) : gather_sorted<true>(cand, sl, cut, below, place);
      const int kth = whole ? k : k - (int)gap.above;
      if (kth <= n) thr = fmaxf(thr, cand.s[kth - 1]);       // else all of them are kept
      if (whole) n_cand = n;
    } else {
      thr = fmaxf(thr, radix_threshold<false>(sh, turn, sl, rank, m, thr, (float)k, gap));
    }
  }
  const float p = top_p ? top_p[b] : 1.f;
  if (p < 1.f && p > 0.f) {
    if (n_cand >= 0) {
      thr = fmaxf(thr, topp_of_sorted(cand, n_cand, m, thr, p, -1.f, 0.f));
    } else if (finite) {
      gap = Bracket();
      if (find_cut<true>(sh, turn, sl, rank, m, lo, thr, p, false, cut, below, denom, gap, place)) {
        const int n = gather_sorted<true>(cand, sl, cut, below, place);
        thr = fmaxf(thr, topp_of_sorted(cand, n, m, thr, p, denom, gap.above));
      } else {
        thr = fmaxf(thr, radix_threshold<true>(sh, turn, sl, rank, m, thr, p * denom, gap));
      }
    }
  }

  // inverse CDF in vocabulary order: segments in order within a CTA, CTAs in rank order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float mine[VT], incl[VT];                              // a segment's mass, and its inclusive scan over its warp of segments
#pragma unroll
  for (int vt = 0; vt < VT; ++vt) {
    const int u = vt * NT + threadIdx.x, i1 = sl.end(u);
    float t = 0.f;
    for (int i = sl.begin(u); i < i1; ++i) {
      const float x = sl.at(i);
      if (x >= thr) t += expf(x - m);
    }
    mine[vt] = incl[vt] = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, incl[vt], o);
      if (lane >= o) incl[vt] += v;
    }
    if (lane == 31) sh.warp_tot[u >> 5] = incl[vt];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < WARPS_OF_SEGMENTS; ++w) s += sh.warp_tot[w];
    sh.blk[0] = s;
  }
  __syncthreads();
  float (*x)[XCH] = exchange(sh, turn, threadIdx.x == 0 ? sh.blk[0] : 0.f, 1, rank);
  float total = 0.f;
#pragma unroll
  for (int r = 0; r < ROW_CTAS; ++r) total += x[r][0];
  const float target = philox_uniform(seeds[b], offsets[b]) * total;
  // the CTA whose share of the cumulative mass reaches the target; beyond the total by rounding: the
  // last CTA that keeps anything, at the end of its share
  int owner = -1, last_nonzero = -1;
  float before = 0.f, before_last = 0.f, run = 0.f;
#pragma unroll
  for (int r = 0; r < ROW_CTAS; ++r) {
    const float t = x[r][0];
    if (t > 0.f) { last_nonzero = r; before_last = run; }
    if (owner < 0 && t > 0.f && run + t >= target) { owner = r; before = run; }
    run += t;
  }
  bool clamp = false;
  if (owner < 0) { owner = last_nonzero; before = before_last; clamp = true; }
  if (owner == (int)rank) {
    // within this CTA: the warp, then the lane, then the entry
    if (threadIdx.x == 0) {
      float cum = before;
      int w_own = -1;
      float w_before = before;
      int w_last = -1;
      float w_before_last = before;
      for (int w = 0; w < WARPS_OF_SEGMENTS; ++w) {
        const float t = sh.warp_tot[w];
        if (t > 0.f) { w_last = w; w_before_last = cum; }
        if (w_own < 0 && !clamp && t > 0.f && cum + t >= target) { w_own = w; w_before = cum; }
        cum += t;
      }
      if (w_own < 0) { w_own = w_last; w_before = w_before_last; sh.pick[2] = 1; } else sh.pick[2] = 0;
      sh.pick[0] = w_own;
      sh.blk[1] = w_before;
    }
    __syncthreads();
#pragma unroll
    for (int vt = 0; vt < VT; ++vt) {
      if (vt * (NT / 32) + warp != sh.pick[0]) continue;
      const bool clamp_w = sh.pick[2] != 0;
      const float base = sh.blk[1];
      const float excl = incl[vt] - mine[vt];            // mass of the segments of the warp before this one
      // the first segment whose inclusive sum reaches the target (or the last one that keeps anything)
      const bool hit = !clamp_w && mine[vt] > 0.f && base + incl[vt] >= target;
      const unsigned hits = __ballot_sync(0xffffffffu, hit);
      const unsigned keeps = __ballot_sync(0xffffffffu, mine[vt] > 0.f);
      int l_own;
      bool clamp_l = false;
      if (hits) l_own = __ffs(hits) - 1;
      else { l_own = 31 - __clz(keeps); clamp_l = true; }
      if (lane == l_own) {
        const int u = vt * NT + threadIdx.x, i1 = sl.end(u);
        float cum = base + excl;
        int last = -1;
        for (int i = sl.begin(u); i < i1; ++i) {
          const float xv = sl.at(i);
          if (xv >= thr) {
            cum += expf(xv - m);
            last = i;
            if (!clamp_l && cum >= target) break;
          }
        }
        out[b] = first + (last < 0 ? 0 : last);
      }
    }
  }
  if (owner < 0 && rank == 0 && threadIdx.x == 0) out[b] = 0;   // nothing kept at all (no finite logit)
}                                                        // (behind the last exchange nobody writes to another any more)

// history of row b: ids[offsets[b] .. offsets[b+1]), the first prompt_len[b] of them the prompt.
__global__ void penalties_kernel(float* __restrict__ logits, int64_t ld, const int* __restrict__ ids,
                                 const int* __restrict__ offsets, const int* __restrict__ prompt_len,
                                 const float* __restrict__ rep, const float* __restrict__ freq,
                                 const float* __restrict__ pres, int vocab) {
  const int b = blockIdx.x;
  const float r = rep[b], f = freq[b], pr = pres[b];
  if (r == 1.f && f == 0.f && pr == 0.f) return;
  float* row = logits + (int64_t)b * ld;
  const int lo = offsets[b], hi = offsets[b + 1], np = prompt_len[b];
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const int t = ids[i];
    if (t < 0 || t >= vocab) continue;
    bool first = true;                       // each distinct token is handled by its first occurrence
    for (int j = lo; j < i; ++j) if (ids[j] == t) { first = false; break; }
    if (!first) continue;
    int cnt = 0;
    for (int j = lo + np; j < hi; ++j) cnt += ids[j] == t;
    float v = row[t];
    if (r != 1.f) v = v > 0.f ? v / r : v * r;
    if (cnt > 0) v -= f * (float)cnt + pr;
    row[t] = v;
  }
}

// logits[rows[i], ids[i]] += bias[i]; a (row, id) pair appears once.
__global__ void logit_bias_kernel(float* __restrict__ logits, int64_t ld, const int* __restrict__ rows,
                                  const int* __restrict__ ids, const float* __restrict__ bias, int n, int vocab) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int t = ids[i];
  if (t >= 0 && t < vocab) logits[(int64_t)rows[i] * ld + t] += bias[i];
}

// Log-probabilities of a row under log_softmax of the logits as given (no temperature, no filter): the chosen
// token's, how many tokens are strictly more likely (its rank), and the k most likely in descending order, ties
// to the lower id.  One CTA per row.  The k best are found one after the other, each as the best entry that comes
// after the last one in that order, so nothing has to be remembered but the last winner.
constexpr int LP_MAX_K = 32;
__global__ void logprobs_kernel(const float* __restrict__ logits, int64_t ld, const int* __restrict__ chosen, int k,
                                int* __restrict__ out_ids, float* __restrict__ out_lp, int* __restrict__ out_rank,
                                int vocab) {
  __shared__ float s_f[BLOCK / 32];
  __shared__ int s_i[BLOCK / 32];
  __shared__ float s_m, s_lse, s_last_v;
  __shared__ int s_last_i;
  const int b = blockIdx.x;
  const float* row = logits + (int64_t)b * ld;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // maximum
  float m = -INFINITY;
  for (int i = threadIdx.x; i < vocab; i += BLOCK) m = fmaxf(m, row[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) s_f[warp] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float v = s_f[0];
    for (int w = 1; w < BLOCK / 32; ++w) v = fmaxf(v, s_f[w]);
    s_m = v;
  }
  __syncthreads();
  m = s_m;
  // log of the sum of exponentials, and the rank of the chosen token (sums in a fixed order)
  const int c = chosen[b];
  const bool c_ok = c >= 0 && c < vocab;
  const float xc = c_ok ? row[c] : -INFINITY;
  float d = 0.f;
  int gt = 0;
  for (int i = threadIdx.x; i < vocab; i += BLOCK) {
    const float v = row[i];
    if (v > -INFINITY) d += expf(v - m);
    gt += v > xc;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    d += __shfl_xor_sync(0xffffffffu, d, o);
    gt += __shfl_xor_sync(0xffffffffu, gt, o);
  }
  if (lane == 0) { s_f[warp] = d; s_i[warp] = gt; }
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = 0.f;
    int cnt = 0;
    for (int w = 0; w < BLOCK / 32; ++w) { sum += s_f[w]; cnt += s_i[w]; }
    s_lse = m + logf(sum);
    out_ids[(int64_t)b * (k + 1)] = c;
    out_lp[(int64_t)b * (k + 1)] = xc - s_lse;
    out_rank[b] = cnt;
    s_last_v = INFINITY;                  // before the first entry of the order
    s_last_i = -1;
  }
  __syncthreads();
  for (int j = 0; j < k; ++j) {
    const float last_v = s_last_v;
    const int last_i = s_last_i;
    ArgMax best{-INFINITY, 0x7fffffff};
    for (int i = threadIdx.x; i < vocab; i += BLOCK) {
      const float v = row[i];
      if (v < last_v || (v == last_v && i > last_i)) best = better(best, ArgMax{v, i});
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      best = better(best, ArgMax{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
    __syncthreads();                      // the last round's readers of s_f / s_i are done
    if (lane == 0) { s_f[warp] = best.v; s_i[warp] = best.i; }
    __syncthreads();
    if (threadIdx.x == 0) {
      ArgMax a{s_f[0], s_i[0]};
      for (int w = 1; w < BLOCK / 32; ++w) a = better(a, ArgMax{s_f[w], s_i[w]});
      const bool any = a.i != 0x7fffffff;  // fewer than k entries in the row: the rest is marked -1
      out_ids[(int64_t)b * (k + 1) + 1 + j] = any ? a.i : -1;
      out_lp[(int64_t)b * (k + 1) + 1 + j] = any ? a.v - s_lse : -INFINITY;
      s_last_v = any ? a.v : -INFINITY;
      s_last_i = any ? a.i : 0x7fffffff;
    }
    __syncthreads();
  }
}

template <typename... KArgs, typename... Args>
int launch_rows(void (*kernel)(KArgs...), int rows, int threads, size_t smem, cudaStream_t stream, const char* what, Args... args) {
  cudaError_t e = launch_pdl_cluster(kernel, dim3(rows * ROW_CTAS), dim3(threads), dim3(ROW_CTAS, 1, 1), smem, stream, args...);
  if (e != cudaSuccess) return refuse((int)e, "%s: launch failed: %s", what, cudaGetErrorString(e));
  return cuda_status(what);
}

}  // namespace

DINFER_DEFINE_LAST_ERROR()

DINFER_API int dinfer_argmax(const float* logits, int64_t ld, int* out, int rows, int vocab, cudaStream_t stream) {
  if (rows < 0 || vocab <= 0 || ld < vocab) return refuse(DINFER_BAD_ARGUMENT, "argmax: bad sizes rows=%d vocab=%d", rows, vocab);
  if (rows == 0) return 0;
  if (rows >= ARGMAX_MANY_ROWS) {
    cudaError_t e = launch_pdl(argmax_many_kernel, dim3(rows), dim3(BLOCK), 0, stream, logits, ld, out, vocab);
    if (e != cudaSuccess) return refuse((int)e, "argmax: launch failed: %s", cudaGetErrorString(e));
    return cuda_status("argmax");
  }
  return launch_rows(argmax_kernel, rows, BLOCK, 0, stream, "argmax", logits, ld, out, vocab);
}

// temperature [rows]; top_k (<=0: off), top_p, min_p may be null; seeds, offsets [rows] uint64.
DINFER_API int dinfer_sample(const float* logits, int64_t ld, const float* temperature, const int* top_k,
                             const float* top_p, const float* min_p, const uint64_t* seeds,
                             const uint64_t* offsets, int* out, int rows, int vocab, cudaStream_t stream) {
  if (rows < 0 || vocab <= 0 || ld < vocab) return refuse(DINFER_BAD_ARGUMENT, "sample: bad sizes rows=%d vocab=%d", rows, vocab);
  if (rows == 0) return 0;
  // a row slice that fits shared memory is kept there (read once); a longer one is read again every pass
  const int per = (vocab + ROW_CTAS - 1) / ROW_CTAS;
  const int cache_slice = per <= MAX_SLICE ? 1 : 0;
  size_t smem = cache_slice ? (size_t)per * sizeof(float) : 0;
  static bool opted = false;
  static int lone_rows = 0;                              // rows whose CTAs all run at once with an SM each
  if (!opted) {
    cudaError_t e = cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SLICE * (int)sizeof(float));
    if (e != cudaSuccess) return refuse((int)e, "sample: shared memory opt-in failed: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(64 * ROW_CTAS); cfg.blockDim = dim3(NT); cfg.dynamicSmemBytes = LONE_SMEM;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = ROW_CTAS; cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    cfg.attrs = &cluster; cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&lone_rows, sample_kernel, &cfg);
    if (e != cudaSuccess) return refuse((int)e, "sample: cluster occupancy query failed: %s", cudaGetErrorString(e));
    opted = true;
  }
  if (rows <= lone_rows && smem < LONE_SMEM) smem = LONE_SMEM;
  return launch_rows(sample_kernel, rows, NT, smem, stream, "sample", logits, ld, temperature, top_k, top_p, min_p, seeds,
                     offsets, out, vocab, cache_slice);
}

DINFER_API int dinfer_penalties(float* logits, int64_t ld, const int* ids, const int* offsets,
                                const int* prompt_len, const float* rep, const float* freq, const float* pres,
                                int rows, int vocab, cudaStream_t stream) {
  if (rows < 0 || vocab <= 0 || ld < vocab) return refuse(DINFER_BAD_ARGUMENT, "penalties: bad sizes rows=%d vocab=%d", rows, vocab);
  if (rows == 0) return 0;
  penalties_kernel<<<rows, 256, 0, stream>>>(logits, ld, ids, offsets, prompt_len, rep, freq, pres, vocab);
  return cuda_status("penalties");
}

// rows, ids, bias [n]: logits[rows[i], ids[i]] += bias[i] (the reference adds its logit_bias before the penalties:
// crates/core/src/sample.rs:104-106).
DINFER_API int dinfer_logit_bias(float* logits, int64_t ld, const int* rows, const int* ids, const float* bias, int n,
                                 int vocab, cudaStream_t stream) {
  if (n < 0 || vocab <= 0 || ld < vocab) return refuse(DINFER_BAD_ARGUMENT, "logit_bias: bad sizes n=%d vocab=%d", n, vocab);
  if (n == 0) return 0;
  logit_bias_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logits, ld, rows, ids, bias, n, vocab);
  return cuda_status("logit_bias");
}

// chosen [rows]; out_ids, out_lp [rows, k + 1]: column 0 the chosen token, then the k most likely, descending;
// out_rank [rows]: tokens strictly more likely than the chosen one (crates/kernels/cuda/sampling.cu:381-430).
DINFER_API int dinfer_logprobs(const float* logits, int64_t ld, const int* chosen, int k, int* out_ids, float* out_lp,
                               int* out_rank, int rows, int vocab, cudaStream_t stream) {
  if (rows < 0 || vocab <= 0 || ld < vocab) return refuse(DINFER_BAD_ARGUMENT, "logprobs: bad sizes rows=%d vocab=%d", rows, vocab);
  if (k < 0 || k > LP_MAX_K) return refuse(DINFER_BAD_ARGUMENT, "logprobs: k must be in [0, %d], got %d", LP_MAX_K, k);
  if (rows == 0) return 0;
  logprobs_kernel<<<rows, BLOCK, 0, stream>>>(logits, ld, chosen, k, out_ids, out_lp, out_rank, vocab);
  return cuda_status("logprobs");
}
