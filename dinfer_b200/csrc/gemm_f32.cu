// C[M, N] = A[M, K] * W[N, K]^T to 32-bit accuracy: the matrix product of the true 32-bit model (no reduced-precision matrix
// mode), and of a bfloat16 model whose file stores a matrix in 32-bit.  A, W and C may each be f32 or bf16 in memory.  Any M,
// N, K.
//
// Three kernels: a tiled one for prompts, on the tensor cores with every 32-bit element taken as three bfloat16 parts
// (split_umma.cuh), and with plain 32-bit multiply-adds a tiled one for short sums and a warp-per-output-column one for the few rows
// of a decode step.  The reference has no 32-bit
// path (its weights are bf16 and its products cuBLASLt: crates/kernels/src/gemm.rs:649-690).
#include "split_umma.cuh"

using namespace dinfer;
using namespace dinfer_umma;
using namespace dinfer_split;

namespace {

constexpr int BN = 128, BK = 32;               // weight rows of a tile (the MMA's rows); k per stage
constexpr int BT = 112;                        // tokens of a tile at most (the MMA's columns, a multiple of 16)
constexpr int STAGES = 3, RAW_STAGES = 4;      // stages of split operands, with an accumulator each; stages of operands as they lie in memory
constexpr int EPI_WARPS = 8, MMA_WARPS = 2, CONV_WARPS = 4, GROUPS = 2;   // warp roles: sums, MMA issue, splitting (a group of warps a stage), TMA
constexpr int MMA_WARP = EPI_WARPS, CONV_WARP = MMA_WARP + MMA_WARPS, TMA_WARP = CONV_WARP + CONV_WARPS * GROUPS;
constexpr int CONV_THREADS = CONV_WARPS * 32;
constexpr int TILE_THREADS = (TMA_WARP + 1) * 32;
constexpr int PIECES = BK / 8;                 // pieces of eight k in a row of a stage
constexpr int UNITS = (BT * PIECES + CONV_THREADS - 1) / CONV_THREADS;   // pieces of the tokens' rows that a thread splits at most
constexpr int ROW_STEP = CONV_THREADS / PIECES;     // rows between them
constexpr int W_COLS = PARTS * BK / 2;         // columns of tensor memory that a stage's split weights take
constexpr int TMEM_COLS = 512;                 // STAGES * (BT + W_COLS), rounded to a power of two
static_assert(STAGES * (BT + W_COLS) <= TMEM_COLS, "tensor memory");
constexpr int HALF = (BT / 2 + 15) / 16 * 16;  // columns of the sums that a warp has at most
constexpr int LDC_S = BN + 4;                  // row stride of the partial tile [token][weight row]
constexpr int MAX_SPLITS = 8;                  // CTAs that may share a tile's K (a portable cluster)
constexpr int MAX_ROWS = 65535 * 128;          // rows of one product

__device__ __forceinline__ float4 ld_cluster_f4(const float* local, uint32_t rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(map_to_rank(smem_u32(local), rank)) : "memory");
  return v;
}

// bfloat16 elements are one part, 32-bit ones three
template <typename T> constexpr int parts_of() { return sizeof(T) == 4 ? PARTS : 1; }
template <typename T> constexpr float unscale() { return sizeof(T) == 4 ? UNSCALE : 1.f; }
template <typename T> constexpr uint32_t raw_row() { return BK * sizeof(T); }
// Eight k of row r from a stage as TMA has laid it down: rows of 128 bytes with the 128-byte swizzle (32-bit), of 64 with the
// 64-byte one (bfloat16)
template <typename T> struct Piece { uint4 v[sizeof(T) / 2]; };
template <typename T>
__device__ __forceinline__ Piece<T> raw_piece(uint32_t raw, int r, int c) {
  Piece<T> p;
  if constexpr (sizeof(T) == 4) {
    p.v[0] = ld_shared16(raw + swizzled128(r, 2 * c));
    p.v[1] = ld_shared16(raw + swizzled128(r, 2 * c + 1));
  } else {
    p.v[0] = ld_shared16(raw + swizzled64(r, c));
  }
  return p;
}
// the same element by element from memory, for rows that TMA cannot address; zeros from `k_end` on
template <typename T>
__device__ __forceinline__ Piece<T> load_piece(const T* __restrict__ row, bool live, int k, int k_end) {
  alignas(16) T e[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) e[i] = live && k + i < k_end ? row[k + i] : from_f32<T>(0.f);
  return *reinterpret_cast<const Piece<T>*>(e);
}
template <typename T, bool FAST>
__device__ __forceinline__ void split_piece(const Piece<T>& p, uint4 (&q)[PARTS]) {
  if constexpr (sizeof(T) == 4) {
    float x[8] = {__uint_as_float(p.v[0].x), __uint_as_float(p.v[0].y), __uint_as_float(p.v[0].z), __uint_as_float(p.v[0].w),
                  __uint_as_float(p.v[1].x), __uint_as_float(p.v[1].y), __uint_as_float(p.v[1].z), __uint_as_float(p.v[1].w)};
    if (!FAST)                                     // (apart: in pairs they would cost that kernel its last registers)
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] *= SCALE;
    split8<FAST>(x, q);
  } else {
    q[0] = p.v[0];
  }
}

// one element again, k after k, for results that are not finite (a sum that is not a number stays one)
template <typename TA, typename TW>
__device__ __noinline__ float plain_sum(const TA* __restrict__ a, const TW* __restrict__ w, int K) {
  float s = 0.f;
  for (int k = 0; k < K && s == s; ++k) s = fmaf(to_f32<TA>(a[k]), to_f32<TW>(w[k]), s);
  return s;
}
__device__ __forceinline__ bool not_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) == 0x7f800000u; }

constexpr size_t MAX_SMEM = 227 * 1024 - 256;               // (the barriers are static)
struct TileParams {
  int64_t lda, ldw, ldc, sa, sw, sc;
  int M, N, K, bt, splits, c_fast;
  int* status;
};

// a stage of split tokens, a stage as it lies in memory (multiples of 1024 bytes: bt is one of 16)
template <typename TA> __host__ __device__ constexpr uint32_t stage_bytes(int bt) { return (uint32_t)(parts_of<TA>() * bt) * BK * 2; }
template <typename TA, typename TW> __host__ __device__ constexpr uint32_t raw_bytes(int bt) {
  return BN * raw_row<TW>() + (uint32_t)bt * raw_row<TA>();
}
// Dynamic shared memory of a launch.  Where CTAs share K they wait for one another, and all of tensor memory is one CTA's: two of them on
// one SM, each ahead of the other's partner on another SM, would wait for good.  So such a CTA takes an SM's shared memory for
// itself (more than half of it), however small its tile is; the others only wait for a CTA in front to end.
constexpr size_t ALONE = 115 * 1024;
template <typename TA, typename TW> __host__ constexpr size_t tile_shared(int bt, int splits) {
  const size_t stages = (size_t)STAGES * stage_bytes<TA>(bt) + RAW_STAGES * raw_bytes<TA, TW>(bt), part = (size_t)bt * LDC_S * 4;
  const size_t own = (stages > part ? stages : part) + 1024;
  return splits > 1 && own < ALONE ? ALONE : own;
}
static_assert(2 * ALONE > 228 * 1024 && ALONE <= MAX_SMEM, "one CTA to an SM");
static_assert(tile_shared<float, float>(BT, 1) <= MAX_SMEM, "fits a CTA");

// The tile kernel: 128 weight rows (the MMA's rows) by up to 112 tokens (its columns, as many as the rows make even tiles of),
// 32 k a stage.  FAST: TMA fetches both operands as they lie in memory (16-byte rows), else the splitting warps read them
// element by element.  Two groups of four warps split a stage in turn: weights to tensor memory (the MMA's A operand), tokens
// to shared memory, which six MMAs a 16 k would otherwise be bound by (both from shared memory: 128 bytes a cycle of its 128).
// A stage's sums leave tensor memory at once and are added in registers, rounded to nearest: the MMA's own sums are cut off, and
// over a whole K that would cost more digits than the parts keep.
//
// Bound by a chain of roles rather than by one of them: while an SM runs, its tensor pipe is busy 41 % of the time and its issue slots
// 59 % (the splits; ncu, 333 x 6144 x 1024), the rest is waits from hand-over to hand-over.  333 x 6144 x 1024 29.8 us (140 TFLOP/s),
// 333 x 1024 x 3072 22.3, 2048 x 6144 x 1024 197; as 64 x 128 tiles of packed 32-bit multiply-adds 129, 81 and 663.  Smaller ones
// gain as well: 100 x 2048 x 1024 12.3 us for 23.8, 33 x 64 x 4096 13.6 for 38.6; rows that TMA cannot address 333 x 6144 x 1030 55 for
// 213, 2048 x 64 x 2045 21 for 61.  Not so where a second round of tiles is nearly empty: 2048 x 1024 x 64 13.5 for 12.0.
//
// Relative errors against 64 bits (2-norm) beside those of the multiply-adds, operands of both signs: K 64 6.2e-8 for 1.1e-7, 1024
// 1.2e-7 for 4.1e-7 (where eight CTAs share K 8.8e-8 for 1.6e-7), 4096 1.1e-7 for 2.9e-7; two bfloat16 operands, whose products are exact,
// K 64 4.7e-8 for 4.3e-8, 512 7.3e-8 for 7.1e-8, from 768 on less.  The MMA cuts its sums off towards zero, and where all products
// have one sign that adds up: K 1024 shared by CTAs 7.2e-8 for 6.0e-8, bfloat16 operands K 512 5.8e-8 for 4.0e-8.
template <typename TA, typename TW, typename TC, bool FAST>
__global__ void __launch_bounds__(TILE_THREADS, 1)
gemm_tile_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const TA* __restrict__ A,
                 const TW* __restrict__ W, TC* __restrict__ C, const TileParams p) {
  extern __shared__ unsigned char smem_dyn[];
  __shared__ __align__(8) uint64_t full_bar[STAGES], free_bar[STAGES], read_bar[STAGES], raw_full[RAW_STAGES], raw_free[RAW_STAGES];
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  const int z = blockIdx.z / p.splits, rank = blockIdx.z % p.splits;
  A += (int64_t)z * p.sa; W += (int64_t)z * p.sw; C += (int64_t)z * p.sc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, bt = p.bt;
  const int n_tiles = (p.N + BN - 1) / BN, t0 = (int)(blockIdx.x / n_tiles) * bt, n0 = (int)(blockIdx.x % n_tiles) * BN;
  const int k_blocks = (p.K + BK - 1) / BK;
  const int first = (int)((int64_t)k_blocks * rank / p.splits), last = (int)((int64_t)k_blocks * (rank + 1) / p.splits);
  const int n_st = last - first;
  const uint32_t a_part = (uint32_t)bt * BK * 2, st_bytes = stage_bytes<TA>(bt), raw = base + STAGES * st_bytes;
  float* partial = reinterpret_cast<float*>(smem_dyn + (base - smem_u32(smem_dyn)));

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), CONV_WARPS);
      mbar_init(smem_u32(&free_bar[s]), 1);
      mbar_init(smem_u32(&read_bar[s]), EPI_WARPS);
    }
    for (int s = 0; s < RAW_STAGES; ++s) {
      mbar_init(smem_u32(&raw_full[s]), 1);
      mbar_init(smem_u32(&raw_free[s]), CONV_WARPS);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_enter();                                                  // (dependents start only now that the tensor memory is ours)
  const uint32_t tmem = s_tmem;

  if (warp == TMA_WARP) {
    if (FAST && lane == 0) {                                   // ---- operands as they lie in memory
      for (int j = 0; j < n_st; ++j) {
        const int s = j % RAW_STAGES;
        if (!mbar_wait(smem_u32(&raw_free[s]), ((j / RAW_STAGES) & 1) ^ 1)) { s_abort = 1; atomicExch(p.status, 44); break; }
        const uint32_t at = raw + s * raw_bytes<TA, TW>(bt), bar = smem_u32(&raw_full[s]);
        mbar_expect_tx(bar, raw_bytes<TA, TW>(bt));
        tma_load_3d(at, &map_w, (first + j) * BK, n0, z, bar);
        tma_load_3d(at + BN * raw_row<TW>(), &map_a, (first + j) * BK, t0, z, bar);
      }
    }
  } else if (warp >= CONV_WARP) {                               // ---- splits: weights to tensor memory, tokens to shared memory
    const int group = (warp - CONV_WARP) / CONV_WARPS, me = (tid - CONV_WARP * 32) % CONV_THREADS;
    const int c = me % PIECES, r = me / PIECES, row = (warp & 3) * 32 + lane;
    const uint32_t w_at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + STAGES * BT;
    const TW* w_row = W + (int64_t)(n0 + row) * p.ldw;
    for (int j = group; j < n_st; j += GROUPS) {
      const int s = j % STAGES, rs = j % RAW_STAGES, k0 = (first + j) * BK;
      const uint32_t at = raw + rs * raw_bytes<TA, TW>(bt), at_a = at + BN * raw_row<TW>(), ta = base + s * st_bytes;
      if (FAST && !mbar_wait(smem_u32(&raw_full[rs]), (j / RAW_STAGES) & 1)) { s_abort = 1; atomicExch(p.status, 45); break; }
      // (all loads of an operand ahead of its first split: one latency instead of four)
      Piece<TW> w[PIECES];
#pragma unroll
      for (int i = 0; i < PIECES; ++i)
        w[i] = FAST ? raw_piece<TW>(at, row, i) : load_piece<TW>(w_row, n0 + row < p.N, k0 + i * 8, p.K);
      if (!mbar_wait(smem_u32(&free_bar[s]), ((j / STAGES) & 1) ^ 1)) { s_abort = 1; atomicExch(p.status, 41); break; }
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < PIECES; i += 2) {
        uint4 q[2][PARTS];
        split_piece<TW, FAST>(w[i], q[0]);
        split_piece<TW, FAST>(w[i + 1], q[1]);
#pragma unroll
        for (int e = 0; e < parts_of<TW>(); ++e) tmem_st8(w_at + s * W_COLS + e * (BK / 2) + i * 4, q[0][e], q[1][e]);
      }
      Piece<TA> x[UNITS];
#pragma unroll
      for (int i = 0; i < UNITS; ++i) {
        const int ra = r + i * ROW_STEP;
        if (ra < bt)
          x[i] = FAST ? raw_piece<TA>(at_a, ra, c) : load_piece<TA>(A + (int64_t)(t0 + ra) * p.lda, t0 + ra < p.M, k0 + c * 8, p.K);
      }
#pragma unroll
      for (int i = 0; i < UNITS; ++i) {
        const int ra = r + i * ROW_STEP;
        if (ra < bt) {
          uint4 q[PARTS];
          split_piece<TA, FAST>(x[i], q);
#pragma unroll
          for (int e = 0; e < parts_of<TA>(); ++e) st_shared16(ta + e * a_part + swizzled64(ra, c), q[e]);
        }
      }
      tmem_st_wait();
      fence_to_mma();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (FAST) mbar_arrive(smem_u32(&raw_free[rs]));
        mbar_arrive(smem_u32(&full_bar[s]));
      }
    }
  } else if (warp >= MMA_WARP) {
    // ---- MMA issue.  Two warps take turns, so that one waits (some 300 cycles a barrier, met or not) while the other's MMAs
    // run: one warp took 1450 cycles a stage whose MMAs take 670.
    const uint32_t idesc = idesc_bf16(BN, bt, 0), lead = elect_lane(), tm = uniform(tmem);
    const uint64_t da0 = desc_k_major64(base);
    for (int j = (int)uniform(warp) - MMA_WARP; j < n_st; j += MMA_WARPS) {
      const int s = j % STAGES;
      if (!mbar_spin(smem_u32(&read_bar[s]), ((j / STAGES) & 1) ^ 1) || !mbar_spin(smem_u32(&full_bar[s]), (j / STAGES) & 1)) {
        s_abort = 1; atomicExch(p.status, 42);
        break;
      }
      tc_fence_after();
      const uint64_t da = da0 + s * (st_bytes >> 4);
      const uint32_t tw = tm + STAGES * BT + s * W_COLS;
      uint32_t accumulate = 0;
#pragma unroll
      for (int i = 0; i < PRODUCTS; ++i) {
        if (part_a(i) >= parts_of<TW>() || part_b(i) >= parts_of<TA>()) continue;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {                     // 16 k: eight columns, 32 bytes (in 16-byte units)
          mma_ts_if(lead, tm + s * BT, tw + part_a(i) * (BK / 2) + 8 * k, da + part_b(i) * (a_part >> 4) + 2 * k, idesc, accumulate);
          accumulate = 1;
        }
      }
      commit_if(lead, smem_u32(&free_bar[s]));                  // the stage is free, its sums are there
    }
  } else {                                                      // ---- a stage's sums leave tensor memory
    // warps 0-3 and 4-7 have half of the tile's columns each; TMEM lanes by warp mod 4
    const int half = warp >> 2, row = (warp & 3) * 32 + lane;
    const int cols = ((bt / 2) + 15) / 16 * 16, c_begin = half * cols, c_end = min(bt, c_begin + cols);
    const uint32_t acc_at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + c_begin;
    uint64_t acc2[HALF / 2];
#pragma unroll
    for (int i = 0; i < HALF / 2; ++i) acc2[i] = 0ull;
    bool ok = true;
    uint32_t s = 0, s_phase = 0;
    for (int j = 0; j < n_st; ++j) {
      ok = mbar_wait(smem_u32(free_bar) + 8 * s, s_phase);
      if (!ok) { s_abort = 1; atomicExch(p.status, 43); break; }
      tc_fence_after();
#pragma unroll
      for (int c0 = 0; c0 < HALF; c0 += 16) {
        if (c_begin + c0 < c_end) {
          uint32_t v[16];
          tmem_ld16(acc_at + s * BT + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int u = 0; u < 16; u += 2)
            acc2[(c0 + u) / 2] = add2(acc2[(c0 + u) / 2], (uint64_t)v[u] | ((uint64_t)v[u + 1] << 32));
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(read_bar) + 8 * s);
      if (++s == STAGES) { s = 0; s_phase ^= 1; }
    }
    if (ok) {
      float acc[HALF];
#pragma unroll
      for (int i = 0; i < HALF; ++i) acc[i] = __uint_as_float((uint32_t)(acc2[i / 2] >> (32 * (i & 1)))) * (unscale<TA>() * unscale<TW>());
      if (p.splits > 1) {                                       // the stages' memory takes the partial tile
#pragma unroll
        for (int i = 0; i < HALF; ++i)
          if (c_begin + i < c_end) partial[(c_begin + i) * LDC_S + row] = acc[i];
      } else {
        const int n = n0 + row, count = min(c_end, p.M - t0) - c_begin;
        if (n < p.N) {
          TC* dst = C + (int64_t)(t0 + c_begin) * p.ldc + n;
          bool finite = true;
#pragma unroll
          for (int i = 0; i < HALF; ++i)
            if (i < count) {
              dst[i * p.ldc] = from_f32<TC>(acc[i]);
              finite = finite && !not_finite(acc[i]);
            }
          if (!finite) {                                        // (read back: a loop over registers by number would spill them)
            for (int i = 0; i < count; ++i)
              if (not_finite(to_f32<TC>(dst[i * p.ldc])))
                dst[i * p.ldc] = from_f32<TC>(plain_sum<TA, TW>(A + (int64_t)(t0 + c_begin + i) * p.lda, W + (int64_t)n * p.ldw, p.K));
          }
        }
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  if (p.splits > 1) {
    cluster_sync_all();
    // all fold the tile in split order, a share of it each
    if (!s_abort) {
      for (int v = rank * TILE_THREADS + tid; v < bt * (BN / 4); v += p.splits * TILE_THREADS) {
        const int r = v / (BN / 4), c = (v % (BN / 4)) * 4;
        const int t = t0 + r, n = n0 + c;
        if (t >= p.M || n >= p.N) continue;
        const float* own = partial + r * LDC_S + c;
        float4 f = ld_cluster_f4(own, 0);
        for (int q = 1; q < p.splits; ++q) {
          const float4 u = ld_cluster_f4(own, q);
          f.x += u.x; f.y += u.y; f.z += u.z; f.w += u.w;
        }
        float e[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (n + u < p.N && not_finite(e[u])) e[u] = plain_sum<TA, TW>(A + (int64_t)t * p.lda, W + (int64_t)(n + u) * p.ldw, p.K);
        TC* dst = C + (int64_t)t * p.ldc + n;
        if (p.c_fast && n + 3 < p.N) {
          if constexpr (sizeof(TC) == 4) {
            *reinterpret_cast<float4*>(dst) = make_float4(e[0], e[1], e[2], e[3]);
          } else {
            __nv_bfloat162 h[2] = {__floats2bfloat162_rn(e[0], e[1]), __floats2bfloat162_rn(e[2], e[3])};
            *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
          }
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (n + u < p.N) dst[u] = from_f32<TC>(e[u]);
        }
      }
    }
    cluster_sync_all();                                         // nobody leaves while others may still read its share
  } else {
    __syncthreads();
  }
  if (warp == MMA_WARP) {
    if (s_abort) {                                              // MMAs in flight land
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// ---- short sums: 64 x 128 tiles of packed 32-bit multiply-adds, all of K in shared memory at once.  Four warps own 32 x 64 of the
// tile each, a lane 8 x 8 (rows ly + 4 i, columns lx + 8 j), and a multiply-add works on two k (even and odd k have a sum of
// their own), so that operands are used as they lie: 16 16-byte loads feed 128 packed multiply-adds.  Bound by one way to
// memory and back; what the tiles above take ahead of their first MMA and behind their last is longer than these sums (times at the
// rule).
constexpr int SHORT_M = 64, SHORT_N = 128, SHORT_THREADS = 128, SHORT_TILE_K = 48;
constexpr int LDK = SHORT_TILE_K + 4;          // row stride of a staged operand: eight rows' 16-byte pieces of one k lie in different banks
constexpr int LDC_SHORT = SHORT_N + 8;
static_assert(SHORT_M * LDC_SHORT <= (SHORT_M + SHORT_N) * LDK, "the result takes the operands' place");

__device__ __forceinline__ void fma2(uint64_t& c, uint64_t a, uint64_t b, bool first) {       // two multiply-adds, each rounded once
  if (first) asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  else asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
// rows [r0, r0 + ROWS) of an operand as [row][k], zeros beyond `rows` and K (a multiple of four is filled); fast: four elements a load
template <typename T, int ROWS>
__device__ __forceinline__ void stage_short(float* dst, const T* __restrict__ src, int64_t ld, int r0, int rows, int K, bool fast) {
  const int pieces = (K + 3) / 4;
  if (fast) {
#pragma unroll 4
    for (int i = threadIdx.x; i < ROWS * pieces; i += SHORT_THREADS) {
      const int r = i / pieces, k = (i % pieces) * 4;
      const bool live = r0 + r < rows;
      const T* p = src + (live ? (int64_t)(r0 + r) * ld + k : 0);
      if constexpr (sizeof(T) == 4) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * LDK + k)), "l"(p), "r"(live ? 16 : 0) : "memory");
      } else {
        const uint2 u = live ? *reinterpret_cast<const uint2*>(p) : make_uint2(0u, 0u);
        *reinterpret_cast<float4*>(dst + r * LDK + k) = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u),
                                                                    __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
      }
    }
    return;
  }
#pragma unroll 4
  for (int i = threadIdx.x; i < ROWS * pieces * 4; i += SHORT_THREADS) {
    const int r = i / (pieces * 4), k = i % (pieces * 4);
    dst[r * LDK + k] = r0 + r < rows && k < K ? to_f32<T>(src[(int64_t)(r0 + r) * ld + k]) : 0.f;
  }
}
template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(SHORT_THREADS, 2)
gemm_short_kernel(const TA* __restrict__ A, int64_t lda, const TW* __restrict__ W, int64_t ldw, TC* __restrict__ C, int64_t ldc, int M,
                  int N, int K, int64_t sa, int64_t sw, int64_t sc, int a_fast, int w_fast, int c_fast) {
  __shared__ __align__(16) float sm[(SHORT_M + SHORT_N) * LDK];
  A += (int64_t)blockIdx.z * sa; W += (int64_t)blockIdx.z * sw; C += (int64_t)blockIdx.z * sc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, m0 = blockIdx.y * SHORT_M, n0 = blockIdx.x * SHORT_N;
  // (lanes 0-7 and 8-15 read the two halves of the columns' pieces: 16 lanes' 16-byte loads then take one pass over the banks)
  const int ly = ((lane >> 2) & 1) | (lane >> 4 << 1), lx = (lane & 3) | ((lane >> 3 & 1) << 2);
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 64;
  stage_short<TA, SHORT_M>(sm, A, lda, m0, M, K, a_fast);
  stage_short<TW, SHORT_N>(sm + SHORT_M * LDK, W, ldw, n0, N, K, w_fast);
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float sum[8][8] = {};
  const float* as = sm + (wr + ly) * LDK;
  const float* ws = sm + (SHORT_M + wc + lx) * LDK;
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 8) {               // (sums of eight, then of those: 0.7 of the error of one sum in order)
    uint64_t acc[8][8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = k0 + 4 * h;
      if (h && k >= K) break;
      ulonglong2 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + 4 * i * LDK + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + 8 * j * LDK + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].x, b.x, h == 0);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].y, b.y, false);    // (a sum's two steps apart: the first takes a while)
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        sum[i][j] += __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) sm[(wr + ly + 4 * i) * LDC_SHORT + wc + lx + 8 * j] = sum[i][j];
  __syncthreads();
  for (int v = tid; v < SHORT_M * (SHORT_N / 4); v += SHORT_THREADS) {
    const int r = v / (SHORT_N / 4), c = (v % (SHORT_N / 4)) * 4, n = n0 + c;
    if (m0 + r >= M || n >= N) continue;
    const float4 t = *reinterpret_cast<const float4*>(sm + r * LDC_SHORT + c);
    const float e[4] = {t.x, t.y, t.z, t.w};
    TC* dst = C + (int64_t)(m0 + r) * ldc + n;
    if (c_fast && n + 3 < N) {
      if constexpr (sizeof(TC) == 4) {
        *reinterpret_cast<float4*>(dst) = t;
      } else {
        __nv_bfloat162 h[2] = {__floats2bfloat162_rn(e[0], e[1]), __floats2bfloat162_rn(e[2], e[3])};
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (n + u < N) dst[u] = from_f32<TC>(e[u]);
    }
  }
}

// The sums over the lanes of acc[m] to C[m * ldc], m < M.  32 rows are halved from step to step, a lane keeping the half with
// its own bit: 31 exchanges instead of 160, the same additions.
template <typename TC, int ROWS>
__device__ __forceinline__ void store_rows(float (&acc)[ROWS], TC* C, int64_t ldc, int M, int lane) {
  if constexpr (ROWS == 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const bool up = lane & o;
        const float send = up ? acc[i] : acc[i + o], keep = up ? acc[i + o] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    if (lane < M) C[(int64_t)lane * ldc] = from_f32<TC>(acc[0]);
  } else {
#pragma unroll
    for (int m = 0; m < ROWS; ++m) {
      const float s = warp_sum(acc[m]);
      if (lane == 0 && m < M) C[(int64_t)m * ldc] = from_f32<TC>(s);
    }
  }
}

// M <= ROWS rows, or with BLOCKS any number in blocks of ROWS (grid.y): one warp per output column n; lanes stride over K, the weight
// row is read once a block.  (Rows counted from blockIdx, not from a parameter: two rows of a 32-bit feed-forward took 94 us instead of 57.)
template <typename TA, typename TW, typename TC, int ROWS, bool BLOCKS = false>
__global__ void __launch_bounds__(256)
gemm_rows_kernel(const TA* __restrict__ A, int64_t lda, const TW* __restrict__ W, int64_t ldw,
                 TC* __restrict__ C, int64_t ldc, int M, int N, int K, int64_t sa, int64_t sw, int64_t sc) {
  A += (int64_t)blockIdx.z * sa; W += (int64_t)blockIdx.z * sw; C += (int64_t)blockIdx.z * sc;
  if constexpr (BLOCKS) {
    A += (int64_t)blockIdx.y * ROWS * lda;
    C += (int64_t)blockIdx.y * ROWS * ldc;
    M = min(ROWS, M - (int)blockIdx.y * ROWS);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * 8 + warp;
  if (n >= N) return;
  const TW* w = W + (int64_t)n * ldw;
  float acc[ROWS];
#pragma unroll
  for (int m = 0; m < ROWS; ++m) acc[m] = 0.f;
  for (int k = lane; k < K; k += 32) {
    const float wv = to_f32<TW>(w[k]);
#pragma unroll
    for (int m = 0; m < ROWS; ++m)
      if (m < M) acc[m] = fmaf(to_f32<TA>(A[(int64_t)m * lda + k]), wv, acc[m]);
  }
  store_rows<TC, ROWS>(acc, C + n, ldc, M, lane);
}

// The same for bfloat16 operands whose rows are 16-byte aligned (K a multiple of 8): every lane takes eight
// consecutive k at once (one 16-byte load of the weight row and one of each A row), four output columns per block,
// so a small K still fills the machine with loads in flight.  Products and sums are 32-bit.
template <typename TC, int ROWS>
__global__ void __launch_bounds__(128)
gemm_rows_bf16x8_kernel(const __nv_bfloat16* __restrict__ A, int64_t lda, const __nv_bfloat16* __restrict__ W, int64_t ldw,
                        TC* __restrict__ C, int64_t ldc, int M, int N, int K, int64_t sa, int64_t sw, int64_t sc) {
  A += (int64_t)blockIdx.z * sa; W += (int64_t)blockIdx.z * sw; C += (int64_t)blockIdx.z * sc;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * 4 + warp;
  if (n >= N) return;
  const __nv_bfloat16* w = W + (int64_t)n * ldw;
  float acc[ROWS];
#pragma unroll
  for (int m = 0; m < ROWS; ++m) acc[m] = 0.f;
  for (int k = lane * 8; k < K; k += 256) {
    const uint4 wv = *reinterpret_cast<const uint4*>(w + k);
    const __nv_bfloat162* wp = reinterpret_cast<const __nv_bfloat162*>(&wv);
    float wf[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(wp[j]); wf[2 * j] = f.x; wf[2 * j + 1] = f.y; }
#pragma unroll
    for (int m = 0; m < ROWS; ++m) {
      if (m < M) {
        const uint4 av = *reinterpret_cast<const uint4*>(A + (int64_t)m * lda + k);
        const __nv_bfloat162* ap = reinterpret_cast<const __nv_bfloat162*>(&av);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(ap[j]);
          acc[m] = fmaf(f.x, wf[2 * j], acc[m]);
          acc[m] = fmaf(f.y, wf[2 * j + 1], acc[m]);
        }
      }
    }
  }
  store_rows<TC, ROWS>(acc, C + n, ldc, M, lane);
}

// A matrix up to which 9 to 32 rows go a warp per output column: one tile or a few leave the SMs idle.  us on a tile and so, 9
// and 32 rows in 32-bit (back to back in a graph): N 48 K 48 4.6 and 2.9, 5.1 and 3.7; N 2048 K 16 5.0 and 2.8, 5.4 and 3.3;
// N 128 K 128 5.5 and 4.8, 6.1 and 6.2; N 2048 K 128 5.9 and 5.5, 6.5 and 7.0; beyond, N 2048 K 192 5.8 and 7.2, 6.4 and 9.6;
// N 4096 K 64 5.1 and 5.7, 5.6 and 6.9.  Errors against 64 bits are alike (7e-8).
constexpr int FEW_ROWS_K = 128, FEW_ROWS_N = 2048;
// Sums up to this long go so beyond 32 rows too, while their blocks (32 rows, 8 columns) are at most three to two SMs: what a tile takes
// ahead of its first MMA and behind its last (5 us) is more than the sums.  us on a tile and so, in 32-bit: 333 x 48 x 16 6.4 and 3.4
// (4.8 on tiles of multiply-adds, as they were), 1000 x 48 x 48 7.3 and 5.3, 200 x 256 x 64 7.0 and 5.4; beyond the line 333 x 256 x
// 16 6.4 and 5.9, x 64 7.0 and 8.2, 100 x 1024 x 64 7.1 and 8.3; longer 1000 x 48 x 96 7.6 and 6.6, 100 x 128 x 128 8.0 and 7.2,
// 2048 x 128 x 128 8.4 and 26; with a bfloat16 operand 64 x 256 x 64 5.1 and 4.8, 33 x 128 x 128 5.6 and 7.3.
constexpr int SHORT_K = 64;
// Beyond those blocks, sums up to which the tiles of multiply-adds are the faster ones: of two 32-bit operands, one, none.  us on the
// tensor cores and so, 333 x 1024, 2048 x 1024 (152 tiles there, two rounds) and 7000 x 128: both 32-bit K 16 6.8 and 4.3, 12.0 and 5.7, 6.9
// and 4.7; K 40 7.5 and 6.4, 13.5 and 9.1, 7.7 and 7.0; one K 16 6.1 and 4.5, 10.7 and
// 5.9, 6.2 and 5.0; K 32 5.9 and 5.8, 10.5 and 7.9, 6.0 and 6.2; K 40 6.4 and 6.7, 11.4 and 9.3, 6.5 and 7.2; none K 16 5.7 and 4.6, 10.4 and
// 6.0, 6.1 and 4.7;
// K 24 5.9 and 5.9, 10.6 and 7.5, 6.2 and 6.0.  Errors against 64 bits are alike (K 4 4.1e-8 for 4.7e-8, K 16 5.6e-8 for 4.8e-8, K 40 6.6e-8 for
// 6.1e-8; bfloat16 operands 2.0e-8 for 2.4e-8).
template <typename TA, typename TW> constexpr int short_tile_k() { return sizeof(TA) + sizeof(TW) == 8 ? 40 : (sizeof(TA) + sizeof(TW) == 6 ? 32 : 16); }
static_assert(short_tile_k<float, float>() <= SHORT_TILE_K, "all of K is staged");

int num_sms() {                                             // of the current device, asked once
  static const int n = [] {
    int dev = 0, v = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

// Clusters of `size` CTAs that run at a time, a CTA to an SM: a cluster stays inside one GPC, so that what a GPC has left over is
// lost (asked once a size, of the current device)
int clusters_resident(int size) {
  static std::atomic<int> known[MAX_SPLITS + 1];
  int n = known[size].load(std::memory_order_relaxed);
  if (n) return n;
  auto k = gemm_tile_kernel<float, float, float, true>;
  const size_t smem = tile_shared<float, float>(BT, size);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(size * num_sms()); cfg.blockDim = dim3(TILE_THREADS); cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = size; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, reinterpret_cast<const void*>(k), &cfg) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = num_sms() / (size + 1);
  }
  known[size].store(n, std::memory_order_relaxed);
  return n;
}

// [batch][rows][K] with row stride ld and `stride` elements between the problems; boxes of BK x box_rows.  false: TMA cannot
// address them (the kernel then reads element by element)
template <typename T>
bool make_map(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int64_t ld, int64_t batch, int64_t stride, int box_rows) {
  static const auto fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
    return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(ok ? f : nullptr);
  }();
  if (!fn || (batch > 1 && stride <= 0)) return false;
  constexpr bool wide = sizeof(T) == 4;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)batch};
  const cuuint64_t strides[2] = {(cuuint64_t)ld * sizeof(T), (cuuint64_t)(batch > 1 ? stride : ld) * sizeof(T)};
  const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1}, step[3] = {1, 1, 1};
  return fn(map, wide ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides,
            box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, wide ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename TA, typename TW> struct both_bf16 { static constexpr bool value = false; };
template <> struct both_bf16<__nv_bfloat16, __nv_bfloat16> { static constexpr bool value = true; };

template <typename TA, typename TW, typename TC>
int launch(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int M, int N,
           int K, int* status, cudaStream_t stream, int batch = 1, int64_t sa = 0, int64_t sw = 0, int64_t sc = 0) {
  if (batch > 65535) return refuse(DINFER_BAD_ARGUMENT, "gemm_f32: batch=%d too large", batch);
  if constexpr (both_bf16<TA, TW>::value) {
    const auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (M <= 32 && (M <= 8 || batch > 1) && K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 && sa % 8 == 0 && sw % 8 == 0 &&
        al(A) && al(W)) {
      const dim3 grid((N + 3) / 4, 1, batch);
      const auto* a = (const __nv_bfloat16*)A;
      const auto* w = (const __nv_bfloat16*)W;
      if (M <= 8) gemm_rows_bf16x8_kernel<TC, 8><<<grid, 128, 0, stream>>>(a, lda, w, ldw, (TC*)C, ldc, M, N, K, sa, sw, sc);
      else if (M <= 16) gemm_rows_bf16x8_kernel<TC, 16><<<grid, 128, 0, stream>>>(a, lda, w, ldw, (TC*)C, ldc, M, N, K, sa, sw, sc);
      else gemm_rows_bf16x8_kernel<TC, 32><<<grid, 128, 0, stream>>>(a, lda, w, ldw, (TC*)C, ldc, M, N, K, sa, sw, sc);
      return cuda_status("gemm_f32");
    }
  }
  if (M <= 8) {
    gemm_rows_kernel<TA, TW, TC, 8><<<dim3((N + 7) / 8, 1, batch), 256, 0, stream>>>(
        (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, sa, sw, sc);
  } else if (M <= 32 && (batch > 1 || (K <= FEW_ROWS_K && N <= FEW_ROWS_N))) {
    // few rows against many small matrices (one per head) or one small one: each weight is read once
    gemm_rows_kernel<TA, TW, TC, 32><<<dim3((N + 7) / 8, 1, batch), 256, 0, stream>>>(
        (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, sa, sw, sc);
  } else if (batch == 1 && K <= SHORT_K && (int64_t)((N + 7) / 8) * ((M + 31) / 32) * 2 <= 3 * num_sms()) {
    gemm_rows_kernel<TA, TW, TC, 32, true><<<dim3((N + 7) / 8, (M + 31) / 32), 256, 0, stream>>>(
        (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, sa, sw, sc);
  } else if (K <= short_tile_k<TA, TW>() && (M + SHORT_M - 1) / SHORT_M <= 65535) {
    const auto fast = [](const void* q, size_t size, int64_t ld, int64_t stride) {
      return (int)((reinterpret_cast<uintptr_t>(q) % (4 * size)) == 0 && ld % 4 == 0 && stride % 4 == 0);
    };
    // (no early start behind the kernel in front: beside its CTAs these share SMs while others idle, 1000 x 1000 x 40 8.3 us for 6.7)
    gemm_short_kernel<TA, TW, TC><<<dim3((N + SHORT_N - 1) / SHORT_N, (M + SHORT_M - 1) / SHORT_M, batch), SHORT_THREADS, 0, stream>>>(
        (const TA*)A, lda, (const TW*)W, ldw, (TC*)C, ldc, M, N, K, sa, sw, sc, fast(A, sizeof(TA), lda, sa) && K % 4 == 0,
        fast(W, sizeof(TW), ldw, sw) && K % 4 == 0, fast(C, sizeof(TC), ldc, sc));
  } else {
    if (!status) return refuse(DINFER_BAD_ARGUMENT, "gemm_f32: a status word is required");
    if (M > MAX_ROWS) return refuse(DINFER_BAD_ARGUMENT, "gemm_f32: M=%d too large", M);
    // as many token tiles as are needed, all of one height
    const int t_tiles = (M + BT - 1) / BT, bt = ((M + t_tiles - 1) / t_tiles + 15) / 16 * 16;
    const int64_t tiles = (int64_t)((N + BN - 1) / BN) * t_tiles * batch;
    if (tiles / batch > 0x7fffffffLL) return refuse(DINFER_BAD_ARGUMENT, "gemm_f32: too many tiles (M=%d N=%d)", M, N);
    // The CTAs that share a tile's K: rounds of clusters that run at once, times a CTA's stages and what a CTA takes besides
    // (some eight stages: the first operands' way, the output; three more for the fold).  333 x 1024 x 3072 is 24 tiles: six
    // CTAs each would fill the SMs, but only five fit into what the GPCs have (24 us, with six 35).
    const int k_blocks = (K + BK - 1) / BK;
    int splits = 1;
    int64_t best = 0;
    for (int n = 1; n <= MAX_SPLITS && n <= k_blocks && (int64_t)batch * n <= 65535; ++n) {
      const int64_t room = n > 1 ? clusters_resident(n) : num_sms();
      const int64_t cost = ((tiles + room - 1) / room) * ((k_blocks + n - 1) / n + 8 + (n > 1 ? 3 : 0));
      if (n == 1 || cost < best) { best = cost; splits = n; }
    }
    const auto fast = [](const void* q, size_t size, int64_t ld, int64_t stride, int piece) {
      return (int)((reinterpret_cast<uintptr_t>(q) % (piece * size)) == 0 && ld % piece == 0 && stride % piece == 0);
    };
    constexpr int EA = 16 / sizeof(TA), EW = 16 / sizeof(TW);
    CUtensorMap ma{}, mw{};
    const bool whole = fast(A, sizeof(TA), lda, sa, EA) && K % EA == 0 && fast(W, sizeof(TW), ldw, sw, EW) && K % EW == 0 &&
                       make_map<TA>(&ma, A, M, K, lda, batch, sa, bt) && make_map<TW>(&mw, W, N, K, ldw, batch, sw, BN);
    const TileParams p{lda, ldw, ldc, sa, sw, sc, M, N, K, bt, splits, fast(C, sizeof(TC), ldc, sc, 4), status};
    auto k = whole ? gemm_tile_kernel<TA, TW, TC, true> : gemm_tile_kernel<TA, TW, TC, false>;
    const size_t smem = tile_shared<TA, TW>(bt, splits);
    static std::atomic<uint64_t> done[2];
    cudaError_t e = allow_shared(k, MAX_SMEM, done[whole]);
    if (e != cudaSuccess) return refuse((int)e, "gemm_f32: shared memory opt-in failed: %s", cudaGetErrorString(e));
    e = launch_pdl_cluster(k, dim3((unsigned)(tiles / batch), 1, batch * splits), dim3(TILE_THREADS), dim3(1, 1, splits), smem, stream,
                           ma, mw, (const TA*)A, (const TW*)W, (TC*)C, p);
    if (e != cudaSuccess) return refuse((int)e, "gemm_f32: launch failed: %s", cudaGetErrorString(e));
  }
  return cuda_status("gemm_f32");
}

}  // namespace

DINFER_DEFINE_LAST_ERROR()

// Dynamic shared memory (bytes) of a launch of tiles of bt tokens whose K `splits` CTAs share, -1: no such launch.
DINFER_API int64_t dinfer_gemm_f32_shared(int a_dtype, int w_dtype, int bt, int splits) {
  if (bt <= 0 || bt > BT || bt % 16 || splits < 1 || splits > MAX_SPLITS) return -1;
  DINFER_DISPATCH_DTYPE(a_dtype, TA,
    DINFER_DISPATCH_DTYPE(w_dtype, TW,
      return (int64_t)tile_shared<TA, TW>(bt, splits)));
  return -1;
}

// A [M, K] row stride lda; W [N, K] row stride ldw; C [M, N] row stride ldc (strides in elements).
DINFER_API int dinfer_gemm_f32(const void* A, int64_t lda, int a_dtype, const void* W, int64_t ldw,
                               int w_dtype, void* C, int64_t ldc, int c_dtype, int M, int N, int K,
                               int* status, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N)
    return refuse(DINFER_BAD_ARGUMENT, "gemm_f32: bad sizes M=%d N=%d K=%d lda=%lld ldw=%lld ldc=%lld", M, N, K,
                  (long long)lda, (long long)ldw, (long long)ldc);
  if (M == 0) return 0;
  DINFER_DISPATCH_DTYPE(a_dtype, TA,
    DINFER_DISPATCH_DTYPE(w_dtype, TW,
      DINFER_DISPATCH_DTYPE(c_dtype, TC,
        return launch<TA, TW, TC>(A, lda, W, ldw, C, ldc, M, N, K, status, stream))));
  return 0;
}

// The same product for `batch` independent problems: problem b reads A + b * sa, W + b * sw and writes C + b * sc
// (strides in elements; the problems of a batch may interleave inside one tensor, e.g. the heads of a row).
DINFER_API int dinfer_gemm_f32_batched(const void* A, int64_t lda, int64_t sa, int a_dtype, const void* W, int64_t ldw,
                                       int64_t sw, int w_dtype, void* C, int64_t ldc, int64_t sc, int c_dtype, int M,
                                       int N, int K, int batch, int* status, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || batch <= 0 || lda < K || ldw < K || ldc < N)
    return refuse(DINFER_BAD_ARGUMENT, "gemm_f32_batched: bad sizes M=%d N=%d K=%d batch=%d lda=%lld ldw=%lld ldc=%lld",
                  M, N, K, batch, (long long)lda, (long long)ldw, (long long)ldc);
  if (M == 0) return 0;
  DINFER_DISPATCH_DTYPE(a_dtype, TA,
    DINFER_DISPATCH_DTYPE(w_dtype, TW,
      DINFER_DISPATCH_DTYPE(c_dtype, TC,
        return launch<TA, TW, TC>(A, lda, W, ldw, C, ldc, M, N, K, status, stream, batch, sa, sw, sc))));
  return 0;
}
