// The state-space mixer's chunks on the tensor cores (see state_space.cu for what they compute): chunks of 128 tokens, every
// 32-bit operand split into three bfloat16 parts (split_umma.cuh).  Included by state_space.cu.
//
//   ssm_sums_umma      per (chunk, a run of a group's heads): B^T (state channel x token) once into tensor memory, then per head
//                      U = B^T (w x); and per (chunk, group) the scores B_s . C_t, stored [s][t]
//   ssm_outputs_umma   per (chunk, run of heads): C (token x state channel) once into tensor memory, then per head
//                      y = exp(c_t) (C S) + A x + D x, A made in registers from the scores, straight into tensor memory
//
// A head's 64 value columns are the MMA's columns; while one head's MMAs run, the next one's operands are split.  Results that
// are not finite are summed again term by term, so that a token's infinity or NaN reaches the tokens behind it and no others (a
// zero of A times it would not be zero).  The weights of x in U and A's elements, which decays make as small as they like, are split
// times 2^16 (split_umma.cuh) at no cost; the layer's own numbers, B, C, x and S, as they are (those below 2^-110, 7e-34, with fewer digits:
// scaled as well, a portion of 400 tokens through 16 heads took 48 us instead of 42).
//
// Bound by a chain, head after head: splitting and making A, then MMAs of 64 columns (54 to 70 cycles each, where 128 x 64 x 16
// would take 32).  ncu, 1500 + 547 tokens of 64 heads of 128 x 64: the outputs' tensor pipe is busy 27 % of the cycles, their issue
// slots 47 %, the sums' 22 and 38; one launch of the sums 43 us, of the walk over the chunks 21, of the outputs 57, on chunks of 64 with
// plain multiply-adds 77, 32 and 112 (the layer 434 -> 346 us).  Where they gain stands at the rule (umma_gains).  Relative errors against
// 64 bits, 16 to 1000 tokens: outputs 0.8e-7 to 1.2e-7 (1.1e-7 to 2.3e-7 with multiply-adds), states 0.6e-7 to 1.2e-7 as with them
// (1.2e-7 for 0.9e-7 at worst: 16 tokens, everything of one sign).
#pragma once

constexpr int CU = 128;                 // tokens of a chunk
constexpr int VT = 64;                  // value columns of a tile
constexpr int UT = 512;                 // threads that split, make A and store; a warp more issues the MMAs
constexpr int MMA_WARP = UT / 32, UMMA_THREADS = UT + 32;
constexpr int MAX_UNITS = 8;            // (head, column tile) pairs of a CTA at most
constexpr uint32_t PART_BYTES = CU * VT * 2, TILE_BYTES = dinfer_split::PARTS * PART_BYTES;   // 128 rows of 64 columns
constexpr int A_COLS = CU / 2, A_ALL = dinfer_split::PARTS * A_COLS;                          // tensor memory columns of an A operand
constexpr int SUM_PARTS = CU / 32;
constexpr int TMEM_ALL = 512;
static_assert(A_ALL + SUM_PARTS * VT <= TMEM_ALL && 2 * A_ALL + 2 * VT <= TMEM_ALL && A_ALL + 2 * CU <= TMEM_ALL, "tensor memory");
constexpr size_t SUMS_SMEM = 2 * TILE_BYTES + 1024 + 16 * 32 * 20 * 4;   // (more than half of an SM's: the tensor memory is one CTA's)
static_assert(SUMS_SMEM > 114 * 1024, "one CTA to an SM");
constexpr size_t OUTPUTS_SMEM = 4 * TILE_BYTES + 1024;
// The MMA cuts its sums off, so that they come out too small: U by 2.4e-8 to 6e-8 of itself, the outputs, whose eight steps lie in one
// sum, by 0.6e-7 to 2e-7 (plain sums and decayed ones, of both signs and of one, 16 to 128 tokens).  The factors that they are
// multiplied by anyhow, the weights of x (rounded from 64 bits) and the outputs' scales, make up for the middle of that.
constexpr double SUMS_CUT = 1.0 + 4e-8;
constexpr float OUTPUTS_CUT = 1.f + 1.1920929e-7f;          // (the next number behind one)
constexpr int STATUS_SUMS = 51, STATUS_OUTPUTS = 52, STATUS_PLACES = 53;

__device__ __forceinline__ int64_t wide_slot(int t_begin, int b, int c) { return (int64_t)(t_begin / CU + b + c); }

// Chunk number `place` of the step's portions (requests with more than one token): its request (-1: there is none) and its number
// in it, by a whole warp.  The launches have no grid dimension for requests, and places for the portions alone: beside 60 single tokens a portion's CTAs would be one in 61, and
// even one that has nothing to do needs an SM's shared memory to itself (700 tokens beside 60: 95 us became 113).
__device__ __forceinline__ int place_of(const int* __restrict__ cu, int B, int place, int& chunk) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int i0 = 0; i0 < B; i0 += 32) {
    const int i = i0 + lane, tokens = i < B ? cu[i + 1] - cu[i] : 0, n = tokens > 1 ? (tokens + CU - 1) / CU : 0;
    int upto = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, d);
      if (lane >= d) upto += v;
    }
    const int all = __shfl_sync(0xffffffffu, upto, 31);
    if (place < before + all) {
      const int src = __ffs(__ballot_sync(0xffffffffu, place >= before + upto - n && place < before + upto)) - 1;
      chunk = place - before - __shfl_sync(0xffffffffu, upto - n, src);
      return i0 + src;
    }
    before += all;
  }
  return -1;
}

// four tokens' numbers of one head for a lane (zeros beyond n)
__device__ __forceinline__ void lane_tokens(const float* __restrict__ src, int64_t ld, int n, float (&v)[4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = 4 * lane + i < n ? src[(int64_t)(4 * lane + i) * ld] : 0.f;
}
// the running sums of the decays' logarithms of up to 128 tokens by one warp, four tokens a lane
__device__ __forceinline__ void wide_log_decay(const float (&la)[4], double (&cum)[4]) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    s += (double)la[i];
    cum[i] = s;
  }
  double before = s;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const double v = __shfl_up_sync(0xffffffffu, before, d);
    if (lane >= d) before += v;
  }
  before = __shfl_up_sync(0xffffffffu, before, 1);
  if (lane > 0)
#pragma unroll
    for (int i = 0; i < 4; ++i) cum[i] += before;
}

// A tile of 128 rows by 64 columns: a thread's pieces of eight, rows below n from memory, else zeros; and their parts to shared
// memory, rows of 128 bytes (times scale[row]).  Apart, so that all loads are on their way before the first split.
constexpr int PIECES = CU * VT / 8 / UT;
struct Pieces { float4 v[PIECES][2]; };
__device__ __forceinline__ void fetch_tile(Pieces& x, const float* __restrict__ src, int64_t ld, int n) {
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int piece = threadIdx.x + i * UT, r = piece >> 3, c = piece & 7;
    x.v[i][0] = x.v[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < n) {
      x.v[i][0] = get4(src + (int64_t)r * ld + c * 8);
      x.v[i][1] = get4(src + (int64_t)r * ld + c * 8 + 4);
    }
  }
}
template <bool SCALED>
__device__ __forceinline__ void stage_tile(uint32_t dst, const Pieces& x, const float* scale) {
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int piece = threadIdx.x + i * UT, r = piece >> 3, c = piece & 7;
    const float4 a = x.v[i][0], b = x.v[i][1];
    const float e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint4 q[dinfer_split::PARTS];
    if (SCALED) dinfer_split::split8_times(e, scale[r], q);     // (0 beyond the chunk's tokens)
    else dinfer_split::split8<false>(e, q);
#pragma unroll
    for (int k = 0; k < dinfer_split::PARTS; ++k) dinfer_split::st_shared16(dst + k * PART_BYTES + dinfer_split::swizzled128(r, c), q[k]);
  }
}
// sixteen k of this thread's lane of an A operand
__device__ __forceinline__ void put_lane(uint32_t at, int unit, const float (&x)[16]) {
  const float lo[8] = {x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]}, hi[8] = {x[8], x[9], x[10], x[11], x[12], x[13], x[14], x[15]};
  uint4 a[dinfer_split::PARTS], b[dinfer_split::PARTS];
  dinfer_split::split8<false>(lo, a);
  dinfer_split::split8<false>(hi, b);
#pragma unroll
  for (int e = 0; e < dinfer_split::PARTS; ++e) dinfer_split::tmem_st8(at + e * A_COLS + unit * 8, a[e], b[e]);
}
// the threads that are not the MMAs' meet
__device__ __forceinline__ void workers_meet() { asm volatile("bar.sync 1, %0;" ::"n"(UT) : "memory"); }

// A row-major operand (rows below `live`, n columns, a multiple of 16, 16-byte rows) into tensor memory, a lane a row, by way of
// shared memory (128 rows of n + 4 floats)
__device__ __forceinline__ void fill_rows(uint32_t at, const float* __restrict__ src, int64_t ld, int live, int n, float* through) {
  const int ldt = n + 4, row = ((threadIdx.x >> 5) & 3) * 32 + (threadIdx.x & 31);
  for (int i0 = threadIdx.x; i0 < CU * (n / 4); i0 += 4 * UT) {     // (CU * n / 4 is a multiple of UT)
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + j * UT, r = i / (n / 4), e = (i % (n / 4)) * 4;
      v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < live) v[j] = get4(src + (int64_t)r * ld + e);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + j * UT, r = i / (n / 4), e = (i % (n / 4)) * 4;
      if (r < CU) put4(through + r * ldt + e, v[j]);
    }
  }
  workers_meet();
  for (int u = threadIdx.x >> 7; u < n / 16; u += UT / 128) {
    float x[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = get4(through + row * ldt + u * 16 + 4 * i);
      x[4 * i] = v.x; x[4 * i + 1] = v.y; x[4 * i + 2] = v.z; x[4 * i + 3] = v.w;
    }
    put_lane(at, u, x);
  }
}
// D = A B over k steps [k0, k1) (at most 8), the six products of parts; B as tiles of 128-byte rows: MN (rows are k), or K-major
// (columns are k: 64 a tile of 128 rows, tiles TILE_BYTES apart)
template <bool MN>
__device__ __forceinline__ void issue(uint32_t lead, uint32_t d, uint32_t a, uint32_t b, int k0, int k1, uint32_t idesc) {
  using namespace dinfer_split;
  const uint64_t b0 = MN ? dinfer_umma::desc_mn_major(b, PART_BYTES) : dinfer_umma::desc_k_major(b);
#pragma unroll
  for (int i = 0; i < PRODUCTS; ++i)
#pragma unroll
    for (int k = 0; k < CU / 16; ++k) {
      if (k < k0 || k >= k1) continue;
      const uint32_t off = part_b(i) * PART_BYTES + (MN ? k * 16 * 128 : (k >> 2) * TILE_BYTES + (k & 3) * 32);
      mma_ts_if(lead, d, a + part_a(i) * A_COLS + 8 * k, b0 + (off >> 4), idesc, i > 0 || k > k0);
    }
}
__device__ __forceinline__ bool finite16(const float (&v)[16]) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 16; ++i) ok = ok && (__float_as_uint(v[i]) & 0x7f800000u) != 0x7f800000u;
  return ok;
}
__device__ __forceinline__ void load_sum(float (&v)[16], uint32_t at) {
  uint32_t r[16];
  dinfer_umma::tmem_ld16(at, r);
  dinfer_umma::tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Sixteen columns of a warp's 32 rows change hands by way of 2560 bytes of shared memory: v is lane `lane`'s row; use(i,
// row, column, four elements) is called for eight rows at a time, a row's 64 bytes by four neighbouring lanes.  (A lane to a row would touch 32
// lines of memory an instruction, a cycle each: 6500 cycles of a head's 17000.)
constexpr int SWAP_LD = 20, SWAP_FLOATS = 32 * SWAP_LD;
template <typename F>
__device__ __forceinline__ void by_rows(float* swap, const float (&v)[16], F use) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 4; ++i) put4(swap + lane * SWAP_LD + 4 * i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 8 * i + (lane >> 2), c = (lane & 3) * 4;
    use(i, r, c, get4(swap + r * SWAP_LD + c));
  }
  __syncwarp();
}
// the units of a CTA: heads of one group by column tiles
struct Run {
  int g, first, count, tiles_v, per_group;
  __device__ __forceinline__ int head(int u, int heads) const { return g * heads + (first + u) / tiles_v; }
  __device__ __forceinline__ int column(int u) const { return (first + u) % tiles_v * VT; }
};

// grid (places of chunks, G * runs of units + G): sums of a run, or a group's scores
__global__ void __launch_bounds__(UMMA_THREADS, 1) ssm_sums_umma_kernel(const Params p, int units, int* status) {
  using namespace dinfer_umma;
  extern __shared__ unsigned char umma_sm[];
  __shared__ __align__(8) uint64_t tiles_bar[2], done_bar[2], read_bar;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ float wgt[MAX_UNITS][CU];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int c = 0;
  const int b = place_of(p.cu, p.B, blockIdx.x, c);
  if (b < 0) return leave(blockIdx.x == 0 && blockIdx.y == 0);
  const int t_begin = p.cu[b], t_end = p.cu[b + 1], t0 = t_begin + c * CU;
  const uint32_t base = (smem_u32(umma_sm) + 1023u) & ~1023u;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&tiles_bar[i]), UT / 32); mbar_init(smem_u32(&done_bar[i]), 1); }
    mbar_init(smem_u32(&read_bar), UT / 32);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_ALL) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_enter();                                     // (dependents start only now that the tensor memory is ours)
  if (blockIdx.y == 0 && blockIdx.x == gridDim.x - 1 && warp == MMA_WARP) {     // a chunk that no CTA takes would go unnoticed
    int beyond;
    if (place_of(p.cu, p.B, gridDim.x, beyond) >= 0 && lane == 0) atomicExch(status, STATUS_PLACES);
  }
  const uint32_t tmem = s_tmem, lead = dinfer_split::elect_lane(), tm = dinfer_split::uniform(tmem), lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const int row = (warp & 3) * 32 + lane, sub = warp >> 2;
  const int n = min(CU, t_end - t0), ch = p.channels(), inner = p.inner(), heads = p.H / p.G;
  const int64_t slot = wide_slot(t_begin, b, c);
  Run run;
  run.tiles_v = p.Pd / VT;
  run.per_group = heads * run.tiles_v;
  const int runs = (run.per_group + units - 1) / units, job = (int)blockIdx.y - p.G * runs;
  float* through = reinterpret_cast<float*>(umma_sm + (base - smem_u32(umma_sm)));
  float* swap = through + (2 * TILE_BYTES) / 4 + warp * SWAP_FLOATS;
  // what this warp has written is there for the MMAs (and it has read what they will overwrite)
  const auto hand_over = [&](uint64_t* bar) {
    tmem_st_wait();
    dinfer_split::fence_to_mma();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(bar));
  };
  if (job >= 0) {
    // ---- scores of group `job`: lanes are tokens s, columns tokens t
    const float* Bp = p.xbc + (int64_t)t0 * ch + inner + job * p.N;
    const float* Cp = Bp + p.G * p.N;
    const int steps = p.N / 16;
    if (warp == MMA_WARP) {
      if (mbar_spin(smem_u32(&tiles_bar[0]), 0)) {
        tc_fence_after();
        issue<false>(lead, tm + A_ALL, tm, base, 0, min(4, steps), idesc_bf16(CU, CU, 0));
        if (steps > 4) issue<false>(lead, tm + A_ALL + CU, tm, base, 4, steps, idesc_bf16(CU, CU, 0));
        dinfer_split::commit_if(lead, smem_u32(&done_bar[0]));
      } else {
        s_abort = 1; atomicExch(status, STATUS_SUMS);
      }
    } else {
      fill_rows(lanes, Bp, ch, n, p.N, through);
      workers_meet();                              // (the tiles take its place)
#pragma unroll 1
      for (int half = 0; half < (p.N + VT - 1) / VT; ++half)
#pragma unroll
        for (int i = 0; i < CU * VT / 8 / UT; ++i) {
          const int piece = tid + i * UT, r = piece >> 3, e = half * VT + (piece & 7) * 8;
          float x[8] = {};
          if (r < n && e < p.N) {
            const float4 u = get4(Cp + (int64_t)r * ch + e), v = get4(Cp + (int64_t)r * ch + e + 4);
            x[0] = u.x; x[1] = u.y; x[2] = u.z; x[3] = u.w; x[4] = v.x; x[5] = v.y; x[6] = v.z; x[7] = v.w;
          }
          uint4 q[dinfer_split::PARTS];
          dinfer_split::split8<false>(x, q);
#pragma unroll
          for (int k = 0; k < dinfer_split::PARTS; ++k)
            dinfer_split::st_shared16(base + half * TILE_BYTES + k * PART_BYTES + dinfer_split::swizzled128(r, piece & 7), q[k]);
        }
      hand_over(&tiles_bar[0]);
      if (mbar_wait(smem_u32(&done_bar[0]), 0)) {
        tc_fence_after();
        float* out = p.cb + (slot * p.G + job) * (int64_t)CU * CU + row * CU;
#pragma unroll 1
        for (int u = 0; u < 2; ++u) {
          const int t = sub * 32 + u * 16;
          float v[16];
          load_sum(v, lanes + A_ALL + t);
          if (steps > 4) {
            float w[16];
            load_sum(w, lanes + A_ALL + CU + t);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += w[i];
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) put4(out + t + 4 * i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
          if (!finite16(v)) {
#pragma unroll 1
            for (int i = 0; i < 16; ++i) {
              float s = 0.f;
              if (row < n && t + i < n)
                for (int e = 0; e < p.N; ++e) s = fmaf(Cp[(int64_t)(t + i) * ch + e], Bp[(int64_t)row * ch + e], s);
              out[t + i] = s;
            }
          }
          __syncwarp();
        }
      } else {
        s_abort = 1; atomicExch(status, STATUS_SUMS);
      }
    }
  } else {
    run.g = (int)blockIdx.y / runs;
    run.first = (int)blockIdx.y % runs * units;
    run.count = min(units, run.per_group - run.first);
    const float* Bp = p.xbc + (int64_t)t0 * ch + inner + run.g * p.N;
    const float* xs = p.xbc + (int64_t)t0 * ch;
    const int steps = (n + 15) / 16;
    if (warp == MMA_WARP) {
      for (int u = 0; u < run.count; ++u) {
        if ((u > 0 && !mbar_spin(smem_u32(&read_bar), (u - 1) & 1)) || !mbar_spin(smem_u32(&tiles_bar[u & 1]), (u >> 1) & 1)) {
          s_abort = 1; atomicExch(status, STATUS_SUMS);
          break;
        }
        tc_fence_after();
        // 32 tokens to a sum, the four of them added in registers: the MMA cuts its sums off, and over 64 tokens a state would be
        // further from 64 bits than with plain multiply-adds (1.56e-7 for 1.41e-7)
#pragma unroll
        for (int q = 0; q < SUM_PARTS; ++q)
          if (2 * q < steps)
            issue<true>(lead, tm + A_ALL + q * VT, tm, base + (u & 1) * TILE_BYTES, 2 * q, min(2 * q + 2, steps), idesc_bf16(CU, VT, 1));
        dinfer_split::commit_if(lead, smem_u32(&done_bar[u & 1]));
      }
    } else {
      float la4[4], dt4[4];
      if (warp < run.count) {
        lane_tokens(p.la + (int64_t)t0 * p.H + run.head(warp, heads), p.H, n, la4);
        lane_tokens(p.dt + (int64_t)t0 * p.H + run.head(warp, heads), p.H, n, dt4);
      }
      // B^T: a lane is a state channel, its k the tokens
      float x[2][16];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int t = (sub + 4 * j) * 16 + i;
          x[j][i] = row < p.N && t < n ? Bp[(int64_t)t * ch + row] : 0.f;
        }
      if (warp < run.count) {
        double cum[4];
        wide_log_decay(la4, cum);
        const double all = __shfl_sync(0xffffffffu, cum[3], 31);     // (nothing is added behind the chunk's last token)
#pragma unroll
        for (int i = 0; i < 4; ++i) wgt[warp][4 * lane + i] = 4 * lane + i < n ? (float)(exp(all - cum[i]) * (double)dt4[i] * SUMS_CUT) : 0.f;
        if (lane == 0 && run.column(warp) == 0) p.decay[slot * p.H + run.head(warp, heads)] = (float)exp(all);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (sub + 4 * j < steps) put_lane(lanes, sub + 4 * j, x[j]);
      workers_meet();                              // the weights are there
      // head u + 1 is staged ahead of head u's results: its tile was read by head u - 1's MMAs, which this warp has waited for
      for (int u = -1; u < run.count; ++u) {
        if (u + 1 < run.count) {
          Pieces x;
          fetch_tile(x, xs + run.head(u + 1, heads) * p.Pd + run.column(u + 1), ch, n);
          stage_tile<true>(base + ((u + 1) & 1) * TILE_BYTES, x, wgt[u + 1]);
          hand_over(&tiles_bar[(u + 1) & 1]);
        }
        if (u < 0) continue;
        if (!s_abort && !mbar_wait(smem_u32(&done_bar[u & 1]), (u >> 1) & 1)) { s_abort = 1; atomicExch(status, STATUS_SUMS); }
        tc_fence_after();
        const int h = run.head(u, heads), c0 = run.column(u) + sub * 16;
        float v[16];
        load_sum(v, lanes + A_ALL + sub * 16);
#pragma unroll
        for (int q = 1; q < SUM_PARTS; ++q)
          if (2 * q < steps) {
            float w[16];
            load_sum(w, lanes + A_ALL + q * VT + sub * 16);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] += w[i];
          }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&read_bar));
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] *= dinfer_split::UNSCALE;
        float* U = p.U + (slot * p.H + h) * (int64_t)p.N * p.Pd + c0;
        by_rows(swap, v, [&](int, int r, int x, const float4& e) {
          const int k = (warp & 3) * 32 + r;
          if (k < p.N) put4(U + (int64_t)k * p.Pd + x, e);
        });
        if (row < p.N && !finite16(v)) {
#pragma unroll 1
          for (int i = 0; i < 16; ++i) {
            float s = 0.f;
            for (int t = 0; t < n; ++t) s = fmaf(Bp[(int64_t)t * ch + row], xs[(int64_t)t * ch + h * p.Pd + c0 + i] * wgt[u][t], s);
            U[(int64_t)row * p.Pd + i] = s;
          }
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    if (s_abort)
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_ALL) : "memory");
  }
}

// grid (places of chunks, G * runs of units)
__global__ void __launch_bounds__(UMMA_THREADS, 1) ssm_outputs_umma_kernel(const Params p, int units, int* status) {
  using namespace dinfer_umma;
  extern __shared__ unsigned char umma_sm[];
  __shared__ __align__(8) uint64_t tiles_bar, a_bar, done_bar;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  __shared__ __align__(16) float c_hi[MAX_UNITS][CU], c_lo[MAX_UNITS][CU], dts[MAX_UNITS][CU];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int c = 0;
  const int b = place_of(p.cu, p.B, blockIdx.x, c);
  if (b < 0) return leave(blockIdx.x == 0 && blockIdx.y == 0);
  const int t_begin = p.cu[b], t_end = p.cu[b + 1], t0 = t_begin + c * CU;
  const uint32_t base = (smem_u32(umma_sm) + 1023u) & ~1023u;
  if (tid == 0) {
    mbar_init(smem_u32(&tiles_bar), UT / 32);
    mbar_init(smem_u32(&a_bar), UT / 32);
    mbar_init(smem_u32(&done_bar), 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(TMEM_ALL) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_enter();
  const uint32_t tmem = s_tmem, lead = dinfer_split::elect_lane(), tm = dinfer_split::uniform(tmem), lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint32_t a_at = A_ALL, d1_at = 2 * A_ALL, d2_at = 2 * A_ALL + VT;
  const int row = (warp & 3) * 32 + lane, sub = warp >> 2;
  const int n = min(CU, t_end - t0), ch = p.channels(), inner = p.inner(), heads = p.H / p.G;
  const int64_t slot = wide_slot(t_begin, b, c);
  Run run;
  run.tiles_v = p.Pd / VT;
  run.per_group = heads * run.tiles_v;
  const int runs = (run.per_group + units - 1) / units;
  run.g = (int)blockIdx.y / runs;
  run.first = (int)blockIdx.y % runs * units;
  run.count = min(units, run.per_group - run.first);
  const float* Cp = p.xbc + (int64_t)t0 * ch + inner + (p.G + run.g) * p.N;
  const float* cb = p.cb + (slot * p.G + run.g) * (int64_t)CU * CU;            // [s][t]
  const float* xs = p.xbc + (int64_t)t0 * ch;
  const int steps_s = p.N / 16, steps_t = (n + 15) / 16;
  const auto S_of = [&](int u) { return p.U + (slot * p.H + run.head(u, heads)) * (int64_t)p.N * p.Pd + run.column(u); };
  const auto stage = [&](int u) {
    Pieces S, x;
    fetch_tile(S, S_of(u), p.Pd, p.N);
    fetch_tile(x, xs + run.head(u, heads) * p.Pd + run.column(u), ch, n);
    if (u > 0) workers_meet();                     // (the tiles' place was where head u - 2's results changed hands)
    stage_tile<false>(base + (u & 1) * 2 * TILE_BYTES, S, nullptr);
    stage_tile<false>(base + (u & 1) * 2 * TILE_BYTES + TILE_BYTES, x, nullptr);
  };
  const auto hand_over = [&](uint64_t* bar) {
    tmem_st_wait();
    dinfer_split::fence_to_mma();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(bar));
  };
  if (warp == MMA_WARP) {
    const uint32_t idesc = idesc_bf16(CU, VT, 1);
    for (int u = 0; u < run.count; ++u) {
      const uint32_t tiles = base + (u & 1) * 2 * TILE_BYTES;
      if (!mbar_spin(smem_u32(&tiles_bar), u & 1)) { s_abort = 1; atomicExch(status, STATUS_OUTPUTS); break; }
      tc_fence_after();
      issue<true>(lead, tm + d1_at, tm, tiles, 0, steps_s, idesc);
      if (!mbar_spin(smem_u32(&a_bar), u & 1)) { s_abort = 1; atomicExch(status, STATUS_OUTPUTS); break; }
      tc_fence_after();
      issue<true>(lead, tm + d2_at, tm + a_at, tiles + TILE_BYTES, 0, steps_t, idesc);
      dinfer_split::commit_if(lead, smem_u32(&done_bar));
    }
  } else {
    float la4[4], dt4[4];
    if (warp < run.count) {
      lane_tokens(p.la + (int64_t)t0 * p.H + run.head(warp, heads), p.H, n, la4);
      lane_tokens(p.dt + (int64_t)t0 * p.H + run.head(warp, heads), p.H, n, dt4);
    }
    // the scores that this thread needs, the same for all heads: its token's with two runs of sixteen s (runs sub and 7 - sub: as
    // many below the diagonal), zeros above
    float score[2][16];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = i ? 7 - sub : sub;
#pragma unroll
      for (int e = 0; e < 16; ++e) score[i][e] = k < steps_t && 16 * k + e <= row ? cb[(16 * k + e) * CU + row] : 0.f;
    }
    stage(0);
    if (warp < run.count) {
      // a running sum, in units of log 2, as two 32-bit numbers: differences of two such are as exact as 32-bit holds them
      double cum[4];
      wide_log_decay(la4, cum);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int s = 4 * lane + i;
        const double sum = cum[i] * 1.4426950408889634;
        const float hi = (float)sum;
        c_hi[warp][s] = hi;
        c_lo[warp][s] = (float)(sum - (double)hi);
        dts[warp][s] = dt4[i] * dinfer_split::SCALE;
      }
    }
    fill_rows(lanes, Cp, ch, n, p.N, reinterpret_cast<float*>(umma_sm + (base - smem_u32(umma_sm)) + 2 * TILE_BYTES));   // (all meet inside)
    hand_over(&tiles_bar);
    for (int u = 0; u < run.count; ++u) {
      // A[t][s] = (C_t . B_s) exp(c_t - c_s) dt_s for s <= t, while C S runs; the last head's MMAs, which read A, have been waited
      // for.  Above the diagonal 0 times a number: the exponent stops at 0 there (a sum that is not a number shows in exp(c_t)).
      const float hi = c_hi[u][row], lo = c_lo[u][row];
      const uint32_t tiles = base + (u & 1) * 2 * TILE_BYTES;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int k = i ? 7 - sub : sub;
        if (k >= steps_t) continue;
        float a[16];
        if (16 * k > (warp & 3) * 32 + 31) {
#pragma unroll
          for (int e = 0; e < 16; ++e) a[e] = 0.f;
        } else {
#pragma unroll
          for (int e = 0; e < 16; e += 4) {
            const int s = 16 * k + e;
            const float4 h4 = get4(&c_hi[u][s]), l4 = get4(&c_lo[u][s]), d4 = get4(&dts[u][s]);
            const float hs[4] = {h4.x, h4.y, h4.z, h4.w}, ls[4] = {l4.x, l4.y, l4.z, l4.w}, ds[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) a[e + j] = score[i][e + j] * exp2f(fminf((hi - hs[j]) + (lo - ls[j]), 0.f)) * ds[j];
          }
        }
        put_lane(lanes + a_at, k, a);
      }
      hand_over(&a_bar);
      if (u + 1 < run.count) stage(u + 1);         // while the MMAs run
      const int h = run.head(u, heads), c0 = run.column(u) + sub * 16;
      const float* x = xs + h * p.Pd + c0;
      float4 xv[4];                                // this lane's four pieces of what by_rows hands out
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = (warp & 3) * 32 + 8 * i + (lane >> 2);
        xv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n) xv[i] = get4(x + (int64_t)t * ch + (lane & 3) * 4);
      }
      // (a warp whose wait runs out goes on without waiting: the others meet it at their barrier)
      if (!s_abort && !mbar_wait(smem_u32(&done_bar), u & 1)) { s_abort = 1; atomicExch(status, STATUS_OUTPUTS); }
      tc_fence_after();
      float v[16], w[16];
      load_sum(v, lanes + d1_at + sub * 16);
      load_sum(w, lanes + d2_at + sub * 16);
      if (u + 1 < run.count) hand_over(&tiles_bar);   // (head u + 1's C S may take the sums' place)
      const float e = exp2f(hi), D = p.D[h], e_cut = e * OUTPUTS_CUT;
      float* y = p.y + (int64_t)t0 * inner + (int64_t)h * p.Pd + c0;
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = fmaf(e_cut, v[i], w[i] * (dinfer_split::UNSCALE * OUTPUTS_CUT));
      by_rows(reinterpret_cast<float*>(umma_sm + (tiles - smem_u32(umma_sm))) + warp * SWAP_FLOATS, v, [&](int i, int r, int col, const float4& o) {
        const int t = (warp & 3) * 32 + r;
        if (t < n)
          put4(y + (int64_t)t * inner + col, make_float4(fmaf(D, xv[i].x, o.x), fmaf(D, xv[i].y, o.y), fmaf(D, xv[i].z, o.z), fmaf(D, xv[i].w, o.w)));
      });
      if (row < n && !finite16(v)) {
        const float* S = S_of(u) + sub * 16;
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
          float r = 0.f;
          for (int k = 0; k < p.N; ++k) r = fmaf(Cp[(int64_t)row * ch + k], S[(int64_t)k * p.Pd + i], r);
          r *= e;
          for (int s = 0; s <= row; ++s)
            r = fmaf(cb[s * CU + row] * exp2f((hi - c_hi[u][s]) + (lo - c_lo[u][s])) * (dts[u][s] * dinfer_split::UNSCALE), xs[(int64_t)s * ch + h * p.Pd + c0 + i], r);
          y[(int64_t)row * inner + i] = fmaf(D, x[(int64_t)row * ch + i], r);
        }
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    if (s_abort)
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_ALL) : "memory");
  }
}

// The units of a CTA: as many as share a group's operand, but so that the CTAs fill the SMs; a CTA takes about 1.2 units' time
// for what its units share
inline int units_of(int chunks, int G, int per_group, int sms) {
  int best = 1;
  int64_t cost = 0;
  for (int u = 1; u <= MAX_UNITS && u <= per_group; ++u) {
    const int64_t ctas = (int64_t)chunks * G * ((per_group + u - 1) / u);
    const int64_t c = (ctas + sms - 1) / sms * (5 * u + 6);
    if (u == 1 || c < cost) { cost = c; best = u; }
  }
  return best;
}
