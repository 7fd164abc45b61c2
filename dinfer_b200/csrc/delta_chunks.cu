// The gated delta rule (see delta_rule.cu) for portions of many tokens, one decay a head: chunks of 32 tokens instead of
// token by token.  With c_t the running sum of the decays' logarithms inside a chunk, Gamma_t = exp(c_t), S the state before
// the chunk, and
//
//     A[t, s] = beta_t exp(c_t - c_s) (k_t . k_s)   for s < t          M[t, s] = exp(c_t - c_s) (q_t . k_s)   for s <= t
//
// the tokens' updates u solve (I + A) U = beta (V - Gamma K S), so
//
//     W_v = (I + A)^-1 (beta V),  W_k = (I + A)^-1 (beta Gamma K)       per (chunk, head): need no state
//     U   = W_v - W_k S,   O = Gamma (Q S) + M U,   S <- exp(c_n) S + sum_s exp(c_n - c_s) k_s u_s^T
//
//   delta_chunk   everything that needs no state, all (chunk, head) side by side, into a workspace
//   delta_walk    per (request, head, 16 value columns) the chunks in order; S in registers and shared memory
//
// What a token's output and what it adds to the state are made of are sums over the tokens up to it and nothing else: an
// infinity or NaN at one token leaves the outputs before it alone, as token by token, where a zero of the triangular matrices
// times it would not.
//
// All arithmetic is 32-bit; the running sums are 64-bit, so that a difference of two large ones is exact; the state's decay is
// S + S expm1(c_n).  An update of the state rounds once a chunk where the token loop rounds 32 times.
//
// What bounds it: the walk, 32-bit multiply-adds on small tiles with every operand from shared memory (1.5 loads of 16 bytes
// for every eight), and the chain of chunks.  2000 tokens of 16 heads of 128 x 128: the token loop 502 us (a chain of 250 ns
// a token), both kernels 199 us (220 with the products of the upper triangles), delta_chunk 44 us of it, delta_walk the rest.
#include <type_traits>

#include "common.cuh"

using namespace dinfer;

namespace {

constexpr int C = 32;              // tokens of a chunk
constexpr int BC = 16;             // value columns of a walk's block
constexpr int THREADS = 256;
constexpr int LDA = C + 4;         // row stride of the 32 x 32 matrices in shared memory
constexpr int SMALL = 2 * C + 4;   // per (chunk, head): Gamma [32], exp(c_n - c_s) [32], expm1(c_n)
constexpr float LOG_FLOOR = -100.f;   // a decay of 0: exp(-100) is 0 beside anything

struct Args {
  const float *q, *k, *v, *beta, *decay;   // [T, G, dk], [T, G, dk], [T, H, dv], [T, H], [T, H] (g - 1)
  float* state; int64_t ld_state;          // S [H, dk, dv] at the start of a row
  const int *cu, *slots, *fresh;
  float* out;                              // [T, H, dv]
  float *wk, *wv, *m, *small;              // [places, H, C, dk], [places, H, C, dv], [places, H, C, C], [places, H, SMALL]
  int B, H, G, dv;
};

__device__ __forceinline__ int warp_inclusive(int v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}
// chunk number `place` of the batch: its request (-1: there is none) and its number in it
__device__ __forceinline__ int request_of_chunk(const int* cu, int B, int place, int lane, int& chunk) {
  int before = 0;
  for (int i0 = 0; i0 < B; i0 += 32) {
    const int i = i0 + lane;
    const int n = i < B ? (cu[i + 1] - cu[i] + C - 1) / C : 0;
    const int incl = warp_inclusive(n, lane);
    const int all = __shfl_sync(0xffffffffu, incl, 31);
    if (place < before + all) {
      const int src = __ffs(__ballot_sync(0xffffffffu, place >= before + incl - n && place < before + incl)) - 1;
      chunk = place - before - __shfl_sync(0xffffffffu, incl - n, src);
      return i0 + src;
    }
    before += all;
  }
  return -1;
}
// chunks of the requests before b
__device__ __forceinline__ int chunks_before(const int* cu, int b, int lane) {
  int sum = 0;
  for (int i = lane; i < b; i += 32) sum += (cu[i + 1] - cu[i] + C - 1) / C;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  return sum;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool live) {     // zeros where not live
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float c) {
  return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c))));
}

// Bound by the reads of shared memory that feed its multiply-adds (a warp's 16-byte read takes four passes whatever its lanes
// share): 4 x 4 sums a thread for the products, 4 x 8 for the columns, which take beta and Gamma with the inverse's columns.
template <int DK>
__global__ void __launch_bounds__(THREADS, 2)
delta_chunk_kernel(const Args a) {
  constexpr int LD = DK + 4, CW = DK / 16;               // columns of a thread
  __shared__ __align__(16) float KQ[2 * C][LD];          // keys, then queries, later values
  __shared__ __align__(16) float As[C][LDA];             // A
  __shared__ __align__(16) float Ts[2][C][LDA];          // the inverse, transposed: Ts[.][s][t], times beta_s; times beta_s Gamma_s
  __shared__ double c_s[C];
  __shared__ float beta_s[C];
  pdl_enter();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int place = blockIdx.x, h = blockIdx.y, g = h / (a.H / a.G);
  int chunk = 0;
  const int b = request_of_chunk(a.cu, a.B, place, lane, chunk);
  if (b < 0) return;
  const int t0 = a.cu[b] + chunk * C, n = min(C, a.cu[b + 1] - t0);
  const int64_t at = (int64_t)place * a.H + h;

  const int64_t nq = (int64_t)a.G * DK;
  for (int i = tid; i < 2 * C * (DK / 4); i += THREADS) {
    const int r = i / (DK / 4), e = (i % (DK / 4)) * 4, t = r & (C - 1);
    const float* src = (r < C ? a.k : a.q) + (t < n ? (t0 + t) * nq + (int64_t)g * DK + e : 0);
    cp_async16(&KQ[r][e], src, t < n);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  float gam = 0.f, be = 0.f;                             // of token `lane`, in warp 0
  if (warp == 0) {
    // the decays' logarithms (0 behind the portion's end), their running sums in 64-bit
    double l = 0.0;
    if (lane < n) {
      l = log1p((double)a.decay[(int64_t)(t0 + lane) * a.H + h]);
      if (l < (double)LOG_FLOOR) l = LOG_FLOOR;            // (not fmax: a NaN stays one, as token by token)
      be = a.beta[(int64_t)(t0 + lane) * a.H + h];
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, l, d);
      if (lane >= d) l += t;
    }
    const double last = __shfl_sync(0xffffffffu, l, 31);
    c_s[lane] = l;
    beta_s[lane] = be;
    gam = expf((float)l);
    float* sm = a.small + at * SMALL;
    sm[lane] = gam;
    sm[C + lane] = expf((float)(last - l));
    if (lane == 0) sm[2 * C] = expm1f((float)last);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  {
    // k_t . k_s and q_t . k_s: rows ty + 16 i of the stacked 64, columns tx + 8 j; half of the key channels to 128 threads.
    // Then the first half of the threads completes the rows of A, the second those of M.
    const int kh = tid >> 7, ty = (tid & 127) >> 3, tx = tid & 7;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 2
    for (int e = kh * (DK / 2); e < (kh + 1) * (DK / 2); e += 4) {
      float4 r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = *reinterpret_cast<const float4*>(&KQ[ty + 16 * i][e]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 s = *reinterpret_cast<const float4*>(&KQ[tx + 8 * j][e]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][j] = dot4(r[i], s, acc[i][j]);
      }
    }
    float (*other)[LDA] = Ts[kh];                          // what the other half of the threads lacks
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) other[ty + 16 * i][tx + 8 * j] = kh ? acc[i][j] : acc[i + 2][j];
    __syncthreads();
    float* m = a.m + at * C * C;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = ty + 16 * i, s = tx + 8 * j;
        const float e = s <= t ? expf((float)(c_s[t] - c_s[s])) : 0.f;
        const float dot = (kh ? acc[i + 2][j] : acc[i][j]) + Ts[kh ^ 1][t][s];
        if (kh == 0) As[t][s] = s < t ? beta_s[t] * e * dot : 0.f;
        else m[t * C + s] = e * dot;
      }
  }
  // nobody reads the queries any more: DK value columns take their place (zeros behind the portion's end)
  auto values = [&](int c0) {
    for (int i = tid; i < C * (DK / 4); i += THREADS) {
      const int t = i / (DK / 4), e = (i % (DK / 4)) * 4;
      const bool live = t < n && c0 + e < a.dv;
      cp_async16(&KQ[C + t][e], a.v + (live ? ((int64_t)(t0 + t) * a.H + h) * a.dv + c0 + e : 0), live);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  values(0);
  __syncthreads();
  if (warp == 0) {
    // column `lane` of (I + A)^-1 by substitution: x_t = [t = lane] - sum_(s < t) A[t, s] x_s
    float x[C];
#pragma unroll
    for (int t = 0; t < C; ++t) {
      float p[4] = {t == lane ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < t; s += 4) {
        const float4 r = *reinterpret_cast<const float4*>(&As[t][s]);
        p[0] = fmaf(-r.x, x[s], p[0]);
        if (s + 1 < t) p[1] = fmaf(-r.y, x[s + 1], p[1]);
        if (s + 2 < t) p[2] = fmaf(-r.z, x[s + 2], p[2]);
        if (s + 3 < t) p[3] = fmaf(-r.w, x[s + 3], p[3]);
      }
      x[t] = (p[0] + p[1]) + (p[2] + p[3]);
    }
#pragma unroll
    for (int t = 0; t < C; t += 4) {
      const float4 v = make_float4(be * x[t], be * x[t + 1], be * x[t + 2], be * x[t + 3]);
      *reinterpret_cast<float4*>(&Ts[0][lane][t]) = v;
      *reinterpret_cast<float4*>(&Ts[1][lane][t]) = make_float4(gam * v.x, gam * v.y, gam * v.z, gam * v.w);
    }
  }
  // [W_v | W_k]: a half of the threads has DK columns, a thread rows rt .. rt + 3 of columns cx + 64 j ..
  const bool keys = tid < 128;
  const int rt = ((tid & 127) >> 4) * 4, cx = (tid & 15) * 4, w0 = (tid & 127) >> 5 << 3;   // (a warp has rows w0 .. w0 + 7)
  for (int c0 = 0; c0 < a.dv; c0 += DK) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (!keys || c0 == 0) {
      const float (*right)[LD] = keys ? KQ : KQ + C;
      const float (*T)[LDA] = Ts[keys];
      float acc[4][CW];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < CW; ++j) acc[i][j] = 0.f;
      auto add = [&](int s, auto diagonal) {
        const float4 t4 = *reinterpret_cast<const float4*>(&T[s][rt]);
        const float t[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
        for (int j = 0; j < CW; j += 4) {
          const float4 r = *reinterpret_cast<const float4*>(&right[s][cx + 16 * j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (diagonal && s > rt + i) continue;          // a later token's value, which may not be finite
            acc[i][j] = fmaf(t[i], r.x, acc[i][j]);
            acc[i][j + 1] = fmaf(t[i], r.y, acc[i][j + 1]);
            acc[i][j + 2] = fmaf(t[i], r.z, acc[i][j + 2]);
            acc[i][j + 3] = fmaf(t[i], r.w, acc[i][j + 3]);
          }
        }
      };
#pragma unroll 4
      for (int s = 0; s < w0; ++s) add(s, std::false_type());
#pragma unroll 4
      for (int u = 0; u < 8; ++u) add(w0 + u, std::true_type());
      float* w = keys ? a.wk + at * C * DK : a.wv + at * C * a.dv + c0;
      const int ld = keys ? DK : a.dv;
#pragma unroll
      for (int j = 0; j < CW; j += 4) {
        const int c = cx + 16 * j;
        if (!keys && c0 + c >= a.dv) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<float4*>(w + (int64_t)(rt + i) * ld + c) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
      }
    }
    if (c0 + DK < a.dv) {
      __syncthreads();
      values(c0 + DK);
    }
  }
}

template <int DK> struct Walk {
  static constexpr int LD = DK + 4, LDS = BC + 4;
  // one chunk's operands: W_k, Q, K | M | W_v | the small ones
  static constexpr int WK = 0, Q = WK + C * LD, K = Q + C * LD, M = K + C * LD, WV = M + C * LDA, SM = WV + C * BC,
                       STAGE = SM + (SMALL + 3) / 4 * 4;
  static constexpr int S = 2 * STAGE, PART = S + DK * LDS, U = PART + 4 * 2 * C * BC, FLOATS = U + 2 * C * BC;
};

template <int DK>
__global__ void __launch_bounds__(THREADS)
delta_walk_kernel(const Args a) {
  using L = Walk<DK>;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int h = blockIdx.y, b = blockIdx.z, g = h / (a.H / a.G);
  const int start = a.cu[b], n = a.cu[b + 1] - start;
  if (n <= 0) return;
  const int c0 = blockIdx.x * BC;
  const int first = chunks_before(a.cu, b, lane), chunks = (n + C - 1) / C;
  const int64_t nq = (int64_t)a.G * DK;
  auto stage = [&](int j) {
    float* s = sm + (j & 1) * L::STAGE;
    const int64_t at = (int64_t)(first + j) * a.H + h;
    const int t0 = start + j * C, m = min(C, n - j * C);
    for (int i = tid; i < C * (DK / 4); i += THREADS) {
      const int t = i / (DK / 4), e = (i % (DK / 4)) * 4;
      cp_async16(s + L::WK + t * L::LD + e, a.wk + (at * C + t) * DK + e, true);
      const int64_t row = t < m ? (t0 + t) * nq + (int64_t)g * DK + e : 0;
      cp_async16(s + L::Q + t * L::LD + e, a.q + row, t < m);
      cp_async16(s + L::K + t * L::LD + e, a.k + row, t < m);
    }
    {
      const int t = tid / (C / 4), e = (tid % (C / 4)) * 4;                    // 32 rows of 8 pieces: a piece a thread
      cp_async16(s + L::M + t * LDA + e, a.m + (at * C + t) * C + e, true);
    }
    if (tid < C * BC / 4) {
      const int t = tid / (BC / 4), e = (tid % (BC / 4)) * 4;
      cp_async16(s + L::WV + t * BC + e, a.wv + (at * C + t) * a.dv + c0 + e, true);
    } else if (tid < C * BC / 4 + SMALL / 4) {
      const int e = (tid - C * BC / 4) * 4;
      cp_async16(s + L::SM + e, a.small + at * SMALL + e, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0);
  // S: threads 0 .. DK - 1 (whole warps) own 4 x 4 of it, rows sr .. sr + 3, columns sc .. sc + 3; a copy for all in
  // shared memory
  const int sr = tid / 4 * 4, sc = tid % 4 * 4;
  const bool owner = tid < DK;
  float* S_s = sm + L::S;
  float* part = sm + L::PART;
  float* U_s = sm + L::U;                                  // U, then exp(c_n - c_s) U
  float* Sg = a.state + (int64_t)a.slots[b] * a.ld_state + (int64_t)h * DK * a.dv + c0;
  float S[4][4];
  if (owner) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) S[i][j] = a.fresh[b] ? 0.f : Sg[(int64_t)(sr + i) * a.dv + sc + j];
      *reinterpret_cast<float4*>(S_s + (sr + i) * L::LDS + sc) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
    }
  }
  // the product [W_k; Q] S: a quarter of the key channels to 64 threads, a thread 4 rows (ry + 16 i) by 4 columns
  const int kg = tid >> 6, ry = (tid & 63) >> 2, cx = (tid & 3) * 4;
  for (int j = 0; j < chunks; ++j) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                       // chunk j is there, S is, and nobody reads chunk j - 1 any more
    if (j + 1 < chunks) stage(j + 1);
    const float* s = sm + (j & 1) * L::STAGE;
    {
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
      const float* rows = s + ry * L::LD + kg * (DK / 4);  // W_k and Q lie one behind the other: rows 0 .. 63
      const float* sk = S_s + kg * (DK / 4) * L::LDS + cx;
#pragma unroll 4
      for (int e = 0; e < DK / 4; e += 4) {
        float4 r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = *reinterpret_cast<const float4*>(rows + 16 * i * L::LD + e);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float4 x = *reinterpret_cast<const float4*>(sk + (e + u) * L::LDS);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float w = u == 0 ? r[i].x : (u == 1 ? r[i].y : (u == 2 ? r[i].z : r[i].w));
            acc[i][0] = fmaf(w, x.x, acc[i][0]);
            acc[i][1] = fmaf(w, x.y, acc[i][1]);
            acc[i][2] = fmaf(w, x.z, acc[i][2]);
            acc[i][3] = fmaf(w, x.w, acc[i][3]);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(part + (kg * 2 * C + ry + 16 * i) * BC + cx) =
            make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    __syncthreads();
    // thread t: row t / 4 of the stacked 64, four columns
    const int row = tid >> 2, t = row & (C - 1);
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 p = *reinterpret_cast<const float4*>(part + (u * 2 * C + row) * BC + cx);
      o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w;
    }
    if (row < C) {
      const float4 w = *reinterpret_cast<const float4*>(s + L::WV + t * BC + cx);
      const float rat = s[L::SM + C + t];
      const float4 u = make_float4(w.x - o.x, w.y - o.y, w.z - o.z, w.w - o.w);
      *reinterpret_cast<float4*>(U_s + t * BC + cx) = u;
      *reinterpret_cast<float4*>(U_s + (C + t) * BC + cx) = make_float4(rat * u.x, rat * u.y, rat * u.z, rat * u.w);
    }
    __syncthreads();
    if (owner) {
      // S <- exp(c_n) S + K^T (exp(c_n - c_s) U)
      const float gm1 = s[L::SM + 2 * C];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) S[i][c] = fmaf(S[i][c], gm1, S[i][c]);
#pragma unroll 8
      for (int u = 0; u < C; ++u) {
        const float4 k = *reinterpret_cast<const float4*>(s + L::K + u * L::LD + sr);
        const float4 x = *reinterpret_cast<const float4*>(U_s + (C + u) * BC + sc);
        const float kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          S[i][0] = fmaf(kk[i], x.x, S[i][0]);
          S[i][1] = fmaf(kk[i], x.y, S[i][1]);
          S[i][2] = fmaf(kk[i], x.z, S[i][2]);
          S[i][3] = fmaf(kk[i], x.w, S[i][3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(S_s + (sr + i) * L::LDS + sc) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
    }
    if (row >= C) {
      // o_t = Gamma_t (q_t S) + sum_(s <= t) M[t, s] u_s
      const float gam = s[L::SM + t];
      o.x *= gam; o.y *= gam; o.z *= gam; o.w *= gam;
      auto add = [&](int u, auto diagonal) {
        const float4 m = *reinterpret_cast<const float4*>(s + L::M + t * LDA + u);
        const float mm[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (diagonal && u + e > t) continue;             // a later token's update, which may not be finite
          const float4 x = *reinterpret_cast<const float4*>(U_s + (u + e) * BC + cx);
          o.x = fmaf(mm[e], x.x, o.x);
          o.y = fmaf(mm[e], x.y, o.y);
          o.z = fmaf(mm[e], x.z, o.z);
          o.w = fmaf(mm[e], x.w, o.w);
        }
      };
      const int w0 = t & ~7;                               // (a warp has rows w0 .. w0 + 7)
#pragma unroll 4
      for (int u = 0; u < w0; u += 4) add(u, std::false_type());
#pragma unroll
      for (int u = 0; u < 8; u += 4) add(w0 + u, std::true_type());
      if (j * C + t < n)
        *reinterpret_cast<float4*>(a.out + ((int64_t)(start + j * C + t) * a.H + h) * a.dv + c0 + cx) = o;
    }
  }
  if (owner) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) Sg[(int64_t)(sr + i) * a.dv + sc + j] = S[i][j];
  }
}

template <int DK>
int launch(const Args& a, int places, cudaStream_t stream) {
  constexpr size_t smem = Walk<DK>::FLOATS * sizeof(float);
  static_assert(smem <= 227 * 1024, "fits a block");
  cudaError_t e = cudaFuncSetAttribute(delta_walk_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return refuse((int)e, "delta_chunks: shared memory opt-in failed: %s", cudaGetErrorString(e));
  launch_pdl(delta_chunk_kernel<DK>, dim3(places, a.H), dim3(THREADS), 0, stream, a);
  if ((e = cudaGetLastError()) != cudaSuccess) return refuse((int)e, "delta_chunks: %s", cudaGetErrorString(e));
  // a plain launch: its blocks are a chain of chunks each and have to be spread evenly over the SMs
  delta_walk_kernel<DK><<<dim3(a.dv / BC, a.H, a.B), dim3(THREADS), smem, stream>>>(a);
  return cuda_status("delta_chunks");
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

DINFER_DEFINE_LAST_ERROR()

DINFER_API int dinfer_delta_chunks_supports(int dk, int dv) { return (dk == 64 || dk == 128) && dv > 0 && dv % BC == 0; }

// As dinfer_delta_recurrence with one decay a head.  work: places * H * (32 (dk + dv) + 32 * 32 + 68) floats, places >=
// the sum over the requests of ceil(tokens / 32).
DINFER_API int dinfer_delta_chunks(const float* q, const float* k, const float* v, const float* beta, const float* decay,
                                   float* state, int64_t ld_state, const int* cu, const int* slots, const int* fresh, float* out,
                                   float* work, int places, int B, int H, int G, int dk, int dv, cudaStream_t stream) {
  if (B <= 0 || H <= 0 || G <= 0 || H % G || places < 0 || H > 65535 || B > 65535 || !dinfer_delta_chunks_supports(dk, dv))
    return refuse(DINFER_BAD_ARGUMENT, "delta_chunks: bad sizes B=%d H=%d G=%d dk=%d dv=%d", B, H, G, dk, dv);
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out) || !aligned16(work))
    return refuse(DINFER_BAD_ARGUMENT, "delta_chunks: 16-byte aligned rows");
  if (places == 0) return 0;
  Args a;
  a.q = q; a.k = k; a.v = v; a.beta = beta; a.decay = decay; a.state = state; a.ld_state = ld_state;
  a.cu = cu; a.slots = slots; a.fresh = fresh; a.out = out; a.B = B; a.H = H; a.G = G; a.dv = dv;
  const int64_t n = (int64_t)places * H;
  a.wk = work; a.wv = a.wk + n * C * dk; a.m = a.wv + n * C * dv; a.small = a.m + n * C * C;
  return dk == 64 ? launch<64>(a, places, stream) : launch<128>(a, places, stream);
}
