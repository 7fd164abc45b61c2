// out[n] = x . W[n, :] for one token in bfloat16, sums in 32-bit: the products of a single chat's decode step.  What such a
// product takes is its way from the input to the output, not the weights' from memory: a tile on the tensor cores (gemm_tc.cu)
// goes through TMA, MMA, commit, tensor memory and a fold over a cluster behind the last kernel's end, this one through shared
// memory, multiply-adds and five exchanges.
//
// A warp takes R weight rows at a time, a lane every 32nd piece of eight k, R * G = 16 pieces in flight a lane.  The first ones are
// asked for before the kernels in front have finished (weights depend on none of them); a piece's registers take the next
// piece as soon as it is used.  The input lies in shared memory in 32-bit.  Three more things it does:
//   * gate: the rows are (gate, up) pairs and out[j] = silu(gate_j) * up_j;
//   * norm: the input is not given but made, by every CTA for itself: h = bfloat16(v * rsqrt(mean(v^2) + eps) * w) of v = residual (+
//     delta), what the norm's kernel would have left; the first CTA writes v to another buffer (others still read the old one);
//   * out in bfloat16 or 32-bit.
//
// Bound by that way: the input's load (behind the weights' on the same path), a barrier or two, 16 pieces' multiply-adds a lane.  A
// step of a 28-layer model of 1024 channels 830 us with tiles and norm kernels, 667 so; figures by size stand at the rule
// (parts/linear.py).  (The input by cp.async: 4.9 us for the first of them instead of 3.5.  Two and four tokens: 5.4 and 9.2.)
//
// The reference's small-M products are mma.sync kernels (crates/kernels/cuda/gemm_small_m.cu:148-285), its norms kernels of their
// own (crates/kernels/cuda/norm.cu:41-116).
#include "common.cuh"

using namespace dinfer;

namespace {

constexpr int THREADS = 256, WARPS = THREADS / 32;
constexpr int MAX_K = 12 * 1024 - 16;              // the input in shared memory in 32-bit beside the warps' sums, no opt-in

struct Params {
  const __nv_bfloat16* w; int64_t ldw;
  const __nv_bfloat16* x;                          // null: from the norm
  void* out;
  int N, K;
  const float* residual;                           // [K]
  const __nv_bfloat16* delta;                      // [K]; null: nothing to add
  float* residual_out;                             // [K], with delta
  const void* norm_w; int norm_w_f32; float eps;
};

__device__ __forceinline__ uint4 load_once(const __nv_bfloat16* p) {           // weights are read once: not into L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float low(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float high(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
// two independent 32-bit multiply-adds, each rounded once
__device__ __forceinline__ void fma2(uint64_t& c, uint32_t u, uint64_t x) {      // u: two bfloat16 elements
  const uint64_t w = (uint64_t)(u << 16) | ((uint64_t)(u & 0xffff0000u) << 32);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(w), "l"(x));
}
template <typename T> __device__ __forceinline__ T cast(float v);
template <> __device__ __forceinline__ float cast<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 cast<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// grid: CTAs of WARPS warps, which share the batches of R rows
template <int R, int G, bool GATED, bool NORM, typename OutT>
__global__ void __launch_bounds__(THREADS, 2) gemv_kernel(const Params p) {
  extern __shared__ __align__(16) float xs[];      // elements 0-3 of every piece, then elements 4-7: [2][pieces][4]
  __shared__ float red[WARPS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pieces = p.K / 8, steps = (pieces + 31) / 32;      // of a row; of a lane
  const int batches = (p.N + R - 1) / R, stride = gridDim.x * WARPS;
  int batch = blockIdx.x * WARPS + warp;
  pdl_launch_dependents();

  uint4 w[G][R];
  const auto fetch = [&](int b, int s, int r) {    // piece s * 32 + lane of row r of batch b
    const int n = b * R + r, piece = s * 32 + lane;
    return b < batches && n < p.N && piece < pieces ? load_once(p.w + (int64_t)n * p.ldw + piece * 8) : make_uint4(0u, 0u, 0u, 0u);
  };
#pragma unroll
  for (int g = 0; g < G; ++g)
#pragma unroll
    for (int r = 0; r < R; ++r) w[g][r] = fetch(batch, g, r);
  const auto at = [&](int k) { return xs + ((k >> 2) & 1) * pieces * 4 + (k >> 3) * 4; };      // four elements from k on
  if constexpr (NORM) {
    // four elements a thread at a time; the first ones stay in registers, the rest of a long row is read again
    constexpr int HOLD = 4;
    float4 v[HOLD], g[HOLD];
    const auto weight = [&](int k) {               // (a weight: ahead of the wait)
      if (p.norm_w_f32) return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.norm_w) + k);
      const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p.norm_w) + k);
      return make_float4(low(u.x), high(u.x), low(u.y), high(u.y));
    };
    const auto value = [&](int k) {
      float4 a = *reinterpret_cast<const float4*>(p.residual + k);
      if (p.delta) {
        const uint2 d = *reinterpret_cast<const uint2*>(p.delta + k);
        a.x += low(d.x); a.y += high(d.x); a.z += low(d.y); a.w += high(d.y);
      }
      return a;
    };
    float ss = 0.f;
    const auto add = [&](int k, const float4& a) {
      ss = fmaf(a.x, a.x, fmaf(a.y, a.y, fmaf(a.z, a.z, fmaf(a.w, a.w, ss))));
      if (p.delta && blockIdx.x == 0) *reinterpret_cast<float4*>(p.residual_out + k) = a;
    };
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int k = (i * THREADS + tid) * 4;
      g[i] = v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < p.K) g[i] = weight(k);
    }
    pdl_wait();
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int k = (i * THREADS + tid) * 4;
      if (k < p.K) v[i] = value(k);
    }
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int k = (i * THREADS + tid) * 4;
      if (k < p.K) add(k, v[i]);
    }
    for (int k = (HOLD * THREADS + tid) * 4; k < p.K; k += THREADS * 4) add(k, value(k));
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < WARPS; ++i) s += red[i];
    const float rinv = rsqrtf(s / (float)p.K + p.eps);
    const auto put = [&](int k, const float4& a, const float4& g4) {
      const auto r = [](float f) { return __bfloat162float(__float2bfloat16_rn(f)); };
      *reinterpret_cast<float4*>(at(k)) = make_float4(r(a.x * rinv * g4.x), r(a.y * rinv * g4.y), r(a.z * rinv * g4.z), r(a.w * rinv * g4.w));
    };
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int k = (i * THREADS + tid) * 4;
      if (k < p.K) put(k, v[i], g[i]);
    }
    for (int k = (HOLD * THREADS + tid) * 4; k < p.K; k += THREADS * 4) put(k, value(k), weight(k));
  } else {
    pdl_wait();
    for (int c = tid; c < pieces; c += THREADS) {
      const uint4 u = *reinterpret_cast<const uint4*>(p.x + c * 8);
      *reinterpret_cast<float4*>(xs + c * 4) = make_float4(low(u.x), high(u.x), low(u.y), high(u.y));
      *reinterpret_cast<float4*>(xs + pieces * 4 + c * 4) = make_float4(low(u.z), high(u.z), low(u.w), high(u.w));
    }
  }
  __syncthreads();

  OutT* out = reinterpret_cast<OutT*>(p.out);
  for (; batch < batches; batch += stride) {
    uint64_t acc[R][2];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = 0ull;
    for (int s0 = 0; s0 < steps; s0 += G) {
      const bool on = s0 + G < steps;
      const int nb = on ? batch : batch + stride, ns = on ? s0 + G : 0;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const int piece = (s0 + g) * 32 + lane;
        ulonglong2 lo = make_ulonglong2(0ull, 0ull), hi = lo;
        if (piece < pieces) {
          lo = *reinterpret_cast<const ulonglong2*>(xs + piece * 4);
          hi = *reinterpret_cast<const ulonglong2*>(xs + pieces * 4 + piece * 4);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          fma2(acc[r][0], w[g][r].x, lo.x);
          fma2(acc[r][1], w[g][r].y, lo.y);
          fma2(acc[r][0], w[g][r].z, hi.x);
          fma2(acc[r][1], w[g][r].w, hi.y);
          w[g][r] = fetch(nb, ns + g, r);
        }
      }
    }
    float sum[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float a = __uint_as_float((uint32_t)acc[r][0]) + __uint_as_float((uint32_t)(acc[r][0] >> 32));
      const float b = __uint_as_float((uint32_t)acc[r][1]) + __uint_as_float((uint32_t)(acc[r][1] >> 32));
      sum[r] = warp_sum(a + b);
    }
    if (lane == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int n = batch * R + r;
        if constexpr (GATED) {
          if (r % 2 == 0 && n + 1 < p.N) out[n >> 1] = cast<OutT>(sum[r] / (1.f + expf(-sum[r])) * sum[r + 1]);
        } else {
          if (n < p.N) out[n] = cast<OutT>(sum[r]);
        }
      }
    }
  }
}

int num_sms() {                                             // of the current device, asked once
  static const int n = [] {
    int dev = 0, v = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

template <int R, int G, bool GATED, bool NORM, typename OutT>
int launch(const Params& p, cudaStream_t stream) {
  const int batches = (p.N + R - 1) / R, warps = 2 * num_sms() * WARPS;
  const int each = (batches + warps - 1) / warps;            // batches of a warp: the same for all, as far as they go
  const int grid = ((batches + each - 1) / each + WARPS - 1) / WARPS;
  const cudaError_t e = launch_pdl(gemv_kernel<R, G, GATED, NORM, OutT>, dim3(grid), dim3(THREADS), (size_t)p.K * 4, stream, p);
  if (e != cudaSuccess) return refuse((int)e, "gemv: launch failed: %s", cudaGetErrorString(e));
  return cuda_status("gemv");
}
template <bool GATED, bool NORM, typename OutT>
int pick(const Params& p, cudaStream_t stream) {
  // Fewer rows a warp keep more warps busy, more of them share the reads of the input.  us a launch with 1, 2 and 4 rows, a chain over
  // more matrices than L2 holds, plain and with the norm (gated products go as those): 1024 x 1024 2.9, 3.0, 3.1 and 3.5, 3.0, 2.8; 1024 x 3072
  // 3.8, 5.0, 5.8 and 4.1, 4.8, 6.2; 2046 x 1024 3.1, 3.2, 3.5 and 3.9, 3.6, 3.0; 2048 x 2048 3.6, 4.1, 5.1 and 4.3, 3.9, 5.0; 2560 x
  // 1024 4.9, 3.4, 3.7 and 5.6, 3.6, 3.0; 4094 x 1024 5.2, 3.6, 4.2 and 5.8, 4.0, 3.7; 4096 x 1536 5.5, 4.4, 5.7 and 6.2, 4.6, 5.6;
  // 5000 x 1024 7.0, 5.3, 4.6 and 7.7, 5.6, 4.5.  So the lines suit K 1024 with the norm in front, as decode steps of such layers have it; a
  // plain product of 2048 to 4096 rows, and K from 1536 on, would do a fifth better with half as many rows.
  if (p.N >= 4096) return launch<4, 4, GATED, NORM, OutT>(p, stream);
  if (p.N >= 2048 || GATED) return launch<2, 8, GATED, NORM, OutT>(p, stream);
  if constexpr (!GATED) return launch<1, 16, false, NORM, OutT>(p, stream);
  return 0;
}
template <bool GATED, bool NORM>
int pick(const Params& p, bool f32, cudaStream_t stream) {
  return f32 ? pick<GATED, NORM, float>(p, stream) : pick<GATED, NORM, __nv_bfloat16>(p, stream);
}

bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

DINFER_DEFINE_LAST_ERROR()

// x [K] bfloat16, or null with residual [K] f32, delta [K] bfloat16 (or null), residual_out [K] f32 (with delta: gets residual +
// delta; not the residual itself), norm_w [K] (f32 or bfloat16) and eps.  w [N, K] bfloat16 (row stride ldw), out [N] (gated: [N /
// 2]) bfloat16 or f32.
DINFER_API int dinfer_gemv(const void* x, const void* w, int64_t ldw, void* out, int out_f32, int N, int K, int gated,
                           const float* residual, const void* delta, float* residual_out, const void* norm_w, int norm_w_f32, float eps,
                           cudaStream_t stream) {
  if (N <= 0 || K <= 0 || K > MAX_K || (gated && (N & 1)) || ldw < K) return refuse(DINFER_BAD_ARGUMENT, "gemv: bad sizes N=%d K=%d", N, K);
  if (K % 8 || ldw % 8 || !al16(w)) return refuse(DINFER_BAD_ARGUMENT, "gemv: weight rows of whole 16-byte pieces");
  if (x ? !al16(x) : (!residual || !norm_w || !al16(residual) || !al16(norm_w) ||
                      (delta && (!al16(delta) || !residual_out || !al16(residual_out) || residual_out == residual))))
    return refuse(DINFER_BAD_ARGUMENT, "gemv: 16-byte aligned vectors, and another buffer for the new residual");
  Params p{};
  p.w = (const __nv_bfloat16*)w; p.ldw = ldw; p.x = (const __nv_bfloat16*)x; p.out = out; p.N = N; p.K = K;
  p.residual = residual; p.delta = (const __nv_bfloat16*)delta; p.residual_out = residual_out;
  p.norm_w = norm_w; p.norm_w_f32 = norm_w_f32; p.eps = eps;
  if (x) return gated ? pick<true, false>(p, out_f32 != 0, stream) : pick<false, false>(p, out_f32 != 0, stream);
  return gated ? pick<true, true>(p, out_f32 != 0, stream) : pick<false, true>(p, out_f32 != 0, stream);
}
