// C[M, N] = A[M, K] * W[N, K]^T with plain 32-bit multiply-adds on the CUDA cores: the matrix
// product of the true 32-bit model (no tensor cores, no reduced-precision matrix mode), and of a
// bfloat16 model whose file stores a matrix in 32-bit.  A, W and C may each be f32 or bf16 in
// memory; every product and sum is f32.  Any M, N, K.
//
// Two kernels: a register-tiled one for prompts (packed multiply-adds, K shared by a cluster where tiles are few), and a
// warp-per-output-column one for the few rows of a decode step.  The reference has no 32-bit path (its weights are bf16 and its
// products cuBLASLt: crates/kernels/src/gemm.rs:649-690).
#include "common.cuh"

using namespace dinfer;

namespace {

constexpr int BM = 64, BN = 128, BK = 16;      // a CTA's tile; k per stage
constexpr int TILE_THREADS = 128;
constexpr int LDK = BK + 4;                    // row stride of a staged operand (floats): eight rows' 16-byte pieces of one k
                                               // lie in different banks
constexpr int STAGES = 3;
constexpr int STAGE_FLOATS = (BM + BN) * LDK;
constexpr int LDC_S = BN + 8;                  // row stride of the partial tile
constexpr int TILE_SMEM = STAGES * STAGE_FLOATS * 4;
static_assert(BM * LDC_S <= STAGES * STAGE_FLOATS, "the partial tile takes the stages' place");
static_assert(TILE_SMEM <= 48 * 1024, "no opt-in");
constexpr int MAX_SPLITS = 8;                  // CTAs that may share a tile's K (a portable cluster)
constexpr int GRID_ROWS = 65535 * BM;          // rows of one launch (row tiles are the grid's y)
constexpr int MAX_ROWS = 65535 * 128;          // rows of one product

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes, or zeros where `live` is false (nothing is read then)
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
// two independent 32-bit multiply-adds, each rounded once (the packed form is one instruction on this machine)
__device__ __forceinline__ void fma2(uint64_t& c, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float4 ld_cluster_f4(const float* local, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
  return v;
}

// Stages rows [r0, r0 + ROWS) of an operand, k in [k0, k0 + BK), as [row][k]; rows from `rows` on and k from `k_end` on are
// zeros.  fast: 32-bit, rows of whole 16-byte pieces (K and the stride multiples of 4, the pointer aligned): cp.async;
// else through registers, element by element.
template <typename T, int ROWS>
__device__ __forceinline__ void stage_rows(float* dst, const T* __restrict__ src, int64_t ld, int r0, int rows, int k0, int k_end,
                                           bool fast) {
  if constexpr (sizeof(T) == 4) {
    if (fast) {
#pragma unroll
      for (int i = 0; i < ROWS * (BK / 4) / TILE_THREADS; ++i) {
        const int idx = threadIdx.x + i * TILE_THREADS;
        const int r = idx / (BK / 4), k = (idx % (BK / 4)) * 4;
        const bool live = r0 + r < rows && k0 + k < k_end;
        cp_async16(dst + r * LDK + k, reinterpret_cast<const float*>(src) + (live ? (int64_t)(r0 + r) * ld + k0 + k : 0), live);
      }
      return;
    }
  }
#pragma unroll 4
  for (int i = 0; i < ROWS * BK / TILE_THREADS; ++i) {
    const int idx = threadIdx.x + i * TILE_THREADS;
    const int r = idx / BK, k = idx % BK;
    dst[r * LDK + k] = (r0 + r < rows && k0 + k < k_end) ? to_f32<T>(src[(int64_t)(r0 + r) * ld + k0 + k]) : 0.f;
  }
}

// The tile kernel.  Bound by the rate of the multiply-adds: four warps own 32 x 64 of the tile each, a lane 8 x 8 (rows ly
// + 4 i, columns lx + 8 j), and a multiply-add works on two k at once (even and odd k have a sum of their own, added at
// the end), so that the operands are used as they lie in shared memory: 16 16-byte loads feed 128 packed multiply-adds.
// Three stages of 16 k.  `splits` CTAs, one cluster, share a tile's K where the tiles alone leave SMs idle (a 333-row
// product of 1024 columns is 48 tiles): each leaves its partial tile in its shared memory and all fold it in split order,
// a share of the tile each.  333 x 6144 x 1024 and 333 x 1024 x 3072 in 32-bit took 884 us with one 128 x 128 x 8 tile per
// CTA (plain multiply-adds, one stage, 24 CTAs on the second), 204 us now (31 TFLOP/s); 2048 x 6144 x 1024 644 us (40).
template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(TILE_THREADS, 2)
gemm_tile_kernel(const TA* __restrict__ A, int64_t lda, const TW* __restrict__ W, int64_t ldw,
                 TC* __restrict__ C, int64_t ldc, int M, int N, int K, int64_t sa, int64_t sw, int64_t sc, int splits,
                 int a_fast, int w_fast, int c_fast) {
  extern __shared__ __align__(16) float sm[];
  const int z = blockIdx.z / splits, rank = blockIdx.z % splits;
  A += (int64_t)z * sa; W += (int64_t)z * sw; C += (int64_t)z * sc;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // (lanes 0-7 and 8-15 read the two halves of the columns' pieces: 16 lanes' 16-byte loads then take one pass over the banks)
  const int ly = ((lane >> 2) & 1) | (lane >> 4 << 1), lx = (lane & 3) | ((lane >> 3 & 1) << 2);
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 64;
  const int tiles = (K + BK - 1) / BK;
  const int first = (int)((int64_t)tiles * rank / splits), last = (int)((int64_t)tiles * (rank + 1) / splits);

  uint64_t acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;

  auto stage = [&](int t) {
    if (t < last) {
      float* s = sm + (t - first) % STAGES * STAGE_FLOATS;
      stage_rows<TA, BM>(s, A, lda, m0, M, t * BK, K, a_fast);
      stage_rows<TW, BN>(s + BM * LDK, W, ldw, n0, N, t * BK, K, w_fast);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int u = 0; u < STAGES - 1; ++u) stage(first + u);
  for (int t = first; t < last; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                       // tile t is there, and nobody reads tile t - 1 any more
    stage(t + STAGES - 1);
    const float* as = sm + (t - first) % STAGES * STAGE_FLOATS + (wr + ly) * LDK;
    const float* ws = sm + (t - first) % STAGES * STAGE_FLOATS + (BM + wc + lx) * LDK;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 a[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + 4 * i * LDK + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + 8 * j * LDK + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < 8; ++i) fma2(acc[i][j], a[i].y, b.y);    // (a sum's two steps apart: the first takes a while)
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                         // the stages' memory takes the partial tile
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float lo = __uint_as_float((uint32_t)acc[i][j]), hi = __uint_as_float((uint32_t)(acc[i][j] >> 32));
      sm[(wr + ly + 4 * i) * LDC_S + wc + lx + 8 * j] = lo + hi;
    }
  if (splits > 1) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  } else {
    __syncthreads();
  }
  for (int v = rank * TILE_THREADS + tid; v < BM * (BN / 4); v += splits * TILE_THREADS) {
    const int r = v / (BN / 4), c = (v % (BN / 4)) * 4;
    const int m = m0 + r, n = n0 + c;
    if (m >= M || n >= N) continue;
    const float* own = sm + r * LDC_S + c;
    float4 t;
    if (splits > 1) {
      t = ld_cluster_f4(own, 0);
      for (int q = 1; q < splits; ++q) {
        const float4 u = ld_cluster_f4(own, q);
        t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
      }
    } else {
      t = *reinterpret_cast<const float4*>(own);
    }
    TC* dst = C + (int64_t)m * ldc + n;
    if (c_fast && n + 3 < N) {
      if constexpr (sizeof(TC) == 4) {
        *reinterpret_cast<float4*>(dst) = t;
      } else {
        __nv_bfloat162 p[2] = {__floats2bfloat162_rn(t.x, t.y), __floats2bfloat162_rn(t.z, t.w)};
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(p);
      }
    } else {
      const float e[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (n + u < N) dst[u] = from_f32<TC>(e[u]);
    }
  }
  if (splits > 1) {                                        // nobody leaves while others may still read its share
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
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

// M <= ROWS rows: one warp per output column n; lanes stride over K, the weight row is read once.
template <typename TA, typename TW, typename TC, int ROWS>
__global__ void __launch_bounds__(256)
gemm_rows_kernel(const TA* __restrict__ A, int64_t lda, const TW* __restrict__ W, int64_t ldw,
                 TC* __restrict__ C, int64_t ldc, int M, int N, int K, int64_t sa, int64_t sw, int64_t sc) {
  A += (int64_t)blockIdx.z * sa; W += (int64_t)blockIdx.z * sw; C += (int64_t)blockIdx.z * sc;
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

// A matrix up to which 9 to 32 rows go a warp per output column.  Two reasons: lanes sum apart, which is 0.7 of a tile's
// rounding error (a model of small 32-bit products amplifies it), and one tile or a few leave the SMs idle.  us on a tile and
// so, 9 and 32 rows in 32-bit: N 48 K 48 6.1 and 3.5, 6.6 and 4.5; N 128 K 128 11.7 and 5.5, 11.9 and 6.8; N 2048 K 128 11.7 and
// 6.1, 12.1 and 7.6; N 2048 K 16 4.5 and 3.7, 4.7 and 4.3 (back to back in a graph; every N and K measured between them alike,
// bfloat16 further apart).  At K 256 a tile is as fast, at 512 it takes 12 us and a warp a column 19 to 25.
constexpr int FEW_ROWS_K = 128, FEW_ROWS_N = 2048;

int num_sms() {                                             // of the current device, asked once
  static const int n = [] {
    int dev = 0, v = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v;
  }();
  return n;
}

template <typename TA, typename TW> struct both_bf16 { static constexpr bool value = false; };
template <> struct both_bf16<__nv_bfloat16, __nv_bfloat16> { static constexpr bool value = true; };

template <typename TA, typename TW, typename TC>
int launch(const void* A, int64_t lda, const void* W, int64_t ldw, void* C, int64_t ldc, int M, int N,
           int K, cudaStream_t stream, int batch = 1, int64_t sa = 0, int64_t sw = 0, int64_t sc = 0) {
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
  } else {
    const int64_t tiles = (int64_t)((N + BN - 1) / BN) * ((M + BM - 1) / BM) * batch;
    // as many CTAs to a tile as find room at once (two to an SM, but a cluster has to fit into what one GPC has left: 48 tiles
    // of 333 x 1024 x 3072 took 79 us with 5 CTAs each and 98 with 6, where the last clusters wait), each with at least eight
    // stages of K to itself
    int splits = 1;
    const int k_tiles = (K + BK - 1) / BK;
    while (splits < MAX_SPLITS && tiles * (splits + 1) <= num_sms() * 5 / 3 && k_tiles / (splits + 1) >= 8 &&
           (int64_t)batch * (splits + 1) <= 65535)
      ++splits;
    if (M > MAX_ROWS) return refuse(DINFER_BAD_ARGUMENT, "gemm_f32: M=%d too large", M);
    const auto fast = [](const void* q, size_t size, int64_t ld, int64_t stride) {
      return (int)((reinterpret_cast<uintptr_t>(q) % (4 * size)) == 0 && ld % 4 == 0 && stride % 4 == 0);
    };
    const int a_fast = fast(A, sizeof(TA), lda, sa) && K % 4 == 0, w_fast = fast(W, sizeof(TW), ldw, sw) && K % 4 == 0;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(TILE_THREADS); cfg.dynamicSmemBytes = TILE_SMEM; cfg.stream = stream;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = splits;
    cfg.attrs = &cluster; cfg.numAttrs = splits > 1 ? 1 : 0;
    for (int r = 0; r < M; r += GRID_ROWS) {                // (one launch up to 4.19 million rows)
      const int rows = M - r < GRID_ROWS ? M - r : GRID_ROWS;
      cfg.gridDim = dim3((N + BN - 1) / BN, (rows + BM - 1) / BM, batch * splits);
      cudaLaunchKernelEx(&cfg, gemm_tile_kernel<TA, TW, TC>, (const TA*)A + r * lda, lda, (const TW*)W, ldw, (TC*)C + r * ldc, ldc,
                         rows, N, K, sa, sw, sc, splits, a_fast, w_fast, fast(C, sizeof(TC), ldc, sc));
    }
  }
  return cuda_status("gemm_f32");
}

}  // namespace

DINFER_DEFINE_LAST_ERROR()

// A [M, K] row stride lda; W [N, K] row stride ldw; C [M, N] row stride ldc (strides in elements).
DINFER_API int dinfer_gemm_f32(const void* A, int64_t lda, int a_dtype, const void* W, int64_t ldw,
                               int w_dtype, void* C, int64_t ldc, int c_dtype, int M, int N, int K,
                               cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N)
    return refuse(DINFER_BAD_ARGUMENT, "gemm_f32: bad sizes M=%d N=%d K=%d lda=%lld ldw=%lld ldc=%lld", M, N, K,
                  (long long)lda, (long long)ldw, (long long)ldc);
  if (M == 0) return 0;
  DINFER_DISPATCH_DTYPE(a_dtype, TA,
    DINFER_DISPATCH_DTYPE(w_dtype, TW,
      DINFER_DISPATCH_DTYPE(c_dtype, TC,
        return launch<TA, TW, TC>(A, lda, W, ldw, C, ldc, M, N, K, stream))));
  return 0;
}

// The same product for `batch` independent problems: problem b reads A + b * sa, W + b * sw and writes C + b * sc
// (strides in elements; the problems of a batch may interleave inside one tensor, e.g. the heads of a row).
DINFER_API int dinfer_gemm_f32_batched(const void* A, int64_t lda, int64_t sa, int a_dtype, const void* W, int64_t ldw,
                                       int64_t sw, int w_dtype, void* C, int64_t ldc, int64_t sc, int c_dtype, int M,
                                       int N, int K, int batch, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || batch <= 0 || lda < K || ldw < K || ldc < N)
    return refuse(DINFER_BAD_ARGUMENT, "gemm_f32_batched: bad sizes M=%d N=%d K=%d batch=%d lda=%lld ldw=%lld ldc=%lld",
                  M, N, K, batch, (long long)lda, (long long)ldw, (long long)ldc);
  if (M == 0) return 0;
  DINFER_DISPATCH_DTYPE(a_dtype, TA,
    DINFER_DISPATCH_DTYPE(w_dtype, TW,
      DINFER_DISPATCH_DTYPE(c_dtype, TC,
        return launch<TA, TW, TC>(A, lda, W, ldw, C, ldc, M, N, K, stream, batch, sa, sw, sc))));
  return 0;
}
