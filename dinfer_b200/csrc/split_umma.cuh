// 32-bit operands on the tensor cores: an element x is the sum of three bfloat16 numbers h + m + l (each the rest rounded
// to nearest; 3 x 8 bits hold the 24 of a 32-bit number), and a product of two such elements is taken as
// h h' + h m' + m h' + m m' + h l' + l h', every one of them exact, summed in 32-bit.  What is left out (m l', m l', l l')
// is at most 2^-23 of the product and 2^-26 on average, less than one rounding of a 32-bit sum.  (The method, with these six of
// the nine products: Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision
// Computations", 2019.)
//
// Elements are split times 2^16, which a kernel takes out of its results again (UNSCALE for each 32-bit operand): the last digit of
// the smallest 32-bit number is then the smallest bfloat16 number's, so that the parts hold every element below 2^112 whole.  An element
// beyond, or one that is infinite or undefined, has parts that are not numbers, and a scaled sum beyond 2^128 is infinite: a
// kernel looks at its results and sums those that are not finite again with plain multiply-adds.
#pragma once
#include <atomic>

#include "umma_attention.cuh"

namespace dinfer_split {

// Lets a kernel take `bytes` of dynamic shared memory on the current device, once a device (the call costs the host a
// microsecond a launch); `done` has a bit a device.
template <typename K>
inline cudaError_t allow_shared(K kernel, size_t bytes, std::atomic<uint64_t>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

constexpr int PARTS = 3;
// the six products, the smallest first: their sums are small while they are added
constexpr int PRODUCTS = 6;
__host__ __device__ constexpr int part_a(int i) { constexpr int t[PRODUCTS] = {1, 2, 0, 1, 0, 0}; return t[i]; }
__host__ __device__ constexpr int part_b(int i) { constexpr int t[PRODUCTS] = {1, 0, 2, 0, 1, 0}; return t[i]; }

// two independent 32-bit sums, each rounded once, in one instruction
__device__ __forceinline__ uint64_t pair(float a, float b) { return (uint64_t)__float_as_uint(a) | ((uint64_t)__float_as_uint(b) << 32); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t c;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {     // a - b (the product by -1 is exact)
  uint64_t c;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(c) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
  return c;
}

// what elements are split times, and back
constexpr float SCALE = 65536.f, UNSCALE = 1.f / SCALE;

// two elements: their parts packed, the first in the lower half.  LOW: what was rounded off the elements joins the rest behind
// their first part.
template <bool LOW = false>
__device__ __forceinline__ void split2(float a, float b, uint32_t (&p)[PARTS], float a_low = 0.f, float b_low = 0.f) {
#pragma unroll
  for (int i = 0; i < PARTS; ++i) {
    p[i] = dinfer_umma::pack_bf16(a, b);
    if (i + 1 < PARTS) {
      uint64_t rest = sub2(pair(a, b), pair(__uint_as_float(p[i] << 16), __uint_as_float(p[i] & 0xffff0000u)));
      if (LOW && i == 0) rest = add2(rest, pair(a_low, b_low));
      a = __uint_as_float((uint32_t)rest);
      b = __uint_as_float((uint32_t)(rest >> 32));
    }
  }
}
// eight elements to the 16 bytes of each part, times SCALE or as they are
template <bool SCALED>
__device__ __forceinline__ void split8(const float (&x)[8], uint4 (&p)[PARTS]) {
  uint32_t q[4][PARTS];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (SCALED) {
      uint64_t v;
      asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(pair(x[2 * i], x[2 * i + 1])), "l"(0x4780000047800000ull));   // (SCALE twice)
      split2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)), q[i]);
    } else {
      split2(x[2 * i], x[2 * i + 1], q[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < PARTS; ++i) p[i] = make_uint4(q[0][i], q[1][i], q[2][i], q[3][i]);
}

// the same of x[i] * w times SCALE, the products' rounding kept
__device__ __forceinline__ void split8_times(const float (&x)[8], float w, uint4 (&p)[PARTS]) {
  uint32_t q[4][PARTS];
  w *= SCALE;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = x[2 * i] * w, b = x[2 * i + 1] * w;
    split2<true>(a, b, q[i], fmaf(x[2 * i], w, -a), fmaf(x[2 * i + 1], w, -b));
  }
#pragma unroll
  for (int i = 0; i < PARTS; ++i) p[i] = make_uint4(q[0][i], q[1][i], q[2][i], q[3][i]);
}

// A whole warp walks the MMAs and one lane issues them, so that descriptors and addresses, the same in all lanes, stay in the
// warp's uniform registers (a branch for one lane alone moves them there for every MMA, 60 to 90 cycles each).
__device__ __forceinline__ uint32_t elect_lane() {
  uint32_t lead;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(lead));
  return lead;
}
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ void mma_ts_if(uint32_t lead, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(lead) : "memory");
}
__device__ __forceinline__ void commit_if(uint32_t lead, uint32_t bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
               "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(lead) : "memory");
}

// where the 16-byte piece c of row r lies in a tile of 128-byte rows with the 128-byte swizzle (c 0..7), and in one of
// 64-byte rows with the 64-byte swizzle (c 0..3)
__device__ __forceinline__ uint32_t swizzled128(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }
__device__ __forceinline__ uint32_t swizzled64(int r, int c) { return (uint32_t)(r * 64 + ((c ^ ((r >> 1) & 3)) << 4)); }
// K-major operand tile with 64-byte rows, 64-byte swizzle: stride between 8-row groups 512 B
__device__ __forceinline__ uint64_t desc_k_major64(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)4 << 61);
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared16(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// eight columns of tensor memory, one lane a thread
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint4& a, const uint4& b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
}
// what this thread has written to shared memory is seen by MMAs that start after the barrier it arrives at next
__device__ __forceinline__ void fence_to_mma() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

}  // namespace dinfer_split
