// Warp-level tensor-core helpers (mma.sync m16n8k16, bfloat16 in, float32 out) and
// the asynchronous-copy and matrix-load instructions the attention kernels use.
#pragma once

#include "common.cuh"

// D = A(16x16, row) * B(16x8, col) + D, float32 accumulate.
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// z / (1 + e^-y) for results that are rounded to bfloat16, as exact as expf and a division leave it: the quotient is a product with the
// approximate reciprocal (an error of about 2^-23), corrected once by what it leaves of z (Newton's step), which squares that error. The
// division branches for divisors beyond 2^126, whose reciprocals are subnormal; here both sides are taken a quarter, an infinite divisor has
// zero for a reciprocal, and what is left beside an infinity is no number and counts as any. 8.4 million of them, with the short convolution
// around: 23.5 us by the division, 15.7 here.
__device__ __forceinline__ float times_logistic(float z, float y) {
  const float divisor = 0.25f * (1.0f + expf(-y)), part = 0.25f * z;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(divisor));
  const float q = part * r;
  return fmaf(fminf(fmaf(-q, divisor, part), 3e38f), r, q);
}
__device__ __forceinline__ float silu_near(float z) { return times_logistic(z, z); }

// x and y as three pairs of bfloat16 terms each, which add up to them (24 bits of mantissa). Two conversions at once and the widening by
// hand: single conversions run on the unit of the exponentials, a quarter as fast.
__device__ __forceinline__ void split3_pair(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = pack_bf16x2(x, y);
    x -= __uint_as_float(t[i] << 16);
    y -= __uint_as_float(t[i] & 0xffff0000u);
  }
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async_16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(smem)), "l"(gmem));
}
// The same copy for bytes that are read once per step (weights): marked to leave L2 first, so that what every
// layer reads again (positions, page tables, rotation tables, gains, the rows in flight) stays there.
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(policy));
  return policy;
}
__device__ __forceinline__ void cp_async_16_stream(void* smem, const void* gmem, uint64_t policy) {
#ifdef KRK_NO_L2_HINT
  (void)policy;
  cp_async_16(smem, gmem);
#else
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;\n" ::"r"(smem_addr(smem)), "l"(gmem), "l"(policy));
#endif
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_addr(smem)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3,
                                                  const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_addr(smem)));
}

// 16-byte global load that does not pollute L1 (weights are read once per step).
__device__ __forceinline__ uint4 ld_stream_16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
