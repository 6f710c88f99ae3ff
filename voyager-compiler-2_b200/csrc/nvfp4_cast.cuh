// Sixteen-element blocks of bfloat16 to e2m1 codes and an e4m3 block scale, shared by the NVFP4 casts.
#pragma once

#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include "quantize_shared.cuh"

namespace vq {

__device__ __forceinline__ float nv_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float nv_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ float nv_bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ uint32_t nv_pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float nv_e4m3_to_float(uint32_t byte) {
  __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)byte, __NV_E4M3);
  return __half2float(*reinterpret_cast<__half*>(&h));
}
// byte offset of a row's four scales of one 64-element group in the 128 x 4 tiles
__device__ __forceinline__ int64_t nv_scale_offset(int64_t row, int64_t k64, int64_t k64_blocks) {
  return ((row >> 7) * k64_blocks + k64) * 512 + (row & 31) * 16 + ((row & 127) >> 5) * 4;
}

// 32 bytes of global memory that nothing writes during the kernel; `wide`: 32-byte aligned (else 16)
struct Words8 { uint32_t w[8]; };
__device__ __forceinline__ Words8 nv_load32(const void* p, bool wide) {
  Words8 r;
  if (wide) {
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]), "=r"(r.w[6]),
                   "=r"(r.w[7]) : "l"(p));
  } else {
    const uint4 a = __ldg(static_cast<const uint4*>(p)), b = __ldg(static_cast<const uint4*>(p) + 1);
    r.w[0] = a.x; r.w[1] = a.y; r.w[2] = a.z; r.w[3] = a.w;
    r.w[4] = b.x; r.w[5] = b.y; r.w[6] = b.z; r.w[7] = b.w;
  }
  return r;
}

// The tensor-wide scale t = max(bf16(bf16(amax) / (6 * 448)), smallest normal float32), NaN kept.
__device__ __forceinline__ float nv_global_scale(float amax) {
  const float r = nv_bf16r(__fdiv_rn(nv_bf16r(amax), 2688.0f));
  const float tiny = 1.17549435e-38f;
  return r < tiny ? tiny : r;
}

struct GlobalScale {
  float t, rcp;
  bool ordinary;
};
__device__ __forceinline__ GlobalScale nv_make_global(float t) { return {t, __frcp_rn(t), ordinary_divisor(t)}; }

// largest |x| bits of sixteen bfloat16 values (NaN patterns order above infinity)
__device__ __forceinline__ uint32_t nv_amax16(const uint32_t (&w)[8]) {
  uint32_t m = w[0] & 0x7FFF7FFFu;
#pragma unroll
  for (int j = 1; j < 8; ++j) m = __vmaxu2(m, w[j] & 0x7FFF7FFFu);
  return max(m & 0xFFFFu, m >> 16);
}

// e4m3 byte of bf16(bf16(amax / 6) / t), 1 where that is not positive; *es = bf16(scale * t) divides the elements
__device__ __forceinline__ uint32_t nv_scale_byte(float q, const GlobalScale& g, float* es) {
  uint32_t sb = (uint32_t)__nv_cvt_float_to_fp8(q, __NV_SATFINITE, __NV_E4M3);
  float s = nv_e4m3_to_float(sb);
  if (!(s > 0.0f)) { s = 1.0f; sb = 0x38u; }
  *es = nv_bf16r(__fmul_rn(s, g.t));
  return sb;
}
__device__ __forceinline__ uint32_t nv_block_scale(uint32_t amax_bits16, const GlobalScale& g, float* es) {
  const float amax = __uint_as_float(amax_bits16 << 16);
  const uint32_t e = amax_bits16 >> 7;
  float q;
  if (g.ordinary && e >= 1u && e <= 254u)
    q = div_to_bf16(div_to_bf16(amax, 6.0f, 1.0f / 6.0f), g.t, g.rcp);   // exact quotients, no true division
  else
    q = nv_bf16r(__fdiv_rn(nv_bf16r(__fdiv_rn(amax, 6.0f)), g.t));
  return nv_scale_byte(q, g, es);
}

static __device__ __noinline__ Words8 nv_quotients_exact(Words8 x, float es) {
  Words8 q;
#pragma unroll
  for (int j = 0; j < 8; ++j) q.w[j] = nv_pack2(__fdiv_rn(nv_lo(x.w[j]), es), __fdiv_rn(nv_hi(x.w[j]), es));
  return q;
}

// bf16(x / es): products with the correctly rounded reciprocal, unless one of the sixteen lies within 2 ulp of a
// bfloat16 midpoint.  (A quotient too small or too large for that argument differs only where no code does.)
__device__ __forceinline__ Words8 nv_quotients(const uint32_t (&w)[8], float es) {
  const float rcp = __frcp_rn(es);
  uint32_t near = 0xFFFFFFFFu;
  Words8 q;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float a = __fmul_rn(nv_lo(w[j]), rcp), b = __fmul_rn(nv_hi(w[j]), rcp);
    near = min(near, min(__float_as_uint(a) * 65536u - 0x7FFD0000u, __float_as_uint(b) * 65536u - 0x7FFD0000u));
    q.w[j] = nv_pack2(a, b);
  }
  if (near <= 0x0006FFFFu || !ordinary_divisor(es)) {
    Words8 x;
#pragma unroll
    for (int j = 0; j < 8; ++j) x.w[j] = w[j];
    q = nv_quotients_exact(x, es);
  }
  return q;
}

// eight code bytes (even element in the low nibble), nearest with ties to even; a zero quotient is +0
__device__ __forceinline__ uint2 nv_nearest(const Words8& q) {
  uint32_t nib[2] = {0, 0};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 f = make_float2(__fadd_rn(nv_lo(q.w[j]), 0.0f), __fadd_rn(nv_hi(q.w[j]), 0.0f));
    nib[j >> 2] |= (uint32_t)__nv_cvt_float2_to_fp4x2(f, __NV_E2M1, cudaRoundNearest) << (8 * (j & 3));
  }
  return make_uint2(nib[0], nib[1]);
}

// Philox4x32-10 on (block index, seed): sixteen random bytes, one per element of the block (philox_byte's bytes)
__device__ __forceinline__ uint4 nv_philox(uint64_t counter, uint64_t seed) {
  uint32_t c0 = (uint32_t)counter, c1 = (uint32_t)(counter >> 32), c2 = 0, c3 = 0;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)c0 * 0xD2511F53ull, p1 = (uint64_t)c2 * 0xCD9E8D57ull;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0, n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
    c0 = n0; c1 = (uint32_t)p1; c2 = n2; c3 = (uint32_t)p0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return make_uint4(c0, c1, c2, c3);
}

// One magnitude of the e2m1 grid 0, .5, 1, 1.5, 2, 3, 4, 6: the level towards zero, or the next one when
// |x| + noise * gap reaches it.  A value on the grid keeps its level (the noise is below one).  A NaN becomes 4 and a
// zero +0, as the level search of the operator leaves them.
__device__ __forceinline__ float nv_stochastic1(float v, uint32_t byte) {
  if (v != v) return 4.0f;
  const float a = fminf(fabsf(v), 6.0f);
  const float gap = a < 2.0f ? 0.5f : (a < 4.0f ? 1.0f : 2.0f), per = a < 2.0f ? 2.0f : (a < 4.0f ? 1.0f : 0.5f);
  const float near = __fmul_rn(floorf(__fmul_rn(a, per)), gap), far = __fadd_rn(near, gap);
  const float noise = __fmul_rn((float)byte, 1.0f / 256.0f);
  const float r = __fadd_rn(a, __fmul_rn(noise, gap)) >= far ? far : near;
  return __fadd_rn(copysignf(r, v), 0.0f);
}
__device__ __forceinline__ uint2 nv_stochastic(const Words8& q, uint64_t block, uint64_t seed) {
  const uint4 rnd = nv_philox(block, seed);
  const uint32_t rw[4] = {rnd.x, rnd.y, rnd.z, rnd.w};
  uint32_t nib[2] = {0, 0};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t two = rw[j >> 1] >> (16 * (j & 1));
    const float2 f = make_float2(nv_stochastic1(nv_lo(q.w[j]), two & 0xFFu), nv_stochastic1(nv_hi(q.w[j]), (two >> 8) & 0xFFu));
    nib[j >> 2] |= (uint32_t)__nv_cvt_float2_to_fp4x2(f, __NV_E2M1, cudaRoundNearest) << (8 * (j & 3));
  }
  return make_uint2(nib[0], nib[1]);
}

}  // namespace vq
