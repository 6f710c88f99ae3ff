// Reading a packed KIVI cache: 2-bit codes (four per byte) of a [outer, T, D] bfloat16 tensor
// back to values,
//
//   out = bf16( bf16(code - zero_point) * scale )
//
// which is quantized_ops::dequantize(codes, scale, zero_point, axes, block) on the unpacked codes
// (reference ops/quantized.py:527-571; the KIVI read of quant_folding.py:2391-2547), every step
// rounded to bfloat16 as that operator does.  Keys are grouped along T (one scale and zero point
// per channel and group of `block` positions: parameters [outer, T / block, D]); values along D
// (one per position and group of `block` channels: [outer, T, D / block]).
//
// The kernels are bound by HBM: 0.25 byte in, 2 bytes out per element.  A thread owns eight
// consecutive channels (two packed bytes in, one 16-byte store out) and decodes two codes at a time
// in packed bfloat16 arithmetic: code - zero_point and the product with the scale each round once,
// as the operator's float32 steps and roundings do (a sum of two bfloat16 numbers that float32 cannot
// hold lies too far from a bfloat16 midpoint for its float32 rounding to matter).  For keys a thread
// keeps its eight scales and zero points in registers and eight threads share a group's positions,
// so that each has a group of 64 in flight as eight independent loads; for values each has four
// vectors in flight.  4 x 8 x 3968 x 128 values: 10.1 us (keys, two threads a group) and 11.6 us
// (values, one vector at a time) before, 6.8 and 6.9 us now (5.3 TB/s).
#include "vq_common.cuh"

namespace vq {
namespace {

__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); }

// four 2-bit code pairs of one 16-bit word, with each pair's zero points and scales
__device__ __forceinline__ uint4 dq8(uint32_t w, const uint32_t (&z)[4], const uint32_t (&s)[4]) {
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    // 128 + code in each half: the codes sit in the low bits of a bfloat16 whose unit is one
    const uint32_t b = ((w >> (4 * j)) & 3u) | ((w << (14 - 4 * j)) & 0x30000u) | 0x43004300u;
    const __nv_bfloat162 c = __hsub2_rn(as_bf162(b), as_bf162(0x43004300u));
    const __nv_bfloat162 r = __hmul2_rn(__hsub2_rn(c, as_bf162(z[j])), as_bf162(s[j]));
    o[j] = *reinterpret_cast<const uint32_t*>(&r);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// groups along T: (group, eight channels) items, eight threads each; four neighbouring items' threads sit side by side
constexpr int kKeyThreads = 8;
__global__ void __launch_bounds__(256)
kivi_read_keys_kernel(const uint8_t* __restrict__ packed, const __nv_bfloat16* __restrict__ scale,
                      const __nv_bfloat16* __restrict__ zero, __nv_bfloat16* __restrict__ out, int64_t groups,
                      int T_block, int D) {
  const int chunks = D >> 3;
  const int64_t item = (int64_t)blockIdx.x * (256 / kKeyThreads) + (threadIdx.x >> 5) * 4 + (threadIdx.x & 3);
  if (item >= groups * chunks) return;
  const int64_t grp = item / chunks;
  const int c = (int)(item - grp * chunks);
  const int first = (threadIdx.x >> 2) & (kKeyThreads - 1);
  const uint4 sv = __ldg(reinterpret_cast<const uint4*>(scale + grp * D + c * 8));
  const uint4 zv = __ldg(reinterpret_cast<const uint4*>(zero + grp * D + c * 8));
  const uint32_t s[4] = {sv.x, sv.y, sv.z, sv.w}, z[4] = {zv.x, zv.y, zv.z, zv.w};
  const int64_t row0 = grp * T_block;                                                   // first position of the group
  const uint8_t* src = packed + (row0 * D >> 2) + c * 2;
  __nv_bfloat16* dst = out + row0 * D + c * 8;
  const int row_bytes = D >> 2;
  int t = first;
  for (; t + 7 * kKeyThreads < T_block; t += 8 * kKeyThreads) {
    uint32_t w[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      w[u] = __ldg(reinterpret_cast<const uint16_t*>(src + (int64_t)(t + u * kKeyThreads) * row_bytes));
#pragma unroll
    for (int u = 0; u < 8; ++u)
      *reinterpret_cast<uint4*>(dst + (int64_t)(t + u * kKeyThreads) * D) = dq8(w[u], z, s);
  }
  for (; t < T_block; t += kKeyThreads)
    *reinterpret_cast<uint4*>(dst + (int64_t)t * D) =
        dq8(__ldg(reinterpret_cast<const uint16_t*>(src + (int64_t)t * row_bytes)), z, s);
}

// groups along D: one vector of eight channels of one position at a time, four per thread; `block` is a power of two
// dividing D, so a vector's group is its flat index shifted
constexpr int kValueUnroll = 4;
__global__ void __launch_bounds__(256)
kivi_read_values_kernel(const uint8_t* __restrict__ packed, const __nv_bfloat16* __restrict__ scale,
                        const __nv_bfloat16* __restrict__ zero, __nv_bfloat16* __restrict__ out, int64_t vectors,
                        int vec_shift) {
  const int64_t base = (int64_t)blockIdx.x * (256 * kValueUnroll) + threadIdx.x;
  uint32_t w[kValueUnroll], s[kValueUnroll], z[kValueUnroll];
#pragma unroll
  for (int u = 0; u < kValueUnroll; ++u) {
    const int64_t v = base + u * 256;
    if (v >= vectors) continue;
    w[u] = __ldg(reinterpret_cast<const uint16_t*>(packed) + v);
    s[u] = __bfloat16_as_ushort(scale[v >> vec_shift]);
    z[u] = __bfloat16_as_ushort(zero[v >> vec_shift]);
  }
#pragma unroll
  for (int u = 0; u < kValueUnroll; ++u) {
    const int64_t v = base + u * 256;
    if (v >= vectors) continue;
    const uint32_t s2 = s[u] | (s[u] << 16), z2 = z[u] | (z[u] << 16);
    const uint32_t sv[4] = {s2, s2, s2, s2}, zv[4] = {z2, z2, z2, z2};
    reinterpret_cast<uint4*>(out)[v] = dq8(w[u], zv, sv);
  }
}

}  // namespace
}  // namespace vq

using namespace vq;

extern "C" int vq_kivi_read_2bit(const void* packed, const void* scale, const void* zero_point, void* out,
                                 int64_t outer, int64_t T, int64_t D, int along_channels, int64_t block,
                                 void* stream) {
  VQ_REQUIRE(outer >= 0 && T >= 0 && D >= 0 && block > 0, "vq_kivi_read_2bit: bad extents");
  if (outer == 0 || T == 0 || D == 0) return VQ_OK;
  VQ_REQUIRE(packed && scale && zero_point && out, "vq_kivi_read_2bit: null argument");
  VQ_REQUIRE(D % 8 == 0 && D < (1 << 20), "vq_kivi_read_2bit: the channel count must be a multiple of 8");
  VQ_REQUIRE(((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(scale) |
               reinterpret_cast<uintptr_t>(zero_point)) & 15) == 0 && (reinterpret_cast<uintptr_t>(packed) & 1) == 0,
             "vq_kivi_read_2bit: buffers must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (along_channels) {
    VQ_REQUIRE(block >= 8 && (block & (block - 1)) == 0 && D % block == 0,
               "vq_kivi_read_2bit: channel groups are a power of two, at least 8, dividing D");
    int shift = 0;
    while ((1ll << shift) < block) ++shift;
    const int64_t vectors = outer * T * (D / 8);
    const int64_t blocks = (vectors + 256 * kValueUnroll - 1) / (256 * kValueUnroll);
    VQ_REQUIRE(blocks < (1ll << 31), "vq_kivi_read_2bit: tensor too large");
    kivi_read_values_kernel<<<(unsigned)blocks, 256, 0, st>>>(static_cast<const uint8_t*>(packed),
                                                              static_cast<const __nv_bfloat16*>(scale),
                                                              static_cast<const __nv_bfloat16*>(zero_point),
                                                              static_cast<__nv_bfloat16*>(out), vectors, shift - 3);
    return check_launch("kivi_read_values_kernel");
  }
  VQ_REQUIRE(T % block == 0 && block < (1 << 20), "vq_kivi_read_2bit: position groups must divide T");
  const int64_t groups = outer * (T / block);
  const int64_t items = groups * (D / 8);
  const int64_t blocks = (items + 256 / kKeyThreads - 1) / (256 / kKeyThreads);
  VQ_REQUIRE(blocks < (1ll << 31), "vq_kivi_read_2bit: tensor too large");
  kivi_read_keys_kernel<<<(unsigned)blocks, 256, 0, st>>>(static_cast<const uint8_t*>(packed),
                                                         static_cast<const __nv_bfloat16*>(scale),
                                                         static_cast<const __nv_bfloat16*>(zero_point),
                                                         static_cast<__nv_bfloat16*>(out), groups, (int)block, (int)D);
  return check_launch("kivi_read_keys_kernel");
}
