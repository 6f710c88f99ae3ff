// NVFP4 operands in the form the block-scaled tensor-core MMA consumes.
//
//   codes : e2m1, two per byte (even element in the low nibble), rows of K/2 bytes
//   scales: e4m3 bytes, one per 16 elements, in 512-byte tiles of 128 rows x 4
//           scales: byte (r % 32) * 16 + (r / 32) * 4 + s of tile
//           (row_block * K/64 + k64_block)
// which is the layout the reference's NVFP4 cast writes for cuBLAS
// (backend/gpu/nvfp4.py:351-372) and what tcgen05.cp moves into tensor memory
// with one 32x128b.warpx4 copy per tile.
//
// Two producers: a fused cast from bfloat16 activations/weights (the arithmetic of
// quantized_ops::quantize_mx with an e2m1 table, e4m3 scale table and a global
// scale, every step rounded to bfloat16 as the op does), and a packer of the
// op's own outputs (bfloat16-valued codes and scales), which also verifies that
// every value is representable.

#include "nvfp4_cast.cuh"

namespace vq {
namespace {

// One thread = one block of 16 elements: a 32-byte load, one scale, eight code bytes; four neighbouring lanes make a
// 64-element group, whose four scale bytes its first lane writes as one word.  Two blocks per thread are in flight.
// The tensor-wide scale is `global_scale`, or follows from `amax` (and is then written to t_out).
//
// Bound by instruction issue (ALU 76 %, DRAM 38 %; 2 bytes in and 0.56 out per element): computing a block's scale once (two threads shared a block
// before) and testing the sixteen quotients' distance from a rounding boundary together took 8192 x 14336 from
// 188 to 82 us (3.7 TB/s).
constexpr int kCastBlocks = 2;
__global__ void __launch_bounds__(256)
quantize_nvfp4_kernel(const char* __restrict__ in, const void* __restrict__ global_scale, int gs_dt,
                      const float* __restrict__ amax, __nv_bfloat16* __restrict__ t_out, uint2* __restrict__ codes,
                      uint8_t* __restrict__ scales, int64_t blocks, int64_t k64_blocks, bool small, bool wide) {
  const GlobalScale g = nv_make_global(amax ? nv_global_scale(*amax) : loadp(global_scale, 0, gs_dt));
  if (t_out && blockIdx.x == 0 && threadIdx.x == 0) *t_out = __float2bfloat16_rn(g.t);
  const int64_t base = (int64_t)blockIdx.x * (256 * kCastBlocks) + threadIdx.x;
  Words8 x[kCastBlocks];
#pragma unroll
  for (int u = 0; u < kCastBlocks; ++u)
    if (base + u * 256 < blocks) x[u] = nv_load32(in + (base + u * 256) * 32, wide);
#pragma unroll
  for (int u = 0; u < kCastBlocks; ++u) {
    const int64_t v = base + u * 256;
    const bool live = v < blocks;   // whole groups of four lanes: the block count is a multiple of four
    uint32_t sb = 0;
    if (live) {
      float es;
      sb = nv_block_scale(nv_amax16(x[u].w), g, &es);
      codes[v] = nv_nearest(nv_quotients(x[u].w, es));
    }
    sb <<= 8 * (threadIdx.x & 3);
    sb |= __shfl_xor_sync(0xFFFFFFFFu, sb, 1);
    sb |= __shfl_xor_sync(0xFFFFFFFFu, sb, 2);
    if (live && (threadIdx.x & 3) == 0) {
      const int64_t grp = v >> 2;
      // 64-bit division is ~100 instructions; almost every tensor fits 32 bits
      const int64_t row = small ? (int64_t)((uint32_t)grp / (uint32_t)k64_blocks) : grp / k64_blocks;
      *reinterpret_cast<uint32_t*>(scales + nv_scale_offset(row, grp - row * k64_blocks, k64_blocks)) = sb;
    }
  }
}

// Pack the operator's outputs: bfloat16-valued e2m1 codes [rows, K] and bfloat16 scales
// [rows, K/16] whose values are e4m3 numbers.  A value that is not representable sets *bad.
__global__ void __launch_bounds__(128)
pack_nvfp4_kernel(const uint4* __restrict__ codes_in, const uint2* __restrict__ scales_in, uint4* __restrict__ codes,
                  uint8_t* __restrict__ scales, int64_t rows, int64_t K, int* __restrict__ bad) {
  const int64_t k64_blocks = K >> 6;
  const int64_t total = rows * k64_blocks;
  bool wrong = false;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = idx / k64_blocks;
    const int64_t k64 = idx - row * k64_blocks;
    const uint4* src = codes_in + idx * 8;
    uint32_t packed[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint4 x = __ldg(src + i);
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
      uint32_t nib = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xFFFF0000u);
        const uint32_t q = (uint32_t)__nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest);
        __half2_raw back = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)q, __NV_E2M1);
        const float2 fb = __half22float2(*reinterpret_cast<__half2*>(&back));
        wrong |= (fb.x != lo) | (fb.y != hi);
        nib |= q << (8 * j);
      }
      packed[i] = nib;
    }
    const uint2 sraw = __ldg(scales_in + idx);  // four bfloat16 scales
    const uint32_t sw[2] = {sraw.x, sraw.y};
    uint32_t sbytes = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float s = __uint_as_float((j & 1) ? (sw[j >> 1] & 0xFFFF0000u) : (sw[j >> 1] << 16));
      const uint32_t sb = (uint32_t)__nv_cvt_float_to_fp8(s, __NV_SATFINITE, __NV_E4M3);
      wrong |= nv_e4m3_to_float(sb) != s;
      sbytes |= sb << (8 * j);
    }
    uint4* dst = codes + idx * 2;
    dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    *reinterpret_cast<uint32_t*>(scales + nv_scale_offset(row, k64, k64_blocks)) = sbytes;
  }
  if (wrong) atomicExch(bad, 1);
}

inline int grid_for_items(int64_t items) {
  int64_t blocks = (items + 127) / 128;
  const int64_t cap = (int64_t)kSmCount * 16;
  return (int)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace
}  // namespace vq

using namespace vq;

extern "C" int64_t vq_nvfp4_scale_bytes(int64_t rows, int64_t K) {
  if (rows < 0 || K < 0) return -1;
  return ((rows + 127) / 128) * ((K + 63) / 64) * 512;
}

static int launch_quantize_nvfp4(const void* in, const void* global_scale, int gs_dt, const float* amax, void* t_out,
                                 void* codes, void* scales, int64_t rows, int64_t K, cudaStream_t st) {
  const int64_t blocks = rows * (K / 16);
  const int64_t ctas = (blocks + 256 * kCastBlocks - 1) / (256 * kCastBlocks);
  VQ_REQUIRE(ctas < (1ll << 31), "quantize_nvfp4: tensor too large");
  quantize_nvfp4_kernel<<<(unsigned)ctas, 256, 0, st>>>(
      static_cast<const char*>(in), global_scale, gs_dt, amax, static_cast<__nv_bfloat16*>(t_out),
      static_cast<uint2*>(codes), static_cast<uint8_t*>(scales), blocks, K / 64, (blocks >> 2) < 0x7FFFFFFFll && K / 64 < 0x7FFFFFFFll,
      (reinterpret_cast<uintptr_t>(in) & 31) == 0);
  return check_launch("quantize_nvfp4_kernel");
}

extern "C" int vq_quantize_nvfp4(const void* in, const void* global_scale, int global_scale_dtype, void* codes,
                                 void* scales, int64_t rows, int64_t K, void* stream) {
  VQ_REQUIRE(rows >= 0 && K >= 0, "vq_quantize_nvfp4: negative extent");
  if (rows == 0 || K == 0) return VQ_OK;
  VQ_REQUIRE(in && global_scale && codes && scales, "vq_quantize_nvfp4: null argument");
  VQ_REQUIRE(K % 64 == 0, "vq_quantize_nvfp4: K must be a multiple of 64");
  VQ_REQUIRE(((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(codes) |
               reinterpret_cast<uintptr_t>(scales)) & 15) == 0, "vq_quantize_nvfp4: misaligned buffers");
  return launch_quantize_nvfp4(in, global_scale, global_scale_dtype, nullptr, nullptr, codes, scales, rows, K,
                               static_cast<cudaStream_t>(stream));
}

extern "C" int vq_cast_nvfp4(const void* in, void* amax, int amax_given, void* codes, void* scales, void* t,
                             int64_t rows, int64_t K, void* stream) {
  VQ_REQUIRE(rows > 0 && K > 0 && K % 64 == 0, "vq_cast_nvfp4: K must be a multiple of 64, the matrix not empty");
  VQ_REQUIRE(in && amax && codes && scales && t, "vq_cast_nvfp4: null argument");
  VQ_REQUIRE(((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(codes) |
               reinterpret_cast<uintptr_t>(scales)) & 15) == 0 && (reinterpret_cast<uintptr_t>(amax) & 3) == 0,
             "vq_cast_nvfp4: misaligned buffers");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (!amax_given) {
    if (cudaMemsetAsync(amax, 0, sizeof(float), st) != cudaSuccess) return fail(VQ_ECUDA, "vq_cast_nvfp4: memset");
    if (int e = vq_amax(in, VQ_BF16, rows * K, static_cast<float*>(amax), stream)) return e;
  }
  // rows past the last full tile have scale bytes of their own
  if (rows % 128 && cudaMemsetAsync(scales, 0, (size_t)vq_nvfp4_scale_bytes(rows, K), st) != cudaSuccess)
    return fail(VQ_ECUDA, "vq_cast_nvfp4: memset");
  return launch_quantize_nvfp4(in, nullptr, 0, static_cast<const float*>(amax), t, codes, scales, rows, K, st);
}

extern "C" int vq_pack_nvfp4(const void* codes_in, const void* scales_in, void* codes, void* scales, int64_t rows,
                             int64_t K, int* bad_flag, void* stream) {
  VQ_REQUIRE(rows >= 0 && K >= 0, "vq_pack_nvfp4: negative extent");
  if (rows == 0 || K == 0) return VQ_OK;
  VQ_REQUIRE(codes_in && scales_in && codes && scales && bad_flag, "vq_pack_nvfp4: null argument");
  VQ_REQUIRE(K % 64 == 0, "vq_pack_nvfp4: K must be a multiple of 64");
  VQ_REQUIRE(((reinterpret_cast<uintptr_t>(codes_in) | reinterpret_cast<uintptr_t>(codes) |
               reinterpret_cast<uintptr_t>(scales)) & 15) == 0 && (reinterpret_cast<uintptr_t>(scales_in) & 7) == 0,
             "vq_pack_nvfp4: misaligned buffers");
  pack_nvfp4_kernel<<<grid_for_items(rows * (K / 64)), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(codes_in), static_cast<const uint2*>(scales_in), static_cast<uint4*>(codes),
      static_cast<uint8_t*>(scales), rows, K, bad_flag);
  return check_launch("pack_nvfp4_kernel");
}
