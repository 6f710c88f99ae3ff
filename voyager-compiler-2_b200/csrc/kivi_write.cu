// Writing a packed KIVI cache: a bfloat16 [outer, T, D] tensor to 2-bit codes (four per byte) with one
// scale and zero point per group, in one pass -- quantized_ops::quantize_affine (reference
// ops/quantized.py:1227-1283) with the codes 0..3, followed by their packing.
//
// Bound by instruction issue on the ALU pipe (80 % busy at 15 to 20 instructions per element, DRAM 34 to 42 %), hence the
// packed pairs and few divisions.  A warp keeps its whole group in registers, so the input is read once and the
// bfloat16-valued codes are never written:
//   * group minima and maxima on packed bfloat16 pairs (NaN propagates, as in torch.amin / amax);
//   * the group's scale and zero point are computed by one lane each and handed round by shuffles;
//   * x / scale as a product with the correctly rounded reciprocal, re-done with a true division only
//     when one of a thread's eight quotients lies within 2 ulp of a bfloat16 midpoint.  Quotients too
//     small for that argument change no code: beside any zero point they round away or give code 0;
//   * the sum with the zero point rounds once in bfloat16 (float32 and then bfloat16 gives the same),
//     is clamped, and adding 128 leaves the rounded code in the low bits.
// Groups whose scale or zero point is not an ordinary number take the element-by-element arithmetic.
//
// 4 x 8 x 3968 x 128 values: 82 us (keys) and 67 us (values) as quantize_affine and pack_codes, 13.3 and 14.8 us
// here; writing and reading back a cache of that size takes 42 us of the device's time and 56 through the Python entry
// points (182 before).
#include "quantize_shared.cuh"

namespace vq {
namespace {

__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); }
__device__ __forceinline__ uint32_t bits_of(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
__device__ __forceinline__ float lo_of(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_of(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// Eight codes, one after the other, for any scale and zero point.
__device__ __noinline__ uint32_t codes8_exact(uint4 x, uint4 s, uint4 z) {
  const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, sw[4] = {s.x, s.y, s.z, s.w}, zw[4] = {z.x, z.y, z.z, z.w};
  uint32_t acc = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float xv = j & 1 ? hi_of(xw[j >> 1]) : lo_of(xw[j >> 1]);
    const float sv = j & 1 ? hi_of(sw[j >> 1]) : lo_of(sw[j >> 1]);
    const float zv = j & 1 ? hi_of(zw[j >> 1]) : lo_of(zw[j >> 1]);
    float y = Elem<VQ_BF16>::round(__fdiv_rn(xv, sv));
    y = Elem<VQ_BF16>::round(__fadd_rn(y, zv));
    acc |= ((uint32_t)__float2int_rn(round_int(y, 0.0f, 3.0f)) & 3u) << (2 * j);
  }
  return acc;
}

// The same for ordinary scales and finite zero points; rcp: the scales' correctly rounded reciprocals.
__device__ __forceinline__ uint32_t codes8(const uint4& x, const uint4& s, const uint4& z, const float (&rcp)[8]) {
  const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, zw[4] = {z.x, z.y, z.z, z.w};
  uint32_t q[4], near = 0xFFFFFFFFu;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a = __fmul_rn(lo_of(xw[j]), rcp[2 * j]), b = __fmul_rn(hi_of(xw[j]), rcp[2 * j + 1]);
    // low sixteen bits in 0x7FFD .. 0x8003: close to a midpoint of two bfloat16 numbers
    near = min(near, min(__float_as_uint(a) * 65536u - 0x7FFD0000u, __float_as_uint(b) * 65536u - 0x7FFD0000u));
    q[j] = bits_of(__floats2bfloat162_rn(a, b));
  }
  if (near <= 0x0006FFFFu) return codes8_exact(x, s, z);
  uint32_t acc = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    __nv_bfloat162 t = __hadd2_rn(as_bf162(q[j]), as_bf162(zw[j]));
    t = __hmin2(__hmax2(t, as_bf162(0u)), as_bf162(0x40404040u));
    const uint32_t u = bits_of(__hadd2_rn(t, as_bf162(0x43004300u)));
    acc |= ((u & 3u) | ((u >> 14) & 12u)) << (4 * j);
  }
  return acc;
}

// Scale and zero point of one group as one word (scale in the low half), its reciprocal, and whether both are ordinary.
__device__ __forceinline__ uint32_t group_params(float low, float high, const Round& sr, float* rcp, bool* plain) {
  float s, z;
  affine_params<VQ_BF16>(low, high, 0.0f, 3.0f, sr, &s, &z);
  *plain = ordinary_divisor(s) && fabsf(z) <= 3.4e38f;
  *rcp = __fdiv_rn(1.0f, s);
  return (__float_as_uint(s) >> 16) | (__float_as_uint(z) & 0xFFFF0000u);
}

__device__ __forceinline__ void min_max(uint32_t& lo, uint32_t& hi, uint32_t lo2, uint32_t hi2) {
  lo = bits_of(__hmin2_nan(as_bf162(lo), as_bf162(lo2)));
  hi = bits_of(__hmax2_nan(as_bf162(hi), as_bf162(hi2)));
}

struct KiviWriteParams {
  const uint4* in;
  uint16_t* scale;
  uint16_t* zero;
  uint16_t* packed;   // eight codes per word
  int64_t units;      // keys: groups x strips; values: vectors of eight
  int row_vecs;       // D / 8
  Round scale_round;
};

// Keys: a warp owns 32 channels of one group of 8 * NP positions.  Lane c + 4 p holds channels 8 c .. 8 c + 7 of
// positions p, p + 8, ...; the four lanes of a row read 64 neighbouring bytes.  After the reduction over p every lane
// has all minima and maxima of its channels, and lane p computes channel p's parameters.
template <int NP>
__global__ void __launch_bounds__(128)
kivi_write_keys_kernel(KiviWriteParams P) {
  __shared__ uint16_t steps[2 * VQ_MAX_STEPS];
  stage_steps(P.scale_round, steps);
  const int lane = threadIdx.x & 31, c = lane & 3, p = lane >> 2;
  const int64_t unit = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (unit >= P.units) return;
  const int strips = P.row_vecs >> 2;
  const int64_t grp = unit / strips;
  const int strip = (int)(unit - grp * strips);
  const int64_t first = (grp * (8 * NP) + p) * P.row_vecs + strip * 4 + c;
  uint4 x[NP];
#pragma unroll
  for (int i = 0; i < NP; ++i) x[i] = __ldg(P.in + first + (int64_t)(i * 8) * P.row_vecs);
  uint32_t lo[4] = {x[0].x, x[0].y, x[0].z, x[0].w}, hi[4] = {x[0].x, x[0].y, x[0].z, x[0].w};
#pragma unroll
  for (int i = 1; i < NP; ++i) {
    min_max(lo[0], hi[0], x[i].x, x[i].x);
    min_max(lo[1], hi[1], x[i].y, x[i].y);
    min_max(lo[2], hi[2], x[i].z, x[i].z);
    min_max(lo[3], hi[3], x[i].w, x[i].w);
  }
#pragma unroll
  for (int off = 4; off < 32; off <<= 1)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      min_max(lo[j], hi[j], __shfl_xor_sync(0xFFFFFFFFu, lo[j], off), __shfl_xor_sync(0xFFFFFFFFu, hi[j], off));
  const uint32_t lp = p & 4 ? (p & 2 ? lo[3] : lo[2]) : (p & 2 ? lo[1] : lo[0]);
  const uint32_t hp = p & 4 ? (p & 2 ? hi[3] : hi[2]) : (p & 2 ? hi[1] : hi[0]);
  float r;
  bool plain;
  const uint32_t sz = group_params(p & 1 ? hi_of(lp) : lo_of(lp), p & 1 ? hi_of(hp) : lo_of(hp), P.scale_round, &r, &plain);
  const int64_t pi = grp * (P.row_vecs * 8) + strip * 32 + c * 8 + p;
  P.scale[pi] = (uint16_t)sz;
  P.zero[pi] = (uint16_t)(sz >> 16);
  float rcp[8];
  uint32_t s[4], z[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t a = __shfl_sync(0xFFFFFFFFu, sz, 8 * j + c), b = __shfl_sync(0xFFFFFFFFu, sz, 8 * j + 4 + c);
    rcp[2 * j] = __shfl_sync(0xFFFFFFFFu, r, 8 * j + c);
    rcp[2 * j + 1] = __shfl_sync(0xFFFFFFFFu, r, 8 * j + 4 + c);
    s[j] = __byte_perm(a, b, 0x5410);
    z[j] = __byte_perm(a, b, 0x7632);
  }
  const uint4 sv = make_uint4(s[0], s[1], s[2], s[3]), zv = make_uint4(z[0], z[1], z[2], z[3]);
  if (__all_sync(0xFFFFFFFFu, plain)) {
#pragma unroll
    for (int i = 0; i < NP; ++i)
      P.packed[first + (int64_t)(i * 8) * P.row_vecs] = (uint16_t)codes8(x[i], sv, zv, rcp);
  } else {
#pragma unroll
    for (int i = 0; i < NP; ++i)
      P.packed[first + (int64_t)(i * 8) * P.row_vecs] = (uint16_t)codes8_exact(x[i], sv, zv);
  }
}

// Values: G = block / 8 neighbouring lanes hold a group; a warp has four runs of 32 vectors in flight, and lane l of a
// group computes the parameters of the run l & 3 (a fourth of the divisions it would take to compute them everywhere).
constexpr int kRuns = 4;
template <int G>
__global__ void __launch_bounds__(256)
kivi_write_values_kernel(KiviWriteParams P) {
  __shared__ uint16_t steps[2 * VQ_MAX_STEPS];
  stage_steps(P.scale_round, steps);
  const int lane = threadIdx.x & 31, l = lane & (G - 1);
  const int64_t base = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * (32 * kRuns) + lane;
  uint4 x[kRuns];
  uint32_t mine = 0;   // (min, max) of the run whose parameters this lane computes
#pragma unroll
  for (int u = 0; u < kRuns; ++u) {
    x[u] = make_uint4(0, 0, 0, 0);
    if (base + u * 32 < P.units) x[u] = __ldg(P.in + base + u * 32);
  }
#pragma unroll
  for (int u = 0; u < kRuns; ++u) {
    uint32_t lo = x[u].x, hi = x[u].x;
    min_max(lo, hi, x[u].y, x[u].y);
    min_max(lo, hi, x[u].z, x[u].z);
    min_max(lo, hi, x[u].w, x[u].w);
    // fold the halves: minimum in the low half, maximum in the high half
    uint32_t mm = __byte_perm(bits_of(__hmin2_nan(as_bf162(lo), as_bf162(lo >> 16))),
                              bits_of(__hmax2_nan(as_bf162(hi), as_bf162(hi >> 16))), 0x5410);
#pragma unroll
    for (int off = 1; off < G; off <<= 1) {
      const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, mm, off);
      mm = __byte_perm(bits_of(__hmin2_nan(as_bf162(mm), as_bf162(other))),
                       bits_of(__hmax2_nan(as_bf162(mm), as_bf162(other))), 0x7610);
    }
    if ((l & (kRuns - 1)) == u) mine = mm;
  }
  float r;
  bool plain;
  const uint32_t sz = group_params(lo_of(mine), hi_of(mine), P.scale_round, &r, &plain);
  if (l < kRuns && base + l * 32 < P.units) {
    const int64_t pi = (base + l * 32) / G;
    P.scale[pi] = (uint16_t)sz;
    P.zero[pi] = (uint16_t)(sz >> 16);
  }
  const bool all_plain = __all_sync(0xFFFFFFFFu, plain);
#pragma unroll
  for (int u = 0; u < kRuns; ++u) {
    const int src = (lane & ~(G - 1)) + u;
    const uint32_t w = __shfl_sync(0xFFFFFFFFu, sz, src);
    const float rv = __shfl_sync(0xFFFFFFFFu, r, src);
    const uint32_t s2 = __byte_perm(w, w, 0x1010), z2 = __byte_perm(w, w, 0x3232);
    const uint4 sv = make_uint4(s2, s2, s2, s2), zv = make_uint4(z2, z2, z2, z2);
    const float rcp[8] = {rv, rv, rv, rv, rv, rv, rv, rv};
    if (base + u * 32 < P.units)
      P.packed[base + u * 32] = (uint16_t)(all_plain ? codes8(x[u], sv, zv, rcp) : codes8_exact(x[u], sv, zv));
  }
}

}  // namespace
}  // namespace vq

using namespace vq;

extern "C" int vq_kivi_write_2bit(const void* in, void* scale, void* zero_point, void* packed, int64_t outer, int64_t T,
                                  int64_t D, int along_channels, int64_t block, const VqRound* scale_round,
                                  void* stream) {
  VQ_REQUIRE(outer >= 0 && T >= 0 && D >= 0 && block > 0, "vq_kivi_write_2bit: bad extents");
  if (outer == 0 || T == 0 || D == 0) return VQ_OK;
  VQ_REQUIRE(in && scale && zero_point && packed, "vq_kivi_write_2bit: null argument");
  if (int e = validate_round(scale_round, "scale rounding")) return e;
  // blocks that fill a warp's registers without a remainder; the rest goes through vq_quantize_affine + vq_pack_codes
  if ((block != 32 && block != 64 && block != 128) || D >= (1 << 20) ||
      (along_channels ? D % block : (T % block || D % 32)) || (reinterpret_cast<uintptr_t>(in) & 15) ||
      (reinterpret_cast<uintptr_t>(packed) & 1))
    return fail(VQ_EUNSUPPORTED, "vq_kivi_write_2bit: not a layout of whole 32-, 64- or 128-element groups");
  KiviWriteParams P{};
  P.in = static_cast<const uint4*>(in);
  P.scale = static_cast<uint16_t*>(scale);
  P.zero = static_cast<uint16_t*>(zero_point);
  P.packed = static_cast<uint16_t*>(packed);
  P.row_vecs = (int)(D / 8);
  P.scale_round = make_round(scale_round);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (along_channels) {
    P.units = outer * T * (D / 8);
    const int64_t blocks = (P.units + 256 * kRuns - 1) / (256 * kRuns);
    VQ_REQUIRE(blocks < (1ll << 31), "vq_kivi_write_2bit: tensor too large");
    if (block == 32) kivi_write_values_kernel<4><<<(unsigned)blocks, 256, 0, st>>>(P);
    else if (block == 64) kivi_write_values_kernel<8><<<(unsigned)blocks, 256, 0, st>>>(P);
    else kivi_write_values_kernel<16><<<(unsigned)blocks, 256, 0, st>>>(P);
    return check_launch("kivi_write_values_kernel");
  }
  P.units = outer * (T / block) * (D / 32);
  const int64_t blocks = (P.units + 3) / 4;
  VQ_REQUIRE(blocks < (1ll << 31), "vq_kivi_write_2bit: tensor too large");
  if (block == 32) kivi_write_keys_kernel<4><<<(unsigned)blocks, 128, 0, st>>>(P);
  else if (block == 64) kivi_write_keys_kernel<8><<<(unsigned)blocks, 128, 0, st>>>(P);
  else kivi_write_keys_kernel<16><<<(unsigned)blocks, 128, 0, st>>>(P);
  return check_launch("kivi_write_keys_kernel");
}
