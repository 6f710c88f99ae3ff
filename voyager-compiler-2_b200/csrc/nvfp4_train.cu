// The casts of an NVFP4 training step: a matrix for its forward GEMM and its transpose for the weight-gradient GEMM
// (optionally rotated and stochastically rounded), and a weight in 16 x 16 blocks packed both ways -- reference
// backend/gpu/nvfp4.py:953-1017, with the arithmetic of quantized_ops::hadamard_rotate, calculate_global_scale and
// quantize_mx (ops/quantized.py:1038-1115), every step rounded to bfloat16 as those operators do.
//
// Each takes two passes over the matrix: the tensor-wide amax (of the rotated transpose too, which is not stored), then
// one kernel that reads 64 x 128 tiles and writes both packed forms.  HBM moves 2 x 2 bytes in and 2 x 0.56 out per
// element and is 10 to 25 % busy: the amax pass waits for its loads, the casts are bound by instruction issue (ALU 61 %;
// 30 instructions per element of a square weight, 78 of a rotated, stochastically rounded pair).  The rotation, 16
// float32 FMAs per element in the operator's order, is issued as f32x2 over two output columns with the matrix
// broadcast from shared memory, once per pass: a stored rotated transpose would cost 4 bytes per element more.
//
// 4096 x 4096: a rotated pair 62 us (96 with both forms stochastically rounded) and a square weight 33 us; as operators
// of their own (rotate, transpose, amax, quantize, pack, the level table rebuilt and read by the host) the three casts
// of a training step of one linear took 1850 us, with 110 launches, and take 200 here.
#include "nvfp4_cast.cuh"

namespace vq {
namespace {

__device__ __forceinline__ uint64_t pair64(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint32_t round2(uint64_t v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return nv_pack2(a, b);
}

// A run of sixteen rows of two neighbouring columns (x[i]: row i, the left column in the low half), as two blocks of
// sixteen.  ROTATE: out[j] = bf16(sum_k x[k] m[k][j]), fp32, k ascending.
template <bool ROTATE>
__device__ __forceinline__ void column_runs(const uint32_t (&x)[16], const float* m, uint32_t (&left)[8],
                                            uint32_t (&right)[8]) {
  if (!ROTATE) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      left[j] = __byte_perm(x[2 * j], x[2 * j + 1], 0x5410);
      right[j] = __byte_perm(x[2 * j], x[2 * j + 1], 0x7632);
    }
    return;
  }
  uint64_t l[8], r[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) l[j] = r[j] = 0ull;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const uint64_t xl = pair64(nv_lo(x[k]), nv_lo(x[k])), xr = pair64(nv_hi(x[k]), nv_hi(x[k]));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const ulonglong2 mm = *reinterpret_cast<const ulonglong2*>(m + k * 16 + j * 4);
      fma2(l[2 * j], xl, mm.x);
      fma2(l[2 * j + 1], xl, mm.y);
      fma2(r[2 * j], xr, mm.x);
      fma2(r[2 * j + 1], xr, mm.y);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    left[j] = round2(l[j]);
    right[j] = round2(r[j]);
  }
}

__device__ __forceinline__ void stage_matrix(float* m, const float* matrix) {
  if (threadIdx.x < 256) m[threadIdx.x] = matrix[threadIdx.x];
}

// amax[0] = max |x| and, for the rotated runs of sixteen rows, amax[1] = max |bf16(rotation)| (atomicMax on zeroed words).
// A thread takes two columns of one run: sixteen independent 4-byte loads, 128 bytes per warp and row.
__global__ void __launch_bounds__(256)
rotated_amax_kernel(const uint32_t* __restrict__ x, const float* __restrict__ matrix, uint32_t* __restrict__ amax,
                    int64_t runs, int pairs) {
  __shared__ __align__(16) float m[256];
  __shared__ uint32_t warp_max[2][8];
  stage_matrix(m, matrix);
  __syncthreads();
  uint32_t plain = 0, turned = 0;
  const int pair = blockIdx.x * 256 + threadIdx.x;
  for (int64_t run = blockIdx.y; run < runs && pair < pairs; run += gridDim.y) {
    const uint32_t* p = x + run * 16 * pairs + pair;
    uint32_t w[16], l[8], r[8];
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = __ldg(p + (int64_t)i * pairs);
#pragma unroll
    for (int i = 0; i < 16; ++i) plain = __vmaxu2(plain, w[i] & 0x7FFF7FFFu);
    column_runs<true>(w, m, l, r);
#pragma unroll
    for (int j = 0; j < 8; ++j) turned = __vmaxu2(turned, __vmaxu2(l[j] & 0x7FFF7FFFu, r[j] & 0x7FFF7FFFu));
  }
  for (int off = 16; off; off >>= 1) {
    plain = __vmaxu2(plain, __shfl_xor_sync(0xFFFFFFFFu, plain, off));
    turned = __vmaxu2(turned, __shfl_xor_sync(0xFFFFFFFFu, turned, off));
  }
  if ((threadIdx.x & 31) == 0) {
    warp_max[0][threadIdx.x >> 5] = plain;
    warp_max[1][threadIdx.x >> 5] = turned;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    uint32_t v = 0;
    for (int w = 0; w < 8; ++w) v = __vmaxu2(v, warp_max[threadIdx.x][w]);
    v = max(v & 0xFFFFu, v >> 16) << 16;   // non-negative float bits order like integers
    if (v > *const_cast<volatile uint32_t*>(amax + threadIdx.x)) atomicMax(amax + threadIdx.x, v);
  }
}

constexpr int kTileM = 64, kTileK = 128;
constexpr int kPitch = kTileK * 2 + 16;      // bytes per staged row: 16-byte accesses of a quarter warp hit every bank once
constexpr int kCodePitch = kTileM / 2 + 8;   // bytes per column of staged transposed codes

struct TrainCastParams {
  const char* in;        // [M, K] bfloat16
  const float* matrix;   // 16 x 16 or null
  const float* amax;     // of the matrix, of its rotated transpose
  const int64_t* seed;
  const int64_t* seed_t;
  uint8_t *codes, *scales, *codes_t, *scales_t;
  __nv_bfloat16 *t, *t_t;
  int64_t M, K;
  bool wide;             // the input is 32-byte aligned
  unsigned col_tiles;    // blockIdx.x counts the tiles row by row (a grid's second extent would end at 4 million rows)
};

struct __align__(16) TrainTile {
  uint8_t x[kTileM * kPitch];
  uint8_t codes[kTileK * kCodePitch];
  uint8_t scales[kTileK * 4];
  float m[256];
};

// Thread's two row blocks: row tid / 4, columns (tid & 3) * 16 and 64 further on.
__device__ __forceinline__ void load_tile(const TrainCastParams& P, TrainTile& s, int64_t m0, int64_t k0, Words8 (&x)[2]) {
  const int row = threadIdx.x >> 2, c = (threadIdx.x & 3) * 16;
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    if (k0 + b * 64 >= P.K) continue;
    x[b] = nv_load32(P.in + ((m0 + row) * P.K + k0 + c + b * 64) * 2, P.wide);
    uint4* dst = reinterpret_cast<uint4*>(s.x + row * kPitch + (c + b * 64) * 2);
    dst[0] = make_uint4(x[b].w[0], x[b].w[1], x[b].w[2], x[b].w[3]);
    dst[1] = make_uint4(x[b].w[4], x[b].w[5], x[b].w[6], x[b].w[7]);
  }
}

// codes and scale byte of row block b; the four lanes of a 64-element group write their scales as one word
__device__ __forceinline__ void store_row_block(const TrainCastParams& P, int64_t m0, int64_t k0, int b, uint2 nib,
                                                uint32_t sb) {
  const int64_t row = m0 + (threadIdx.x >> 2), k = k0 + b * 64;
  *reinterpret_cast<uint2*>(P.codes + (row * P.K + k) / 2 + (threadIdx.x & 3) * 8) = nib;
  sb <<= 8 * (threadIdx.x & 3);
  sb |= __shfl_xor_sync(0xFFFFFFFFu, sb, 1);
  sb |= __shfl_xor_sync(0xFFFFFFFFu, sb, 2);
  if ((threadIdx.x & 3) == 0)
    *reinterpret_cast<uint32_t*>(P.scales + nv_scale_offset(row, k >> 6, P.K >> 6)) = sb;
}

__device__ __forceinline__ void stage_column(TrainTile& s, int col, int run, uint2 nib, uint32_t sb) {
  *reinterpret_cast<uint2*>(s.codes + col * kCodePitch + run * 8) = nib;
  s.scales[col * 4 + run] = (uint8_t)sb;
}

// the tile's transposed codes (32 bytes per column) and scales (one word per column: a whole 512-byte tile)
__device__ __forceinline__ void store_columns(const TrainCastParams& P, const TrainTile& s, int64_t m0, int64_t k0) {
  for (int i = threadIdx.x; i < kTileK * 4; i += 256) {
    const int col = i >> 2, part = i & 3;
    if (k0 + col < P.K)
      *reinterpret_cast<uint2*>(P.codes_t + ((k0 + col) * P.M + m0) / 2 + part * 8) =
          *reinterpret_cast<const uint2*>(s.codes + col * kCodePitch + part * 8);
  }
  if (threadIdx.x < kTileK && k0 + threadIdx.x < P.K)
    *reinterpret_cast<uint32_t*>(P.scales_t + nv_scale_offset(k0 + threadIdx.x, m0 >> 6, P.M >> 6)) =
        *reinterpret_cast<const uint32_t*>(s.scales + threadIdx.x * 4);
}

template <bool ROTATE, bool SEED, bool SEED_T>
__global__ void __launch_bounds__(256, 3)
cast_pair_kernel(const __grid_constant__ TrainCastParams P) {
  __shared__ TrainTile s;
  const int64_t k0 = (int64_t)(blockIdx.x % P.col_tiles) * kTileK, m0 = (int64_t)(blockIdx.x / P.col_tiles) * kTileM;
  if (ROTATE) stage_matrix(s.m, P.matrix);
  Words8 x[2];
  load_tile(P, s, m0, k0, x);
  const GlobalScale g = nv_make_global(nv_global_scale(P.amax[0]));
  const GlobalScale gt = ROTATE ? nv_make_global(nv_global_scale(P.amax[1])) : g;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *P.t = __float2bfloat16_rn(g.t);
    *P.t_t = __float2bfloat16_rn(gt.t);
  }
  const uint64_t seed = SEED ? (uint64_t)*P.seed : 0, seed_t = SEED_T ? (uint64_t)*P.seed_t : 0;
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    if (k0 + b * 64 >= P.K) continue;
    float es;
    const uint32_t sb = nv_block_scale(nv_amax16(x[b].w), g, &es);
    const Words8 q = nv_quotients(x[b].w, es);
    const uint64_t flat = (uint64_t)((m0 + (threadIdx.x >> 2)) * P.K + k0 + b * 64 + (threadIdx.x & 3) * 16);
    store_row_block(P, m0, k0, b, SEED ? nv_stochastic(q, flat >> 4, seed) : nv_nearest(q), sb);
  }
  __syncthreads();
  const int pair = threadIdx.x & 63, run = threadIdx.x >> 6;
  if (k0 + pair * 2 < P.K) {
    uint32_t w[16], col[2][8];
#pragma unroll
    for (int i = 0; i < 16; ++i)
      w[i] = *reinterpret_cast<const uint32_t*>(s.x + (run * 16 + i) * kPitch + pair * 4);
    column_runs<ROTATE>(w, s.m, col[0], col[1]);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float es;
      const uint32_t sb = nv_block_scale(nv_amax16(col[c]), gt, &es);
      const Words8 q = nv_quotients(col[c], es);
      const uint64_t flat = (uint64_t)((k0 + pair * 2 + c) * P.M + m0 + run * 16);
      stage_column(s, pair * 2 + c, run, SEED_T ? nv_stochastic(q, flat >> 4, seed_t) : nv_nearest(q), sb);
    }
  }
  __syncthreads();
  store_columns(P, s, m0, k0);
}

// 16 x 16 blocks: a block's scale e4m3(min(bf16(bf16(amax * (1 / 6)) / t), 448)); its elements once by rows, once by columns.
__global__ void __launch_bounds__(256, 3)
cast_square_kernel(const __grid_constant__ TrainCastParams P) {
  __shared__ TrainTile s;
  __shared__ uint16_t row_max[kTileM][8];
  __shared__ float block_es[4][8];
  __shared__ uint32_t block_sb[4][8];
  const int64_t k0 = (int64_t)(blockIdx.x % P.col_tiles) * kTileK, m0 = (int64_t)(blockIdx.x / P.col_tiles) * kTileM;
  const int row = threadIdx.x >> 2;
  Words8 x[2];
  load_tile(P, s, m0, k0, x);
  const GlobalScale g = nv_make_global(nv_global_scale(P.amax[0]));
  if (blockIdx.x == 0 && threadIdx.x == 0) *P.t = __float2bfloat16_rn(g.t);
#pragma unroll
  for (int b = 0; b < 2; ++b)
    if (k0 + b * 64 < P.K) row_max[row][b * 4 + (threadIdx.x & 3)] = (uint16_t)nv_amax16(x[b].w);
  __syncthreads();
  if (threadIdx.x < 32) {
    const int run = threadIdx.x >> 3, c = threadIdx.x & 7;
    if (k0 + c * 16 < P.K) {
      uint32_t m = 0;
#pragma unroll
      for (int i = 0; i < 16; ++i) m = max(m, (uint32_t)row_max[run * 16 + i][c]);
      const float sixth = nv_bf16r(__fmul_rn(__uint_as_float(m << 16), 1.0f / 6.0f));
      block_sb[run][c] = nv_scale_byte(nv_bf16r(__fdiv_rn(sixth, g.t)), g, &block_es[run][c]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    if (k0 + b * 64 >= P.K) continue;
    const int c = b * 4 + (threadIdx.x & 3);
    store_row_block(P, m0, k0, b, nv_nearest(nv_quotients(x[b].w, block_es[row >> 4][c])), block_sb[row >> 4][c]);
  }
  const int pair = threadIdx.x & 63, run = threadIdx.x >> 6;
  if (k0 + pair * 2 < P.K) {
    uint32_t w[16], col[2][8];
#pragma unroll
    for (int i = 0; i < 16; ++i)
      w[i] = *reinterpret_cast<const uint32_t*>(s.x + (run * 16 + i) * kPitch + pair * 4);
    column_runs<false>(w, nullptr, col[0], col[1]);
#pragma unroll
    for (int c = 0; c < 2; ++c)
      stage_column(s, pair * 2 + c, run, nv_nearest(nv_quotients(col[c], block_es[run][pair >> 3])),
                   block_sb[run][pair >> 3]);
  }
  __syncthreads();
  store_columns(P, s, m0, k0);
}

// scale bytes of the rows that fill up a last tile of 128
int zero_ragged_scales(void* scales, int64_t rows, int64_t K, cudaStream_t st) {
  if (rows % 128 && cudaMemsetAsync(scales, 0, (size_t)vq_nvfp4_scale_bytes(rows, K), st) != cudaSuccess)
    return fail(VQ_ECUDA, "NVFP4 cast: memset");
  return VQ_OK;
}

int64_t tile_count(const TrainCastParams& P) { return P.M / kTileM * P.col_tiles; }

int check_train_cast(const TrainCastParams& P, const char* what) {
  VQ_REQUIRE(P.M > 0 && P.K > 0 && P.M % 64 == 0 && P.K % 64 == 0, "%s: both extents must be positive multiples of 64", what);
  VQ_REQUIRE(P.K < (1ll << 31) && tile_count(P) < (1ll << 31), "%s: matrix too large", what);
  VQ_REQUIRE(P.in && P.amax && P.codes && P.scales && P.codes_t && P.scales_t && P.t, "%s: null argument", what);
  VQ_REQUIRE(((reinterpret_cast<uintptr_t>(P.in) | reinterpret_cast<uintptr_t>(P.codes) | reinterpret_cast<uintptr_t>(P.scales) |
               reinterpret_cast<uintptr_t>(P.codes_t) | reinterpret_cast<uintptr_t>(P.scales_t)) & 15) == 0 &&
             (reinterpret_cast<uintptr_t>(P.amax) & 3) == 0, "%s: misaligned buffers", what);
  return VQ_OK;
}

}  // namespace
}  // namespace vq

using namespace vq;

extern "C" int vq_cast_nvfp4_pair(const void* in, const float* matrix, const int64_t* seed, const int64_t* seed_t,
                                  float* amax, void* codes, void* scales, void* t, void* codes_t, void* scales_t,
                                  void* t_t, int64_t M, int64_t K, void* stream) {
  TrainCastParams P{static_cast<const char*>(in), matrix, amax, seed, seed_t, static_cast<uint8_t*>(codes),
                    static_cast<uint8_t*>(scales), static_cast<uint8_t*>(codes_t), static_cast<uint8_t*>(scales_t),
                    static_cast<__nv_bfloat16*>(t), static_cast<__nv_bfloat16*>(t_t), M, K,
                    (reinterpret_cast<uintptr_t>(in) & 31) == 0, (unsigned)((K + kTileK - 1) / kTileK)};
  if (int e = check_train_cast(P, "vq_cast_nvfp4_pair")) return e;
  VQ_REQUIRE(t_t, "vq_cast_nvfp4_pair: null argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(amax, 0, 2 * sizeof(float), st) != cudaSuccess) return fail(VQ_ECUDA, "vq_cast_nvfp4_pair: memset");
  if (int e = zero_ragged_scales(scales, M, K, st)) return e;
  if (int e = zero_ragged_scales(scales_t, K, M, st)) return e;
  if (matrix) {
    const int64_t runs = M / 16;
    const dim3 grid((unsigned)((K / 2 + 255) / 256), (unsigned)(runs < 65535 ? runs : 65535));
    rotated_amax_kernel<<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(in), matrix,
                                              reinterpret_cast<uint32_t*>(amax), runs, (int)(K / 2));
    if (int e = check_launch("rotated_amax_kernel")) return e;
  } else if (int e = vq_amax(in, VQ_BF16, M * K, amax, stream)) {
    return e;
  }
  const unsigned grid = (unsigned)tile_count(P);
#define VQ_PAIR(R) \
  (seed ? (seed_t ? cast_pair_kernel<R, true, true><<<grid, 256, 0, st>>>(P) : cast_pair_kernel<R, true, false><<<grid, 256, 0, st>>>(P)) \
        : (seed_t ? cast_pair_kernel<R, false, true><<<grid, 256, 0, st>>>(P) : cast_pair_kernel<R, false, false><<<grid, 256, 0, st>>>(P)))
  if (matrix) VQ_PAIR(true);
  else VQ_PAIR(false);
#undef VQ_PAIR
  return check_launch("cast_pair_kernel");
}

extern "C" int vq_cast_nvfp4_square(const void* in, float* amax, void* codes, void* scales, void* codes_t,
                                    void* scales_t, void* t, int64_t N, int64_t K, void* stream) {
  TrainCastParams P{static_cast<const char*>(in), nullptr, amax, nullptr, nullptr, static_cast<uint8_t*>(codes),
                    static_cast<uint8_t*>(scales), static_cast<uint8_t*>(codes_t), static_cast<uint8_t*>(scales_t),
                    static_cast<__nv_bfloat16*>(t), nullptr, N, K,
                    (reinterpret_cast<uintptr_t>(in) & 31) == 0, (unsigned)((K + kTileK - 1) / kTileK)};
  if (int e = check_train_cast(P, "vq_cast_nvfp4_square")) return e;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(amax, 0, sizeof(float), st) != cudaSuccess) return fail(VQ_ECUDA, "vq_cast_nvfp4_square: memset");
  if (int e = zero_ragged_scales(scales, N, K, st)) return e;
  if (int e = zero_ragged_scales(scales_t, K, N, st)) return e;
  if (int e = vq_amax(in, VQ_BF16, N * K, amax, stream)) return e;
  cast_square_kernel<<<(unsigned)tile_count(P), 256, 0, st>>>(P);
  return check_launch("cast_square_kernel");
}
