// A 128 x 128 float32 product tile on the FMA pipes, for the GPTQ solve's updates and factorisation (their arithmetic
// is float32 throughout: no tensor-core format keeps it).
//
// 256 threads, 8 x 8 accumulators each, as f32x2 pairs along the columns (half the issue slots of single FMAs, the rest
// feed the pipe); operands pass through two shared-memory buffers of 16 contraction steps, the next one loading into
// registers meanwhile.  Each accumulator adds its products in ascending order of the contraction.
#pragma once

#include "vq_common.cuh"

namespace vq {

constexpr int kGt = 128;          // tile edge
constexpr int kGtK = 16;          // contraction steps per buffer
constexpr int kGtPitch = kGt + 4;

struct GtSmem {
  float a[2][kGtK][kGtPitch];
  float b[2][kGtK][kGtPitch];
};

__device__ __forceinline__ uint64_t gt_pair(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 gt_split(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// acc[i][j]: rows ty * 8 + i, columns tx * 4 + 2 j (j < 2) and 64 + tx * 4 + 2 (j - 2), tx = tid % 16, ty = tid / 16.
// A: [rows][depth] with leading dimension lda; B: [depth][cols] (BT false) or [cols][depth] (BT true).  Rows, columns and
// depth past `rows`, `cols`, `depth` count as zeros; depth and (BT false) cols are multiples of 4, rows 16-byte aligned.
template <bool BT>
__device__ __forceinline__ void gt_multiply(uint64_t (&acc)[8][4], GtSmem& s, const float* __restrict__ A, int64_t lda,
                                            const float* __restrict__ B, int64_t ldb, int rows, int cols, int depth) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  float4 ra[2], rb[2];
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = (tid >> 2) + 64 * u, k = k0 + (tid & 3) * 4;        // 128 rows x 16 deep
      ra[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && k < depth) ra[u] = *reinterpret_cast<const float4*>(A + r * lda + k);
      rb[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (BT) {
        if (r < cols && k < depth) rb[u] = *reinterpret_cast<const float4*>(B + r * ldb + k);
      } else {
        const int kk = k0 + (tid >> 5) + 8 * u, c = (tid & 31) * 4;     // 16 deep x 128 columns
        if (kk < depth && c < cols) rb[u] = *reinterpret_cast<const float4*>(B + kk * ldb + c);
      }
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = (tid >> 2) + 64 * u, k = (tid & 3) * 4;
      s.a[buf][k][r] = ra[u].x; s.a[buf][k + 1][r] = ra[u].y; s.a[buf][k + 2][r] = ra[u].z; s.a[buf][k + 3][r] = ra[u].w;
      if (BT) {
        s.b[buf][k][r] = rb[u].x; s.b[buf][k + 1][r] = rb[u].y; s.b[buf][k + 2][r] = rb[u].z; s.b[buf][k + 3][r] = rb[u].w;
      } else {
        *reinterpret_cast<float4*>(&s.b[buf][(tid >> 5) + 8 * u][(tid & 31) * 4]) = rb[u];
      }
    }
  };
  load(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < depth; k0 += kGtK) {
    const bool more = k0 + kGtK < depth;
    if (more) load(k0 + kGtK);
#pragma unroll
    for (int k = 0; k < kGtK; ++k) {
      const float4 a0 = *reinterpret_cast<const float4*>(&s.a[buf][k][ty * 8]);
      const float4 a1 = *reinterpret_cast<const float4*>(&s.a[buf][k][ty * 8 + 4]);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&s.b[buf][k][tx * 4]);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&s.b[buf][k][64 + tx * 4]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const uint64_t bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint64_t aa = gt_pair(av[i], av[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(aa), "l"(bv[j]));
      }
    }
    if (more) {
      store(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
}

// For each of the thread's row pieces: fn(row, column, four neighbouring values).
template <typename F>
__device__ __forceinline__ void gt_each(const uint64_t (&acc)[8][4], F fn) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 x = gt_split(acc[i][2 * h]), y = gt_split(acc[i][2 * h + 1]);
      fn(ty * 8 + i, 64 * h + tx * 4, make_float4(x.x, x.y, y.x, y.y));
    }
}

}  // namespace vq
