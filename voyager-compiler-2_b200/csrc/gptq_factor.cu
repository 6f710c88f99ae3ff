// The factor a GPTQ sweep walks along: U upper triangular with U^T U = H^-1 (hessian_inverse_chol, reference
// quantization/gptq.py:37-75), in one elimination.
//
// With J the exchange of rows and columns and J H J = L L^T, U = J L^-1 J: one Cholesky factorisation and one triangular
// inverse, k^3 / 3 multiply-adds each, where factor - invert - factor again takes four times that.  Both
// run here as one blocked Gauss-Jordan elimination in place on W = J H J (lower triangle): step j, for 128-row blocks,
//   diag    W[j,j] = L_jj^-1                                         (one CTA)
//   panel   P[i] = W[i,j] L_jj^-T for i > j;  W[j,k] = L_jj^-1 W[j,k] for k < j
//   update  W[i,k] -= P[i] P[k]^T for j < k <= i;  W[i,j] = -P[i] L_jj^-1;  W[i,k] -= P[i] W[j,k] for k < j
// and leaves L^-1 in W.  All of it is float32 FMAs: the update is bound by them, the diagonal blocks (one after the
// other, 128 columns each) by latency.  K = 4096: 2.9 ms (diag 33 us, panel 17 us, update 42 us a
// step on average); factor, inverse and second factor from the library took 12 ms.
#include "gptq_tile.cuh"

namespace vq {
namespace {

// W = J h^T J from the lower triangle of h (element (i, j) at i * rs + j * cs), zeros above the diagonal, an identity
// behind row k.  Tiles of 32 x 32 turned in shared memory, so that reads run along h's denser axis and writes along W's
// rows.  K = 4096: 40 us; reversing the transpose, copying it into rows and masking took 161 as tensor operators.
__global__ void __launch_bounds__(256)
factor_load_kernel(const float* __restrict__ h, int64_t rs, int64_t cs, float* __restrict__ W, int64_t k, int64_t n) {
  __shared__ float s[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t a0 = (int64_t)blockIdx.y * 32, b0 = (int64_t)blockIdx.x * 32;
  const bool along_rows = cs <= rs;
#pragma unroll
  for (int u = 0; u < 32; u += 8) {
    const int al = along_rows ? tx : ty + u, bl = along_rows ? ty + u : tx;
    const int64_t a = a0 + al, b = b0 + bl;
    float v = a == b ? 1.0f : 0.0f;
    if (a < k && b < k) v = b <= a ? __ldg(h + (k - 1 - b) * rs + (k - 1 - a) * cs) : 0.0f;
    s[al][bl] = v;
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 32; u += 8) W[(a0 + ty + u) * n + b0 + tx] = s[ty + u][tx];
}

// One 128 x 128 block: 512 threads own 4 x 8 elements each in registers, a warp 16 x 64.  Column c's raw values and row
// c's go through shared memory (two buffers, one barrier per column); then every thread eliminates its own elements: a
// factor of zero leaves the finished rows alone.  Warps whose rows are all finished, or lie above the diagonal, only
// keep the barriers.
__global__ void __launch_bounds__(512, 1)
factor_diag_kernel(float* __restrict__ W, int64_t n, int j, int* __restrict__ info) {
  __shared__ __align__(16) float col[2][128], row[2][128];
  float* base = W + ((int64_t)j * 128) * n + (int64_t)j * 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
  const int last_row = (warp >> 1) * 16 + 15;
  const bool above = (warp & 1) * 64 > last_row;
  float w[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 x = *reinterpret_cast<const float4*>(base + (ty * 4 + i) * n + tx * 8);
    const float4 y = *reinterpret_cast<const float4*>(base + (ty * 4 + i) * n + tx * 8 + 4);
    w[i][0] = x.x; w[i][1] = x.y; w[i][2] = x.z; w[i][3] = x.w;
    w[i][4] = y.x; w[i][5] = y.y; w[i][6] = y.z; w[i][7] = y.w;
  }
  bool bad = false;
  for (int cb = 0; cb < 16; ++cb) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int c = cb * 8 + u;
      float* pc = col[u & 1];
      float* pr = row[u & 1];
      if (tx == cb) {
        *reinterpret_cast<float4*>(pc + ty * 4) = make_float4(w[0][u], w[1][u], w[2][u], w[3][u]);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i][u] = 0.0f;
      }
      const bool row_owner = ty == cb * 2 + (u >> 2);
      if (row_owner) {
        *reinterpret_cast<float4*>(pr + tx * 8) = make_float4(w[u & 3][0], w[u & 3][1], w[u & 3][2], w[u & 3][3]);
        *reinterpret_cast<float4*>(pr + tx * 8 + 4) = make_float4(w[u & 3][4], w[u & 3][5], w[u & 3][6], w[u & 3][7]);
      }
      __syncthreads();
      if (last_row < c || above) continue;
      const float pivot = pc[c];
      bad |= !(pivot > 0.0f);
      // 1 / sqrt(pivot): the approximation and one Newton step
      float inv = rsqrtf(pivot);
      inv = fmaf(0.5f * inv, fmaf(-pivot * inv, inv, 1.0f), inv);
      // columns right of c: L's column (by symmetry); left of it: row c of the inverse
      const float4 lc = *reinterpret_cast<const float4*>(pc + ty * 4);
      const float* vs = tx > cb ? pc : pr;
      const float4 v0 = *reinterpret_cast<const float4*>(vs + tx * 8), v1 = *reinterpret_cast<const float4*>(vs + tx * 8 + 4);
      float l[4] = {lc.x, lc.y, lc.z, lc.w}, v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
      if (tx == cb) {
#pragma unroll
        for (int k = u; k < 8; ++k) v[k] = k == u ? 1.0f : pc[cb * 8 + k];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) l[i] = ty * 4 + i > c ? l[i] * inv : 0.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] *= inv;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 8; ++k) w[i][k] = fmaf(-l[i], v[k], w[i][k]);
      if (row_owner) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (tx * 8 + k <= c) w[u & 3][k] = v[k];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (tx * 8 + k > ty * 4 + i) w[i][k] = 0.0f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    *reinterpret_cast<float4*>(base + (ty * 4 + i) * n + tx * 8) = make_float4(w[i][0], w[i][1], w[i][2], w[i][3]);
    *reinterpret_cast<float4*>(base + (ty * 4 + i) * n + tx * 8 + 4) = make_float4(w[i][4], w[i][5], w[i][6], w[i][7]);
  }
  if (bad) atomicExch(info, 1);
}

// blockIdx.x < nb - j - 1: P[i] = W[i,j] L_jj^-T, i = j + 1 + blockIdx.x; the others: W[j,k] = L_jj^-1 W[j,k].
__global__ void __launch_bounds__(256, 2)
factor_panel_kernel(float* __restrict__ W, float* __restrict__ P, int64_t n, int j) {
  __shared__ __align__(16) GtSmem s;
  const int nb = (int)(n / 128), below = nb - j - 1;
  const float* inv = W + ((int64_t)j * 128) * n + (int64_t)j * 128;
  uint64_t acc[8][4];
  if ((int)blockIdx.x < below) {
    const int i = j + 1 + blockIdx.x;
    gt_multiply<true>(acc, s, W + ((int64_t)i * 128) * n + (int64_t)j * 128, n, inv, n, 128, 128, 128);
    float* out = P + (int64_t)i * 128 * 128;
    gt_each(acc, [&](int r, int c, float4 v) { *reinterpret_cast<float4*>(out + r * 128 + c) = v; });
  } else {
    float* tile = W + ((int64_t)j * 128) * n + (int64_t)(blockIdx.x - below) * 128;
    gt_multiply<false>(acc, s, inv, n, tile, n, 128, 128, 128);
    __syncthreads();   // the tile has been read
    gt_each(acc, [&](int r, int c, float4 v) { *reinterpret_cast<float4*>(tile + r * n + c) = v; });
  }
}

// One tile (i, k), i > j, k <= i: blockIdx.x counts them row by row.
__global__ void __launch_bounds__(256, 2)
factor_update_kernel(float* __restrict__ W, const float* __restrict__ P, int64_t n, int j) {
  __shared__ __align__(16) GtSmem s;
  int i = j + 1, k = blockIdx.x;
  while (k > i) { k -= i + 1; ++i; }
  float* tile = W + ((int64_t)i * 128) * n + (int64_t)k * 128;
  const float* p = P + (int64_t)i * 128 * 128;
  uint64_t acc[8][4];
  if (k > j) gt_multiply<true>(acc, s, p, 128, P + (int64_t)k * 128 * 128, 128, 128, 128, 128);
  else gt_multiply<false>(acc, s, p, 128, W + ((int64_t)j * 128) * n + (int64_t)k * 128, n, 128, 128, 128);
  const bool fresh = k == j;   // the panel's place: what stood here is in P
  gt_each(acc, [&](int r, int c, float4 v) {
    float4* dst = reinterpret_cast<float4*>(tile + r * n + c);
    const float4 old = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *dst;
    *dst = make_float4(old.x - v.x, old.y - v.y, old.z - v.z, old.w - v.w);
  });
}

}  // namespace
}  // namespace vq

using namespace vq;

extern "C" int vq_gptq_factor_load(const float* h, int64_t row_stride, int64_t col_stride, float* W, int64_t k, int64_t n,
                                   void* stream) {
  VQ_REQUIRE(k >= 0 && n >= k && n % 128 == 0 && n <= (1 << 20) && row_stride >= 0 && col_stride >= 0,
             "vq_gptq_factor_load: bad extents");
  if (n == 0) return VQ_OK;
  VQ_REQUIRE(W && (h || k == 0), "vq_gptq_factor_load: null argument");
  const unsigned tiles = (unsigned)(n / 32);
  factor_load_kernel<<<dim3(tiles, tiles), 256, 0, static_cast<cudaStream_t>(stream)>>>(h, row_stride, col_stride, W, k, n);
  return check_launch("factor_load_kernel");
}

extern "C" int vq_gptq_factor(float* W, float* panel, int64_t n, int* info, void* stream) {
  VQ_REQUIRE(n >= 0 && n % 128 == 0 && n <= (1 << 20), "vq_gptq_factor: the extent must be a multiple of 128");
  if (n == 0) return VQ_OK;
  VQ_REQUIRE(W && panel && info, "vq_gptq_factor: null argument");
  VQ_REQUIRE(((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(panel)) & 15) == 0, "vq_gptq_factor: misaligned buffers");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(info, 0, sizeof(int), st) != cudaSuccess) return fail(VQ_ECUDA, "vq_gptq_factor: memset");
  const int nb = (int)(n / 128);
  for (int j = 0; j < nb; ++j) {
    factor_diag_kernel<<<1, 512, 0, st>>>(W, n, j, info);
    if (nb > 1) factor_panel_kernel<<<nb - 1, 256, 0, st>>>(W, panel, n, j);
    // tiles (i, 0 .. i) for i = j + 1 .. nb - 1
    const int64_t tiles = (int64_t)nb * (nb + 1) / 2 - (int64_t)(j + 1) * (j + 2) / 2;
    if (tiles > 0) factor_update_kernel<<<(unsigned)tiles, 256, 0, st>>>(W, panel, n, j);
  }
  return check_launch("gptq factor");
}
