// GPTQ column sweep against a block-scaled grid, on the device.
//
// For one block of `bs` input channels (columns) of a weight [rows, K]:
//   1. each row takes its scale from the current, already compensated values
//      (microscaling: amax / quant_max through the scale table; or group-wise
//      affine: (max - min) / (qmax - qmin) with a zero point);
//   2. the block's columns are rounded one after the other; each column's
//      error over its pivot U[c][c] is propagated into the block's later
//      columns with U's row c (U = upper Cholesky factor of the inverse Hessian);
//   3. the trailing columns receive  work[:, end:] -= deltas @ U[start:end, end:].
// Rows never interact.  Eight lanes share a row, each with four neighbouring columns of every 32 in registers; U's
// diagonal tile stands in shared memory, and every arithmetic step is a separately rounded fp32 operation in
// the order the reference's column loop performs them.  The columns are a serial chain -- quotient, rounding,
// difference, quotient by the pivot, broadcast, update -- and that latency is what the kernel's time is: 128 columns
// of 4096 rows take 38 us, 387 us with a thread per row and its 128 values updated one by one.

#include "gptq_tile.cuh"
#include "quantize_shared.cuh"

namespace vq {
namespace {

constexpr float kEps = 1e-12f;  // the reference's EPS clamp on scales and pivots
constexpr int kMaxBlock = 128;
constexpr int kBlockThreads = 128;
constexpr int kRowsPerCta = kBlockThreads / 8;
constexpr int kShrinkCandidates = 5;

struct GptqBlockParams {
  float* work;          // [rows, K] fp32, updated in place inside the block
  float* out;           // [rows, K] fp32, receives the block's grid values
  float* deltas;        // [rows, bs] fp32
  const float* U;       // [K, K] fp32 upper triangular
  const float* salience;  // [K] fp32 (shrink search weights) or null
  int64_t rows, K;
  int start, n;         // block = columns [start, start + n)
  int affine;           // 0: microscaling scale; 1: group-wise affine (scale + zero point)
  float quant_min, quant_max;
  int shrink;
  int vec;              // rows of work, out and deltas are whole 16-byte pieces
  Round scale_round;    // rounding of the scale (microscaling)
  Round round;          // element grid
};

template <int MODE>
__device__ __forceinline__ float grid_value(const Round& r, float w, float scale, float zero, bool affine) {
  // quantize(w / scale [+ zero]) then back to the weight's units
  float y = __fdiv_rn(w, scale);
  if (affine) y = __fadd_rn(y, zero);
  float code = apply_round<MODE>(r, y, 0);
  if (affine) code = __fsub_rn(code, zero);
  return __fmul_rn(code, scale);
}

// NQ: groups of 32 columns.  MODE: the element grid's rounding at compile time, or -1.
template <int NQ, int MODE>
__global__ void __launch_bounds__(kBlockThreads)
gptq_block_kernel(const __grid_constant__ GptqBlockParams p) {
  constexpr int W = 32 * NQ;
  extern __shared__ __align__(16) float tile[];  // strictly upper part of U[start:start+n, start:start+n], W x W
  __shared__ uint16_t s_steps[2][2 * VQ_MAX_STEPS];
  __shared__ float s_pivot[W];
  Round round = p.round, scale_round = p.scale_round;
  stage_steps(round, s_steps[0]);
  stage_steps(scale_round, s_steps[1]);
  const int n = p.n;
  for (int t = threadIdx.x; t < W * W; t += kBlockThreads) {
    const int r = t / W, c = t - r * W;
    tile[t] = r < c && c < n ? p.U[(int64_t)(p.start + r) * p.K + p.start + c] : 0.0f;
  }
  for (int t = threadIdx.x; t < W; t += kBlockThreads)
    s_pivot[t] = t < n ? fmaxf(p.U[(int64_t)(p.start + t) * p.K + p.start + t], kEps) : 1.0f;
  __syncthreads();
  const int lane = threadIdx.x & 31, l = lane & 7, first = lane & 24;
  const int64_t row = (int64_t)blockIdx.x * kRowsPerCta + (threadIdx.x >> 3);
  const bool live = row < p.rows;

  float w[4 * NQ];   // column 32 q + 4 l + e
  const float* wrow = p.work + (live ? row : p.rows - 1) * p.K + p.start;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int c = 32 * q + 4 * l;
    if (p.vec) {
      const float4 v = c < n ? *reinterpret_cast<const float4*>(wrow + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) w[4 * q + e] = c + e < n ? wrow[c + e] : 0.0f;
    }
  }

  // ---- per-row scale (and zero point) from the block as compensated so far ----
  const bool affine = p.affine != 0;
  float scale, zero = 0.0f;
  if (affine) {
    float lo = __uint_as_float(0x7FC00000u), hi = lo;   // a NaN is no minimum or maximum
#pragma unroll
    for (int i = 0; i < 4 * NQ; ++i)
      if (32 * (i >> 2) + 4 * l + (i & 3) < n) { lo = fminf(lo, w[i]); hi = fmaxf(hi, w[i]); }
    for (int off = 1; off < 8; off <<= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, off));
      hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, off));
    }
    scale = __fdiv_rn(__fsub_rn(hi, lo), __fsub_rn(p.quant_max, p.quant_min));
    scale = scale > 0.0f ? scale : 1.0f;
    zero = __fadd_rn(__fdiv_rn(-lo, scale), p.quant_min);
  } else {
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4 * NQ; ++i) m = max(m, abs_bits(w[i]));   // columns past the block are zeros
    for (int off = 1; off < 8; off <<= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, off));
    float base = __fdiv_rn(__uint_as_float(m), p.quant_max);
    if (scale_round.mode != VQ_ROUND_NONE) base = apply_round(scale_round, base, 0);
    base = base > 0.0f ? base : 1.0f;
    base = fmaxf(base, kEps);
    scale = base;
    if (p.shrink) {
      // try scales below amax / quant_max; keep the one with the least salience-weighted error
      const float factors[kShrinkCandidates] = {1.0f, 0.93f, 0.86f, 0.79f, 0.72f};
      float best_err = 0.0f;
      for (int f = 0; f < kShrinkCandidates; ++f) {
        float s = base;
        if (f > 0) {
          s = __bfloat162float(__float2bfloat16_rn(__fmul_rn(base, factors[f])));
          s = apply_round(scale_round, s, 0);
          s = fmaxf(s, kEps);
        }
        float err = 0.0f;   // the columns' terms in ascending order
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
          float term[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = 32 * q + 4 * l + e;
            const float d = __fsub_rn(w[4 * q + e], grid_value<MODE>(round, w[4 * q + e], s, 0.0f, false));
            term[e] = c < n ? __fmul_rn(__fmul_rn(d, d), p.salience[p.start + c]) : 0.0f;
          }
          for (int ll = 0; ll < 8; ++ll)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float t = __shfl_sync(0xFFFFFFFFu, term[e], first + ll);
              if (32 * q + 4 * ll + e < n) err = __fadd_rn(err, t);
            }
        }
        if (f == 0 || err < best_err) { best_err = err; scale = s; }
      }
    }
  }

  // ---- column sweep ----
  float level[4 * NQ], step[4 * NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
#pragma unroll 1
    for (int ll = 0; ll < 8; ++ll) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 32 * q + 4 * ll + e;   // lane ll of the row has it
        float4 u[NQ];   // fetched before the quotients, which it does not depend on; zeros up to column c itself
#pragma unroll
        for (int q2 = q; q2 < NQ; ++q2) u[q2] = *reinterpret_cast<const float4*>(tile + c * W + 4 * l + 32 * q2);
        const float pivot = s_pivot[c];
        const float g = grid_value<MODE>(round, w[4 * q + e], scale, zero, affine);
        const float mine = __fdiv_rn(__fsub_rn(w[4 * q + e], g), pivot);
        const float delta = __shfl_sync(0xFFFFFFFFu, mine, first + ll);
        if (l == ll) { level[4 * q + e] = g; step[4 * q + e] = mine; }
#pragma unroll
        for (int q2 = q; q2 < NQ; ++q2) {
          w[4 * q2] = __fsub_rn(w[4 * q2], __fmul_rn(delta, u[q2].x));
          w[4 * q2 + 1] = __fsub_rn(w[4 * q2 + 1], __fmul_rn(delta, u[q2].y));
          w[4 * q2 + 2] = __fsub_rn(w[4 * q2 + 2], __fmul_rn(delta, u[q2].z));
          w[4 * q2 + 3] = __fsub_rn(w[4 * q2 + 3], __fmul_rn(delta, u[q2].w));
        }
      }
    }
  }
  if (!live) return;
  float* orow = p.out + row * p.K + p.start;
  float* drow = p.deltas + row * n;
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int c = 32 * q + 4 * l;
    if (p.vec) {
      if (c < n) {
        *reinterpret_cast<float4*>(orow + c) = make_float4(level[4 * q], level[4 * q + 1], level[4 * q + 2], level[4 * q + 3]);
        *reinterpret_cast<float4*>(drow + c) = make_float4(step[4 * q], step[4 * q + 1], step[4 * q + 2], step[4 * q + 3]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + e < n) { orow[c + e] = level[4 * q + e]; drow[c + e] = step[4 * q + e]; }
    }
  }
}

// The same update on whole 16-byte pieces: 128 x 128 tiles, the sums in the same order.  Averaged over
// the 31 updates of a 4096 x 4096 sweep: 55 us (40 TFLOP/s), 95 us as 64 x 64 tiles.
__global__ void __launch_bounds__(256, 2)
gptq_update_tiles_kernel(float* __restrict__ work, const float* __restrict__ deltas, const float* __restrict__ U,
                         int64_t rows, int64_t K, int start, int n, int end) {
  __shared__ __align__(16) GtSmem s;
  const int64_t r0 = (int64_t)blockIdx.y * kGt, j0 = (int64_t)end + (int64_t)blockIdx.x * kGt;
  const int live_rows = (int)min((int64_t)kGt, rows - r0), live_cols = (int)min((int64_t)kGt, K - j0);
  uint64_t acc[8][4];
  gt_multiply<false>(acc, s, deltas + r0 * n, n, U + (int64_t)start * K + j0, K, live_rows, live_cols, n);
  gt_each(acc, [&](int r, int c, float4 v) {
    if (r >= live_rows || c >= live_cols) return;
    float4* dst = reinterpret_cast<float4*>(work + (r0 + r) * K + j0 + c);
    const float4 old = *dst;
    *dst = make_float4(__fsub_rn(old.x, v.x), __fsub_rn(old.y, v.y), __fsub_rn(old.z, v.z), __fsub_rn(old.w, v.w));
  });
}

// work[r][end + j] -= sum_c deltas[r][c] * U[start + c][end + j], c ascending, fp32.
// A CTA computes a 64-row x 64-column patch; deltas and U's rows are staged in
// shared memory in chunks of 32 c.
constexpr int kUpdTile = 64;
__global__ void __launch_bounds__(256)
gptq_update_kernel(float* __restrict__ work, const float* __restrict__ deltas, const float* __restrict__ U,
                   int64_t rows, int64_t K, int start, int n, int end) {
  __shared__ float sd[kUpdTile][33];
  __shared__ float su[32][kUpdTile + 1];
  const int64_t r0 = (int64_t)blockIdx.y * kUpdTile;
  const int64_t j0 = (int64_t)end + (int64_t)blockIdx.x * kUpdTile;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;  // 16 x 16 threads, 4 x 4 outputs each
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;
  for (int c0 = 0; c0 < n; c0 += 32) {
    for (int t = threadIdx.x; t < kUpdTile * 32; t += 256) {
      const int r = t >> 5, c = t & 31;
      sd[r][c] = (r0 + r < rows && c0 + c < n) ? deltas[(r0 + r) * n + c0 + c] : 0.0f;
    }
    for (int t = threadIdx.x; t < 32 * kUpdTile; t += 256) {
      const int c = t / kUpdTile, j = t - c * kUpdTile;
      su[c][j] = (c0 + c < n && j0 + j < K) ? U[(int64_t)(start + c0 + c) * K + j0 + j] : 0.0f;
    }
    __syncthreads();
#pragma unroll 8
    for (int c = 0; c < 32; ++c) {
      float d[4], u[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) d[a] = sd[ty * 4 + a][c];
#pragma unroll
      for (int b = 0; b < 4; ++b) u[b] = su[c][tx * 4 + b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fmaf(d[a], u[b], acc[a][b]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int64_t r = r0 + ty * 4 + a;
    if (r >= rows) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int64_t j = j0 + tx * 4 + b;
      if (j < K) work[r * K + j] = __fsub_rn(work[r * K + j], acc[a][b]);
    }
  }
}

}  // namespace
}  // namespace vq

using namespace vq;

extern "C" int vq_gptq_block(float* work, float* out, float* deltas, const float* U, const float* salience,
                             int64_t rows, int64_t K, int64_t start, int64_t n, int affine, float quant_min,
                             float quant_max, int shrink, const VqRound* scale_round, const VqRound* round,
                             void* stream) {
  VQ_REQUIRE(rows >= 0 && K > 0 && start >= 0 && n > 0 && start + n <= K, "vq_gptq_block: bad block");
  if (rows == 0) return VQ_OK;
  VQ_REQUIRE(work && out && deltas && U && round, "vq_gptq_block: null argument");
  VQ_REQUIRE(n <= kMaxBlock, "vq_gptq_block: blocks of more than %d columns are not supported", kMaxBlock);
  VQ_REQUIRE(!shrink || (salience && !affine && scale_round && scale_round->mode != VQ_ROUND_NONE),
             "vq_gptq_block: the shrink search needs salience weights and a scale table");
  VQ_REQUIRE(affine ? quant_max > quant_min : quant_max > 0.0f, "vq_gptq_block: bad code range");
  if (int e = validate_round(scale_round, "scale rounding")) return e;
  if (int e = validate_round(round, "element rounding")) return e;
  GptqBlockParams p{};
  p.work = work; p.out = out; p.deltas = deltas; p.U = U; p.salience = salience;
  p.rows = rows; p.K = K; p.start = (int)start; p.n = (int)n;
  p.affine = affine; p.quant_min = quant_min; p.quant_max = quant_max; p.shrink = shrink;
  p.scale_round = make_round(scale_round);
  p.round = make_round(round);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int grid = (int)((rows + kRowsPerCta - 1) / kRowsPerCta);
  p.vec = K % 4 == 0 && start % 4 == 0 && n % 4 == 0 &&
          ((reinterpret_cast<uintptr_t>(work) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(deltas)) & 15) == 0;
  static unsigned long long configured = 0;
  if (first_call_on_device(&configured)) {
    cudaFuncSetAttribute(gptq_block_kernel<4, VQ_ROUND_INT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 128 * 4);
    cudaFuncSetAttribute(gptq_block_kernel<4, -1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 128 * 4);
  }
  const int width = n <= 32 ? 32 : n <= 64 ? 64 : 128;
  const size_t smem = (size_t)width * width * sizeof(float);
#define VQ_BLOCK(NQ)                                                                                    \
  (p.round.mode == VQ_ROUND_INT ? gptq_block_kernel<NQ, VQ_ROUND_INT><<<grid, kBlockThreads, smem, st>>>(p) \
                                : gptq_block_kernel<NQ, -1><<<grid, kBlockThreads, smem, st>>>(p))
  if (width == 32) VQ_BLOCK(1);
  else if (width == 64) VQ_BLOCK(2);
  else VQ_BLOCK(4);
#undef VQ_BLOCK
  return check_launch("gptq_block_kernel");
}

extern "C" int vq_gptq_update(float* work, const float* deltas, const float* U, int64_t rows, int64_t K,
                              int64_t start, int64_t n, void* stream) {
  VQ_REQUIRE(rows >= 0 && K > 0 && start >= 0 && n > 0 && start + n <= K, "vq_gptq_update: bad block");
  const int64_t end = start + n;
  if (rows == 0 || end == K) return VQ_OK;
  VQ_REQUIRE(work && deltas && U, "vq_gptq_update: null argument");
  if (K % 4 == 0 && start % 4 == 0 && n % 4 == 0 && rows < (1ll << 22) &&
      ((reinterpret_cast<uintptr_t>(work) | reinterpret_cast<uintptr_t>(deltas) | reinterpret_cast<uintptr_t>(U)) & 15) == 0) {
    const dim3 tiles((unsigned)((K - end + kGt - 1) / kGt), (unsigned)((rows + kGt - 1) / kGt));
    gptq_update_tiles_kernel<<<tiles, 256, 0, static_cast<cudaStream_t>(stream)>>>(work, deltas, U, rows, K, (int)start,
                                                                                   (int)n, (int)end);
    return check_launch("gptq_update_tiles_kernel");
  }
  dim3 grid((unsigned)((K - end + kUpdTile - 1) / kUpdTile), (unsigned)((rows + kUpdTile - 1) / kUpdTile));
  gptq_update_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(work, deltas, U, rows, K, (int)start,
                                                                          (int)n, (int)end);
  return check_launch("gptq_update_kernel");
}

// ---------------------------------------------------------------------------
// One GPTQ block step for callers that cannot allocate device memory
// ---------------------------------------------------------------------------
// vq_gptq_block + vq_gptq_update hand the per-column errors from the sweep to the
// trailing update through a caller-provided [rows, n] fp32 buffer.  Some hosts of
// this library have no allocator to get that buffer from: a runtime that drives
// the solve from inside a fixed, pre-planned memory arena (every byte of the pool
// already assigned to tensors), or a plugin loaded into a process whose policy
// forbids cudaMalloc after start-up.  For them the errors live in the array below,
// which is part of the library image: every GPU that loads the library holds these
// 8 MiB until the process exits.
constexpr int64_t kStaticDeltaFloats = 2 * 1024 * 1024;  // 8 MiB: e.g. 16384 rows x 128 columns
static __device__ __align__(256) float g_static_deltas[kStaticDeltaFloats];

// In host code `g_static_deltas` is only a handle for the symbol, not a device
// address; the address is looked up once per device, with that device current.
static float* static_deltas_for_current_device(int* status) {
  constexpr int kMaxDevices = 64;
  static float* address[kMaxDevices] = {};
  int device = -1;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess || device < 0 || device >= kMaxDevices) {
    *status = fail(VQ_ECUDA, "vq_gptq_block_step_static: cannot identify the current device");
    return nullptr;
  }
  if (address[device] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_static_deltas);
    if (e != cudaSuccess || p == nullptr) {
      *status = fail(VQ_ECUDA, "vq_gptq_block_step_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      return nullptr;
    }
    address[device] = p;
  }
  *status = VQ_OK;
  return address[device];
}

extern "C" int vq_gptq_block_step_static(float* work, float* out, const float* U, const float* salience,
                                         int64_t rows, int64_t K, int64_t start, int64_t n, int affine,
                                         float quant_min, float quant_max, int shrink, const VqRound* scale_round,
                                         const VqRound* round, void* stream) {
  VQ_REQUIRE(rows >= 0 && n > 0, "vq_gptq_block_step_static: bad block");
  VQ_REQUIRE(rows <= kStaticDeltaFloats / n,   // not rows * n: an absurd row count must not wrap around
             "vq_gptq_block_step_static: %lld rows x %lld block columns exceeds the built-in buffer of %lld values "
             "(8 MiB); split the rows or use vq_gptq_block / vq_gptq_update with your own buffer",
             (long long)rows, (long long)n, (long long)kStaticDeltaFloats);
  int status = VQ_OK;
  float* deltas = static_deltas_for_current_device(&status);
  if (deltas == nullptr) return status;
  // Every value of the [rows, n] region is rewritten by the sweep before the update
  // reads it, so nothing left over from an earlier call is ever consumed.
  if (int e = vq_gptq_block(work, out, deltas, U, salience, rows, K, start, n, affine, quant_min, quant_max, shrink,
                            scale_round, round, stream))
    return e;
  return vq_gptq_update(work, deltas, U, rows, K, start, n, stream);
}
