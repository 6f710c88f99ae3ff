// Weight-streaming linear for a decode step: a few activation rows (M <= 32) against a weight
// stored PACKED -- two 4-bit codebook indices per byte plus one scale per block of K -- which is
// what a `lut4_to_int6, bs=64, scale=fp8_e5m3` weight costs in memory (0.53 bytes per parameter
// here, against 2 for the bfloat16-valued index tensor the operator contract passes around).
//
//   Y[m][n] = alpha * sum_k a[m][k] * w[n][k] + bias[n]
//   a[m][k] = bf16(levels_a[A[m][k]] * scale_a[m][k / bs])     (or A itself when it has no scale / codebook)
//   w[n][k] = bf16(levels_w[code(n, k)] * scale_w[n][k / bs])
//
// Both operands are rounded to bfloat16 exactly as quantized_ops::linear_mx's read-back does
// (reference ops/quantized.py:574-591), the products are exact in float32 and the sum is float32:
// the result differs from the operator's dequantize-then-matmul in summation order only.
//
// The kernel is bound by HBM (the weight bytes) and, next, by shared-memory lookups and instruction
// issue (decoding a weight is a table lookup and a multiply), so every SM streams the same share of the
// weight from its first cycle to its last:
//   * the weight is a flat list of (32-row tile, 128 weights of K) steps -- one list per K slice, as many
//     slices as the decoded activations need to fit in shared memory (2048 of K for M <= 8, 1024 for 16 and 32
//     rows) -- and the list is cut evenly over CTAs and then over a CTA's sixteen warps, wherever in a tile
//     the cut falls;
//   * each warp has a ring of two steps of its own in shared memory, filled by TMA (32 rows x 64 bytes, and 16 bytes
//     of block scales per row), so the strided rows cost the load/store pipe, which the lookups need, nothing: loading
//     them with 16-byte loads straight into registers held that pipe at 32 us for gate/up.  A step is read into
//     registers at once and its slot refilled, across tiles; the first two are in flight before the prologue;
//   * prologue: the activation slice is decoded into shared memory once (the four elements a lane needs per
//     MMA step stored so that a warp's loads touch every bank once) and a 256-entry table maps a packed
//     byte to its two codebook values as a bfloat16 pair -- one copy per lane (32 random indices into a
//     single table would collide on banks about 3.5-fold), rows 256 bytes apart at a 64 KB-aligned shared
//     address, which makes a lookup three instructions: byte-permute (address), load, packed multiply (scale);
//   * the weights are the MMA's 16-row operand, so that up to 8 activation rows cost one MMA and one load per
//     256 weights, and four rows of a lane share a load;
//   * weights in the operator's own storage (bfloat16-valued codes, 2 bytes each: WIDE) stream the same way, 32 of K
//     per step; their codes are the values themselves or indices that the same table decodes in pairs;
//   * a tile that several warps of a CTA share is added up in shared memory, one that several CTAs share
//     through a workspace by the last to arrive (a counter per tile, cleared by the call), each in a fixed order.
//
// 4096 x 4096 from bfloat16 codes with blocks of 16, 7 rows (34 MB): 16.7 us; the tensor-core GEMM's 256-row tiles
// gave 16 CTA pairs work for 68 us.
//
// gate/up projection of Llama-3.1-8B (28672 x 4096, 62 MB): 24.8 us for one row (44 with CTAs of 256 rows x 1024
// weights of K that each decoded the activations and met at a barrier per tile), 39 us for 16 rows (57 before);
// down projection (4096 x 14336): 18.4 and 32 us (25 and 41 before).
// What is left beside HBM (11 us for gate/up) is the latency of lookup, multiply and MMA at four warps a scheduler.

#include <cuda.h>
#include <cuda_bf16.h>
#include <string.h>

#include "sm100_ptx.cuh"
#include "vq_common.cuh"

namespace vq {
namespace {

using namespace sm100;

constexpr int L4_WARPS = 16;
constexpr int L4_THREADS = 32 * L4_WARPS;
// weights of K per step and row: 64 bytes
template <bool WIDE> struct L4Step { static constexpr int value = WIDE ? 32 : 128; };
// The byte table: one 256-byte row per byte value, lane l reading word l of the row.  It sits at
// shared-memory address 0x10000, so that a lookup address is the lane's base address with its second
// byte replaced by the packed byte -- one byte-permute instruction, no shift, mask or add.
constexpr uint32_t L4_TABLE_ADDR = 0x10000u;
constexpr int L4_TABLE_BYTES = 256 * 256;
constexpr int L4_APAD = 16;                            // bfloat16 elements of padding per activation row (bank spread)

struct Lut4Params {
  const void* a;            // [M, K] bfloat16: values, or codebook indices when a_levels != null
  const void* a_scale;      // [M, K / bs] bfloat16 or null
  const void* a_levels;     // [n_a_levels] bfloat16 or null
  int n_a_levels;
  const uint8_t* w;         // packed: [N, K / 2]
  const void* w_scale;      // [N, K / bs] bfloat16
  const void* w_levels;     // [16] bfloat16; wide codes: null when the codes are the values
  void* out;
  int out_dt;
  int M, N, K, bs;
  int64_t lda;              // elements between activation rows
  const void* alpha;
  int alpha_dt;
  const void* bias;
  int bias_dt;
  float* workspace;         // [tiles][max_parts][accumulators of a tile]
  int* counters;            // [tiles], cleared before each launch
  int tiles;                // row tiles
  int steps;                // K / step
  int slices;               // K slices: slice s holds steps s * steps / slices .. (s + 1) * steps / slices
  int ctas;                 // CTAs per slice
  int max_parts;            // workspace slots per tile
  int lda_s;                // elements per activation row in shared memory
  int bs_shift;
  int small;                // every product of the cut's arithmetic fits 32 bits
  int tma_scales;           // the scale rows are whole 16-byte pieces: map_s covers them
};

__device__ int g_lut4_error;

__device__ __forceinline__ float lparam(const void* p, int64_t i, int dt) {
  if (dt == VQ_F32) return static_cast<const float*>(p)[i];
  if (dt == VQ_BF16) return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
  return __half2float(static_cast<const __half*>(p)[i]);
}

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t v, uint32_t s) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(s));
  return r;
}

// first step of slice `s`.  `small`: steps * slices fits 32 bits (K below 11 million in any plan; 64-bit divisions took
// half of a tile's finishing)
__host__ __device__ inline int l4_slice_begin(int s, int steps, int slices, bool small) {
  return small ? (int)((uint32_t)s * (uint32_t)steps / (uint32_t)slices) : (int)((uint64_t)s * (uint64_t)steps / (uint64_t)slices);
}
// part `i` of `n` equal parts of `total` begins here, and the part that holds step f.  `small`: total * n fits 32 bits.
__device__ inline int l4_cut(uint32_t i, uint32_t total, uint32_t n, bool small) {
  return small ? (int)(i * total / n) : (int)((uint64_t)i * total / n);
}
__device__ inline int l4_part_of(uint32_t f, uint32_t total, uint32_t n, bool small) {
  return small ? (int)(((f + 1) * n - 1) / total) : (int)(((uint64_t)(f + 1) * n - 1) / total);
}

// One code's codebook entry as the generic read-back indexes it (truncate, wrap a negative once, clamp).
__device__ __forceinline__ int code_index(float v, int n) {
  long long i = (long long)v;
  i = i < 0 ? i + n : i;
  return (int)(i < 0 ? 0 : (i >= n ? n - 1 : i));
}
// a vector of wide codes with something other than 0..15 in it
__device__ __noinline__ uint4 decode_odd(uint4 raw, const __nv_bfloat16* __restrict__ levels, uint32_t scale2) {
  const float s = __uint_as_float(scale2 << 16);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float a = __bfloat162float(levels[code_index(__uint_as_float(w[j] << 16), 16)]);
    const float b = __bfloat162float(levels[code_index(__uint_as_float(w[j] & 0xFFFF0000u), 16)]);
    const __nv_bfloat162 h = __floats2bfloat162_rn(__fmul_rn(a, s), __fmul_rn(b, s));
    o[j] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Clears the tiles' counters before the product that counts in them.  A kernel, with the product launched as its
// programmatic dependent (that launch and the product's prologue overlap this one): the decode step of one sequence, four
// products, takes 133 us in a graph, 146 with a memset node before each, 127 with counters that nothing clears and 130
// where the step clears all four products' at once.
__global__ void __launch_bounds__(256) clear_counters_kernel(int* counters, int n) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) counters[i] = 0;
}

// NT: activation rows in tiles of 8 (1..4).  RG: row groups of 8 per weight tile (4, or 2 beside many activation rows).
template <bool WIDE, int NT, int RG>
__global__ void __launch_bounds__(L4_THREADS, 1)
gemm_lut4_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_s,
                 const __grid_constant__ Lut4Params p) {
  constexpr int L4_STEP = L4Step<WIDE>::value;
  constexpr int TILE = 8 * RG;                  // weight rows per tile
  constexpr int RT = RG / 2;                    // 16-row MMA tiles of it
  constexpr int E = RT * NT * 4;                // accumulators per lane
  extern __shared__ __align__(16) uint8_t l4_smem[];
  // dynamic shared memory starts a little above the window's first kilobyte; the table is placed so that
  // its shared address is exactly L4_TABLE_ADDR, the scale slots and the partial tiles before it, the activations
  // and the weight ring behind it
  const uint32_t dyn_base = (uint32_t)__cvta_generic_to_shared(l4_smem);
  const uint32_t table_offset = L4_TABLE_ADDR - dyn_base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t* table = reinterpret_cast<uint32_t*>(l4_smem + table_offset);           // [256][64 words], 32 used
  uint8_t* slots = l4_smem + ((128u - (dyn_base & 127u)) & 127u) + warp * (2 * TILE * 16);   // this warp's [2][TILE][16]
  float* heads = reinterpret_cast<float*>(l4_smem + ((128u - (dyn_base & 127u)) & 127u) + L4_WARPS * 2 * TILE * 16);   // [warps][E][32]
  uint8_t* rings = l4_smem + table_offset + L4_TABLE_BYTES;                        // [warps][2][TILE][64]
  uint8_t* ring = rings + warp * (2 * TILE * 64);
  __nv_bfloat16* sa = reinterpret_cast<__nv_bfloat16*>(rings + L4_WARPS * 2 * TILE * 64);   // [NT * 8][lda_s]
  // a warp's unfinished last tile lies in its own ring, which is empty by then
  auto tails = [&](int w) { return reinterpret_cast<float*>(rings + w * (2 * TILE * 64)); };
  __shared__ __align__(8) uint64_t bars[L4_WARPS][2];
  __shared__ int s_abort;
  volatile int* abort_flag = &s_abort;
  __shared__ float a_levels[256];                                                  // the activation's codebook
  __shared__ uint16_t w_levels[16];

  const int g = lane >> 2, t = lane & 3;
  const int slice = blockIdx.y;
  const bool small = p.small != 0;
  const int step0 = l4_slice_begin(slice, p.steps, p.slices, small);
  const int steps = l4_slice_begin(slice + 1, p.steps, p.slices, small) - step0;  // of K, per tile
  const int total = p.tiles * steps;
  const int cta0 = l4_cut(blockIdx.x, total, p.ctas, small), cta1 = l4_cut(blockIdx.x + 1, total, p.ctas, small);
  const int f0 = cta0 + l4_cut(warp, cta1 - cta0, L4_WARPS, small), f1 = cta0 + l4_cut(warp + 1, cta1 - cta0, L4_WARPS, small);

  if (threadIdx.x < L4_WARPS * 2) mbar_init(&bars[0][0] + threadIdx.x, 1);
  if (threadIdx.x == 0) s_abort = 0;
  fence_barrier_init();
  __syncthreads();

  // ---- the weight stream of this warp ----
  const int blocks_per_row = p.K >> p.bs_shift;
  // 16 bytes of scales hold eight blocks; a step's blocks lie in one such piece
  auto scale_piece = [&](int step) { return ((step0 + step) * L4_STEP) >> (p.bs_shift + 3); };
  int ft = f0 / steps, fk = f0 - ft * steps;               // next step to fetch
  int to_fetch = f1 - f0, fetch_slot = 1, fetched_piece = -1;
  struct Scales { uint32_t s[RG]; };
  auto fetch = [&](int stage, Scales& sc, bool early) {
    if (to_fetch <= 0) return;
    --to_fetch;
    if (p.tma_scales) {
      const int piece = scale_piece(fk);
      const bool fresh = fk == 0 || piece != fetched_piece;
      fetched_piece = piece;
      if (fresh) fetch_slot ^= 1;
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[warp][stage], TILE * 64 + (fresh ? TILE * 16 : 0));
        tma_load_3d(ring + stage * (TILE * 64), &map_w, &bars[warp][stage], (step0 + fk) * 64, ft * TILE, 0);
        if (fresh) tma_load_3d(slots + fetch_slot * (TILE * 16), &map_s, &bars[warp][stage], piece * 8, ft * TILE, 0);
      }
    } else {
      if (lane == 0) {
        mbar_arrive_expect_tx(&bars[warp][stage], TILE * 64);
        tma_load_3d(ring + stage * (TILE * 64), &map_w, &bars[warp][stage], (step0 + fk) * 64, ft * TILE, 0);
      }
#pragma unroll
      for (int j = 0; j < RG; ++j) {   // rows past the end of the weight read row N - 1's scales; their results are never stored
        const uint16_t* src = static_cast<const uint16_t*>(p.w_scale) + (int64_t)min(ft * TILE + 8 * j + g, p.N - 1) * blocks_per_row +
                              (((step0 + fk) * L4_STEP + t * (L4_STEP / 4)) >> p.bs_shift);
        sc.s[j] = early ? __ldcg(src) : __ldg(src);
      }
    }
    if (++fk == steps) { fk = 0; ++ft; }
  };
  Scales sc0, sc1;
  fetch(0, sc0, true);
  fetch(1, sc1, true);

  // ---- prologue: byte table and the decoded activation slice ----
  // It runs beside the clearing of the counters.  That kernel began after everything before it in the stream had ended, so
  // the operands are in the L2; loads go there (TMA, ld.cg), not to an L1 that an earlier kernel may have filled.
  if (threadIdx.x < 16 && p.w_levels) w_levels[threadIdx.x] = __ldcg(static_cast<const uint16_t*>(p.w_levels) + threadIdx.x);
  if (p.a_levels != nullptr && (int)threadIdx.x < p.n_a_levels)
    a_levels[threadIdx.x] = __uint_as_float((uint32_t)__ldcg(static_cast<const uint16_t*>(p.a_levels) + threadIdx.x) << 16);
  __syncthreads();
  for (int i = threadIdx.x; i < 256 * 32 && p.w_levels; i += L4_THREADS) {
    const int byte = i >> 5;
    table[byte * 64 + (i & 31)] = (uint32_t)w_levels[byte & 15] | ((uint32_t)w_levels[byte >> 4] << 16);   // even element low
  }
  {
    const __nv_bfloat16* A = static_cast<const __nv_bfloat16*>(p.a);
    const uint16_t* S = static_cast<const uint16_t*>(p.a_scale);
    const bool coded = p.a_levels != nullptr;
    const int k0 = step0 * L4_STEP;
    const int groups = steps * (L4_STEP / 8);                                      // 8 elements per thread and step
    constexpr int BATCH = 4;                                                       // loads in flight per thread
    for (int base = 0; base < NT * 8 * groups; base += BATCH * L4_THREADS) {
      uint4 raw[BATCH];
      float scl[BATCH];
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int idx = base + u * L4_THREADS + threadIdx.x;
        const int m = idx / groups, kk = (idx - m * groups) << 3;
        raw[u] = make_uint4(0, 0, 0, 0);
        scl[u] = 1.0f;
        if (idx < NT * 8 * groups && m < p.M) {
          raw[u] = __ldcg(reinterpret_cast<const uint4*>(A + (int64_t)m * p.lda + k0 + kk));
          if (S) scl[u] = __uint_as_float((uint32_t)__ldcg(S + (int64_t)m * blocks_per_row + ((k0 + kk) >> p.bs_shift)) << 16);
        }
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int idx = base + u * L4_THREADS + threadIdx.x;
        if (idx >= NT * 8 * groups) continue;
        const int m = idx / groups, kk = (idx - m * groups) << 3;
        uint4 packed = raw[u];
        if (m < p.M && (S != nullptr || coded)) {
          const uint32_t w4[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
          uint32_t o4[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float v0 = __uint_as_float(w4[q] << 16), v1 = __uint_as_float(w4[q] & 0xFFFF0000u);
            if (coded && WIDE) {
              v0 = a_levels[code_index(v0, p.n_a_levels)];
              v1 = a_levels[code_index(v1, p.n_a_levels)];
            } else if (coded) {   // indices are exact small integers in bfloat16
              v0 = a_levels[min(max((int)v0, 0), p.n_a_levels - 1)];
              v1 = a_levels[min(max((int)v1, 0), p.n_a_levels - 1)];
            }
            const __nv_bfloat162 h = __floats2bfloat162_rn(v0 * scl[u], v1 * scl[u]);   // one rounding of the exact product
            o4[q] = *reinterpret_cast<const uint32_t*>(&h);
          }
          packed = make_uint4(o4[0], o4[1], o4[2], o4[3]);
        }
        if (WIDE) {   // a lane takes eight neighbouring elements of a step: they stay in order
          *reinterpret_cast<uint4*>(sa + m * p.lda_s + kk) = packed;
          continue;
        }
        // element 128 i + 32 t + 4 s + e of the slice lives at column 128 i + 16 s + 4 t + e: lane t of a warp
        // reads its four elements of step s eight bytes after lane t - 1's
        const int seg = kk & 127, tt = seg >> 5, ss = (seg & 31) >> 2;              // ss is even: steps ss and ss + 1
        __nv_bfloat16* dst = sa + m * p.lda_s + (kk & ~127) + 16 * ss + 4 * tt;
        *reinterpret_cast<uint2*>(dst) = make_uint2(packed.x, packed.y);
        *reinterpret_cast<uint2*>(dst + 16) = make_uint2(packed.z, packed.w);
      }
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");   // the counters are clear; nothing was written to global memory before
  __syncthreads();

  // This lane's column of the table as a 32-bit shared address; its second byte is zero.
  const uint32_t tb_lane = L4_TABLE_ADDR + 4u * lane;
  // the table entry of byte `which` (0..3) of `word`: address = tb_lane with byte 1 replaced by that byte
  auto lookup = [&](uint32_t word, int which) {
    uint32_t r;
    // not volatile: the table is constant once the CTA has passed its barrier, and the scheduler may then
    // hoist a step's lookups ahead of the MMAs that consume them
    asm("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(__byte_perm(word, tb_lane, 0x7604u | ((uint32_t)which << 4))));
    return r;
  };
  float acc[RT][NT][4];
  auto clear = [&]() {
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][n][e] = 0.0f;
  };
  // the eight MMAs deep contraction of one step: MMA s takes bytes 2 s and 2 s + 1 of each row's 16-byte vector, i.e.
  // elements k = 32 t + 4 s + {0..3}, as its (k, k + 1) and (k + 8, k + 9) pairs
  auto compute = [&](int k, const uint4 (&w8)[RG], const uint32_t (&sc)[RG]) {
    const __nv_bfloat16* a_it = sa + g * p.lda_s + k * L4_STEP + t * 4;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      uint2 af[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n) af[n] = *reinterpret_cast<const uint2*>(a_it + n * 8 * p.lda_s + 16 * s);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        uint32_t b[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4& w = w8[2 * r + h];
          const uint32_t word = s < 2 ? w.x : s < 4 ? w.y : s < 6 ? w.z : w.w;
          b[h][0] = mul_bf16x2(lookup(word, 2 * (s & 1)), sc[2 * r + h]);
          b[h][1] = mul_bf16x2(lookup(word, 2 * (s & 1) + 1), sc[2 * r + h]);
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) mma_bf16_16816(acc[r][n], b[0][0], b[1][0], b[0][1], b[1][1], af[n].x, af[n].y);
      }
    }
  };

  // One step of wide codes: lane t has elements k = 8 t + {0..7} of each row, the first four for one MMA and the last
  // four for another, as their (k, k + 1) and (k + 8, k + 9) pairs.
  auto compute_wide = [&](int k, const uint4 (&w8)[RG], const uint32_t (&sc)[RG]) {
    uint4 af[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n)
      af[n] = *reinterpret_cast<const uint4*>(sa + (n * 8 + g) * p.lda_s + k * L4_STEP + t * 8);
    uint4 b[RG];
#pragma unroll
    for (int j = 0; j < RG; ++j) {
      uint32_t w[4] = {w8[j].x, w8[j].y, w8[j].z, w8[j].w};
      uint32_t odd = 0;
      if (p.w_levels) {
        const __nv_bfloat162 bias2 = __float2bfloat162_rn(128.0f);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // 128 + code leaves an index in the low bits of each half, exactly for 0..15
          const __nv_bfloat162 c = __hadd2_rn(*reinterpret_cast<const __nv_bfloat162*>(&w[q]), bias2);
          const __nv_bfloat162 back = __hsub2_rn(c, bias2);
          const uint32_t cb = *reinterpret_cast<const uint32_t*>(&c);
          odd |= ((cb ^ 0x43004300u) & 0xFFF0FFF0u) | (*reinterpret_cast<const uint32_t*>(&back) ^ w[q]);
          w[q] = lookup((cb & 0xFu) | ((cb >> 12) & 0xF0u), 0);
        }
      }
      b[j] = make_uint4(mul_bf16x2(w[0], sc[j]), mul_bf16x2(w[1], sc[j]), mul_bf16x2(w[2], sc[j]), mul_bf16x2(w[3], sc[j]));
      if (odd) b[j] = decode_odd(w8[j], static_cast<const __nv_bfloat16*>(p.w_levels), sc[j]);
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        mma_bf16_16816(acc[r][n], b[2 * r].x, b[2 * r + 1].x, b[2 * r].y, b[2 * r + 1].y, af[n].x, af[n].y);
        mma_bf16_16816(acc[r][n], b[2 * r].z, b[2 * r + 1].z, b[2 * r].w, b[2 * r + 1].w, af[n].z, af[n].w);
      }
  };

  // ---- the finished sum of one tile over this CTA's part of this slice ----
  // accumulator e of MMA tile (r, n): weight row 16 r + g (+ 8 for e >= 2), activation row 8 n + 2 t + (e & 1)
  auto output = [&](int tile) {
    const float alpha = p.alpha ? lparam(p.alpha, 0, p.alpha_dt) : 1.0f;
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = tile * TILE + 16 * r + 8 * h + g;
        if (row >= p.N) continue;
        const float bias = p.bias ? lparam(p.bias, row, p.bias_dt) : 0.0f;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int m = 8 * n + 2 * t + e;
            if (m >= p.M) continue;
            float sum = acc[r][n][2 * h + e];
            if (p.alpha) sum = __fmul_rn(sum, alpha);
            if (p.bias) sum = __fadd_rn(sum, bias);
            const int64_t o = (int64_t)m * p.N + row;
            if (p.out_dt == VQ_F32) static_cast<float*>(p.out)[o] = sum;
            else if (p.out_dt == VQ_BF16) static_cast<__nv_bfloat16*>(p.out)[o] = __float2bfloat16_rn(sum);
            else static_cast<__half*>(p.out)[o] = __float2half_rn(sum);
          }
      }
  };
  auto finish = [&](int tile) {
    // the parts of this tile, over all slices and CTAs; mine is number `mine`
    int parts = 0, mine = 0;
    for (int s = lane; s < p.slices; s += 32) {
      const int n = l4_slice_begin(s + 1, p.steps, p.slices, small) - l4_slice_begin(s, p.steps, p.slices, small);
      const int first = l4_part_of(tile * n, p.tiles * n, p.ctas, small);
      const int last = l4_part_of((tile + 1) * n - 1, p.tiles * n, p.ctas, small);
      parts += last - first + 1;
      if (s < slice) mine += last - first + 1;
      if (s == slice) mine += blockIdx.x - first;
    }
    parts = __reduce_add_sync(0xFFFFFFFFu, parts);
    mine = __reduce_add_sync(0xFFFFFFFFu, mine);
    if (parts > 1) {
      float* slots = p.workspace + (int64_t)tile * p.max_parts * (E * 32) + lane;
      float* my = slots + (int64_t)mine * (E * 32);
#pragma unroll
      for (int e = 0; e < E; ++e) __stcg(my + e * 32, acc[e / (NT * 4)][(e / 4) % NT][e % 4]);
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0) last = atomicAdd(&p.counters[tile], 1) == parts - 1;
      if (!__shfl_sync(0xFFFFFFFFu, last, 0)) return;
      __threadfence();
      clear();
      for (int q = 0; q < parts; ++q)
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e / (NT * 4)][(e / 4) % NT][e % 4] += __ldcg(slots + (int64_t)q * (E * 32) + e * 32);
    }
    output(tile);
  };

  // ---- main loop ----
  clear();
  int ct = f0 / steps, ck = f0 - ct * steps;
  bool whole = ck == 0;                          // this warp has the tile from its first step
  int left = f1 - f0, read_slot = 1, read_piece = -1;
  uint32_t phase = 0;
  auto step = [&](int stage, Scales& next) {
    if (!__all_sync(0xFFFFFFFFu, mbar_wait(&bars[warp][stage], phase, abort_flag))) return false;
    uint4 w8[RG];
    uint32_t sc[RG];
#pragma unroll
    for (int j = 0; j < RG; ++j)
      w8[j] = *reinterpret_cast<const uint4*>(ring + stage * (TILE * 64) + (8 * j + g) * 64 + t * 16);
    if (p.tma_scales) {
      const int piece = scale_piece(ck);
      if (ck == 0 || piece != read_piece) read_slot ^= 1;
      read_piece = piece;
      const int blk = (((step0 + ck) * L4_STEP + t * (L4_STEP / 4)) >> p.bs_shift) & 7;
#pragma unroll
      for (int j = 0; j < RG; ++j)
        sc[j] = *reinterpret_cast<const uint16_t*>(slots + read_slot * (TILE * 16) + (8 * j + g) * 16 + blk * 2) * 0x10001u;
    } else {
#pragma unroll
      for (int j = 0; j < RG; ++j) sc[j] = next.s[j] * 0x10001u;
    }
    __syncwarp();   // the step is in registers: its slot may be refilled
    fetch(stage, next, false);
    if constexpr (WIDE) compute_wide(ck, w8, sc);
    else compute(ck, w8, sc);
    --left;
    if (++ck == steps || left == 0) {
      if (whole && ck == steps) {
        finish(ct);
      } else {
        float* slot = (whole ? tails(warp) : heads + warp * (E * 32)) + lane;
#pragma unroll
        for (int e = 0; e < E; ++e) slot[e * 32] = acc[e / (NT * 4)][(e / 4) % NT][e % 4];
      }
      clear();
      whole = true;
      ck = 0;
      ++ct;
    }
    return true;
  };
  bool ok = true;
  while (left > 0) {
    if (!(ok = step(0, sc0))) break;
    if (left > 0 && !(ok = step(1, sc1))) break;
    phase ^= 1;
  }
  if (!ok) {   // a load never arrived: let what is in flight end (waiting again with a limit) and report it
    for (int i = 0; i < 2; ++i)
      for (int spin = 0; spin < (1 << 20) && !mbar_try_wait(&bars[warp][i], phase); ++spin) {}
    if (lane == 0) atomicExch(&g_lut4_error, VQ_ETIMEOUT);
  }
  __syncthreads();

  // ---- tiles that several warps, or this CTA's first or last warp and another CTA, share ----
  if (cta0 == cta1 || *abort_flag) return;
  const int len = cta1 - cta0;
  const int tile_first = cta0 / steps, tile_last = (cta1 - 1) / steps;
  for (int tile = tile_first + warp; tile <= tile_last; tile += L4_WARPS) {
    const int b = tile * steps, e = b + steps;
    const int lo = max(b, cta0), hi = min(e, cta1);
    int w = l4_part_of(lo - cta0, len, L4_WARPS, small);
    if (cta0 + l4_cut(w, len, L4_WARPS, small) <= b && cta0 + l4_cut(w + 1, len, L4_WARPS, small) >= e) continue;   // one warp had it all
    const int w_last = l4_part_of(hi - 1 - cta0, len, L4_WARPS, small);
    clear();
    for (; w <= w_last; ++w) {
      const int begin = cta0 + l4_cut(w, len, L4_WARPS, small);
      if (begin == cta0 + l4_cut(w + 1, len, L4_WARPS, small)) continue;   // a warp without steps
      const float* slot = (begin <= b ? tails(w) : heads + w * (E * 32)) + lane;
#pragma unroll
      for (int q = 0; q < E; ++q) acc[q / (NT * 4)][(q / 4) % NT][q % 4] += slot[q * 32];
    }
    finish(tile);
  }
}

// Pack bfloat16-valued codebook indices (0..15) two per byte, even element in the low nibble.
__global__ void pack_lut4_kernel(const __nv_bfloat16* __restrict__ codes, uint8_t* __restrict__ out, int64_t bytes,
                                 int* bad) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= bytes) return;
  const float lo = __bfloat162float(codes[2 * i]), hi = __bfloat162float(codes[2 * i + 1]);
  const int a = (int)lo, b = (int)hi;
  if (!(lo == (float)a && hi == (float)b && a >= 0 && a < 16 && b >= 0 && b < 16)) atomicExch(bad, 1);
  out[i] = (uint8_t)((a & 15) | ((b & 15) << 4));
}

}  // namespace
}  // namespace vq

using namespace vq;

// Boxes of box_x elements x box_rows rows of a dense [rows, cols] matrix, unswizzled (eight lanes read 128 neighbouring
// bytes); rows past the end arrive as zeros.
static int lut4_map(CUtensorMap* map, const void* base, CUtensorMapDataType type, int elem, int64_t cols, int64_t rows,
                    int box_x, int box_rows) {
  typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeFn enc = nullptr;
  if (!enc) {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      return fail(VQ_ECUDA, "cuTensorMapEncodeTiled is not available from this driver");
    enc = reinterpret_cast<EncodeFn>(sym);
  }
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, 1};
  const cuuint64_t strides[2] = {(cuuint64_t)(cols * elem), (cuuint64_t)(cols * elem * rows)};
  const cuuint32_t box[3] = {(cuuint32_t)box_x, (cuuint32_t)box_rows, 1}, unit[3] = {1, 1, 1};
  const CUresult r = enc(map, type, 3, const_cast<void*>(base), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(VQ_ECUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return VQ_OK;
}

// whether a launch gave up waiting for a load (read by vq_gemm_status)
namespace vq {
int lut4_status(int reset) {
  int value = 0;
  if (cudaMemcpyFromSymbol(&value, g_lut4_error, sizeof(int)) != cudaSuccess) return VQ_ECUDA;
  if (reset && value) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_lut4_error, &zero, sizeof(int));
  }
  return value;
}
}  // namespace vq

extern "C" int vq_clear_counters(int* counters, int64_t n, void* stream) {
  VQ_REQUIRE(n >= 0 && n < (1ll << 31), "vq_clear_counters: bad extent");
  if (n == 0) return VQ_OK;
  VQ_REQUIRE(counters, "vq_clear_counters: null argument");
  clear_counters_kernel<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(counters, (int)n);
  return check_launch("clear_counters_kernel");
}

// How a product is cut: 8 * NT activation rows, weight tiles of 8 * RG rows, K slices, CTAs per slice.
struct Lut4Plan {
  int nt, rg, tiles, steps, slices, ctas, max_parts, lda_s;
  bool small;   // every product of the cut's arithmetic fits 32 bits
};
static Lut4Plan lut4_plan(int64_t M, int64_t N, int64_t K, bool wide) {
  const int step = wide ? L4Step<true>::value : L4Step<false>::value;
  Lut4Plan q{};
  q.nt = (int)((M + 7) / 8);
  q.rg = q.nt <= 2 ? 4 : 2;                                  // partial tiles of both sets beside the activations
  q.tiles = (int)((N + 8 * q.rg - 1) / (8 * q.rg));
  q.steps = (int)(K / step);
  // elements of an activation row that fit behind table and ring
  static const int longest[2][5] = {{0, 2048, 1024, 1280, 1024}, {0, 2048, 1024, 1280, 896}};
  const int fits = longest[wide][q.nt] / step, least_slices = (q.steps + fits - 1) / fits;
  // as few slices as that allows, or up to a quarter more where they use more of the SMs
  q.slices = least_slices;
  for (int n = least_slices + 1; n <= least_slices + least_slices / 4 && n <= kSmCount; ++n)
    if (kSmCount / n * n > kSmCount / q.slices * q.slices) q.slices = n;
  // one CTA per SM; a small weight has a step for each warp of a CTA at least
  const int64_t total = (int64_t)q.tiles * (q.steps / q.slices);
  int64_t ctas = kSmCount / q.slices, most = (total + L4_WARPS - 1) / L4_WARPS;
  if (ctas > most) ctas = most;
  q.ctas = ctas < 1 ? 1 : (int)ctas;
  const int slice_max = (q.steps + q.slices - 1) / q.slices;
  // the rows' pitch spreads the lanes of a load over the banks: 32 bytes apart (packed, 8 bytes a lane), 64 (wide, 16)
  q.lda_s = wide ? slice_max * step + (slice_max % 2 ? 64 : 32) : slice_max * step + L4_APAD;
  // a CTA has at least floor(total / ctas) consecutive steps of a slice, and a slice at most slice_max of a tile
  const int64_t least = total / q.ctas < 1 ? 1 : total / q.ctas;
  const int64_t per_slice = (slice_max - 1) / least + 2;
  q.max_parts = (int)(q.slices * (per_slice < q.ctas ? per_slice : q.ctas));
  const int64_t most_ctas = q.ctas > L4_WARPS ? q.ctas : L4_WARPS;
  q.small = ((int64_t)q.tiles * q.steps + 1) * most_ctas < (1ll << 32) && (int64_t)q.steps * q.slices < (1ll << 32);
  return q;
}

// Slices lie along the grid's second extent, a slice's steps are counted in an int.
static bool lut4_launchable(const Lut4Plan& q) { return q.slices <= 65535 && (int64_t)q.tiles * q.steps < (1ll << 31); }

// The cut, tensor maps and launch of a product whose operands stand in `p`.
template <bool WIDE>
static int launch_row_stream(Lut4Params p, bool clear, cudaStream_t st) {
  const int64_t M = p.M, N = p.N, K = p.K;
  const Lut4Plan q = lut4_plan(M, N, K, WIDE);
  p.tiles = q.tiles; p.steps = q.steps; p.slices = q.slices; p.ctas = q.ctas; p.max_parts = q.max_parts; p.lda_s = q.lda_s;
  while ((1 << p.bs_shift) < p.bs) ++p.bs_shift;
  VQ_REQUIRE(lut4_launchable(q), "row stream: weight too large");
  p.small = q.small;
  // Shared memory: the table must sit at shared address L4_TABLE_ADDR.  Dynamic memory starts somewhere in
  // [1 KB, 4 KB) of the window (system + static variables), so reserving up to the table's end measured from
  // 1 KB always suffices; scale slots and partial tiles (16 + 32 KB at most) fit before the table.
  const int tile = q.rg * 8;
  const int a_bytes = q.nt * 8 * q.lda_s * (int)sizeof(__nv_bfloat16);
  const size_t smem = (size_t)L4_TABLE_ADDR + L4_TABLE_BYTES - 1024 + a_bytes + L4_WARPS * 2 * tile * 64;
  constexpr int kMostSmem = (int)L4_TABLE_ADDR + L4_TABLE_BYTES - 1024 + 100352;   // 16 rows of 1088 elements + 64 KB
  VQ_REQUIRE((int)smem <= kMostSmem, "row stream: internal error: %d bytes of shared memory", (int)smem);
  CUtensorMap map_w, map_s;
  if (int e = lut4_map(&map_w, p.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, WIDE ? K * 2 : K / 2, N, 64, tile)) return e;
  memset(&map_s, 0, sizeof(map_s));
  p.tma_scales = (K / p.bs) % 8 == 0 && (reinterpret_cast<uintptr_t>(p.w_scale) & 15) == 0;
  if (p.tma_scales)
    if (int e = lut4_map(&map_s, p.w_scale, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, K / p.bs, N, 8, tile)) return e;
  static unsigned long long configured = 0;
  if (first_call_on_device(&configured)) {
    cudaFuncSetAttribute(gemm_lut4_kernel<WIDE, 1, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
    cudaFuncSetAttribute(gemm_lut4_kernel<WIDE, 2, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
    cudaFuncSetAttribute(gemm_lut4_kernel<WIDE, 3, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
    cudaFuncSetAttribute(gemm_lut4_kernel<WIDE, 4, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
  }
  // cleared for every launch and not by the last one's tiles: a launch that gave up leaves some of them counted in part
  if (clear)
    if (int e = vq_clear_counters(p.counters, q.tiles, st)) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)q.ctas, (unsigned)q.slices);
  cfg.blockDim = dim3(L4_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = clear ? 1 : 0;
  const cudaError_t e = q.nt == 1   ? cudaLaunchKernelEx(&cfg, gemm_lut4_kernel<WIDE, 1, 4>, map_w, map_s, p)
                        : q.nt == 2 ? cudaLaunchKernelEx(&cfg, gemm_lut4_kernel<WIDE, 2, 4>, map_w, map_s, p)
                        : q.nt == 3 ? cudaLaunchKernelEx(&cfg, gemm_lut4_kernel<WIDE, 3, 2>, map_w, map_s, p)
                                    : cudaLaunchKernelEx(&cfg, gemm_lut4_kernel<WIDE, 4, 2>, map_w, map_s, p);
  if (e != cudaSuccess) return fail(VQ_ECUDA, "gemm_lut4_kernel: %s", cudaGetErrorString(e));
  return check_launch("gemm_lut4_kernel");
}

extern "C" {

int vq_row_stream_slice(int64_t M, int64_t N, int64_t K, int packed, int64_t slice, int64_t* steps, int64_t* slices,
                        int64_t* begin, int64_t* end) {
  VQ_REQUIRE(M > 0 && M <= 32 && N > 0 && N < (1ll << 31) && K > 0 && K < (1ll << 31) && K % (packed ? 128 : 32) == 0,
             "vq_row_stream_slice: bad extents");
  VQ_REQUIRE(steps && slices && begin && end, "vq_row_stream_slice: null argument");
  const Lut4Plan q = lut4_plan(M, N, K, !packed);
  VQ_REQUIRE(slice >= 0 && slice < q.slices, "vq_row_stream_slice: there are %d slices", q.slices);
  *steps = q.steps;
  *slices = q.slices;
  *begin = l4_slice_begin((int)slice, q.steps, q.slices, q.small);
  *end = l4_slice_begin((int)slice + 1, q.steps, q.slices, q.small);
  return VQ_OK;
}

int64_t vq_gemm_lut4_workspace_floats(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K <= 0 || M > 32 || K % 128) return 0;
  const Lut4Plan q = lut4_plan(M, N, K, false);
  return (int64_t)q.tiles * q.max_parts * (q.nt * 8) * (q.rg * 8);
}

int64_t vq_gemm_lut4_counters(int64_t N) { return N <= 0 ? 0 : (N + 15) / 16; }

int64_t vq_gemm_mx_rows_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K <= 0 || M > 32 || K % 32) return 0;
  const Lut4Plan q = lut4_plan(M, N, K, true);
  if (!lut4_launchable(q)) return 0;
  return ((int64_t)q.tiles * q.max_parts * (q.nt * 8) * (q.rg * 8) + q.tiles) * 4;
}

int vq_gemm_mx_rows(const void* a, const void* a_scale, const void* a_levels, int n_a_levels, const void* w,
                    const void* w_scale, const void* w_levels, int64_t block_size, void* out, int out_dtype, int64_t M,
                    int64_t N, int64_t K, const void* alpha, int alpha_dtype, const void* bias, int bias_dtype,
                    void* workspace, void* stream) {
  VQ_REQUIRE(M >= 0 && N >= 0 && K >= 0, "vq_gemm_mx_rows: negative extent");
  if (M == 0 || N == 0) return VQ_OK;
  VQ_REQUIRE(M <= 32 && K > 0 && K % 32 == 0, "vq_gemm_mx_rows: at most 32 activation rows, K a positive multiple of 32");
  VQ_REQUIRE(block_size >= 8 && block_size < (1 << 30) && (block_size & (block_size - 1)) == 0 && K % block_size == 0,
             "vq_gemm_mx_rows: the block size must be a power of two, at least 8, that divides K");
  VQ_REQUIRE(a && a_scale && w && w_scale && out && workspace, "vq_gemm_mx_rows: null argument");
  VQ_REQUIRE(((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(workspace)) & 15) == 0,
             "vq_gemm_mx_rows: operands must be 16-byte aligned");
  VQ_REQUIRE(a_levels == nullptr || (n_a_levels > 0 && n_a_levels <= 256),
             "vq_gemm_mx_rows: an activation codebook has 1 to 256 entries");
  VQ_REQUIRE(out_dtype >= VQ_BF16 && out_dtype <= VQ_F32, "vq_gemm_mx_rows: bad output dtype");
  VQ_REQUIRE(N < (1ll << 31) && K < (1ll << 30), "vq_gemm_mx_rows: extent too large");
  Lut4Params p{};
  p.a = a; p.a_scale = a_scale; p.a_levels = a_levels; p.n_a_levels = n_a_levels;
  p.w = static_cast<const uint8_t*>(w); p.w_scale = w_scale; p.w_levels = w_levels;
  p.out = out; p.out_dt = out_dtype;
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.bs = (int)block_size; p.lda = K;
  p.alpha = alpha; p.alpha_dt = alpha_dtype; p.bias = bias; p.bias_dt = bias_dtype;
  // the tiles' counters belong to this call: products of several streams may run at the same time
  p.counters = static_cast<int*>(workspace);
  p.workspace = reinterpret_cast<float*>(p.counters + lut4_plan(M, N, K, true).tiles);
  return launch_row_stream<true>(p, true, static_cast<cudaStream_t>(stream));
}

int vq_pack_lut4(const void* codes, void* packed, int64_t rows, int64_t K, int* bad, void* stream) {
  VQ_REQUIRE(rows >= 0 && K >= 0 && K % 2 == 0, "vq_pack_lut4: K must be even");
  const int64_t bytes = rows * (K / 2);
  if (bytes == 0) return VQ_OK;
  VQ_REQUIRE(codes && packed && bad, "vq_pack_lut4: null argument");
  pack_lut4_kernel<<<(unsigned)((bytes + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(codes), static_cast<uint8_t*>(packed), bytes, bad);
  return check_launch("pack_lut4_kernel");
}

static int gemm_lut4(bool clear, const void* a, int64_t lda, const void* a_scale, const void* a_levels, int n_a_levels, int64_t M,
                 const void* w_packed, const void* w_scale, const void* w_levels, int block_size, void* out,
                 int out_dtype, int64_t N, int64_t K, const void* alpha, int alpha_dtype, const void* bias,
                 int bias_dtype, float* workspace, int* counters, void* stream) {
  VQ_REQUIRE(M >= 0 && N >= 0 && K >= 0, "vq_gemm_lut4: negative extent");
  if (M == 0 || N == 0) return VQ_OK;
  VQ_REQUIRE(M <= 32, "vq_gemm_lut4: at most 32 activation rows (a decode step); larger products take linear_mx's GEMM");
  VQ_REQUIRE(K > 0 && K % 128 == 0, "vq_gemm_lut4: K must be a positive multiple of 128");
  VQ_REQUIRE(block_size >= 32 && (block_size & (block_size - 1)) == 0 && K % block_size == 0,
             "vq_gemm_lut4: the block size must be a power of two, at least 32, that divides K");
  VQ_REQUIRE(a && w_packed && w_scale && w_levels && out && workspace && counters, "vq_gemm_lut4: null argument");
  VQ_REQUIRE(lda >= K && lda % 8 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(w_packed) & 15) == 0,
             "vq_gemm_lut4: operands must be 16-byte aligned with rows a multiple of 8 elements apart");
  VQ_REQUIRE(out_dtype >= VQ_BF16 && out_dtype <= VQ_F32, "vq_gemm_lut4: bad output dtype");
  VQ_REQUIRE(a_levels == nullptr || (n_a_levels > 0 && n_a_levels <= 256),
             "vq_gemm_lut4: an activation codebook has 1 to 256 entries");
  VQ_REQUIRE(N < (1ll << 31) && K < (1ll << 31), "vq_gemm_lut4: extent too large");
  Lut4Params p{};
  p.a = a; p.a_scale = a_scale; p.a_levels = a_levels; p.n_a_levels = n_a_levels;
  p.w = static_cast<const uint8_t*>(w_packed); p.w_scale = w_scale; p.w_levels = w_levels;
  p.out = out; p.out_dt = out_dtype;
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.bs = block_size; p.lda = lda;
  p.alpha = alpha; p.alpha_dt = alpha_dtype; p.bias = bias; p.bias_dt = bias_dtype;
  p.workspace = workspace; p.counters = counters;
  return launch_row_stream<false>(p, clear, static_cast<cudaStream_t>(stream));
}

int vq_gemm_lut4(const void* a, int64_t lda, const void* a_scale, const void* a_levels, int n_a_levels, int64_t M,
                 const void* w_packed, const void* w_scale, const void* w_levels, int block_size, void* out,
                 int out_dtype, int64_t N, int64_t K, const void* alpha, int alpha_dtype, const void* bias,
                 int bias_dtype, float* workspace, int* counters, void* stream) {
  return gemm_lut4(true, a, lda, a_scale, a_levels, n_a_levels, M, w_packed, w_scale, w_levels, block_size, out, out_dtype, N, K,
                   alpha, alpha_dtype, bias, bias_dtype, workspace, counters, stream);
}

int vq_gemm_lut4_cleared(const void* a, int64_t lda, const void* a_scale, const void* a_levels, int n_a_levels, int64_t M,
                         const void* w_packed, const void* w_scale, const void* w_levels, int block_size, void* out,
                         int out_dtype, int64_t N, int64_t K, const void* alpha, int alpha_dtype, const void* bias,
                         int bias_dtype, float* workspace, int* counters, void* stream) {
  return gemm_lut4(false, a, lda, a_scale, a_levels, n_a_levels, M, w_packed, w_scale, w_levels, block_size, out, out_dtype, N, K,
                   alpha, alpha_dtype, bias, bias_dtype, workspace, counters, stream);
}

}  // extern "C"
