// FP8 (e4m3) training kernels for sm_100a: block-scaled quantisation and a tcgen05 GEMM with
// per-128-K-block scale promotion.
//
// The reference trains in bf16 only (src/nanoplm/pretraining/pure_pipeline.py:485-487 sets a bf16
// MixedPrecisionPolicy); this file serves the `pretraining.fp8` extension: activations scaled per
// 1 x 128 (row x K-block), weights per 128 x 128, e4m3 operands for forward, data gradient and
// weight gradient, fp32 accumulation.
//
// Scale layout. Every quantised operand is K-major (contraction axis contiguous) and carries
// fp32 scales stored K-block-major: scale[kb * rows + r] for row-scaled operands (1 x 128) and
// scale[kb * row_blocks + r / 128] for block-scaled ones (128 x 128). value = q * scale.
//
// GEMM. C[M,N] (+)= sum_kb (A_kb * sa[.,kb]) (B_kb * sb[.,kb])^T. One pipeline stage holds one
// 128-wide K block of A (128 rows) and B (256 or 128 rows) as 128-byte swizzled rows; the MMA warp issues
// four kind::f8f6f4 UMMAs (K = 32 each) per stage into one of the TMEM buffers and the eight
// epilogue warps read each partial product, multiply by the scales of that K block and add it to
// fp32 registers ("promotion"), so the scales never have to be folded into 8-bit data.
#include <cuda_fp8.h>

#include "common.cuh"

namespace nplm {

constexpr float E4M3_MAX = 448.f;

__device__ __forceinline__ uint32_t pack_e4m3x4(float a, float b, float c, float d) {
  const __nv_fp8x2_storage_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const __nv_fp8x2_storage_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
}

// ------------------------------------------------------------------ quantise, no transpose
// x bf16 [R][K] (row stride ldx) -> q e4m3 [R][K], 1 x 128 scales [K/128][R]. 16 threads per
// (row, K block), 8 elements each.
__global__ void __launch_bounds__(256)
quant_rows_kernel(const __nv_bfloat16* __restrict__ x, int R, int K, int ldx, uint8_t* __restrict__ q,
                  float* __restrict__ scale) {
  grid_chain();
  const int KB = K / 128;
  const long long groups = static_cast<long long>(R) * KB;
  const int sub = threadIdx.x & 15;
  const long long warp_global = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> 5;
  const long long warps_total = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  // two groups per warp and iteration; the loop bound is warp-uniform (full-mask shuffles inside)
  for (long long gw = warp_global * 2; gw < groups; gw += warps_total * 2) {
    const long long g = gw + ((threadIdx.x >> 4) & 1);
    const bool valid = g < groups;
    const int r = valid ? static_cast<int>(g / KB) : 0, kb = valid ? static_cast<int>(g % KB) : 0;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (valid) v = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(r) * ldx + kb * 128 + sub * 8);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&v);
    float f[8];
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 t = unpack_bf16x2(w[i]);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
      amax = fmaxf(amax, fmaxf(fabsf(t.x), fabsf(t.y)));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float s = fmaxf(amax, 1e-12f) / E4M3_MAX;
    const float inv = 1.f / s;
    if (valid) {
      uint2 o2;
      o2.x = pack_e4m3x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
      o2.y = pack_e4m3x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
      *reinterpret_cast<uint2*>(q + static_cast<size_t>(r) * K + kb * 128 + sub * 8) = o2;
      if (sub == 0) scale[static_cast<size_t>(kb) * R + r] = s;
    }
  }
}

// ------------------------------------------------------------------ 128 x 128 tile kernel
// One CTA per 128 x 128 tile of x bf16 [R][K] (R, K multiples of 128).
//   TRANSPOSE = false, BLOCK = true : q [R][K],  scale[(k/128) * (R/128) + r/128]   (weights)
//   TRANSPOSE = true,  BLOCK = true : q [K][R],  scale[(r/128) * (K/128) + k/128]   (weights^T)
//   TRANSPOSE = true,  BLOCK = false: q [K][R],  scale[(r/128) * K + k]  (1 x 128 along the old row
//                                     axis: operands of the weight-gradient GEMM)
template <bool TRANSPOSE, bool BLOCK>
__global__ void __launch_bounds__(256)
quant_tile_kernel(const __nv_bfloat16* __restrict__ x, int R, int K, int ldx, uint8_t* __restrict__ q,
                  float* __restrict__ scale) {
  grid_chain();
  __shared__ __nv_bfloat16 tile[128][130];
  __shared__ float s_red[128];
  const int r0 = blockIdx.y * 128, k0 = blockIdx.x * 128;
  const int tid = threadIdx.x;
  // load: 128 rows x 16 chunks of 8
  for (int i = tid; i < 128 * 16; i += 256) {
    const int r = i >> 4, c = (i & 15) * 8;
    float f[8];
    if (r0 + r < R) {
      const uint4 v = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(r0 + r) * ldx + k0 + c);
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = unpack_bf16x2(w[j]);
        f[2 * j] = t.x;
        f[2 * j + 1] = t.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) tile[r][c + j] = __float2bfloat16(f[j]);
  }
  __syncthreads();
  // amax: per column of the tile (1 x 128 along rows) or of the whole tile
  if (tid < 128) {
    float m = 0.f;
#pragma unroll 8
    for (int r = 0; r < 128; ++r) m = fmaxf(m, fabsf(__bfloat162float(tile[r][tid])));
    s_red[tid] = m;
  }
  __syncthreads();
  if (BLOCK) {
    if (tid < 32) {
      float m = fmaxf(fmaxf(s_red[tid], s_red[tid + 32]), fmaxf(s_red[tid + 64], s_red[tid + 96]));
      m = warp_max(m);
      if (tid == 0) s_red[0] = fmaxf(m, 1e-12f) / E4M3_MAX;
    }
    __syncthreads();
    const float s = s_red[0];
    if (tid == 0) {
      if (TRANSPOSE)
        scale[static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x] = s;
      else
        scale[static_cast<size_t>(blockIdx.x) * gridDim.y + blockIdx.y] = s;
    }
  } else {
    if (tid < 128) {
      const float s = fmaxf(s_red[tid], 1e-12f) / E4M3_MAX;
      s_red[tid] = s;
      scale[static_cast<size_t>(blockIdx.y) * K + k0 + tid] = s;
    }
    __syncthreads();
  }
  // store 128 output rows x 8 chunks of 16 bytes
  for (int i = tid; i < 128 * 8; i += 256) {
    const int orow = i >> 3, oc = (i & 7) * 16;
    uint32_t pk[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = oc + 4 * j + e;
        const float val = __bfloat162float(TRANSPOSE ? tile[c][orow] : tile[orow][c]);
        const float s = BLOCK ? s_red[0] : s_red[TRANSPOSE ? orow : c];
        v[e] = val / s;
      }
      pk[j] = pack_e4m3x4(v[0], v[1], v[2], v[3]);
    }
    if (TRANSPOSE) {
      // output [K][R]: row k0 + orow, columns r0 + oc ..
      if (r0 + oc < R)
        *reinterpret_cast<uint4*>(q + static_cast<size_t>(k0 + orow) * R + r0 + oc) =
            make_uint4(pk[0], pk[1], pk[2], pk[3]);
    } else {
      if (r0 + orow < R)
        *reinterpret_cast<uint4*>(q + static_cast<size_t>(r0 + orow) * K + k0 + oc) =
            make_uint4(pk[0], pk[1], pk[2], pk[3]);
    }
  }
}

// ------------------------------------------------------------------ both forms of an operand in one pass
// A 128 x 128 tile of a bf16 operand [R][K] (R, K multiples of 128) -> what quant_rows_kernel and
// quant_tile_kernel<true, false> give, bit for bit: qr [R][K] with scales sr[(k/128) * R + r], qt [K][R] with scales
// st[(r/128) * K + k]. A warp holds eight rows x 128 columns of the tile in registers (a lane four columns, so a row is one
// 256-byte request): row maxima by warp reduction, column maxima through shared memory; the transposed bytes cross the
// block in shared memory (16-byte chunks swizzled against bank conflicts) and leave as whole 128-byte lines. Two blocks of
// 512 threads a multiprocessor: 55 424 x 1024 in 43 us (5.2 TB/s), SwiGLU form below 125, against 50 and 145 with 16 rows a
// warp in two blocks of 256 (44 and 148 in three).
constexpr int DUAL_ROWS = 8, DUAL_THREADS = 32 * 128 / DUAL_ROWS;

struct DualSmem {
  alignas(16) uint8_t tile[128 * 128];
  float cmax[128 / DUAL_ROWS][128];
};

__device__ __forceinline__ void quant_dual_tile(const uint2 (&v)[DUAL_ROWS], DualSmem& sm, int r0, int k0, int R, int K,
                                                uint8_t* __restrict__ qr, float* __restrict__ sr,
                                                uint8_t* __restrict__ qt, float* __restrict__ st) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  float cm[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int i = 0; i < DUAL_ROWS; ++i) {
    const float2 a = unpack_bf16x2(v[i].x), b = unpack_bf16x2(v[i].y);
    const float m[4] = {fabsf(a.x), fabsf(a.y), fabsf(b.x), fabsf(b.y)};
    float rm = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      cm[j] = fmaxf(cm[j], m[j]);
      rm = fmaxf(rm, m[j]);
    }
    // magnitudes order like their bit patterns
    rm = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(rm)));
    const float s = fmaxf(rm, 1e-12f) / E4M3_MAX;
    const float inv = 1.f / s;
    *reinterpret_cast<uint32_t*>(qr + static_cast<size_t>(r0 + w * DUAL_ROWS + i) * K + k0 + 4 * l) =
        pack_e4m3x4(a.x * inv, a.y * inv, b.x * inv, b.y * inv);
    if (l == i) sr[static_cast<size_t>(k0 >> 7) * R + r0 + w * DUAL_ROWS + i] = s;
  }
  *reinterpret_cast<float4*>(&sm.cmax[w][4 * l]) = make_float4(cm[0], cm[1], cm[2], cm[3]);
  __syncthreads();
  if (threadIdx.x < 128) {
    float m = sm.cmax[0][threadIdx.x];
#pragma unroll
    for (int j = 1; j < 128 / DUAL_ROWS; ++j) m = fmaxf(m, sm.cmax[j][threadIdx.x]);
    const float s = fmaxf(m, 1e-12f) / E4M3_MAX;
    sm.cmax[0][threadIdx.x] = s;
    st[static_cast<size_t>(r0 >> 7) * K + k0 + threadIdx.x] = s;
  }
  __syncthreads();
  const float4 s4 = *reinterpret_cast<const float4*>(&sm.cmax[0][4 * l]);
  const float ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t pk[DUAL_ROWS / 4];
#pragma unroll
    for (int q = 0; q < DUAL_ROWS / 4; ++q) {
      float f[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 t = unpack_bf16x2(j < 2 ? v[q * 4 + u].x : v[q * 4 + u].y);
        f[u] = ((j & 1) ? t.y : t.x) / ss[j];
      }
      pk[q] = pack_e4m3x4(f[0], f[1], f[2], f[3]);
    }
    uint8_t* row = sm.tile + (4 * l + j) * 128;
    *reinterpret_cast<uint2*>(row + (((w >> 1) ^ (l & 7)) << 4) + ((w & 1) << 3)) = make_uint2(pk[0], pk[1]);
  }
  __syncthreads();
#pragma unroll
  for (int i = threadIdx.x; i < 128 * 8; i += DUAL_THREADS) {
    const int col = i >> 3, c = i & 7;
    *reinterpret_cast<uint4*>(qt + static_cast<size_t>(k0 + col) * R + r0 + c * 16) =
        *reinterpret_cast<const uint4*>(sm.tile + col * 128 + ((c ^ ((col >> 2) & 7)) << 4));
  }
}

// Bound by memory: 2 bytes read and 2 written an element, against 6 for the two kernels.
__global__ void __launch_bounds__(DUAL_THREADS, 2)
quant_dual_kernel(const __nv_bfloat16* __restrict__ x, int R, int K, int ldx, uint8_t* __restrict__ qr,
                  float* __restrict__ sr, uint8_t* __restrict__ qt, float* __restrict__ st) {
  grid_chain();
  __shared__ DualSmem sm;
  const int r0 = blockIdx.y * 128, k0 = blockIdx.x * 128;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  uint2 v[DUAL_ROWS];
#pragma unroll
  for (int i = 0; i < DUAL_ROWS; ++i)
    v[i] = __ldg(reinterpret_cast<const uint2*>(x + static_cast<size_t>(r0 + w * DUAL_ROWS + i) * ldx + k0 + 4 * l));
  quant_dual_tile(v, sm, r0, k0, R, K, qr, sr, qt, st);
}

// Both forms of the gradient of an un-rotated QKV projection from that of the rotated one (x, bf16 [R][K]): 64-wide heads
// that start below rope_cols are rotated back (in fp32, rounded to bf16, as the separate pass does it in place) on the
// way. A lane's partner channels, 32 on, are eight lanes away. A warp copies the cos and sin lines of its eight rows to
// shared memory while its loads of x are in flight (cos lies where the transposed bytes go later). 55 424 x 3072: 165 us in
// place of 78 + 123; 187 with the lines read row by row behind the row's position, 210 with several tiles a block that
// share the lines (112 bytes of spills).
__global__ void __launch_bounds__(DUAL_THREADS, 2)
rope_quant_dual_kernel(const __nv_bfloat16* __restrict__ x, int R, int K, int ldx, const int* __restrict__ pos,
                       const float* __restrict__ cos_t, const float* __restrict__ sin_t, int rope_cols,
                       uint8_t* __restrict__ qr, float* __restrict__ sr, uint8_t* __restrict__ qt, float* __restrict__ st) {
  grid_chain();
  __shared__ DualSmem sm;
  __shared__ alignas(16) float sin_rows[128 * 32];
  float* cos_rows = reinterpret_cast<float*>(sm.tile);
  const int r0 = blockIdx.y * 128, k0 = blockIdx.x * 128;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int row_pos = __ldg(pos + r0 + w * DUAL_ROWS + (l & (DUAL_ROWS - 1)));
  uint2 v[DUAL_ROWS];
#pragma unroll
  for (int i = 0; i < DUAL_ROWS; ++i)
    v[i] = __ldg(reinterpret_cast<const uint2*>(x + static_cast<size_t>(r0 + w * DUAL_ROWS + i) * ldx + k0 + 4 * l));
  if (k0 < rope_cols) {
#pragma unroll
    for (int j = 0; j < DUAL_ROWS; j += 4) {   // four rows at a time, a 16-byte chunk a lane
      const int i = j + (l >> 3);
      const size_t from = static_cast<size_t>(__shfl_sync(0xffffffffu, row_pos, i)) * 32 + (l & 7) * 4;
      const int to = (w * DUAL_ROWS + i) * 32 + (l & 7) * 4;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(cos_rows + to)), "l"(cos_t + from) : "memory");
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(sin_rows + to)), "l"(sin_t + from) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();     // (the other lanes' chunks)
    const bool rotate = k0 + (l >> 4) * 64 < rope_cols;
    const bool second = (l & 8) != 0;           // this lane holds the second halves of the pairs
#pragma unroll
    for (int i = 0; i < DUAL_ROWS; ++i) {
      const uint2 o = make_uint2(__shfl_xor_sync(0xffffffffu, v[i].x, 8), __shfl_xor_sync(0xffffffffu, v[i].y, 8));
      if (rotate) {
        const int at = (w * DUAL_ROWS + i) * 32 + (l & 7) * 4;
        const float4 c = *reinterpret_cast<const float4*>(cos_rows + at);
        float4 s = *reinterpret_cast<const float4*>(sin_rows + at);
        s = make_float4(-s.x, -s.y, -s.z, -s.w);
        const float2 m0 = unpack_bf16x2(v[i].x), m1 = unpack_bf16x2(v[i].y), p0 = unpack_bf16x2(o.x), p1 = unpack_bf16x2(o.y);
        if (second) {
          v[i].x = pack_bf16x2(m0.x * c.x + p0.x * s.x, m0.y * c.y + p0.y * s.y);
          v[i].y = pack_bf16x2(m1.x * c.z + p1.x * s.z, m1.y * c.w + p1.y * s.w);
        } else {
          v[i].x = pack_bf16x2(m0.x * c.x - p0.x * s.x, m0.y * c.y - p0.y * s.y);
          v[i].y = pack_bf16x2(m1.x * c.z - p1.x * s.z, m1.y * c.w - p1.y * s.w);
        }
      }
    }
  }
  quant_dual_tile(v, sm, r0, k0, R, K, qr, sr, qt, st);
}

// Both forms of h = bf16(silu(gate) * value) straight from pre = [value | gate] (bf16 [R][2 I]): h, which only e4m3 products
// read, is neither written nor read back (6 bytes an element of h instead of 10 in two passes; 55 424 x 2048 115 + 105 us ->
// 125, 5.4 TB/s).
__global__ void __launch_bounds__(DUAL_THREADS, 2)
swiglu_quant_dual_kernel(const __nv_bfloat16* __restrict__ pre, int R, int I, uint8_t* __restrict__ qr,
                         float* __restrict__ sr, uint8_t* __restrict__ qt, float* __restrict__ st) {
  grid_chain();
  __shared__ DualSmem sm;
  const int r0 = blockIdx.y * 128, k0 = blockIdx.x * 128;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const __nv_bfloat16* src = pre + static_cast<size_t>(r0 + w * DUAL_ROWS) * 2 * I + k0 + 4 * l;
  uint2 v[DUAL_ROWS];
  uint2 g[DUAL_ROWS];
#pragma unroll
  for (int i = 0; i < DUAL_ROWS; ++i) {
    const __nv_bfloat16* p = src + static_cast<size_t>(i) * 2 * I;
    v[i] = __ldg(reinterpret_cast<const uint2*>(p));
    g[i] = __ldg(reinterpret_cast<const uint2*>(p + I));
  }
#pragma unroll
  for (int i = 0; i < DUAL_ROWS; ++i) {
    const float2 a0 = unpack_bf16x2(v[i].x), a1 = unpack_bf16x2(v[i].y);
    const float2 b0 = unpack_bf16x2(g[i].x), b1 = unpack_bf16x2(g[i].y);
    v[i].x = pack_bf16x2(b0.x / (1.f + __expf(-b0.x)) * a0.x, b0.y / (1.f + __expf(-b0.y)) * a0.y);
    v[i].y = pack_bf16x2(b1.x / (1.f + __expf(-b1.x)) * a1.x, b1.y / (1.f + __expf(-b1.y)) * a1.y);
  }
  quant_dual_tile(v, sm, r0, k0, R, I, qr, sr, qt, st);
}

// Both forms of the gradient of pre = [value | gate] from that of h (bf16 [R][I]): [dh silu(gate) | dh value silu'(gate)],
// rounded to bf16 as the separate pass did, quantised without leaving the registers (10 bytes an element of h read and
// written instead of 18). A block makes the value tile and the gate tile of the same 128 columns; the gate tile waits in
// shared memory, since both do not fit the 64 registers that two blocks leave a thread (245 us for 55 424 x 2048, 4.6 TB/s;
// one block a multiprocessor 276).
struct SwigluBwdSmem {
  DualSmem dual;
  uint2 gate[DUAL_ROWS][DUAL_THREADS];
};

__device__ __forceinline__ void swiglu_grad(uint32_t& value, uint32_t& gate, uint32_t dh) {
  const float2 a = unpack_bf16x2(value), b = unpack_bf16x2(gate), c = unpack_bf16x2(dh);
  const float s0 = 1.f / (1.f + __expf(-b.x)), s1 = 1.f / (1.f + __expf(-b.y));
  value = pack_bf16x2(c.x * b.x * s0, c.y * b.y * s1);
  gate = pack_bf16x2(c.x * a.x * s0 * (1.f + b.x * (1.f - s0)), c.y * a.y * s1 * (1.f + b.y * (1.f - s1)));
}

__global__ void __launch_bounds__(DUAL_THREADS, 2)
swiglu_bwd_quant_dual_kernel(const __nv_bfloat16* __restrict__ pre, const __nv_bfloat16* __restrict__ dh, int R, int I,
                             uint8_t* __restrict__ qr, float* __restrict__ sr, uint8_t* __restrict__ qt,
                             float* __restrict__ st) {
  grid_chain();
  extern __shared__ __align__(16) uint8_t swiglu_bwd_smem[];
  SwigluBwdSmem& sm = *reinterpret_cast<SwigluBwdSmem*>(swiglu_bwd_smem);
  const int r0 = blockIdx.y * 128, k0 = blockIdx.x * 128;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  const size_t row = static_cast<size_t>(r0 + w * DUAL_ROWS);
  const __nv_bfloat16* src = pre + row * 2 * I + k0 + 4 * l;
  const __nv_bfloat16* dsrc = dh + row * I + k0 + 4 * l;
  uint2 v[DUAL_ROWS];
  {
    uint2 g[DUAL_ROWS], d[DUAL_ROWS];
#pragma unroll
    for (int i = 0; i < DUAL_ROWS; ++i) {
      v[i] = __ldg(reinterpret_cast<const uint2*>(src + static_cast<size_t>(i) * 2 * I));
      g[i] = __ldg(reinterpret_cast<const uint2*>(src + static_cast<size_t>(i) * 2 * I + I));
      d[i] = __ldg(reinterpret_cast<const uint2*>(dsrc + static_cast<size_t>(i) * I));
    }
#pragma unroll
    for (int i = 0; i < DUAL_ROWS; ++i) {
      swiglu_grad(v[i].x, g[i].x, d[i].x);
      swiglu_grad(v[i].y, g[i].y, d[i].y);
      sm.gate[i][threadIdx.x] = g[i];
    }
  }
  quant_dual_tile(v, sm.dual, r0, k0, R, 2 * I, qr, sr, qt, st);
#pragma unroll
  for (int i = 0; i < DUAL_ROWS; ++i) v[i] = sm.gate[i][threadIdx.x];   // (this thread's own)
  __syncthreads();
  quant_dual_tile(v, sm.dual, r0, I + k0, R, 2 * I, qr, sr, qt, st);
}

// ------------------------------------------------------------------ GEMM
constexpr int F8_BM = 128, F8_BK = 128;  // BK in elements = bytes
// Warpgroup 0: TMA warp, MMA warp, two idle warps, 40 registers a thread. Warpgroups 1 and 2: 8 epilogue warps (2 per
// TMEM lane quarter), which hold 128 sums a thread: at the 168 registers an even split gives they spilled inside
// the promotion loop (6 100 cycles per K block of a weight gradient instead of under 1 000).
constexpr int F8_THREADS = 384;
constexpr int F8_REGS_LAUNCH = 168, F8_REGS_LIGHT = 40, F8_REGS_HEAVY = 232;
static_assert(128 * F8_REGS_LIGHT + 256 * F8_REGS_HEAVY <= F8_THREADS * F8_REGS_LAUNCH,
              "setmaxnreg.inc would wait forever for registers the CTA does not own");

// 256-wide tiles: a K block is 512 cycles of MMAs, and reading its partial products out of tensor memory about 1 024 (see
// the promotion loop), which bounds the kernel: the MMAs of a block hide behind the promotion of the one before (two
// TMEM buffers). 128-wide tiles load 4/3 of the bytes per FLOP and were bound by that and by the serial
// wait -> read -> add -> release chain. They remain for narrow outputs and for weight shards that do not hold whole 256-row
// tiles.
template <int BN>
struct F8Cfg {
  static constexpr int ACC = 512 / BN;                             // TMEM partial-product buffers (all of TMEM)
  static constexpr int STAGE_BYTES = (F8_BM + BN) * F8_BK;
  static constexpr int STAGES = BN == 256 ? 3 : 5;
  static constexpr int HC = BN / 2;                                // columns per epilogue thread
  // 8 warps x 2 output tiles of 32 rows x 128 B. The CTAs finish their tiles together and their stores leave at the
  // rate L2 takes them; with the whole bf16 tile staged the warps go on to the next one meanwhile (K = 1024: the
  // stores took 4 200 of 13 600 cycles a tile with half of that and a fourth operand stage)
  static constexpr int OFF_EPI = STAGES * STAGE_BYTES;
  static constexpr int OFF_SB = OFF_EPI + 8 * 8192;                // [2][BN] scales of B (row-scaled form)
  static constexpr int OFF_BAR = OFF_SB + 2 * BN * 4;
  static constexpr int SMEM = OFF_BAR + 512;
};

__device__ __forceinline__ float2 bf16_rounded(float2 v) { return unpack_bf16x2(pack_bf16x2(v.x, v.y)); }

// What the epilogue does with the finished sums (forms 1 and 2: block-scaled B, bf16 output, plain launches).
enum : int { F8_PLAIN = 0, F8_ADD = 1, F8_ROPE = 2 };

struct Fp8Args {
  const float* sa;   // [KB][M]
  const float* sb;   // [KB][N] (b_block == 0) or [KB][ceil(N/128)] (b_block == 1)
  int M, N, K, ldc;
  int b_block;
  int out_mode;      // 0: bf16 store, 1: fp32 store, 2: fp32 reduce-add (all through tmC)
  int splits;        // out_mode 2: the K blocks of a tile are cut into this many work items (0: the launch chooses)
  int* status;
  // F8_ROPE: position of every row, cos / sin tables [max_pos][32]; 64-wide heads that start below rope_cols are rotated
  const int* rope_pos;
  const float* rope_cos;
  const float* rope_sin;
  int rope_cols;
  // All-gather mode (ag_world > 1, block-scaled B only): B's rows and the matching scale columns
  // are sharded over the ranks. The epilogue warps of all CTAs first copy the other ranks' e4m3
  // rows (half the bytes of a bf16 gather) and scales out of peer memory into the local full-size
  // buffers, bump ag_flags[shard], and both the TMA producer and the epilogue wait (bounded) on a
  // shard's flag before touching it. Tiles are visited shard by shard, the local shard first.
  int ag_world, ag_rank, ag_rows;
  const uint8_t* ag_src[8];   // peer r's shard rows (ag_rows x K bytes)
  const float* ag_ssrc[8];    // peer r's full-size scale buffer [KB][N/128]
  uint8_t* ag_dst;            // local full B
  float* ag_sdst;             // local full scale buffer
  unsigned* ag_flags;         // [ag_world], zeroed before the launch
};

__device__ __forceinline__ bool f8_wait_shard(const Fp8Args& args, int shard, unsigned target) {
  const long long t0 = clock64();
  while (ld_acquire_gpu(args.ag_flags + shard) < target) {
    if (clock64() - t0 > WAIT_LIMIT_CYCLES) return false;
    __nanosleep(100);
  }
  return true;
}

// The forms start from the product rounded to bf16, which is what the passes that they replace read: e4m3 training
// amplifies a last bit of one activation to per cents of a small batch's gradients, so the forms keep every bit.
// F8_ADD: the residual's tiles (tmR) travel through TMA into the staging tiles while the products run, are added to the
// product and overwritten by the results. F8_ROPE: a thread holds whole heads of its row (64 columns), so the
// rotation is register arithmetic on the row's 32 cos / sin pairs, which wait in the staging tiles too (read from global
// memory there and then, 32 rows apart, they cost 150 us). 55 424 rows, us: 1024 columns of K = 1024 79 plain, 95 with the
// residual, 3072 of 1024 225 plain, 266 rotated; the passes over the output that they replace took 57 and 78.
template <int BN, bool B_BLOCK, int FORM>
__global__ void __launch_bounds__(F8_THREADS, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmR, const Fp8Args args) {
  using C8 = F8Cfg<BN>;
  constexpr int STAGES = C8::STAGES, ACC = C8::ACC, HC = C8::HC;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {  // the swizzled tiles need a 1024-byte aligned base
    grid_wait();
    if (threadIdx.x == 0) atomicExch(args.status, ST_BAD_ARG);
    return;
  }
  float* sb_tile = reinterpret_cast<float*>(smem + C8::OFF_SB);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C8::OFF_BAR);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tfull_bar = bars + 2 * STAGES;
  uint64_t* tempty_bar = bars + 2 * STAGES + ACC;
  uint64_t* res_bar = bars + 2 * STAGES + 2 * ACC;   // F8_ADD: [8 epilogue warps][2 staging tiles]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_bar + 16);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int M = args.M, N = args.N;
  const int num_m = (M + F8_BM - 1) / F8_BM, num_n = (N + BN - 1) / BN;
  const int KB = args.K / F8_BK;
  const int n_blocks = (N + 127) / 128;      // columns of a block-scaled B's scale table
  const int kb_per = (KB + args.splits - 1) / args.splits;
  const int total = num_m * num_n * args.splits;
  // work item -> tile origin and K blocks (all-gather mode: shard by shard, the local one first). Tiles run
  // fastest: the items of one wave walk the same K blocks and share operand panels through L2
  auto tile_of = [&](int w, int& m0, int& n0, int& kb0, int& kb1) {
    const int tiles = num_m * num_n;
    const int split = w / tiles, t = w % tiles;
    kb0 = split * kb_per;
    kb1 = min(KB, kb0 + kb_per);
    if (args.ag_world > 1) {
      const int n_per = args.ag_rows / BN;
      const int per_shard = num_m * n_per;
      const int shard = (args.ag_rank + t / per_shard) % args.ag_world;
      const int rem = t % per_shard;
      m0 = (rem / n_per) * F8_BM;
      n0 = shard * args.ag_rows + (rem % n_per) * BN;
    } else {
      m0 = (t / num_n) * F8_BM;
      n0 = (t % num_n) * BN;
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < ACC; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 8);
    }
    if (FORM == F8_ADD)
      for (int i = 0; i < 16; ++i) mbar_init(&res_bar[i], 1);
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
  }
  grid_wait();
  if (warp == 1) {
    tmem_alloc(tmem_slot, ACC * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (args.ag_world <= 1) grid_release();

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F8_REGS_LIGHT));
  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      uint32_t ag_seen = 0;
      for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
        int m0, n0, kb0, kb1;
        tile_of(w, m0, n0, kb0, kb1);
        if (args.ag_world > 1) {
          const int shard = n0 / args.ag_rows;
          if (shard != args.ag_rank && !((ag_seen >> shard) & 1u)) {
            if (!f8_wait_shard(args, shard, gridDim.x)) {
              atomicExch(args.status, ST_TIMEOUT_PEER);
              ok = false;
              break;
            }
            ag_seen |= 1u << shard;
            fence_proxy_async_global();
          }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
            atomicExch(args.status, ST_TIMEOUT_EMPTY);
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * C8::STAGE_BYTES;
          uint8_t* sb = sa + F8_BM * F8_BK;
          mbar_arrive_expect_tx(&full_bar[stage], C8::STAGE_BYTES);
          tma_load_2d(sa, &tmA, &full_bar[stage], kb * F8_BK, m0);
          tma_load_2d(sb, &tmB, &full_bar[stage], kb * F8_BK, n0);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_e4m3(F8_BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < total && ok; w += gridDim.x) {
        int m0, n0, kb0, kb1;
        tile_of(w, m0, n0, kb0, kb1);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&tempty_bar[acc], acc_phase ^ 1)) {
            atomicExch(args.status, ST_TIMEOUT_TMEM_EMPTY);
            ok = false;
            break;
          }
          if (!mbar_wait(&full_bar[stage], phase)) {
            atomicExch(args.status, ST_TIMEOUT_FULL);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * C8::STAGE_BYTES);
          const uint32_t sb = sa + F8_BM * F8_BK;
          const uint32_t d_tmem = tmem_base + acc * BN;
#pragma unroll
          for (int k = 0; k < F8_BK / 32; ++k)
            umma_f8(d_tmem, make_smem_desc(sa + k * 32, 16, 1024), make_smem_desc(sb + k * 32, 16, 1024),
                    idesc, k > 0 ? 1u : 0u);
          umma_commit(&empty_bar[stage]);
          umma_commit(&tfull_bar[acc]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
          if (++acc == ACC) {
            acc = 0;
            acc_phase ^= 1;
          }
        }
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(F8_REGS_HEAVY));
    // warp w owns TMEM lanes 32 * (w % 4) .. +31 (hardware rule) and the column half (w - 4) / 4
    const int quarter = warp & 3;
    const int half = (warp - 4) >> 2;
    const int et = threadIdx.x - 128;  // 0..255 over the eight epilogue warps
    uint8_t* stage_out = smem + C8::OFF_EPI + (warp - 4) * 8192;
    int toggle = 0;                      // which of this warp's two staging tiles is next
    uint32_t res_phase = 0;
    uint32_t ag_seen = 0;
    if (args.ag_world > 1) {
      const long long shard_vecs = static_cast<long long>(args.ag_rows) * args.K / 16;
      const long long per_cta = (shard_vecs + gridDim.x - 1) / gridDim.x;
      const long long v0 = per_cta * blockIdx.x, v1 = min(shard_vecs, v0 + per_cta);
      const int nb_shard = args.ag_rows / 128;
      for (int d = 1; d < args.ag_world; ++d) {
        const int shard = (args.ag_rank + d) % args.ag_world;
        const uint4* src = reinterpret_cast<const uint4*>(args.ag_src[shard]);
        uint4* dst = reinterpret_cast<uint4*>(args.ag_dst + static_cast<size_t>(shard) * args.ag_rows * args.K);
        for (long long v = v0 + et; v < v1; v += 256) dst[v] = src[v];
        if (blockIdx.x == 0) {   // the scale columns of this shard, every K block
          for (int i = et; i < KB * nb_shard; i += 256) {
            const int idx = (i / nb_shard) * n_blocks + shard * nb_shard + (i % nb_shard);
            args.ag_sdst[idx] = args.ag_ssrc[shard][idx];
          }
        }
        __threadfence();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        if (et == 0) red_release_gpu_add(args.ag_flags + shard, 1u);
      }
    }
    int acc = 0;
    uint32_t acc_phase = 0;
    uint32_t it = 0;          // K blocks so far: the scale buffers alternate across work items too
    bool ok = true;
    // (with a row-scaled B a warp whose wait ran out goes on to the barriers the other warps need)
    for (int w = blockIdx.x; w < total && (ok || !B_BLOCK); w += gridDim.x) {
      int m0, n0, kb0, kb1;
      tile_of(w, m0, n0, kb0, kb1);
      if (args.ag_world > 1) {
        const int shard = n0 / args.ag_rows;
        if (shard != args.ag_rank && !((ag_seen >> shard) & 1u)) {
          if (!f8_wait_shard(args, shard, gridDim.x)) {   // scales of this shard must have landed
            if (lane == 0) atomicExch(args.status, ST_TIMEOUT_PEER);
            ok = false;
            break;
          }
          ag_seen |= 1u << shard;
        }
      }
      const int nh = n0 + half * HC;            // first of this thread's columns
      const int row = m0 + quarter * 32 + lane;
      const bool row_ok = row < M;
      const int nb = min(nh >> 7, n_blocks - 1);
      // The item's second operand goes into the staging tiles once the previous item's results have left them. That takes a few
      // thousand cycles, which pass while the first K blocks are added up.
      int rope_at = 0;
      if constexpr (FORM == F8_ROPE) rope_at = row_ok ? __ldg(args.rope_pos + row) * 32 : 0;
      auto second_operand = [&] {
        if (elect_one()) tma_store_wait_read<0>();
        __syncwarp();
        if constexpr (FORM == F8_ADD) {
          if (m0 + quarter * 32 < M && elect_one()) {
#pragma unroll
            for (int q = 0; q < HC / 64; ++q) {
              if (nh + q * 64 < N) {
                mbar_arrive_expect_tx(&res_bar[(warp - 4) * 2 + q], 4096);
                tma_load_2d(stage_out + q * 4096, &tmR, &res_bar[(warp - 4) * 2 + q], nh + q * 64, m0 + quarter * 32);
              }
            }
          }
          __syncwarp();
        } else if (nh < args.rope_cols) {
          // 32 rows x [32 cos | 32 sin]: sixteen 16-byte pieces a row, piece c of row r at place c ^ (r & 7)
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int r = 2 * i + (lane >> 4), piece = lane & 15;
            const int at = __shfl_sync(0xffffffffu, rope_at, r);
            const float* src = (piece < 8 ? args.rope_cos : args.rope_sin) + at + (piece & 7) * 4;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(stage_out + r * 256 +
                                                                                    ((piece ^ (r & 7)) << 4))),
                         "l"(src)
                         : "memory");
          }
          asm volatile("cp.async.commit_group;" ::: "memory");
        }
      };
      float2 c[HC / 2];
#pragma unroll
      for (int j = 0; j < HC / 2; ++j) c[j] = make_float2(0.f, 0.f);
      // Scales of the item's first K block; those of block kb + 1 are fetched while block kb is being awaited (two
      // or four blocks ahead measured no faster). Row-scaled B: thread et carries the scale of tile column et (BN =
      // 128: the first 128 threads) to shared memory, where every thread reads the scales of its columns.
      const bool sb_mine = !B_BLOCK && et < BN && n0 + et < N;
      float sa_n = row_ok ? args.sa[static_cast<size_t>(kb0) * M + row] : 0.f;
      float sb_n = B_BLOCK ? __ldcg(args.sb + static_cast<size_t>(kb0) * n_blocks + nb)
                           : (sb_mine ? __ldg(args.sb + static_cast<size_t>(kb0) * N + n0 + et) : 0.f);
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const float sa = sa_n;
        const float sblk = sb_n * sa;
        float* sb_cur = sb_tile + (it & 1) * BN;
        if (!B_BLOCK) {
          // the buffer's readers (two blocks ago) are behind the barrier of the block in between
          if (et < BN) sb_cur[et] = sb_n;
          asm volatile("bar.sync 1, 256;" ::: "memory");
        }
        if (kb + 1 < kb1) {
          sa_n = row_ok ? args.sa[static_cast<size_t>(kb + 1) * M + row] : 0.f;
          if (B_BLOCK) sb_n = __ldcg(args.sb + static_cast<size_t>(kb + 1) * n_blocks + nb);
          else sb_n = sb_mine ? __ldg(args.sb + static_cast<size_t>(kb + 1) * N + n0 + et) : 0.f;
        }
        if (ok && !mbar_wait(&tfull_bar[acc], acc_phase)) {
          if (lane == 0) atomicExch(args.status, ST_TIMEOUT_TMEM_FULL);
          ok = false;
        }
        if (!ok) {
          if (B_BLOCK) break;
          continue;
        }
        if (FORM != F8_PLAIN && kb == min(kb0 + 1, kb1 - 1)) second_operand();
        tc_fence_after();
        const uint32_t taddr = tmem_base + acc * BN + half * HC + (static_cast<uint32_t>(quarter * 32) << 16);
        const float2 sa2 = make_float2(sa, sa), sblk2 = make_float2(sblk, sblk);
        // Reading the partial products (128 KB a block) takes 1 024 cycles, tensor memory gives about 128 bytes a
        // clock and SM: that, not the MMAs, bounds this kernel (without the arithmetic 224 us for 55 424 x 1024 x
        // 4096). So the next 32 columns are on their way while these are scaled and added.
        uint32_t r[2][32];
        tmem_ld32(taddr, r[0]);
#pragma unroll
        for (int q = 0; q < HC / 32; ++q) {
          tmem_ld_wait();
          if (q + 1 < HC / 32) {
            tmem_ld32(taddr + (q + 1) * 32, r[(q + 1) & 1]);
          } else {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty_bar[acc]);
          }
          const uint32_t (&v)[32] = r[q & 1];
          if (B_BLOCK) {
#pragma unroll
            for (int e = 0; e < 16; ++e)
              c[q * 16 + e] = fma2(make_float2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])), sblk2,
                                   c[q * 16 + e]);
          } else {
            const float4* sp = reinterpret_cast<const float4*>(sb_cur + half * HC + q * 32);
#pragma unroll
            for (int e4 = 0; e4 < 8; ++e4) {
              const float4 s4 = sp[e4];
              const int e = e4 * 2;
              c[q * 16 + e] = fma2(mul2(make_float2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])), sa2),
                                   make_float2(s4.x, s4.y), c[q * 16 + e]);
              c[q * 16 + e + 1] =
                  fma2(mul2(make_float2(__uint_as_float(v[2 * e + 2]), __uint_as_float(v[2 * e + 3])), sa2),
                       make_float2(s4.z, s4.w), c[q * 16 + e + 1]);
            }
          }
        }
        if (++acc == ACC) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
      if (!ok) continue;
      // 128 bytes of every row at a time (64 bf16 or 32 fp32 columns) through this warp's staging tile and one TMA
      // store or reduce-add; rows and columns past the end are clipped by the tensor map. (Adds issued from the
      // registers touch 32 rows an instruction: a fifth of a weight gradient's time.)
      const int y0 = m0 + quarter * 32;
      const bool bf = args.out_mode == 0;
      if constexpr (FORM == F8_ROPE) {
        if (nh < args.rope_cols) {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {     // pairs (4i .. 4i + 3) and their partners 32 columns on, in each of the thread's heads
            const float4 cs = *reinterpret_cast<const float4*>(stage_out + lane * 256 + ((i ^ (lane & 7)) << 4));
            const float4 sn = *reinterpret_cast<const float4*>(stage_out + lane * 256 + (((8 + i) ^ (lane & 7)) << 4));
#pragma unroll
            for (int q = 0; q < HC / 64; ++q) {
              if (nh + q * 64 < args.rope_cols) {
                float2 *a = c + q * 32 + 2 * i, *b = a + 16;
                const float2 a0 = bf16_rounded(a[0]), a1 = bf16_rounded(a[1]);
                const float2 b0 = bf16_rounded(b[0]), b1 = bf16_rounded(b[1]);
                a[0] = make_float2(fmaf(a0.x, cs.x, -__fmul_rn(b0.x, sn.x)), fmaf(a0.y, cs.y, -__fmul_rn(b0.y, sn.y)));
                b[0] = make_float2(fmaf(b0.x, cs.x, __fmul_rn(a0.x, sn.x)), fmaf(b0.y, cs.y, __fmul_rn(a0.y, sn.y)));
                a[1] = make_float2(fmaf(a1.x, cs.z, -__fmul_rn(b1.x, sn.z)), fmaf(a1.y, cs.w, -__fmul_rn(b1.y, sn.w)));
                b[1] = make_float2(fmaf(b1.x, cs.z, __fmul_rn(a1.x, sn.z)), fmaf(b1.y, cs.w, __fmul_rn(a1.y, sn.w)));
              }
            }
          }
          __syncwarp();     // every lane has read its row before the results overwrite the tiles
        }
      }
#pragma unroll
      for (int q = 0; q < HC / 32; ++q) {
        if (bf && q >= HC / 64) break;
        const int x = nh + q * (bf ? 64 : 32);
        if constexpr (FORM == F8_ADD) {
          if (q < HC / 64 && y0 < M && x < N) {
            uint8_t* rb = stage_out + (q % (HC / 64)) * 4096;
            if (!mbar_wait(&res_bar[(warp - 4) * 2 + (q % (HC / 64))], (res_phase >> q) & 1u)) {
              if (lane == 0) atomicExch(args.status, ST_TIMEOUT_MISC);
            }
            res_phase ^= 1u << q;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint4* at = reinterpret_cast<uint4*>(rb + lane * 128 + ((j ^ (lane & 7)) << 4));
              uint4 o = *at;
              uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
              const float2* v = c + (q % (HC / 64)) * 32 + j * 4;
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 t = unpack_bf16x2(ow[e]);
                const float2 p = bf16_rounded(v[e]);
                ow[e] = pack_bf16x2(p.x + t.x, p.y + t.y);
              }
              *at = o;
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (elect_one()) {
              tma_store_2d(&tmC, rb, x, y0);
              tma_store_commit();
            }
          }
          continue;
        }
        if (y0 < M && x < N) {
          if (elect_one()) tma_store_wait_read<1>();
          __syncwarp();
          uint8_t* tile_out = stage_out + toggle * 4096;
          toggle ^= 1;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint4 o;
            if (bf) {
              const float2* v = c + (q % (HC / 64)) * 32 + j * 4;
              o = make_uint4(pack_bf16x2(v[0].x, v[0].y), pack_bf16x2(v[1].x, v[1].y), pack_bf16x2(v[2].x, v[2].y),
                             pack_bf16x2(v[3].x, v[3].y));
            } else {
              const float2* v = c + q * 16 + j * 2;
              o = make_uint4(__float_as_uint(v[0].x), __float_as_uint(v[0].y), __float_as_uint(v[1].x),
                             __float_as_uint(v[1].y));
            }
            *reinterpret_cast<uint4*>(tile_out + lane * 128 + ((j ^ (lane & 7)) << 4)) = o;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            if (args.out_mode == 2) tma_reduce_add_2d(&tmC, tile_out, x, y0);
            else tma_store_2d(&tmC, tile_out, x, y0);
            tma_store_commit();
          }
        }
      }
    }
    if (elect_one()) tma_store_wait<0>();
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ACC * BN);
  }
}

typedef CUresult (*EncodeTiledFn8)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn8 f8_encode_fn() {
  static EncodeTiledFn8 fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn8>(p);
  }
  return fn;
}

// uint8 [rows][K] row-major, box 128 bytes x box_rows rows, 128-byte swizzle
static int f8_make_map(CUtensorMap* map, const void* base, uint64_t K, uint64_t rows, uint32_t box_rows) {
  EncodeTiledFn8 fn = f8_encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = nplm::with_context([&] { return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE); });
  return r == CUDA_SUCCESS ? 0 : -2;
}

// bf16 or fp32 [rows][cols] output, boxes of 32 rows x 128 bytes
static int f8_make_out_map(CUtensorMap* map, void* base, uint64_t cols, uint64_t rows, uint64_t ld, bool bf16) {
  EncodeTiledFn8 fn = f8_encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * (bf16 ? 2 : 4)};
  cuuint32_t box[2] = {bf16 ? 64u : 32u, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = nplm::with_context([&] { return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE); });
  return r == CUDA_SUCCESS ? 0 : -2;
}

// Work items a tile is cut into when the output is accumulated (weight gradients: few tiles, a long contraction
// over tokens): the smallest number that fills the last wave of SMs best, at least 16 K blocks (2 048 tokens) each.
// 55 424 tokens: a 1024 x 1024 gradient is 32 tiles, i.e. 116 of 148 SMs idle without it.
static int f8_splits(int tiles, int kb, int sms) {
  int best = 1;
  double best_eff = 0.0;
  for (int s = 1; s <= 9 && (s == 1 || kb / s >= 16); ++s) {
    const int work = tiles * s;
    const double eff = static_cast<double>(work) / (static_cast<double>((work + sms - 1) / sms) * sms);
    if (eff > best_eff + 0.02) {
      best = s;
      best_eff = eff;
    }
  }
  return best;
}

template <int BN, bool B_BLOCK, int FORM = F8_PLAIN>
static int f8_launch_form(const void* A, const void* B, void* C, const void* R, int ldr, Fp8Args& args, bool coop,
                          cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmC, tmR;
  int rc = f8_make_map(&tmA, A, args.K, args.M, F8_BM);
  if (rc) return rc;
  rc = f8_make_map(&tmB, B, args.K, args.N, BN);
  if (rc) return rc;
  rc = f8_make_out_map(&tmC, C, args.N, args.M, args.ldc, args.out_mode == 0);
  if (rc) return rc;
  tmR = tmC;
  if (FORM == F8_ADD) {
    rc = f8_make_out_map(&tmR, const_cast<void*>(R), args.N, args.M, ldr, true);
    if (rc) return rc;
  }
  auto kern = gemm_fp8_kernel<BN, B_BLOCK, FORM>;
  static bool configured_on[nplm::MAX_DEVICES];
  const int dev_slot = nplm::current_device_slot();
  if (dev_slot < 0) return -4;
  bool& configured = configured_on[dev_slot];
  if (!configured) {
    NPLM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, F8Cfg<BN>::SMEM));
    configured = true;
  }
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_slot);
  const int tiles = ((args.M + F8_BM - 1) / F8_BM) * ((args.N + BN - 1) / BN);
  if (args.out_mode != 2) args.splits = 1;
  else if (args.splits == 0) args.splits = f8_splits(tiles, args.K / F8_BK, sms);
  const int total = tiles * args.splits;
  const int grid = total < sms ? total : sms;
  if (coop) {
    void* params[] = {&tmA, &tmB, &tmC, &tmR, &args};
    return static_cast<int>(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(grid), dim3(F8_THREADS),
                                                        params, F8Cfg<BN>::SMEM, stream));
  }
  launch_chained(kern, grid, F8_THREADS, F8Cfg<BN>::SMEM, stream, tmA, tmB, tmC, tmR, args);
  return static_cast<int>(cudaGetLastError());
}

template <int BN>
static int f8_launch(const void* A, const void* B, void* C, Fp8Args& args, bool coop, cudaStream_t stream) {
  return args.b_block ? f8_launch_form<BN, true>(A, B, C, nullptr, 0, args, coop, stream)
                      : f8_launch_form<BN, false>(A, B, C, nullptr, 0, args, coop, stream);
}

static int f8_grid(long long threads_needed, int block) {
  long long g = (threads_needed + block - 1) / block;
  if (g < 1) g = 1;
  if (g > 148 * 16) g = 148 * 16;
  return static_cast<int>(g);
}

}  // namespace nplm

using namespace nplm;

// x bf16 [R][K] -> q e4m3 [R][K], scales fp32 [K/128][R]
extern "C" int nplm_fp8_quant_rows(const void* x, int R, int K, int ldx, void* q, float* scale,
                                   cudaStream_t stream) {
  if (R <= 0 || K <= 0) return 0;
  if ((K % 128) || (ldx % 8)) return -3;
  const long long threads = static_cast<long long>(R) * (K / 128) * 16;
  launch_chained(quant_rows_kernel, f8_grid(threads, 256), 256, 0, stream,
      reinterpret_cast<const __nv_bfloat16*>(x), R, K, ldx, reinterpret_cast<uint8_t*>(q), scale);
  return static_cast<int>(cudaGetLastError());
}

// 128 x 128 tile quantisation of x bf16 [R][K]; see quant_tile_kernel for the three forms.
//   transpose = 0, block = 1: R, K multiples of 128
//   transpose = 1: K multiple of 128, R multiple of 16 (rows beyond R count as zeros)
extern "C" int nplm_fp8_quant_tile(const void* x, int R, int K, int ldx, int transpose, int block,
                                   void* q, float* scale, cudaStream_t stream) {
  if (R <= 0 || K <= 0) return 0;
  if ((K % 128) || (ldx % 8) || (R % 16)) return -3;
  if (!transpose && (!block || (R % 128))) return -3;
  dim3 grid(K / 128, (R + 127) / 128);
  const __nv_bfloat16* xp = reinterpret_cast<const __nv_bfloat16*>(x);
  uint8_t* qp = reinterpret_cast<uint8_t*>(q);
  if (!transpose)
    launch_chained(quant_tile_kernel<false, true>, grid, 256, 0, stream, xp, R, K, ldx, qp, scale);
  else if (block)
    launch_chained(quant_tile_kernel<true, true>, grid, 256, 0, stream, xp, R, K, ldx, qp, scale);
  else
    launch_chained(quant_tile_kernel<true, false>, grid, 256, 0, stream, xp, R, K, ldx, qp, scale);
  return static_cast<int>(cudaGetLastError());
}

// Row form and transposed row form of x bf16 [R][K] in one pass, R and K multiples of 128; see quant_dual_kernel.
extern "C" int nplm_fp8_quant_dual(const void* x, int R, int K, int ldx, void* qr, float* sr, void* qt, float* st,
                                   cudaStream_t stream) {
  if (R <= 0 || K <= 0) return 0;
  if ((K % 128) || (R % 128) || (ldx % 4) || (reinterpret_cast<uintptr_t>(x) & 7)) return -3;
  if (R / 128 > 65535) return -3;
  launch_chained(quant_dual_kernel, dim3(K / 128, R / 128), DUAL_THREADS, 0, stream,
      reinterpret_cast<const __nv_bfloat16*>(x), R, K, ldx, reinterpret_cast<uint8_t*>(qr), sr,
      reinterpret_cast<uint8_t*>(qt), st);
  return static_cast<int>(cudaGetLastError());
}

// Row and transposed row form of x bf16 [R][K] with the rotary embedding of its 64-wide heads below column rope_cols
// undone; R and K multiples of 128, rope_cols of 64, cos / sin fp32 [max_pos][32].
extern "C" int nplm_fp8_rope_quant_dual(const void* x, int R, int K, int ldx, const int* pos, const float* cos_t,
                                        const float* sin_t, int rope_cols, void* qr, float* sr, void* qt, float* st,
                                        cudaStream_t stream) {
  if (R <= 0 || K <= 0) return 0;
  if ((K % 128) || (R % 128) || (ldx % 4) || (reinterpret_cast<uintptr_t>(x) & 7) || R / 128 > 65535 || (rope_cols % 64) ||
      ((reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15))
    return -3;
  launch_chained(rope_quant_dual_kernel, dim3(K / 128, R / 128), DUAL_THREADS, 0, stream,
                 reinterpret_cast<const __nv_bfloat16*>(x), R, K, ldx, pos, cos_t, sin_t, rope_cols,
                 reinterpret_cast<uint8_t*>(qr), sr, reinterpret_cast<uint8_t*>(qt), st);
  return static_cast<int>(cudaGetLastError());
}

// Both e4m3 forms of h = silu(gate) * value, pre = [value | gate] bf16 [R][2 I] contiguous; R, I multiples of 128.
extern "C" int nplm_fp8_swiglu_quant_dual(const void* pre, int R, int I, void* qr, float* sr, void* qt, float* st,
                                          cudaStream_t stream) {
  if (R <= 0 || I <= 0) return 0;
  if ((I % 128) || (R % 128) || (reinterpret_cast<uintptr_t>(pre) & 7) || R / 128 > 65535) return -3;
  launch_chained(swiglu_quant_dual_kernel, dim3(I / 128, R / 128), DUAL_THREADS, 0, stream,
                 reinterpret_cast<const __nv_bfloat16*>(pre), R, I, reinterpret_cast<uint8_t*>(qr), sr,
                 reinterpret_cast<uint8_t*>(qt), st);
  return static_cast<int>(cudaGetLastError());
}

// Both e4m3 forms of the gradient of pre (bf16 [R][2 I]) from dh (bf16 [R][I]), all contiguous; R, I multiples of 128.
extern "C" int nplm_fp8_swiglu_bwd_quant_dual(const void* pre, const void* dh, int R, int I, void* qr, float* sr, void* qt,
                                              float* st, cudaStream_t stream) {
  if (R <= 0 || I <= 0) return 0;
  if ((I % 128) || (R % 128) || ((reinterpret_cast<uintptr_t>(pre) | reinterpret_cast<uintptr_t>(dh)) & 7) ||
      R / 128 > 65535)
    return -3;
  static bool configured_on[nplm::MAX_DEVICES];
  const int dev_slot = nplm::current_device_slot();
  if (dev_slot < 0) return -4;
  if (!configured_on[dev_slot]) {
    NPLM_CUDA_CHECK(cudaFuncSetAttribute(swiglu_bwd_quant_dual_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(SwigluBwdSmem))));
    configured_on[dev_slot] = true;
  }
  launch_chained(swiglu_bwd_quant_dual_kernel, dim3(I / 128, R / 128), DUAL_THREADS, sizeof(SwigluBwdSmem), stream,
                 reinterpret_cast<const __nv_bfloat16*>(pre), reinterpret_cast<const __nv_bfloat16*>(dh), R, I,
                 reinterpret_cast<uint8_t*>(qr), sr, reinterpret_cast<uint8_t*>(qt), st);
  return static_cast<int>(cudaGetLastError());
}

// Tile width of a plain product: few rows run on 128-wide tiles as long as those fit one wave of 148, where they finish
// sooner. Graph-timed us, wide / narrow: 256 rows, 2048 columns of 512 6.9 / 5.8; 1 536 rows, 1024 columns of 1024
// 8.9 / 7.8. Past a wave the wide ones are ahead (2 432 rows of the latter 9.2; the earlier kernel, all 128-wide, 14.0, and
// 8.6 - 8.9 below a wave). Both sum a tile's K blocks in the same order. Accumulated outputs fill the chip by
// splitting the contraction instead.
static bool f8_wide(int M, int N, int out_mode) {
  const long long wide_tiles = (M + 127LL) / 128 * ((N + 255LL) / 256);
  return N > 128 && (out_mode == 2 || 2 * wide_tiles > 148);
}

static Fp8Args f8_plain_args(const float* sa, const float* sb, int M, int N, int K, int ldc, int b_block, int out_mode,
                             int* status) {
  Fp8Args args = {};
  args.sa = sa;
  args.sb = sb;
  args.M = M;
  args.N = N;
  args.K = K;
  args.ldc = ldc;
  args.b_block = b_block;
  args.out_mode = out_mode;
  args.status = status;
  return args;
}

// C[M][N] (+)= (A * sa) (B * sb)^T, A e4m3 [M][K], B e4m3 [N][K] (both K-major, K % 128 == 0).
// sa fp32 [K/128][M]; sb fp32 [K/128][N] (b_block = 0) or [K/128][ceil(N/128)] (b_block = 1).
// out_mode 0: bf16 C; 1: fp32 C; 2: fp32 C accumulated by TMA reduce-adds, several work items a tile in any order unless
// whole_tiles is set.
extern "C" int nplm_gemm_fp8(const void* A, const void* B, void* C, const float* sa, const float* sb,
                             int M, int N, int K, int ldc, int b_block, int out_mode, int whole_tiles, int* status,
                             cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((K % 128) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15))
    return -3;
  if (out_mode == 0 ? ((N % 8) || (ldc % 8)) : ((N % 4) || (ldc % 4))) return -5;
  if (!b_block && (N % 4)) return -5;
  Fp8Args args = f8_plain_args(sa, sb, M, N, K, ldc, b_block, out_mode, status);
  args.splits = whole_tiles ? 1 : 0;
  return f8_wide(M, N, out_mode) ? f8_launch<256>(A, B, C, args, false, stream)
                                 : f8_launch<128>(A, B, C, args, false, stream);
}

// bf16 C[M][N] = (A * sa) (B * sb)^T with block-scaled B, plus R (bf16, row stride ldr; may be null), or with the rotary
// embedding applied to the 64-wide heads that start below rope_cols (rope_pos not null). Either starts from the product
// rounded to bf16.
extern "C" int nplm_gemm_fp8_form(const void* A, const void* B, void* C, const void* R, const float* sa, const float* sb,
                                  int M, int N, int K, int ldc, int ldr, const int* rope_pos, const float* rope_cos,
                                  const float* rope_sin, int rope_cols, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((K % 128) || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15) || (N % 8) || (ldc % 8))
    return -3;
  if ((R != nullptr) == (rope_pos != nullptr)) return -3;
  if (R != nullptr && ((ldr % 8) || (reinterpret_cast<uintptr_t>(R) & 15))) return -3;
  if (rope_pos != nullptr && (rope_cos == nullptr || rope_sin == nullptr || (N % 64) || (rope_cols % 64) ||
                              (reinterpret_cast<uintptr_t>(rope_cos) & 15) || (reinterpret_cast<uintptr_t>(rope_sin) & 15)))
    return -3;
  Fp8Args args = f8_plain_args(sa, sb, M, N, K, ldc, 1, 0, status);
  args.rope_pos = rope_pos;
  args.rope_cos = rope_cos;
  args.rope_sin = rope_sin;
  args.rope_cols = rope_cols;
  const bool wide = f8_wide(M, N, 0);
  if (R != nullptr)
    return wide ? f8_launch_form<256, true, F8_ADD>(A, B, C, R, ldr, args, false, stream)
                : f8_launch_form<128, true, F8_ADD>(A, B, C, R, ldr, args, false, stream);
  return wide ? f8_launch_form<256, true, F8_ROPE>(A, B, C, nullptr, 0, args, false, stream)
              : f8_launch_form<128, true, F8_ROPE>(A, B, C, nullptr, 0, args, false, stream);
}

// All-gather fused into the fp8 GEMM. b_ptrs[r] / sb_ptrs[r]: rank r's full-size e4m3 weight buffer
// [N][K] and block-scale buffer [K/128][N/128] in peer-mapped memory; on entry only the rows (and
// scale columns) of shard r are valid in buffer r. N / world must be a multiple of 128. On return
// this rank's buffers hold the whole quantised weight. flags: 8 device words.
extern "C" int nplm_gemm_fp8_ag(const void* A, void* const* b_ptrs, void* C, const float* sa,
                                void* const* sb_ptrs, int M, int N, int K, int ldc, int out_mode,
                                int rank, int world, unsigned* flags, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (world < 2 || world > 8 || rank < 0 || rank >= world || (N % world) || ((N / world) % 128) ||
      (K % 128) || flags == nullptr)
    return -10;
  if (out_mode == 0 ? ((N % 8) || (ldc % 8)) : ((N % 4) || (ldc % 4))) return -5;
  Fp8Args args = {};
  args.sa = sa;
  args.sb = reinterpret_cast<const float*>(sb_ptrs[rank]);
  args.M = M;
  args.N = N;
  args.K = K;
  args.ldc = ldc;
  args.b_block = 1;
  args.splits = 0;
  args.out_mode = out_mode;
  args.status = status;
  args.ag_world = world;
  args.ag_rank = rank;
  args.ag_rows = N / world;
  args.ag_dst = reinterpret_cast<uint8_t*>(b_ptrs[rank]);
  args.ag_sdst = reinterpret_cast<float*>(sb_ptrs[rank]);
  args.ag_flags = flags;
  for (int r = 0; r < 8; ++r) {
    args.ag_src[r] = r < world ? reinterpret_cast<const uint8_t*>(b_ptrs[r]) + static_cast<size_t>(r) * args.ag_rows * K
                               : nullptr;
    args.ag_ssrc[r] = r < world ? reinterpret_cast<const float*>(sb_ptrs[r]) : nullptr;
  }
  NPLM_CUDA_CHECK(cudaMemsetAsync(flags, 0, 8 * sizeof(unsigned), stream));
  return args.ag_rows % 256 == 0 ? f8_launch<256>(A, b_ptrs[rank], C, args, true, stream)
                                 : f8_launch<128>(A, b_ptrs[rank], C, args, true, stream);
}
