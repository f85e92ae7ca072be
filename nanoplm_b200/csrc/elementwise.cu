// Memory-bound kernels for the encoder: LayerNorm / RMSNorm (fwd, bwd), embedding gather +
// norm, RoPE, SwiGLU, GELU backward, fused MLM-head cross-entropy (V <= 32), row gather /
// scatter, fused AdamW with on-device gradient clipping, sum of squares.
//
// They replace the ATen / Inductor-generated kernels the reference gets from
// src/nanoplm/pretraining/models/modern_bert/modeling.py:112-131 (RoPE), :219-223 (embedding +
// LayerNorm), :300-302 (SwiGLU), :555-559 (head), :659-664 (decoder + cross entropy) and
// src/nanoplm/pretraining/pure_pipeline.py:755-764 (clip + AdamW).
//
// Activations are bf16, statistics and gradients of parameters are fp32. All kernels are
// plain grid-stride / warp-per-row kernels: none of them waits on anything.
#include <stdlib.h>

#include "common.cuh"
#include "entry_points.h"

namespace nplm {

constexpr int MAX_CHUNKS = 16;  // a warp keeps a row of up to 16*256 = 4096 channels in registers

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 t = unpack_bf16x2(w[e]);
    f[2 * e] = t.x;
    f[2 * e + 1] = t.y;
  }
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 t = unpack_bf16x2(w[e]);
    f[2 * e] = t.x;
    f[2 * e + 1] = t.y;
  }
}

__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) w[e] = pack_bf16x2(f[2 * e], f[2 * e + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

// ------------------------------------------------------------------ norm forward
// One warp per row. ids != nullptr: the row is gathered from table[ids[row]] (embedding).
// rms = 0: LayerNorm without bias, rms = 1: RMSNorm. w == nullptr means weight 1.
template <int CHUNKS>
__global__ void __launch_bounds__(256)
norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ ids,
                const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                float* __restrict__ mean_out, float* __restrict__ rstd_out, int T, int C, float eps,
                int rms) {
  grid_chain();
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (int row = blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < T;
       row += gridDim.x * warps_per_block) {
    const __nv_bfloat16* src =
        ids ? x + static_cast<size_t>(ids[row]) * C : x + static_cast<size_t>(row) * C;
    float v[CHUNKS][8];
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) {
        load8(src + i, v[c]);
#pragma unroll
        for (int e = 0; e < 8; ++e) s += v[c][e];
      }
    }
    float mean = 0.f;
    if (!rms) mean = warp_sum(s) / C;
    float q = 0.f;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float d = v[c][e] - mean;
          q += d * d;
        }
      }
    }
    const float rstd = rsqrtf(warp_sum(q) / C + eps);
    if (lane == 0) {
      if (mean_out) mean_out[row] = mean;
      if (rstd_out) rstd_out[row] = rstd;
    }
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) {
        float wv[8];
        if (w) {
          load8(w + i, wv);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) wv[e] = 1.f;
        }
        float o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = (v[c][e] - mean) * rstd * wv[e];
        store8(y + static_cast<size_t>(row) * C + i, o);
      }
    }
  }
}

// ------------------------------------------------------------------ norm backward
// dx = [dres +] rstd * (g - mean(g) - xhat * mean(g * xhat)),  g = dy * w   (LayerNorm)
// dx = [dres +] rstd * (g - xhat * mean(g * xhat))                           (RMSNorm)
// dw (fp32) accumulates sum_rows dy * xhat: registers per warp -> shared per block -> atomics.
// ids != nullptr (embedding): x rows are gathered from the table, dx is not written, and the
// row gradient is accumulated into dtable[ids[row]] (fp32) instead.
template <int CHUNKS>
__global__ void __launch_bounds__(256, 2)
norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                const int* __restrict__ ids, const __nv_bfloat16* __restrict__ w,
                const float* __restrict__ mean_in, const float* __restrict__ rstd_in,
                const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                float* __restrict__ dw, float* __restrict__ dtable, int T, int C, int rms) {
  grid_chain();
  __shared__ __align__(16) float sm_dw[8][256];  // one 256-channel chunk of every warp's sums
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;

  float acc[CHUNKS][8];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[c][e] = 0.f;

  for (int row = blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < T;
       row += gridDim.x * warps_per_block) {
    const __nv_bfloat16* src =
        ids ? x + static_cast<size_t>(ids[row]) * C : x + static_cast<size_t>(row) * C;
    // Every global load of the row (x, dy and the skip gradient) is issued before the first use and
    // kept packed (bf16) in registers, so a warp has 6 KB in flight; the second pass unpacks again.
    uint4 xr[CHUNKS], dr[CHUNKS], rr[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      xr[c] = dr[c] = rr[c] = make_uint4(0u, 0u, 0u, 0u);
      if (i < C) {
        xr[c] = __ldg(reinterpret_cast<const uint4*>(src + i));
        dr[c] = __ldg(reinterpret_cast<const uint4*>(dy + static_cast<size_t>(row) * C + i));
        if (dres) rr[c] = __ldg(reinterpret_cast<const uint4*>(dres + static_cast<size_t>(row) * C + i));
      }
    }
    const float mean = rms ? 0.f : mean_in[row];
    const float rstd = rstd_in[row];
    float sg = 0.f, sgx = 0.f;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) {
        float xv[8], dv[8], wv[8];
        unpack8(xr[c], xv);
        unpack8(dr[c], dv);
        if (w) {
          load8(w + i, wv);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) wv[e] = 1.f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = (xv[e] - mean) * rstd;
          const float g = dv[e] * wv[e];
          sg += g;
          sgx += g * xh;
          acc[c][e] += dv[e] * xh;
        }
      }
    }
    sg = rms ? 0.f : warp_sum(sg) / C;
    sgx = warp_sum(sgx) / C;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) {
        float xv[8], dv[8], wv[8], o[8];
        unpack8(xr[c], xv);
        unpack8(dr[c], dv);
        if (w) {
          load8(w + i, wv);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) wv[e] = 1.f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float xh = (xv[e] - mean) * rstd;
          o[e] = rstd * (dv[e] * wv[e] - sg - xh * sgx);
        }
        if (ids) {
          float* dst = dtable + static_cast<size_t>(ids[row]) * C + i;
#pragma unroll
          for (int e = 0; e < 8; ++e) atomicAdd(dst + e, o[e]);
        } else {
          if (dres) {
            float r[8];
            unpack8(rr[c], r);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] += r[e];
          }
          store8(dx + static_cast<size_t>(row) * C + i, o);
        }
      }
    }
  }
  if (dw) {
    // The warps' sums meet in shared memory chunk by chunk and without atomics (fp32 adds there are compare-and-swap
    // loops, and all eight warps wanted the same words: 8 704 x 1024 21.3 -> 15.6 us, 55 424 x
    // 1024 91.7 -> 85.9)
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (c) __syncthreads();
      float4* mine = reinterpret_cast<float4*>(&sm_dw[threadIdx.x >> 5][lane * 8]);
      mine[0] = make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
      mine[1] = make_float4(acc[c][4], acc[c][5], acc[c][6], acc[c][7]);
      __syncthreads();
      const int i = c * 256 + threadIdx.x;
      if (i < C) {
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) sum += sm_dw[j][threadIdx.x];
        atomicAdd(&dw[i], sum);
      }
    }
  }
}

// The same without ids for rows of up to 1024 channels, and with its bits (the sums in its order, the skip gradient added to a
// rounded product). Bytes and instructions of a row take about equally long, so the two have to overlap: each lane copies
// its channels of the warp's next rows (x, dy and the skip gradient) to a ring in shared memory, two rows ahead, and the
// arithmetic is on packed pairs. Held in registers the loads of a row were waited for with nothing else to do, and 48 of
// the 128 registers were theirs. With the skip gradient, us before / after: 55 424 x 1024 86.5 / 78.1 (5.8 TB/s), 8 704 x 1024
// 19.1 / 16.5, 17 024 x 512 18.7 / 14.1, x 768 24.1 / 20.2; one bulk copy a row and part instead of the lanes' own 78.3, 16.3,
// 14.5, 20.4; three rows ahead, which is one block a multiprocessor, 78.2, 18.0, 16.3, 22.9.
constexpr int NB_WARPS = 8, NB_STAGES = 2;

// 16 bytes from global to shared memory, in flight until this thread waits for their group.
__device__ __forceinline__ void cp_async_16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int CHUNKS, bool RMS, bool RES>
__global__ void __launch_bounds__(NB_WARPS * 32, 2)
norm_bwd_ring_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                     const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean_in,
                     const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres,
                     __nv_bfloat16* __restrict__ dx, float* __restrict__ dw, int T, int C) {
  constexpr int PARTS = RES ? 3 : 2;
  extern __shared__ __align__(128) uint8_t nb_smem[];   // [warps][stages][parts][C] bf16
  __shared__ __align__(16) float sm_dw[NB_WARPS][256];  // one 256-channel chunk of every warp's sums
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t row_bytes = static_cast<uint32_t>(C) * 2;
  uint8_t* ring = nb_smem + static_cast<size_t>(warp) * NB_STAGES * PARTS * row_bytes;
  grid_chain();
  const int stride = gridDim.x * NB_WARPS;
  const int row0 = blockIdx.x * NB_WARPS + warp;
  auto load = [&](int row, int stage) {   // every iteration commits one group, so the oldest is the one waited for
    if (row < T) {
      uint8_t* d = ring + static_cast<size_t>(stage) * PARTS * row_bytes;
      const size_t at = static_cast<size_t>(row) * C;
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) {
        const int i = c * 256 + lane * 8;
        if (i < C) {
          cp_async_16(d + i * 2, x + at + i);
          cp_async_16(d + row_bytes + i * 2, dy + at + i);
          if (RES) cp_async_16(d + 2 * row_bytes + i * 2, dres + at + i);
        }
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int i = 0; i < NB_STAGES; ++i) load(row0 + i * stride, i);
  uint4 wr[CHUNKS];   // weights of this lane's channels
  float2 acc[CHUNKS][4];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const int i = c * 256 + lane * 8;
    const uint32_t one = 0x3f803f80u;
    wr[c] = w && i < C ? __ldg(reinterpret_cast<const uint4*>(w + i)) : make_uint4(one, one, one, one);
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[c][e] = make_float2(0.f, 0.f);
  }
  float mean_n = 0.f, rstd_n = 0.f;
  if (row0 < T) {
    mean_n = RMS ? 0.f : mean_in[row0];
    rstd_n = rstd_in[row0];
  }
  int stage = 0;
  for (int row = row0; row < T; row += stride) {
    const float mean = mean_n, rstd = rstd_n;
    if (row + stride < T) {
      mean_n = RMS ? 0.f : mean_in[row + stride];
      rstd_n = rstd_in[row + stride];
    }
    cp_async_wait<NB_STAGES - 1>();
    const uint8_t* sx = ring + static_cast<size_t>(stage) * PARTS * row_bytes;
    const float2 nm = make_float2(-mean, -mean), rs = make_float2(rstd, rstd);
    float sg = 0.f, sgx = 0.f;   // (element by element)
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) {
        const uint4 xr = *reinterpret_cast<const uint4*>(sx + i * 2);
        const uint4 dr = *reinterpret_cast<const uint4*>(sx + row_bytes + i * 2);
        const uint32_t *xw = &xr.x, *dww = &dr.x, *ww = &wr[c].x;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 d = unpack_bf16x2(dww[e]);
          float2 xh = unpack_bf16x2(xw[e]);
          if (!RMS) xh = add2(xh, nm);
          xh = mul2(xh, rs);
          const float2 wv = unpack_bf16x2(ww[e]);
          const float2 g = mul2(d, wv);
          if (!RMS) {
            sg += g.x;
            sg += g.y;
          }
          sgx = fmaf(g.x, xh.x, sgx);
          sgx = fmaf(g.y, xh.y, sgx);
          acc[c][e] = fma2(d, xh, acc[c][e]);
        }
      }
    }
    sg = RMS ? 0.f : warp_sum(sg) / C;
    sgx = warp_sum(sgx) / C;
    const float2 nsg = make_float2(-sg, -sg), nsgx = make_float2(-sgx, -sgx);
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) {
        const uint4 xr = *reinterpret_cast<const uint4*>(sx + i * 2);
        const uint4 dr = *reinterpret_cast<const uint4*>(sx + row_bytes + i * 2);
        uint4 rr = make_uint4(0u, 0u, 0u, 0u);
        if (RES) rr = *reinterpret_cast<const uint4*>(sx + 2 * row_bytes + i * 2);
        const uint32_t *xw = &xr.x, *dww = &dr.x, *ww = &wr[c].x, *rw = &rr.x;
        uint4 out;
        uint32_t* ow = &out.x;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float2 xh = unpack_bf16x2(xw[e]);
          if (!RMS) xh = add2(xh, nm);
          xh = mul2(xh, rs);
          float2 g = mul2(unpack_bf16x2(dww[e]), unpack_bf16x2(ww[e]));
          if (!RMS) g = add2(g, nsg);
          g = mul2(fma2(xh, nsgx, g), rs);
          if (RES) {
            const float2 r = unpack_bf16x2(rw[e]);
            g = make_float2(__fadd_rn(g.x, r.x), __fadd_rn(g.y, r.y));
          }
          ow[e] = pack_bf16x2(g.x, g.y);
        }
        *reinterpret_cast<uint4*>(dx + static_cast<size_t>(row) * C + i) = out;
      }
    }
    load(row + NB_STAGES * stride, stage);
    if (++stage == NB_STAGES) stage = 0;
  }
  if (dw) {
    // the warps' sums meet in shared memory chunk by chunk, without atomics there
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (c) __syncthreads();
      float4* mine = reinterpret_cast<float4*>(&sm_dw[warp][lane * 8]);
      mine[0] = make_float4(acc[c][0].x, acc[c][0].y, acc[c][1].x, acc[c][1].y);
      mine[1] = make_float4(acc[c][2].x, acc[c][2].y, acc[c][3].x, acc[c][3].y);
      __syncthreads();
      const int i = c * 256 + threadIdx.x;
      if (i < C) {
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < NB_WARPS; ++j) sum += sm_dw[j][threadIdx.x];
        atomicAdd(&dw[i], sum);
      }
    }
  }
}

template <int CHUNKS, bool RMS, bool RES>
static int norm_bwd_ring(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w, const float* mean,
                         const float* rstd, const __nv_bfloat16* dres, __nv_bfloat16* dx, float* dw, int T, int C,
                         cudaStream_t st) {
  auto kern = norm_bwd_ring_kernel<CHUNKS, RMS, RES>;
  constexpr int most = NB_WARPS * NB_STAGES * (RES ? 3 : 2) * CHUNKS * 256 * 2;
  static bool configured_on[nplm::MAX_DEVICES];
  const int dev_slot = nplm::current_device_slot();
  if (dev_slot < 0) return -4;
  if (!configured_on[dev_slot]) {
    NPLM_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    configured_on[dev_slot] = true;
  }
  int blocks = (T + NB_WARPS - 1) / NB_WARPS;
  if (blocks > 148 * 2) blocks = 148 * 2;   // more blocks only add contention on the dw atomics
  launch_when(static_cast<long long>(T) * C <= CHAIN_ELEMENTS, kern, blocks, NB_WARPS * 32,
      static_cast<size_t>(NB_WARPS) * NB_STAGES * (RES ? 3 : 2) * C * 2, st, dy, x, w, mean, rstd, dres, dx, dw, T, C);
  return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------------ embedding + norm backward
// Rows with the same token have the same x, mean and rstd, and the norm's backward pass is linear in dy: the gradient of a
// table row is the norm backward of S[v] = sum of dy over the rows of token v. So a first kernel reads dy once and only adds
// (bound by that read: 2 C bytes a token), a second one applies the norm's backward pass to the V sums. One norm backward
// per token row, its two reductions behind block barriers and the sums in shared-memory atomics of one block a
// multiprocessor, took 286 us for 55 424 x 1024 and 33 for 2 600 x 256, mostly the flush of 148 whole tables; this takes 92
// and 14.
//
// A warp walks rows of a 128-channel slice, a lane owns four channels and adds them into the warp's own table in shared
// memory [V][128] (nobody else's, so plain adds); the block's tables meet at the end and leave as 16-byte reductions.
// sums: fp32 [V][C], then int [V] = 1 + a row that holds the token (0: none), all zero before the launch.
constexpr int EMB_SLICE = 128, EMB_ROWS = 16;

__global__ void __launch_bounds__(512)
embed_grad_sums_kernel(const __nv_bfloat16* __restrict__ dy, const int* __restrict__ ids,
                       float* __restrict__ sums, int T, int C, int V) {
  grid_chain();
  extern __shared__ __align__(16) float emb_tables[];   // [warps][V][128]
  const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int table = V * EMB_SLICE;
  for (int i = threadIdx.x * 4; i < warps * table; i += blockDim.x * 4)
    *reinterpret_cast<float4*>(emb_tables + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  const int c = blockIdx.x * EMB_SLICE + lane * 4;
  const bool on = c < C;
  float* mine = emb_tables + warp * table + lane * 4;
  int* some_row = reinterpret_cast<int*>(sums + static_cast<size_t>(V) * C);
  const int step = gridDim.y * warps;
  for (int row0 = blockIdx.y * warps + warp; row0 < T; row0 += step * EMB_ROWS) {
    uint2 d[EMB_ROWS];
    int id[EMB_ROWS];
#pragma unroll
    for (int k = 0; k < EMB_ROWS; ++k) {
      const int row = row0 + k * step;
      d[k] = make_uint2(0u, 0u);
      id[k] = -1;
      if (row < T) {
        id[k] = __ldg(ids + row);
        if (on) d[k] = __ldg(reinterpret_cast<const uint2*>(dy + static_cast<size_t>(row) * C + c));
      }
    }
#pragma unroll
    for (int k = 0; k < EMB_ROWS; ++k) {
      if (id[k] >= 0) {
        float4* t = reinterpret_cast<float4*>(mine + id[k] * EMB_SLICE);
        const float2 a = unpack_bf16x2(d[k].x), b = unpack_bf16x2(d[k].y);
        float4 v = *t;
        v.x += a.x;
        v.y += a.y;
        v.z += b.x;
        v.w += b.y;
        *t = v;
        if (blockIdx.x == 0 && lane == 0) some_row[id[k]] = 1 + row0 + k * step;   // (any of them: see above)
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < V * (EMB_SLICE / 4); i += blockDim.x) {
    const int v = i / (EMB_SLICE / 4), ch = blockIdx.x * EMB_SLICE + (i % (EMB_SLICE / 4)) * 4;
    if (ch >= C) continue;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int w = 0; w < warps; ++w) {
      const float4 t = *reinterpret_cast<const float4*>(emb_tables + w * table + i * 4);
      s.x += t.x;
      s.y += t.y;
      s.z += t.z;
      s.w += t.w;
    }
    if (s.x != 0.f || s.y != 0.f || s.z != 0.f || s.w != 0.f)
      atomicAdd(reinterpret_cast<float4*>(sums + static_cast<size_t>(v) * C + ch), s);
  }
}

// One block a token: dtable[v] += norm backward of S[v], dw += S[v] * xhat[v].
__global__ void __launch_bounds__(256)
embed_grad_finish_kernel(const float* __restrict__ sums, const __nv_bfloat16* __restrict__ table,
                         const __nv_bfloat16* __restrict__ w, const float* __restrict__ mean_in,
                         const float* __restrict__ rstd_in, float* __restrict__ dtable, float* __restrict__ dw, int C,
                         int V, int rms) {
  grid_chain();
  __shared__ float red[8][2];
  const int v = blockIdx.x;
  const int row = reinterpret_cast<const int*>(sums + static_cast<size_t>(V) * C)[v] - 1;
  if (row < 0) return;   // the token does not occur (the whole block leaves)
  const float mean = rms ? 0.f : mean_in[row], rstd = rstd_in[row];
  const float* S = sums + static_cast<size_t>(v) * C;
  const __nv_bfloat16* x = table + static_cast<size_t>(v) * C;
  float sg = 0.f, sgx = 0.f;
  for (int c = threadIdx.x; c < C; c += 256) {
    const float xh = (__bfloat162float(x[c]) - mean) * rstd;
    const float g = S[c] * (w ? __bfloat162float(w[c]) : 1.f);
    sg += g;
    sgx += g * xh;
  }
  sg = warp_sum(sg);
  sgx = warp_sum(sgx);
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5][0] = sg;
    red[threadIdx.x >> 5][1] = sgx;
  }
  __syncthreads();
  sg = sgx = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    sg += red[k][0];
    sgx += red[k][1];
  }
  sg = rms ? 0.f : sg / C;
  sgx /= C;
  for (int c = threadIdx.x; c < C; c += 256) {
    const float xh = (__bfloat162float(x[c]) - mean) * rstd;
    const float g = S[c] * (w ? __bfloat162float(w[c]) : 1.f);
    dtable[static_cast<size_t>(v) * C + c] += rstd * (g - sg - xh * sgx);
    if (dw) atomicAdd(&dw[c], S[c] * xh);
  }
}

// ------------------------------------------------------------------ RoPE (in place on packed qkv)
// qkv: [T][3][H][D] bf16. Rotates q and k: out = x*cos + rotate_half(x)*sin with
// cos/sin[pos][D/2] fp32 (the two halves of the reference table are identical). sign = -1
// applies the transpose (backward).
__global__ void __launch_bounds__(256)
rope_kernel(__nv_bfloat16* __restrict__ qkv, const int* __restrict__ pos,
            const float* __restrict__ cos_t, const float* __restrict__ sin_t, int T, int H, int D,
            float sign) {
  grid_chain();
  const int half = D >> 1;
  const int vec_per_head = half >> 3;  // 8 elements per thread from each half
  const long long total = static_cast<long long>(T) * 2 * H * vec_per_head;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int vv = static_cast<int>(idx % vec_per_head);
    long long r = idx / vec_per_head;
    const int h = static_cast<int>(r % H);
    r /= H;
    const int qk = static_cast<int>(r % 2);
    const int t = static_cast<int>(r / 2);
    __nv_bfloat16* base = qkv + ((static_cast<size_t>(t) * 3 + qk) * H + h) * D + vv * 8;
    const int p = pos[t];
    const float* cp = cos_t + static_cast<size_t>(p) * half + vv * 8;
    const float* sp = sin_t + static_cast<size_t>(p) * half + vv * 8;
    float x1[8], x2[8], o1[8], o2[8];
    load8(base, x1);
    load8(base + half, x2);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float c = cp[e], s = sign * sp[e];
      o1[e] = x1[e] * c - x2[e] * s;
      o2[e] = x2[e] * c + x1[e] * s;
    }
    store8(base, o1);
    store8(base + half, o2);
  }
}

// ------------------------------------------------------------------ SwiGLU
// pre: [T][2I] = [value | gate]; out[T][I] = silu(gate) * value
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ pre, __nv_bfloat16* __restrict__ out,
                  long long T, int I) {
  grid_chain();
  const int vec = I >> 3;
  const long long total = T * vec;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = idx / vec;
    const int i = static_cast<int>(idx % vec) * 8;
    float v[8], g[8], o[8];
    load8(pre + t * 2 * I + i, v);
    load8(pre + t * 2 * I + I + i, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = g[e] / (1.f + __expf(-g[e])) * v[e];
    store8(out + t * I + i, o);
  }
}

// dpre[T][2I] from dout[T][I]: dvalue = dout*silu(g), dgate = dout*v*sig(g)*(1+g*(1-sig(g)))
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ pre, const __nv_bfloat16* __restrict__ dout,
                  __nv_bfloat16* __restrict__ dpre, long long T, int I) {
  grid_chain();
  const int vec = I >> 3;
  const long long total = T * vec;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long t = idx / vec;
    const int i = static_cast<int>(idx % vec) * 8;
    float v[8], g[8], d[8], dv[8], dg[8];
    load8(pre + t * 2 * I + i, v);
    load8(pre + t * 2 * I + I + i, g);
    load8(dout + t * I + i, d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sg = 1.f / (1.f + __expf(-g[e]));
      dv[e] = d[e] * g[e] * sg;
      dg[e] = d[e] * v[e] * sg * (1.f + g[e] * (1.f - sg));
    }
    store8(dpre + t * 2 * I + i, dv);
    store8(dpre + t * 2 * I + I + i, dg);
  }
}

// ------------------------------------------------------------------ activations
// act: 0 gelu(erf), 1 relu, 2 silu
__global__ void __launch_bounds__(256)
act_fwd_kernel(const __nv_bfloat16* __restrict__ pre, __nv_bfloat16* __restrict__ out,
               long long n8, int act) {
  grid_chain();
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < n8;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    float p[8], o[8];
    load8(pre + idx * 8, p);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      o[e] = act == 0 ? gelu_erf(p[e]) : act == 1 ? fmaxf(p[e], 0.f) : p[e] / (1.f + __expf(-p[e]));
    }
    store8(out + idx * 8, o);
  }
}

__global__ void __launch_bounds__(256)
act_bwd_kernel(const __nv_bfloat16* __restrict__ pre, const __nv_bfloat16* __restrict__ dout,
               __nv_bfloat16* __restrict__ dpre, long long n8, int act) {
  grid_chain();
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < n8;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    float p[8], d[8], o[8];
    load8(pre + idx * 8, p);
    load8(dout + idx * 8, d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float gr;
      if (act == 0) {
        gr = gelu_erf_grad(p[e]);
      } else if (act == 1) {
        gr = p[e] > 0.f ? 1.f : 0.f;
      } else {
        const float sg = 1.f / (1.f + __expf(-p[e]));
        gr = sg * (1.f + p[e] * (1.f - sg));
      }
      o[e] = d[e] * gr;
    }
    store8(dpre + idx * 8, o);
  }
}

// ------------------------------------------------------------------ row gather / scatter
__global__ void __launch_bounds__(256)
gather_rows_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ idx,
                   __nv_bfloat16* __restrict__ dst, int n, int C) {
  grid_chain();
  const int vec = C >> 3;
  const long long total = static_cast<long long>(n) * vec;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / vec);
    const int c = static_cast<int>(i % vec) * 8;
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(r) * C + c) =
        *reinterpret_cast<const uint4*>(src + static_cast<size_t>(idx[r]) * C + c);
  }
}

// dst[idx[r]] = src[r] (indices are unique); rows not named keep their contents.
__global__ void __launch_bounds__(256)
scatter_rows_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ idx,
                    __nv_bfloat16* __restrict__ dst, int n, int C) {
  grid_chain();
  const int vec = C >> 3;
  const long long total = static_cast<long long>(n) * vec;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / vec);
    const int c = static_cast<int>(i % vec) * 8;
    *reinterpret_cast<uint4*>(dst + static_cast<size_t>(idx[r]) * C + c) =
        *reinterpret_cast<const uint4*>(src + static_cast<size_t>(r) * C + c);
  }
}

// ------------------------------------------------------------------ fused MLM-head cross entropy
// One warp per row. h: [n][C] bf16 (output of the head norm), W: [V][C] bf16 (tied decoder),
// bias: [V] bf16 or null, labels: [n] int (ignore_index = -100). V <= 32.
// Writes dlogits[n][32] fp32 = (softmax - onehot) * inv_count (0 for ignored rows), optional
// logits[n][V] fp32, and accumulates loss_sum += -log p[label] * inv_count.
// inv_count is read from device memory (1 / number of valid labels).
constexpr int CE_WARPS = 8;

// inv[0] = 1 / max(number of labels >= 0, 1), loss[0] = 0: one small launch for what were six (comparison, sum, clamp,
// conversion, division, zeros).
__global__ void __launch_bounds__(1024)
ce_count_kernel(const int* __restrict__ labels, int n, float* __restrict__ inv, float* __restrict__ loss) {
  grid_chain();
  __shared__ int part[32];
  int valid = 0;
  for (int i = threadIdx.x; i < n; i += 1024) valid += labels[i] >= 0;
  valid = __reduce_add_sync(0xffffffffu, valid);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = valid;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int total = __reduce_add_sync(0xffffffffu, part[threadIdx.x]);
    if (threadIdx.x == 0) {
      inv[0] = __fdiv_rn(1.f, static_cast<float>(max(total, 1)));
      loss[0] = 0.f;
    }
  }
}

template <int CHUNKS>
__global__ void __launch_bounds__(CE_WARPS * 32)
ce_fwd_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ W,
              const __nv_bfloat16* __restrict__ bias, const int* __restrict__ labels,
              const float* __restrict__ inv_count, float* __restrict__ dlogits,
              float* __restrict__ logits_out, float* __restrict__ loss_sum, int n, int C, int V) {
  grid_chain();
  extern __shared__ __nv_bfloat16 sW[];  // [V][C]
  for (int i = threadIdx.x * 8; i < V * C; i += blockDim.x * 8)
    *reinterpret_cast<uint4*>(sW + i) = *reinterpret_cast<const uint4*>(W + i);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const float invc = *inv_count;
  float block_loss = 0.f;
  for (int row = blockIdx.x * CE_WARPS + (threadIdx.x >> 5); row < n; row += gridDim.x * CE_WARPS) {
    float hv[CHUNKS][8];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int i = c * 256 + lane * 8;
      if (i < C) load8(h + static_cast<size_t>(row) * C + i, hv[c]);
    }
    float part[32];
#pragma unroll
    for (int v = 0; v < 32; ++v) {
      float s = 0.f;
      if (v < V) {
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
          const int i = c * 256 + lane * 8;
          if (i < C) {
            float wv[8];
            load8(sW + v * C + i, wv);
#pragma unroll
            for (int e = 0; e < 8; ++e) s += hv[c][e] * wv[e];
          }
        }
      }
      part[v] = s;
    }
    // transpose-reduce: after the 5 steps lane l holds the full sum for vocab entry l
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
      const bool upper = (lane & step) != 0;
#pragma unroll
      for (int j = 0; j < step; ++j) {
        const float send = upper ? part[j] : part[j + step];
        const float keep = upper ? part[j + step] : part[j];
        part[j] = keep + __shfl_xor_sync(0xffffffffu, send, step);
      }
    }
    float logit = part[0];
    if (lane < V) {
      if (bias) logit += __bfloat162float(bias[lane]);
    } else {
      logit = -INFINITY;
    }
    if (logits_out && lane < V) logits_out[static_cast<size_t>(row) * V + lane] = logit;
    const float mx = warp_max(logit);
    const float ex = lane < V ? __expf(logit - mx) : 0.f;
    const float se = warp_sum(ex);
    const int lab = labels[row];
    float dl = 0.f;
    if (lab >= 0) {
      const float p = ex / se;
      dl = (p - (lane == lab ? 1.f : 0.f)) * invc;
      const float lab_logit = __shfl_sync(0xffffffffu, logit, lab);
      if (lane == 0) block_loss += (mx + __logf(se) - lab_logit) * invc;
    }
    dlogits[static_cast<size_t>(row) * 32 + lane] = dl;
  }
  if (lane == 0 && block_loss != 0.f) atomicAdd(loss_sum, block_loss);
}

// Backward: dh[row] = g * sum_v dl[row][v] W[v];  dW[v] += g * sum_rows dl[row][v] h[row];
// dbias[v] += g * sum_rows dl[row][v].  g = *gscale (upstream gradient of the loss).
// Bound by its 2 x 32 fp32 multiply-adds an element of h. A thread owns two channels: W and the sums dW of all 32 entries
// of the vocabulary stay in registers (128 of them, three blocks a multiprocessor), the dlogits of 16 rows are read as
// broadcasts from shared memory, doubled for the packed multiply-adds. A block takes 256 channels of `rows` rows, so that
// 1 300 rows already fill the chip: 1 300 x 1024 11.5 us, 8 300 x 1024 42, where a block a 32-row tile took 95 and 170.
// The 32 products of an element of dh are one chain in the vocabulary's order: its bits reach e4m3 training.
// A row whose dlogits are all zero (an ignored label) has a zero gradient and its h is not read: an infinity or a NaN there
// reaches nothing.
constexpr int CE_ROWS = 16;

__global__ void __launch_bounds__(128, 3)
ce_bwd_kernel(const __nv_bfloat16* __restrict__ h, const __nv_bfloat16* __restrict__ W,
              const float* __restrict__ dlogits, const float* __restrict__ gscale,
              __nv_bfloat16* __restrict__ dh, float* __restrict__ dW, float* __restrict__ dbias,
              int n, int C, int V, int rows) {
  grid_chain();
  __shared__ __align__(16) float2 sd[CE_ROWS][32];
  __shared__ __align__(16) uint8_t live[CE_ROWS];
  const int tid = threadIdx.x;
  const int ch = blockIdx.x * 256 + tid * 2;
  const bool own = ch < C;
  const int r1 = min(n, (static_cast<int>(blockIdx.y) + 1) * rows);
  const float g = *gscale;
  float2 w[32], acc[32];
#pragma unroll
  for (int v = 0; v < 32; ++v) {
    w[v] = own && v < V ? unpack_bf16x2(__ldg(reinterpret_cast<const uint32_t*>(W + static_cast<size_t>(v) * C + ch)))
                        : make_float2(0.f, 0.f);
    acc[v] = make_float2(0.f, 0.f);
  }
  float db = 0.f;
  for (int base = blockIdx.y * rows; base < r1; base += CE_ROWS) {
    __syncthreads();   // the previous rows are consumed
#pragma unroll
    for (int i = tid; i < CE_ROWS * 32; i += 128) {
      const int r = base + (i >> 5);
      const float d = r < r1 && (i & 31) < V ? dlogits[static_cast<size_t>(r) * 32 + (i & 31)] * g : 0.f;
      sd[i >> 5][i & 31] = make_float2(d, d);
      const int any = __any_sync(0xffffffffu, d != 0.f);      // (a warp holds one row)
      if ((i & 31) == 0) live[i >> 5] = any ? 1 : 0;
    }
    __syncthreads();
    // bit r: row base + r has a gradient (four bytes of 0 or 1 gathered into the top nibble by each product)
    const uint4 all = *reinterpret_cast<const uint4*>(live);
    const uint32_t rows_on = (all.x * 0x10204080u >> 28) | (all.y * 0x10204080u >> 28 << 4) |
                             (all.z * 0x10204080u >> 28 << 8) | (all.w * 0x10204080u >> 28 << 12);
    if (blockIdx.x == 0 && tid < 32) {
#pragma unroll
      for (int r = 0; r < CE_ROWS; ++r) db += sd[r][tid].x;
    }
#pragma unroll 1
    for (int r = 0; r < CE_ROWS && base + r < r1; r += 4) {
      float2 hv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        hv[q] = own && (rows_on >> (r + q) & 1u)
                    ? unpack_bf16x2(__ldg(reinterpret_cast<const uint32_t*>(h + static_cast<size_t>(base + r + q) * C + ch)))
                    : make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 o = make_float2(0.f, 0.f);
#pragma unroll
        for (int v = 0; v < 32; v += 2) {
          const float4 d = *reinterpret_cast<const float4*>(&sd[r + q][v]);
          const float2 d0 = make_float2(d.x, d.y), d1 = make_float2(d.z, d.w);
          o = fma2(d0, w[v], o);
          o = fma2(d1, w[v + 1], o);
          acc[v] = fma2(d0, hv[q], acc[v]);
          acc[v + 1] = fma2(d1, hv[q], acc[v + 1]);
        }
        if (own && base + r + q < r1)
          *reinterpret_cast<uint32_t*>(dh + static_cast<size_t>(base + r + q) * C + ch) =
              (rows_on >> (r + q) & 1u) ? pack_bf16x2(o.x, o.y) : 0u;
      }
    }
  }
  if (own) {
#pragma unroll
    for (int v = 0; v < 32; ++v)
      if (v < V && (acc[v].x != 0.f || acc[v].y != 0.f)) {
        float* dst = dW + static_cast<size_t>(v) * C + ch;
        if ((reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
          atomicAdd(reinterpret_cast<float2*>(dst), acc[v]);
        } else {
          atomicAdd(dst, acc[v].x);
          atomicAdd(dst + 1, acc[v].y);
        }
      }
  }
  if (dbias && blockIdx.x == 0 && tid < V && db != 0.f) atomicAdd(&dbias[tid], db);
}

// ------------------------------------------------------------------ optimizer
// sum of squares of an fp32 buffer, accumulated into out[0]
__global__ void __launch_bounds__(256)
sumsq_kernel(const float* __restrict__ x, long long n, float* __restrict__ out) {
  grid_chain();
  float s = 0.f;
  const long long n4 = n >> 2;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float4 v = reinterpret_cast<const float4*>(x)[i];
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    for (long long i = n4 << 2; i < n; ++i) s += x[i] * x[i];
  s = warp_sum(s);
  __shared__ float ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < (blockDim.x >> 5); ++i) t += ws[i];
    atomicAdd(out, t);
  }
}

// AdamW on fp32 master weights with decoupled weight decay; the gradient is scaled by
// grad_scale * min(1, max_norm / (sqrt(*sumsq * grad_scale^2) + 1e-6)) (clip_grad_norm_
// semantics), read on the device so no host round trip is needed. Writes the bf16 compute copy
// and, when zero_grad != 0, clears the gradient for the next accumulation window.
// hyper: [lr, beta1, beta2, eps, weight_decay, bias_corr1, bias_corr2, grad_scale, max_norm]
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
             float* __restrict__ g, __nv_bfloat16* __restrict__ p_bf16,
             const float* __restrict__ hyper, const float* __restrict__ sumsq, long long n,
             int zero_grad) {
  grid_chain();
  const float lr = hyper[0], b1 = hyper[1], b2 = hyper[2], eps = hyper[3], wd = hyper[4];
  const float bc1 = hyper[5], bc2 = hyper[6], gs = hyper[7], max_norm = hyper[8];
  float scale = gs;
  if (sumsq != nullptr && max_norm > 0.f) {
    const float norm = sqrtf(*sumsq) * gs;
    scale = gs * fminf(1.f, max_norm / (norm + 1e-6f));
  }
  const float step_size = lr / bc1;
  const float inv_sqrt_bc2 = rsqrtf(bc2);
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float gr = g[i] * scale;
    float pv = p[i];
    pv *= (1.f - lr * wd);
    const float mv = b1 * m[i] + (1.f - b1) * gr;
    const float vv = b2 * v[i] + (1.f - b2) * gr * gr;
    const float denom = sqrtf(vv) * inv_sqrt_bc2 + eps;
    pv -= step_size * mv / denom;
    p[i] = pv;
    m[i] = mv;
    v[i] = vv;
    if (p_bf16) p_bf16[i] = __float2bfloat16(pv);
    if (zero_grad) g[i] = 0.f;
  }
}

// ---- Muon (matrices of one shape, addressed through a table of flat offsets) -----------------
// gradient scale shared by the optimizer kernels: grad_scale and clip_grad_norm_ by the global norm
__device__ __forceinline__ float clip_scale(const float* sumsq, float gs, float max_norm) {
  if (sumsq == nullptr || max_norm <= 0.f) return gs;
  return gs * fminf(1.f, max_norm / (sqrtf(*sumsq) * gs + 1e-6f));
}

// Momentum of matrix blockIdx.y (numel elements at flat offset off[y]) and the bf16 update that
// enters the Newton-Schulz iterations:  m <- mu m + g,  u = nesterov ? g + mu m : m,
// upd[y] = bf16(u),  usq[y] += sum of the rounded u^2 (its Frobenius norm normalises the iteration).
__global__ void __launch_bounds__(256)
muon_momentum_kernel(const float* __restrict__ g, float* __restrict__ m,
                     const long long* __restrict__ off, long long numel,
                     __nv_bfloat16* __restrict__ upd, float* __restrict__ usq,
                     const float* __restrict__ sumsq, float gs, float max_norm, float mu, int nesterov) {
  grid_chain();
  const float scale = clip_scale(sumsq, gs, max_norm);
  const long long base = off[blockIdx.y];
  const float4* g4 = reinterpret_cast<const float4*>(g + base);
  float4* m4 = reinterpret_cast<float4*>(m + base);
  uint2* u4 = reinterpret_cast<uint2*>(upd + static_cast<long long>(blockIdx.y) * numel);
  float acc = 0.f;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < (numel >> 2);
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float4 gv = g4[i];
    float4 mv = m4[i];
    gv.x *= scale; gv.y *= scale; gv.z *= scale; gv.w *= scale;
    mv.x = mu * mv.x + gv.x; mv.y = mu * mv.y + gv.y; mv.z = mu * mv.z + gv.z; mv.w = mu * mv.w + gv.w;
    m4[i] = mv;
    float4 u = mv;
    if (nesterov) { u.x = gv.x + mu * mv.x; u.y = gv.y + mu * mv.y; u.z = gv.z + mu * mv.z; u.w = gv.w + mu * mv.w; }
    uint2 pk;
    pk.x = pack_bf16x2(u.x, u.y);
    pk.y = pack_bf16x2(u.z, u.w);
    u4[i] = pk;
    const float2 a = unpack_bf16x2(pk.x), b = unpack_bf16x2(pk.y);
    acc += a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y;
  }
  acc = warp_sum(acc);
  __shared__ float ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int i = 0; i < 8; ++i) t += ws[i];
    atomicAdd(&usq[blockIdx.y], t);
  }
}

// Applies the orthogonalised update O[y] (bf16) to matrix y: decoupled weight decay (cautious:
// only where the update and the weight agree in sign), p <- p - lr O, and the bf16 compute copy.
__global__ void __launch_bounds__(256)
muon_apply_kernel(float* __restrict__ p, __nv_bfloat16* __restrict__ p16,
                  const long long* __restrict__ off, long long numel,
                  const __nv_bfloat16* __restrict__ O, float lr, float wd, int cautious) {
  grid_chain();
  const long long base = off[blockIdx.y];
  float4* p4 = reinterpret_cast<float4*>(p + base);
  uint2* q4 = p16 ? reinterpret_cast<uint2*>(p16 + base) : nullptr;
  const uint2* o4 = reinterpret_cast<const uint2*>(O + static_cast<long long>(blockIdx.y) * numel);
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < (numel >> 2);
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float4 pv = p4[i];
    const uint2 ov = o4[i];
    const float2 oa = unpack_bf16x2(ov.x), ob = unpack_bf16x2(ov.y);
    const float o[4] = {oa.x, oa.y, ob.x, ob.y};
    float* pe = reinterpret_cast<float*>(&pv);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float x = pe[e];
      if (wd > 0.f) {
        if (cautious) x -= (o[e] * x > 0.f) ? lr * wd * x : 0.f;
        else x *= (1.f - lr * wd);
      }
      pe[e] = x - lr * o[e];
    }
    p4[i] = pv;
    if (q4) {
      uint2 pk;
      pk.x = pack_bf16x2(pv.x, pv.y);
      pk.y = pack_bf16x2(pv.z, pv.w);
      q4[i] = pk;
    }
  }
}

// AdamW over a table of parameter tensors of one flat buffer (tensor y: numel[y] elements at
// offset off[y], weight decay only where decay[y] != 0); same update as adamw_kernel.
__global__ void __launch_bounds__(256)
adamw_slots_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                   const float* __restrict__ g, __nv_bfloat16* __restrict__ p16,
                   const long long* __restrict__ off, const long long* __restrict__ numel,
                   const int* __restrict__ decay, const float* __restrict__ sumsq, float gs, float max_norm,
                   float lr, float b1, float b2, float eps, float wd, float bc1, float bc2) {
  grid_chain();
  const float scale = clip_scale(sumsq, gs, max_norm);
  const long long base = off[blockIdx.y], n = numel[blockIdx.y];
  const float decay_mul = decay[blockIdx.y] ? (1.f - lr * wd) : 1.f;
  const float step_size = lr / bc1, inv_sqrt_bc2 = rsqrtf(bc2);
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long j = base + i;
    const float gr = g[j] * scale;
    float pv = p[j] * decay_mul;
    const float mv = b1 * m[j] + (1.f - b1) * gr;
    const float vv = b2 * v[j] + (1.f - b2) * gr * gr;
    pv -= step_size * mv / (sqrtf(vv) * inv_sqrt_bc2 + eps);
    p[j] = pv;
    m[j] = mv;
    v[j] = vv;
    if (p16) p16[j] = __float2bfloat16(pv);
  }
}

__global__ void __launch_bounds__(256)
cast_f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                        long long n) {
  grid_chain();
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    dst[i] = __float2bfloat16(src[i]);
}

// masked MSE for embedding distillation: loss = sum_{valid tokens} sum_c (s-t)^2 / max(1, n_valid)
// (src/nanoplm/distillation/trainer.py:30-40). ds = 2 (s-t) * inv_count for valid rows, else 0.
__global__ void __launch_bounds__(256)
masked_mse_kernel(const __nv_bfloat16* __restrict__ s, const __nv_bfloat16* __restrict__ t,
                  const int* __restrict__ valid, const long long* __restrict__ rows, const float* __restrict__ inv_count,
                  __nv_bfloat16* __restrict__ ds, float* __restrict__ loss_sum, int T, int C) {
  grid_chain();
  const int vec = C >> 3;
  const long long total = static_cast<long long>(T) * vec;
  const float invc = *inv_count;
  float acc = 0.f;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / vec);
    const int c = static_cast<int>(i % vec) * 8;
    float o[8];
    if (valid == nullptr || valid[r]) {
      float a[8], b[8];
      load8(s + static_cast<size_t>(r) * C + c, a);
      load8(t + static_cast<size_t>(rows == nullptr ? r : rows[r]) * C + c, b);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = a[e] - b[e];
        acc += d * d;
        o[e] = 2.f * d * invc;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = 0.f;
    }
    if (ds) store8(ds + static_cast<size_t>(r) * C + c, o);
  }
  acc = warp_sum(acc);
  __shared__ float ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tsum = 0.f;
    for (int i = 0; i < (blockDim.x >> 5); ++i) tsum += ws[i];
    atomicAdd(loss_sum, tsum * invc);
  }
}

static int grid_for(long long work_items, int threads) {
  long long b = (work_items + threads - 1) / threads;
  const long long cap = 148LL * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace nplm

using namespace nplm;

#define NPLM_CHUNK_DISPATCH(C_, CALL)                      \
  do {                                                     \
    const int chunks_ = ((C_) + 255) / 256;                \
    if (chunks_ <= 1) { CALL(1); }                         \
    else if (chunks_ <= 2) { CALL(2); }                    \
    else if (chunks_ <= 3) { CALL(3); }                    \
    else if (chunks_ <= 4) { CALL(4); }                    \
    else if (chunks_ <= 8) { CALL(8); }                    \
    else if (chunks_ <= 16) { CALL(16); }                  \
    else return -3;                                        \
  } while (0)

extern "C" int nplm_norm_fwd(const void* x, const int* ids, const void* w, void* y, float* mean,
                             float* rstd, int T, int C, float eps, int rms, cudaStream_t st) {
  if (T <= 0) return 0;
  if (C % 8) return -3;
  const int blocks = (T + 7) / 8 < 148 * 8 ? (T + 7) / 8 : 148 * 8;
#define CALL(N_)                                                                               \
  launch_when(static_cast<long long>(T) * C <= CHAIN_ELEMENTS, norm_fwd_kernel<N_>, blocks, 256, 0, st,                       \
      reinterpret_cast<const __nv_bfloat16*>(x), ids,                                                                         \
                                              reinterpret_cast<const __nv_bfloat16*>(w),       \
                                              reinterpret_cast<__nv_bfloat16*>(y), mean, rstd, \
                                              T, C, eps, rms)
  NPLM_CHUNK_DISPATCH(C, CALL);
#undef CALL
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_norm_bwd(const void* dy, const void* x, const int* ids, const void* w,
                             const float* mean, const float* rstd, const void* dres, void* dx,
                             float* dw, float* dtable, int T, int C, int V, int rms, cudaStream_t st) {
  if (T <= 0) return 0;
  if (C % 8) return -3;
  if (ids == nullptr && C <= 1024) {
    const auto go = [&](auto kern) {
      return kern(reinterpret_cast<const __nv_bfloat16*>(dy), reinterpret_cast<const __nv_bfloat16*>(x),
                  reinterpret_cast<const __nv_bfloat16*>(w), mean, rstd, reinterpret_cast<const __nv_bfloat16*>(dres),
                  reinterpret_cast<__nv_bfloat16*>(dx), dw, T, C, st);
    };
#define RING(N_)                                                                                   \
  return rms ? (dres ? go(norm_bwd_ring<N_, true, true>) : go(norm_bwd_ring<N_, true, false>))     \
             : (dres ? go(norm_bwd_ring<N_, false, true>) : go(norm_bwd_ring<N_, false, false>))
    if (C <= 256) RING(1);
    if (C <= 512) RING(2);
    if (C <= 768) RING(3);
    RING(4);
#undef RING
  }
  int blocks = (T + 7) / 8;
  if (blocks > 148 * 2) blocks = 148 * 2;
#define CALL(N_)                                                                              \
  launch_when(static_cast<long long>(T) * C <= CHAIN_ELEMENTS, norm_bwd_kernel<N_>, blocks, 256, 0, st,                                                 \
      reinterpret_cast<const __nv_bfloat16*>(dy), reinterpret_cast<const __nv_bfloat16*>(x),  \
      ids, reinterpret_cast<const __nv_bfloat16*>(w), mean, rstd,                             \
      reinterpret_cast<const __nv_bfloat16*>(dres), reinterpret_cast<__nv_bfloat16*>(dx), dw, \
      dtable, T, C, rms)
  NPLM_CHUNK_DISPATCH(C, CALL);
#undef CALL
  return static_cast<int>(cudaGetLastError());
}

// Embedding + norm backward (x = table[ids]): dtable (fp32 [V][C]) and dw (fp32 [C], may be null) are added to. scratch: fp32
// [V * (C + 1)], cleared here. A block keeps one table of 512 V bytes a warp in shared memory, so up to V = 200 at least
// two warps fit; larger vocabularies return -3 (nplm_norm_bwd with ids takes them).
extern "C" int nplm_embed_bwd(const void* dy, const void* table, const int* ids, const void* w, const float* mean,
                              const float* rstd, float* dw, float* dtable, float* scratch, int T, int C, int V, int rms,
                              cudaStream_t st) {
  if (T <= 0) return 0;
  if ((C % 8) || V < 1 || V > 200 || (reinterpret_cast<uintptr_t>(dy) & 7) || (reinterpret_cast<uintptr_t>(scratch) & 15))
    return -3;
  const int table_bytes = V * EMB_SLICE * 4;
  int warps = 200 * 1024 / table_bytes;
  if (warps > 12) warps = 12;
  const int slices = (C + EMB_SLICE - 1) / EMB_SLICE;
  // one block a multiprocessor; with few tokens fewer blocks, so that a warp has at least one full set of loads
  int by = 148 / slices;
  if (by < 1) by = 1;
  const int full = (T + warps * EMB_ROWS - 1) / (warps * EMB_ROWS);
  if (by > full) by = full;
  NPLM_CUDA_CHECK(cudaMemsetAsync(scratch, 0, static_cast<size_t>(V) * (C + 1) * sizeof(float), st));
  static bool configured_on[nplm::MAX_DEVICES];
  const int dev_slot = nplm::current_device_slot();
  if (dev_slot < 0) return -4;
  if (!configured_on[dev_slot]) {
    NPLM_CUDA_CHECK(cudaFuncSetAttribute(embed_grad_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    configured_on[dev_slot] = true;
  }
  launch_when(static_cast<long long>(T) * C <= CHAIN_ELEMENTS, embed_grad_sums_kernel, dim3(slices, by), 32 * warps,
      static_cast<size_t>(warps) * table_bytes, st,
                 reinterpret_cast<const __nv_bfloat16*>(dy), ids, scratch, T, C, V);
  launch_chained(embed_grad_finish_kernel, V, 256, 0, st, scratch, reinterpret_cast<const __nv_bfloat16*>(table),
                 reinterpret_cast<const __nv_bfloat16*>(w), mean, rstd, dtable, dw, C, V, rms);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_rope(void* qkv, const int* pos, const float* cos_t, const float* sin_t, int T,
                         int H, int D, int backward, cudaStream_t st) {
  if (T <= 0) return 0;
  if (D % 16) return -3;
  const long long total = static_cast<long long>(T) * 2 * H * (D / 16);
  launch_when(static_cast<long long>(T) * 2 * H * D <= CHAIN_ELEMENTS, rope_kernel, grid_for(total, 256), 256, 0, st,
      reinterpret_cast<__nv_bfloat16*>(qkv), pos, cos_t, sin_t, T, H, D, backward ? -1.f : 1.f);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_swiglu_fwd(const void* pre, void* out, long long T, int I, cudaStream_t st) {
  if (T <= 0) return 0;
  if (I % 8) return -3;
  launch_when(T * I <= CHAIN_ELEMENTS, swiglu_fwd_kernel, grid_for(T * (I / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(pre), reinterpret_cast<__nv_bfloat16*>(out), T, I);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_swiglu_bwd(const void* pre, const void* dout, void* dpre, long long T, int I,
                               cudaStream_t st) {
  if (T <= 0) return 0;
  if (I % 8) return -3;
  launch_when(T * I <= CHAIN_ELEMENTS, swiglu_bwd_kernel, grid_for(T * (I / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(pre), reinterpret_cast<const __nv_bfloat16*>(dout),
      reinterpret_cast<__nv_bfloat16*>(dpre), T, I);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_act_fwd(const void* pre, void* out, long long n, int act, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -3;
  launch_when(n <= CHAIN_ELEMENTS, act_fwd_kernel, grid_for(n / 8, 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(pre), reinterpret_cast<__nv_bfloat16*>(out), n / 8, act);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_act_bwd(const void* pre, const void* dout, void* dpre, long long n, int act,
                            cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -3;
  launch_when(n <= CHAIN_ELEMENTS, act_bwd_kernel, grid_for(n / 8, 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(pre), reinterpret_cast<const __nv_bfloat16*>(dout),
      reinterpret_cast<__nv_bfloat16*>(dpre), n / 8, act);
  return static_cast<int>(cudaGetLastError());
}

// y[b][j][i] = x[b][i][j] * scale[b] (bf16 [B][R][C] -> [B][C][R], scale bf16 or null; R and C multiples of 64). A block
// moves a 64 x 64 tile through shared memory, 16 bytes a lane on both sides, rows of 66 elements against bank
// conflicts. Bound by memory: the strided copy it replaces took 234 us for 16 matrices of 4096 x 1024 (268 MB), this
// and its 3072 x 1024 like 41 us on average.
namespace nplm {
__global__ void __launch_bounds__(256)
transpose_scale_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ scale,
                       __nv_bfloat16* __restrict__ y, int R, int C) {
  grid_chain();
  __shared__ __nv_bfloat16 tile[64][66];
  const size_t base = static_cast<size_t>(blockIdx.z) * R * C;
  const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
  const int row = threadIdx.x >> 3, ch = (threadIdx.x & 7) * 8;
  const float s = scale != nullptr ? __bfloat162float(scale[blockIdx.z]) : 1.f;
#pragma unroll
  for (int h = 0; h < 64; h += 32) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(x + base + static_cast<size_t>(r0 + row + h) * C + c0 + ch));
    const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 t = unpack_bf16x2(w[e]);
      *reinterpret_cast<uint32_t*>(&tile[row + h][ch + 2 * e]) = pack_bf16x2(t.x * s, t.y * s);
    }
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 64; h += 32) {
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = tile[ch + e][row + h];
    *reinterpret_cast<uint4*>(y + base + static_cast<size_t>(c0 + row + h) * R + r0 + ch) =
        *reinterpret_cast<const uint4*>(v);
  }
}
}  // namespace nplm

extern "C" int nplm_transpose_scale(const void* x, const void* scale, void* y, int B, int R, int C, cudaStream_t st) {
  if (B <= 0 || R <= 0 || C <= 0) return 0;
  if ((R % 64) || (C % 64) || B > 65535 || R / 64 > 65535 || (reinterpret_cast<uintptr_t>(x) & 15) ||
      (reinterpret_cast<uintptr_t>(y) & 15))
    return -3;
  launch_chained(nplm::transpose_scale_kernel, dim3(C / 64, R / 64, B), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(scale),
      reinterpret_cast<__nv_bfloat16*>(y), R, C);
  return static_cast<int>(cudaGetLastError());
}

// out[b][c] = mean over rows cu[b] .. cu[b + 1] - drop_last of x[row][c] (bf16 in, fp32 sums and result; no rows: NaN,
// as an empty mean is). A block takes 64 channels of one sequence: 8 threads cover a 128-byte line of a row, 32
// row groups walk the sequence, so one protein still fills C / 64 blocks. Bound by reading x once (2 C bytes a
// token); what it replaces is a reduction, a count and two copies per sequence (13.5 + 3.5 + 3.2 + 2.9 us each
// and as many launches and host synchronisations).
namespace nplm {
__global__ void __launch_bounds__(256)
segment_mean_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ cu, float* __restrict__ out,
                    int C, int drop_last) {
  grid_chain();
  __shared__ float part[32][64];
  const int b = blockIdx.x, g = threadIdx.x >> 3, l = threadIdx.x & 7;
  const int c = blockIdx.y * 64 + l * 8;
  const int lo = cu[b], hi = cu[b + 1] - drop_last;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c < C) {
    for (int r = lo + g; r < hi; r += 32) {
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(x + static_cast<size_t>(r) * C + c));
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 t = unpack_bf16x2(w[e]);
        acc[2 * e] += t.x;
        acc[2 * e + 1] += t.y;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) part[g][l * 8 + e] = acc[e];
  __syncthreads();
  const int col = blockIdx.y * 64 + threadIdx.x;
  if (threadIdx.x < 64 && col < C) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) s += part[i][threadIdx.x];
    out[static_cast<size_t>(b) * C + col] = s / static_cast<float>(max(hi - lo, 0));
  }
}
}  // namespace nplm

extern "C" int nplm_segment_mean(const void* x, const int* cu, float* out, int B, int C, int drop_last,
                                 cudaStream_t st) {
  if (B <= 0) return 0;
  if ((C % 8) || (reinterpret_cast<uintptr_t>(x) & 15)) return -3;
  launch_chained(nplm::segment_mean_kernel, dim3(B, (C + 63) / 64), 256, 0, st, reinterpret_cast<const __nv_bfloat16*>(x),
      cu, out, C, drop_last);
  return static_cast<int>(cudaGetLastError());
}

// ------------------------------------------------------------------ padded batches
// What a padded [B][S] batch needs before its first layer: the kept positions, their ids, the position of each inside its
// sequence and the sequences' offsets. Three launches and one wait for the token count; composed of tensor operations it was
// fifteen launches with the GPU idle between them (0.25 ms before the first layer of 9 x 1001 positions). A mask
// may have holes: a token's position is its rank among the kept ones of its row, as the composition had it.
namespace nplm {
template <typename M>
__global__ void __launch_bounds__(256)
unpad_count_kernel(const M* __restrict__ mask, int S, int* __restrict__ counts) {
  grid_chain();
  __shared__ int part[8];
  const M* row = mask + static_cast<size_t>(blockIdx.x) * S;
  int n = 0;
  for (int s = threadIdx.x; s < S; s += 256) n += row[s] != 0;
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
    for (int i = 0; i < 8; ++i) total += part[i];
    counts[blockIdx.x] = total;
  }
}

// cu[0 .. B] = running sums of counts[0 .. B - 1], one block
__global__ void __launch_bounds__(1024)
running_sum_kernel(const int* __restrict__ counts, int B, int* __restrict__ cu) {
  grid_chain();
  __shared__ int warp_sum_[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int before = 0;
  if (threadIdx.x == 0) cu[0] = 0;
  for (int b0 = 0; b0 < B; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    int v = b < B ? counts[b] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    if (lane == 31) warp_sum_[warp] = v;
    __syncthreads();
    int add = before;
    for (int i = 0; i < warp; ++i) add += warp_sum_[i];
    if (b < B) cu[b + 1] = v + add;
    for (int i = 0; i < 32; ++i) before += warp_sum_[i];
    __syncthreads();
  }
}

template <typename M, typename I>
__global__ void __launch_bounds__(256)
unpad_fill_kernel(const M* __restrict__ mask, const I* __restrict__ ids, const int* __restrict__ cu, int S,
                  long long* __restrict__ index, I* __restrict__ flat, int* __restrict__ pos) {
  grid_chain();
  __shared__ int part[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t row = static_cast<size_t>(blockIdx.x) * S;
  const int first = cu[blockIdx.x];
  int before = 0;
  for (int s0 = 0; s0 < S; s0 += 256) {
    const int s = s0 + threadIdx.x;
    const bool keep = s < S && mask[row + s] != 0;
    const unsigned votes = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) part[warp] = __popc(votes);
    __syncthreads();
    int rank = before + __popc(votes & ((1u << lane) - 1u));
    for (int i = 0; i < 8; ++i) {
      if (i < warp) rank += part[i];
      before += part[i];
    }
    if (keep) {
      index[first + rank] = static_cast<long long>(row + s);
      flat[first + rank] = ids[row + s];
      pos[first + rank] = rank;
    }
    __syncthreads();
  }
}

template <typename M>
static int unpad_fill(const void* mask, const void* ids, int id_bytes, const int* cu, int B, int S, long long* index,
                      void* flat, int* pos, cudaStream_t st) {
  if (id_bytes == 8)
    launch_chained(unpad_fill_kernel<M, long long>, B, 256, 0, st, static_cast<const M*>(mask),
                   static_cast<const long long*>(ids), cu, S, index, static_cast<long long*>(flat), pos);
  else
    launch_chained(unpad_fill_kernel<M, int>, B, 256, 0, st, static_cast<const M*>(mask), static_cast<const int*>(ids), cu,
                   S, index, static_cast<int*>(flat), pos);
  return static_cast<int>(cudaGetLastError());
}
}  // namespace nplm

// mask [B][S] (mask_bytes 1, 4 or 8: bool / integers, kept where not zero); counts: int [B] scratch, cu: int [B + 1].
extern "C" int nplm_unpad_count(const void* mask, int mask_bytes, int B, int S, int* counts, int* cu, cudaStream_t st) {
  if (B <= 0 || S <= 0) return -3;
  if (mask_bytes == 1) launch_chained(unpad_count_kernel<signed char>, B, 256, 0, st,
      static_cast<const signed char*>(mask), S, counts);
  else if (mask_bytes == 4) launch_chained(unpad_count_kernel<int>, B, 256, 0, st, static_cast<const int*>(mask), S, counts);
  else if (mask_bytes == 8) launch_chained(unpad_count_kernel<long long>, B, 256, 0, st,
      static_cast<const long long*>(mask), S, counts);
  else return -3;
  launch_chained(running_sum_kernel, 1, 1024, 0, st, counts, B, cu);
  return static_cast<int>(cudaGetLastError());
}

// ids [B][S] (id_bytes 4 or 8) -> flat ids, int64 indices into B * S and int positions of the kept tokens.
extern "C" int nplm_unpad_fill(const void* mask, int mask_bytes, const void* ids, int id_bytes, const int* cu, int B, int S,
                               long long* index, void* flat, int* pos, cudaStream_t st) {
  if (B <= 0 || S <= 0 || (id_bytes != 4 && id_bytes != 8)) return -3;
  if (mask_bytes == 1) return nplm::unpad_fill<signed char>(mask, ids, id_bytes, cu, B, S, index, flat, pos, st);
  if (mask_bytes == 4) return nplm::unpad_fill<int>(mask, ids, id_bytes, cu, B, S, index, flat, pos, st);
  if (mask_bytes == 8) return nplm::unpad_fill<long long>(mask, ids, id_bytes, cu, B, S, index, flat, pos, st);
  return -3;
}

extern "C" int nplm_gather_rows(const void* src, const int* idx, void* dst, int n, int C,
                                cudaStream_t st) {
  if (n <= 0) return 0;
  if (C % 8) return -3;
  launch_when(static_cast<long long>(n) * C <= CHAIN_ELEMENTS, gather_rows_kernel,
      grid_for(static_cast<long long>(n) * (C / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(src), idx, reinterpret_cast<__nv_bfloat16*>(dst), n, C);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_scatter_rows(const void* src, const int* idx, void* dst, int n, int C,
                                 cudaStream_t st) {
  if (n <= 0) return 0;
  if (C % 8) return -3;
  launch_when(static_cast<long long>(n) * C <= CHAIN_ELEMENTS, scatter_rows_kernel,
      grid_for(static_cast<long long>(n) * (C / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(src), idx, reinterpret_cast<__nv_bfloat16*>(dst), n, C);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_ce_count(const int* labels, int n, float* inv, float* loss, cudaStream_t st) {
  if (n < 0) return -3;
  launch_chained(ce_count_kernel, 1, 1024, 0, st, labels, n, inv, loss);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_ce_fwd(const void* h, const void* W, const void* bias, const int* labels,
                           const float* inv_count, float* dlogits, float* logits, float* loss_sum,
                           int n, int C, int V, cudaStream_t st) {
  if (n <= 0) return 0;
  if (V > 32 || V < 1 || (C % 8)) return -3;
  const size_t smem = static_cast<size_t>(V) * C * 2;
  if (smem > 200 * 1024) return -4;
  int blocks = (n + CE_WARPS - 1) / CE_WARPS;
  if (blocks > 148 * 2) blocks = 148 * 2;
#define CALL(N_)                                                                                   \
  do {                                                                                             \
    cudaFuncSetAttribute(ce_fwd_kernel<N_>, cudaFuncAttributeMaxDynamicSharedMemorySize,           \
                         static_cast<int>(smem));                                                  \
    launch_chained(ce_fwd_kernel<N_>, blocks, CE_WARPS * 32, smem, st,                                         \
        reinterpret_cast<const __nv_bfloat16*>(h), reinterpret_cast<const __nv_bfloat16*>(W),      \
        reinterpret_cast<const __nv_bfloat16*>(bias), labels, inv_count, dlogits, logits, loss_sum, \
        n, C, V);                                                                                  \
  } while (0)
  NPLM_CHUNK_DISPATCH(C, CALL);
#undef CALL
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_ce_bwd(const void* h, const void* W, const float* dlogits, const float* gscale,
                           void* dh, float* dW, float* dbias, int n, int C, int V,
                           cudaStream_t st) {
  if (n <= 0) return 0;
  if (V > 32 || V < 1 || (C % 8)) return -3;
  if ((reinterpret_cast<uintptr_t>(h) & 3) || (reinterpret_cast<uintptr_t>(W) & 3) ||
      (reinterpret_cast<uintptr_t>(dh) & 3))
    return -3;
  // three blocks a multiprocessor, at least 16 rows each
  const int slices = (C + 255) / 256;
  int by = (148 * 3 + slices - 1) / slices;
  int rows = ((n + by - 1) / by + CE_ROWS - 1) / CE_ROWS * CE_ROWS;
  by = (n + rows - 1) / rows;
  launch_chained(ce_bwd_kernel, dim3(slices, by), 128, 0, st, reinterpret_cast<const __nv_bfloat16*>(h),
                 reinterpret_cast<const __nv_bfloat16*>(W), dlogits, gscale, reinterpret_cast<__nv_bfloat16*>(dh), dW,
                 dbias, n, C, V, rows);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_sumsq(const float* x, long long n, float* out, cudaStream_t st) {
  if (n <= 0) return 0;
  if (reinterpret_cast<uintptr_t>(x) & 15) return -3;
  launch_when(n <= CHAIN_ELEMENTS, sumsq_kernel, grid_for(n / 4 + 1, 256), 256, 0, st, x, n, out);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_adamw(float* p, float* m, float* v, float* g, void* p_bf16, const float* hyper,
                          const float* sumsq, long long n, int zero_grad, cudaStream_t st) {
  if (n <= 0) return 0;
  launch_when(n <= CHAIN_ELEMENTS, adamw_kernel, grid_for(n, 256), 256, 0, st, p, m, v, g,
      reinterpret_cast<__nv_bfloat16*>(p_bf16), hyper, sumsq, n, zero_grad);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_muon_momentum(const float* g, float* m, const long long* off, int n_mat, long long numel,
                                  void* upd, float* usq, const float* sumsq, float gs, float max_norm,
                                  float mu, int nesterov, cudaStream_t st) {
  if (n_mat <= 0 || numel <= 0) return 0;
  if (numel & 3) return -3;
  int bx = grid_for(numel / 4, 256);
  if (bx > 592) bx = 592;
  launch_when(n_mat * numel <= CHAIN_ELEMENTS, muon_momentum_kernel, dim3(bx, n_mat), 256, 0, st, g, m, off, numel,
      reinterpret_cast<__nv_bfloat16*>(upd), usq, sumsq, gs, max_norm, mu, nesterov);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_muon_apply(float* p, void* p16, const long long* off, int n_mat, long long numel,
                               const void* O, float lr, float wd, int cautious, cudaStream_t st) {
  if (n_mat <= 0 || numel <= 0) return 0;
  if (numel & 3) return -3;
  int bx = grid_for(numel / 4, 256);
  if (bx > 592) bx = 592;
  launch_when(n_mat * numel <= CHAIN_ELEMENTS, muon_apply_kernel, dim3(bx, n_mat), 256, 0, st, p,
      reinterpret_cast<__nv_bfloat16*>(p16), off, numel, reinterpret_cast<const __nv_bfloat16*>(O), lr, wd, cautious);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_adamw_slots(float* p, float* m, float* v, const float* g, void* p16, const long long* off,
                                const long long* numel, const int* decay, int n_slots, long long max_numel,
                                const float* sumsq, float gs, float max_norm, float lr, float b1, float b2,
                                float eps, float wd, float bc1, float bc2, cudaStream_t st) {
  if (n_slots <= 0 || max_numel <= 0) return 0;
  int bx = grid_for(max_numel, 256);
  if (bx > 64) bx = 64;
  launch_when(n_slots * max_numel <= CHAIN_ELEMENTS, adamw_slots_kernel, dim3(bx, n_slots), 256, 0, st, p, m, v, g,
      reinterpret_cast<__nv_bfloat16*>(p16), off, numel, decay, sumsq, gs, max_norm, lr, b1, b2, eps, wd, bc1, bc2);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_cast_f32_bf16(const float* src, void* dst, long long n, cudaStream_t st) {
  if (n <= 0) return 0;
  launch_when(n <= CHAIN_ELEMENTS, cast_f32_to_bf16_kernel, grid_for(n, 256), 256, 0, st, src,
      reinterpret_cast<__nv_bfloat16*>(dst), n);
  return static_cast<int>(cudaGetLastError());
}

// rows (may be null): row r of s is compared with row rows[r] of t
extern "C" int nplm_masked_mse(const void* s, const void* t, const int* valid, const long long* rows,
                               const float* inv_count, void* ds, float* loss_sum, int T, int C,
                               cudaStream_t st) {
  if (T <= 0) return 0;
  if (C % 8) return -3;
  launch_when(static_cast<long long>(T) * C <= CHAIN_ELEMENTS, masked_mse_kernel,
      grid_for(static_cast<long long>(T) * (C / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(s), reinterpret_cast<const __nv_bfloat16*>(t), valid,
      rows, inv_count, reinterpret_cast<__nv_bfloat16*>(ds), loss_sum, T, C);
  return static_cast<int>(cudaGetLastError());
}
