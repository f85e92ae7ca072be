// Kernels for the optional encoder blocks: varlen depthwise convolution and hyper-connection
// (mHC) stream mixing. The reference has neither; semantics are defined here.
//
// Varlen depthwise conv (kernel size KS, odd, "same" centring): for packed tokens x[T][C],
//   y[t][c] = bias[c] + sum_{k} w[c][k] * x[t + k - KS/2][c]   over taps that stay inside the
// sequence of token t (seq_start[t] <= t + k - KS/2 < seq_end[t]); taps that would cross a
// sequence boundary contribute zero.
//   dx[t][c] = sum_k w[c][k] * dy[t - (k - KS/2)][c]            (same boundary rule, flipped taps)
//   dw[c][k] = sum_t dy[t][c] * x[t + k - KS/2][c],  dbias[c] = sum_t dy[t][c]
//
// mHC mixing on streams X[T][n][C] with per-token coefficients:
//   read : h[t][:]     = sum_i alpha[t][i] * X[t][i][:]
//   write: Xn[t][i][:] = sum_j R[t][i][j] * X[t][j][:] + beta[t][i] * y[t][:]
// plus the backward of both (gradients w.r.t. X, y and the coefficients).
#include "common.cuh"

namespace nplm {

__device__ __forceinline__ void ld8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 t = unpack_bf16x2(w[e]);
    f[2 * e] = t.x;
    f[2 * e + 1] = t.y;
  }
}

__device__ __forceinline__ void unpack8x(const uint4& u, float (&f)[8]) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 t = unpack_bf16x2(w[e]);
    f[2 * e] = t.x;
    f[2 * e + 1] = t.y;
  }
}

__device__ __forceinline__ void st8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  uint32_t* w = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) w[e] = pack_bf16x2(f[2 * e], f[2 * e + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

constexpr int MAX_KS = 9;

// flip = 0: forward (tap k reads t + k - r);  flip = 1: input gradient (tap k reads t - (k - r))
// skip: y = x + the convolution rounded to bf16 (forward of the residual block, and its input gradient with x the output's)
__global__ void __launch_bounds__(256)
dwconv_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
              const __nv_bfloat16* __restrict__ bias, const int* __restrict__ s_start,
              const int* __restrict__ s_end, __nv_bfloat16* __restrict__ y, int T, int C, int KS, int flip, int skip) {
  grid_chain();
  const int vec = C >> 3;
  const int r = KS >> 1;
  const long long total = static_cast<long long>(T) * vec;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(idx / vec);
    const int c = static_cast<int>(idx % vec) * 8;
    const int a = s_start[t], b = s_end[t];
    float acc[8];
    if (bias != nullptr && !flip) {
      ld8(bias + c, acc);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    }
    for (int k = 0; k < KS; ++k) {
      const int src = flip ? t - (k - r) : t + (k - r);
      if (src < a || src >= b) continue;
      float xv[8];
      ld8(x + static_cast<size_t>(src) * C + c, xv);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += xv[e] * __bfloat162float(w[(c + e) * KS + k]);
    }
    if (skip) {
      float xv[8];
      ld8(x + static_cast<size_t>(t) * C + c, xv);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = xv[e] + __bfloat162float(__float2bfloat16_rn(acc[e]));
    }
    st8(y + static_cast<size_t>(t) * C + c, acc);
  }
}

// Kernel size known at compile time: a warp owns 128 channels (a lane four: one 256-byte request a row) of a run of
// consecutive tokens and slides over them, the KS rows around a token and the weights in registers, four rows loaded
// ahead (eight: 17.5 us, fewer warps fit). Every row is read once but for KS - 1 at the ends of a run; tokens whose whole
// window lies inside their sequence (all but KS - 1 of it) take no masks. 17 024 x 768, 7 taps: 24.8 -> 16.4 us; 55 424 x
// 1024 110 -> 83 (2.7 TB/s: bound by the latency of the rows, 16 warps a multiprocessor). The form before, eight channels x
// eight tokens a thread, read 14 rows for eight and ran one block of 243 registers a multiprocessor.
constexpr int DW_CH = 4, DW_AHEAD = 4;

__device__ __forceinline__ void ld4(const __nv_bfloat16* p, float2 (&f)[2]) {
  const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
  f[0] = unpack_bf16x2(u.x);
  f[1] = unpack_bf16x2(u.y);
}

// rows[j] = x[t - R + j] of this lane's channels for j in [from, KS - 1 + DW_AHEAD), zero outside the tensor
template <int KS, int FROM>
__device__ __forceinline__ void dw_load(const __nv_bfloat16* __restrict__ x, int t, int T, int C, int c,
                                        float2 (&rows)[KS - 1 + DW_AHEAD][2]) {
#pragma unroll
  for (int j = FROM; j < KS - 1 + DW_AHEAD; ++j) {
    const int src = t - KS / 2 + j;
    if (src >= 0 && src < T) ld4(x + static_cast<size_t>(src) * C + c, rows[j]);
    else rows[j][0] = rows[j][1] = make_float2(0.f, 0.f);
  }
}

template <int KS>
__global__ void __launch_bounds__(256, 2)
dwconv_run_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                  const __nv_bfloat16* __restrict__ bias, const int* __restrict__ s_start,
                  const int* __restrict__ s_end, __nv_bfloat16* __restrict__ y, int T, int C, int flip, int skip, int run) {
  grid_chain();
  constexpr int R = KS / 2;
  const int lane = threadIdx.x & 31;
  const int c = (blockIdx.y * 32 + lane) * DW_CH;
  const bool on = c < C;
  const int cc = on ? c : 0;          // (every lane takes part in the shuffles below)
  const int t0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * run, t1 = min(T, t0 + run);
  if (t0 >= t1) return;
  float2 wt[KS][2], b4[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int k = 0; k < KS; ++k) {
    const __nv_bfloat16* p = w + static_cast<size_t>(cc) * KS + (flip ? KS - 1 - k : k);
    wt[k][0] = make_float2(__bfloat162float(p[0]), __bfloat162float(p[KS]));
    wt[k][1] = make_float2(__bfloat162float(p[2 * KS]), __bfloat162float(p[3 * KS]));
  }
  if (bias != nullptr && !flip) {
    b4[0] = make_float2(__bfloat162float(bias[cc]), __bfloat162float(bias[cc + 1]));
    b4[1] = make_float2(__bfloat162float(bias[cc + 2]), __bfloat162float(bias[cc + 3]));
  }
  float2 rows[KS - 1 + DW_AHEAD][2];
  dw_load<KS, 0>(x, t0, T, C, cc, rows);
  for (int t = t0; t < t1; t += DW_AHEAD) {
    int lo = 0, hi = 0;
    if (lane < DW_AHEAD && t + lane < t1) {
      lo = s_start[t + lane];
      hi = s_end[t + lane];
    }
#pragma unroll
    for (int i = 0; i < DW_AHEAD; ++i) {
      const int a = __shfl_sync(0xffffffffu, lo, i), b = __shfl_sync(0xffffffffu, hi, i);
      if (t + i < t1) {
        float2 acc[2] = {b4[0], b4[1]};
        if (t + i - R >= a && t + i + R < b) {
#pragma unroll
          for (int k = 0; k < KS; ++k)
#pragma unroll
            for (int e = 0; e < 2; ++e) acc[e] = fma2(rows[i + k][e], wt[k][e], acc[e]);
        } else {
#pragma unroll
          for (int k = 0; k < KS; ++k) {
            const int src = t + i + k - R;
            if (src >= a && src < b) {
#pragma unroll
              for (int e = 0; e < 2; ++e) acc[e] = fma2(rows[i + k][e], wt[k][e], acc[e]);
            }
          }
        }
        uint2 out = make_uint2(pack_bf16x2(acc[0].x, acc[0].y), pack_bf16x2(acc[1].x, acc[1].y));
        if (skip) {     // (the row itself is the middle tap's)
          const float2 o0 = add2(unpack_bf16x2(out.x), rows[i + R][0]), o1 = add2(unpack_bf16x2(out.y), rows[i + R][1]);
          out = make_uint2(pack_bf16x2(o0.x, o0.y), pack_bf16x2(o1.x, o1.y));
        }
        if (on) *reinterpret_cast<uint2*>(y + static_cast<size_t>(t + i) * C + c) = out;
      }
    }
    if (t + DW_AHEAD < t1) {
#pragma unroll
      for (int j = 0; j < KS - 1; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) rows[j][e] = rows[j + DW_AHEAD][e];
      dw_load<KS, KS - 1>(x, t + DW_AHEAD, T, C, cc, rows);
    }
  }
}

// dw[c][k] += sum_t dy[t][c] x[t+k-r][c];  dbias[c] += sum_t dy[t][c]. One block handles a slab of
// tokens for 32 channels x 8 token lanes and reduces through shared memory before the atomics.
__global__ void __launch_bounds__(256)
dwconv_bwd_w_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                    const int* __restrict__ s_start, const int* __restrict__ s_end,
                    float* __restrict__ dw, float* __restrict__ dbias, int T, int C, int KS,
                    int tokens_per_block) {
  grid_chain();
  __shared__ float red[8][32][MAX_KS + 1];
  const int cl = threadIdx.x & 31;       // channel lane
  const int tl = threadIdx.x >> 5;       // token lane
  const int c = blockIdx.y * 32 + cl;
  const int r = KS >> 1;
  float acc[MAX_KS + 1];
#pragma unroll
  for (int k = 0; k <= MAX_KS; ++k) acc[k] = 0.f;
  const int t0 = blockIdx.x * tokens_per_block;
  const int t1 = min(T, t0 + tokens_per_block);
  if (c < C) {
    for (int t = t0 + tl; t < t1; t += 8) {
      const float g = __bfloat162float(dy[static_cast<size_t>(t) * C + c]);
      const int a = s_start[t], b = s_end[t];
      acc[MAX_KS] += g;
#pragma unroll
      for (int k = 0; k < MAX_KS; ++k) {
        if (k < KS) {
          const int src = t + k - r;
          if (src >= a && src < b) acc[k] += g * __bfloat162float(x[static_cast<size_t>(src) * C + c]);
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k <= MAX_KS; ++k) red[tl][cl][k] = acc[k];
  __syncthreads();
  if (tl == 0 && c < C) {
    for (int k = 0; k <= MAX_KS; ++k) {
      float s = 0.f;
      for (int j = 0; j < 8; ++j) s += red[j][cl][k];
      if (k < KS) atomicAdd(&dw[c * KS + k], s);
      else if (k == MAX_KS && dbias != nullptr) atomicAdd(&dbias[c], s);
    }
  }
}

// Weight gradient with the kernel size known at compile time: warps slide over runs of tokens as above, with the 4 x (KS +
// 1) sums of a lane's channels in registers; the eight warps of a block meet in shared memory. 17 024 x 768, 7 taps: 51 ->
// 18.6 us, 55 424 x 1024 220 -> 91; with one channel a lane a warp's requests were 64 bytes and its loads waited for one another.
template <int KS>
__global__ void __launch_bounds__(256, 2)
dwconv_bwd_w_run_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                        const int* __restrict__ s_start, const int* __restrict__ s_end,
                        float* __restrict__ dw, float* __restrict__ dbias, int T, int C, int run) {
  grid_chain();
  constexpr int R = KS / 2;
  __shared__ float4 red[8][KS + 1][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = (blockIdx.y * 32 + lane) * DW_CH;
  const int cc = c < C ? c : 0;
  const int t0 = (blockIdx.x * 8 + warp) * run, t1 = min(T, t0 + run);
  float2 acc[KS + 1][2];
#pragma unroll
  for (int k = 0; k <= KS; ++k) acc[k][0] = acc[k][1] = make_float2(0.f, 0.f);
  if (t0 < t1) {
    float2 rows[KS - 1 + DW_AHEAD][2];
    dw_load<KS, 0>(x, t0, T, C, cc, rows);
    for (int t = t0; t < t1; t += DW_AHEAD) {
      uint2 g[DW_AHEAD];
#pragma unroll
      for (int i = 0; i < DW_AHEAD; ++i)
        g[i] = t + i < t1 ? __ldg(reinterpret_cast<const uint2*>(dy + static_cast<size_t>(t + i) * C + cc))
                          : make_uint2(0u, 0u);
      int lo = 0, hi = 0;
      if (lane < DW_AHEAD && t + lane < t1) {
        lo = s_start[t + lane];
        hi = s_end[t + lane];
      }
#pragma unroll
      for (int i = 0; i < DW_AHEAD; ++i) {
        const int a = __shfl_sync(0xffffffffu, lo, i), b = __shfl_sync(0xffffffffu, hi, i);
        const float2 gv[2] = {unpack_bf16x2(g[i].x), unpack_bf16x2(g[i].y)};
        if (t + i < t1) {
#pragma unroll
          for (int e = 0; e < 2; ++e) acc[KS][e] = add2(acc[KS][e], gv[e]);
          if (t + i - R >= a && t + i + R < b) {
#pragma unroll
            for (int k = 0; k < KS; ++k)
#pragma unroll
              for (int e = 0; e < 2; ++e) acc[k][e] = fma2(gv[e], rows[i + k][e], acc[k][e]);
          } else {
#pragma unroll
            for (int k = 0; k < KS; ++k) {
              const int src = t + i + k - R;
              if (src >= a && src < b) {
#pragma unroll
                for (int e = 0; e < 2; ++e) acc[k][e] = fma2(gv[e], rows[i + k][e], acc[k][e]);
              }
            }
          }
        }
      }
      if (t + DW_AHEAD < t1) {
#pragma unroll
        for (int j = 0; j < KS - 1; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) rows[j][e] = rows[j + DW_AHEAD][e];
        dw_load<KS, KS - 1>(x, t + DW_AHEAD, T, C, cc, rows);
      }
    }
  }
#pragma unroll
  for (int k = 0; k <= KS; ++k) red[warp][k][lane] = make_float4(acc[k][0].x, acc[k][0].y, acc[k][1].x, acc[k][1].y);
  __syncthreads();
  for (int i = threadIdx.x; i < (KS + 1) * 32 * DW_CH; i += 256) {
    const int k = i / (32 * DW_CH), ch = blockIdx.y * 32 * DW_CH + i % (32 * DW_CH);
    if (ch >= C) continue;
    const float* p = reinterpret_cast<const float*>(&red[0][k][0]) + i % (32 * DW_CH);
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += p[j * (KS + 1) * 32 * DW_CH];
    if (k < KS) atomicAdd(&dw[ch * KS + k], sum);
    else if (dbias != nullptr) atomicAdd(&dbias[ch], sum);
  }
}

// Tokens a warp walks: as many as leave the two blocks of eight warps that a multiprocessor holds (more blocks wait for a
// second round: 17 024 x 768 22 us with three), in whole batches of rows loaded ahead, 16 at least (a run reads KS - 1
// rows more than it has) and 256 at most.
static int dw_run(int T, int C) {
  const long long groups = (C + 127) / 128;
  long long run = (T * groups + 148 * 2 * 8 - 1) / (148 * 2 * 8);
  run = (run + DW_AHEAD - 1) / DW_AHEAD * DW_AHEAD;
  return static_cast<int>(run < 16 ? 16 : (run > 256 ? 256 : run));
}

// ---------------------------------------------------------------------------- mHC
constexpr int MAX_STREAMS = 8;

// h[t][:] = sum_i alpha[t][i] X[t][i][:]
__global__ void __launch_bounds__(256)
mhc_read_kernel(const __nv_bfloat16* __restrict__ X, const float* __restrict__ alpha,
                __nv_bfloat16* __restrict__ h, int T, int n, int C) {
  grid_chain();
  const int vec = C >> 3;
  const long long total = static_cast<long long>(T) * vec;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(idx / vec);
    const int c = static_cast<int>(idx % vec) * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < n; ++i) {
      float xv[8];
      ld8(X + (static_cast<size_t>(t) * n + i) * C + c, xv);
      const float a = alpha[t * n + i];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += a * xv[e];
    }
    st8(h + static_cast<size_t>(t) * C + c, acc);
  }
}

// Xn[t][i][:] = sum_j R[t][i][j] X[t][j][:] + beta[t][i] y[t][:]
// N = number of streams (compile-time, so every per-stream array stays in registers).
// MEAN: also z[t][:] = (1/N) sum_i Xn[t][i][:] of the rounded streams, which mhc_mean_kernel would read them back for
// (17 024 x 4 x 768: 50 us, 71 in two passes).
template <int N, bool MEAN>
__global__ void __launch_bounds__(256)
mhc_write_kernel(const __nv_bfloat16* __restrict__ X, const __nv_bfloat16* __restrict__ y,
                 const float* __restrict__ R, const float* __restrict__ beta,
                 __nv_bfloat16* __restrict__ Xn, __nv_bfloat16* __restrict__ z, int T, int C) {
  grid_chain();
  const int vec = C >> 3;
  const long long total = static_cast<long long>(T) * vec;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(idx / vec);
    const int c = static_cast<int>(idx % vec) * 8;
    uint4 xr[N];
#pragma unroll
    for (int j = 0; j < N; ++j)
      xr[j] = __ldg(reinterpret_cast<const uint4*>(X + (static_cast<size_t>(t) * N + j) * C + c));
    float yv[8];
    ld8(y + static_cast<size_t>(t) * C + c, yv);
    float acc[N][8];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float bt = beta[t * N + i];
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[i][e] = bt * yv[e];
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
      float xv[8];
      unpack8x(xr[j], xv);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float rr = R[(t * N + i) * N + j];
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[i][e] += rr * xv[e];
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) st8(Xn + (static_cast<size_t>(t) * N + i) * C + c, acc[i]);
    if constexpr (MEAN) {
      float m[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) m[e] += __bfloat162float(__float2bfloat16_rn(acc[i][e]));
#pragma unroll
      for (int e = 0; e < 8; ++e) m[e] *= 1.f / static_cast<float>(N);
      st8(z + static_cast<size_t>(t) * C + c, m);
    }
  }
}

// Sum of V <= 32 per-lane values over the warp: lane l (l < 32) returns the total of value l.
// Five exchange rounds that halve the number of live values (31 shuffles instead of 5 per value).
template <int V>
__device__ __forceinline__ float warp_transpose_sum(float (&v)[32], int lane) {
#pragma unroll
  for (int i = V; i < 32; ++i) v[i] = 0.f;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < off; ++i) {
      const float keep = upper ? v[i + off] : v[i];
      const float send = upper ? v[i] : v[i + off];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return v[0];
}

// Backward of read and / or write, one warp per token (dXn == null: read part only, dh == null:
// write part only; outputs of the missing part are not touched):
//   given dXn[t][i][:] (gradient of the written streams) and dh[t][:] (gradient of the read),
//   dX[t][j][:]  = sum_i R[t][i][j] dXn[t][i][:] + alpha[t][j] dh[t][:]
//   dy[t][:]     = sum_i beta[t][i] dXn[t][i][:]
//   dR[t][i][j]  = <dXn[t][i], X[t][j]>,  dbeta[t][i] = <dXn[t][i], y[t]>,  dalpha[t][j] = <dh[t], X[t][j]>
// All loads of a 256-channel slice are issued before the first use and kept packed in registers.
// JOIN (with WRITE alone): the written streams are the ones of the next site, whose gradient mhc_dx_combine_kernel forms from
// dXn (here the next site's own write), its alpha and dh and the gradient dz of its stream mean; formed here, with the same
// bits, it is neither written nor read back (17 024 x 4 x 768: 77 us, 112 in two passes).
// WRITE / READ: which parts there are. As run-time flags the read part alone (what a training step asks for beside the
// write part) carried the write part's N x N sums along, on zeros: 17 024 x 4 x 768 53 -> 27 us, the write part alone 70 -> 61.
template <int N, bool WRITE, bool READ, bool JOIN = false>
__global__ void __launch_bounds__(256, 2)
mhc_bwd_kernel(const __nv_bfloat16* __restrict__ X, const __nv_bfloat16* __restrict__ y,
               const float* __restrict__ R, const float* __restrict__ alpha, const float* __restrict__ beta,
               const __nv_bfloat16* __restrict__ dXn, const __nv_bfloat16* __restrict__ dh,
               const __nv_bfloat16* __restrict__ dz, __nv_bfloat16* __restrict__ dX, __nv_bfloat16* __restrict__ dy,
               float* __restrict__ dR, float* __restrict__ dalpha, float* __restrict__ dbeta, int T, int C) {
  grid_chain();
  static_assert(!JOIN || (WRITE && !READ), "the joined form is the write part's");
  static_assert(N * N + 2 * N <= 32, "too many streams for the warp-transpose reduction");
  const int lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5;
  constexpr bool has_w = WRITE, has_r = READ;
  for (int t = blockIdx.x * warps + (threadIdx.x >> 5); t < T; t += gridDim.x * warps) {
    // sums[i * N + j] = dR[i][j], sums[N*N + i] = dbeta[i], sums[N*N + N + j] = dalpha[j]
    float sums[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) sums[i] = 0.f;
    float rc[N][N], bt[N], al[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      bt[i] = has_w ? beta[t * N + i] : 0.f;
      al[i] = has_r || JOIN ? alpha[t * N + i] : 0.f;
#pragma unroll
      for (int j = 0; j < N; ++j) rc[i][j] = has_w ? R[(t * N + i) * N + j] : 0.f;
    }
#pragma unroll 1
    for (int c = lane * 8; c < C; c += 256) {
      uint4 xr[N], gr[N], yr = make_uint4(0u, 0u, 0u, 0u), hr = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int j = 0; j < N; ++j) {
        xr[j] = __ldg(reinterpret_cast<const uint4*>(X + (static_cast<size_t>(t) * N + j) * C + c));
        gr[j] = has_w ? __ldg(reinterpret_cast<const uint4*>(dXn + (static_cast<size_t>(t) * N + j) * C + c))
                      : make_uint4(0u, 0u, 0u, 0u);
      }
      if (has_w) yr = __ldg(reinterpret_cast<const uint4*>(y + static_cast<size_t>(t) * C + c));
      if (has_r || JOIN) hr = __ldg(reinterpret_cast<const uint4*>(dh + static_cast<size_t>(t) * C + c));
      float yv[8], hv[8];
      if constexpr (JOIN) {
        float zv[8];
        unpack8x(__ldg(reinterpret_cast<const uint4*>(dz + static_cast<size_t>(t) * C + c)), zv);
        unpack8x(hr, hv);
#pragma unroll
        for (int e = 0; e < 8; ++e) zv[e] *= 1.f / static_cast<float>(N);
#pragma unroll
        for (int i = 0; i < N; ++i) {
          float gv[8];
          unpack8x(gr[i], gv);
#pragma unroll
          for (int e = 0; e < 8; ++e) gv[e] += fmaf(al[i], hv[e], zv[e]);
          gr[i] = make_uint4(pack_bf16x2(gv[0], gv[1]), pack_bf16x2(gv[2], gv[3]), pack_bf16x2(gv[4], gv[5]),
                             pack_bf16x2(gv[6], gv[7]));
        }
      }
      unpack8x(yr, yv);
      unpack8x(hr, hv);
      float dyv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      float o[N][8];
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int e = 0; e < 8; ++e) o[j][e] = has_r ? al[j] * hv[e] : 0.f;
#pragma unroll
      for (int j = 0; j < N; ++j) {
        float xv[8];
        unpack8x(xr[j], xv);
        if constexpr (has_r) {
#pragma unroll
          for (int e = 0; e < 8; ++e) sums[N * N + N + j] += hv[e] * xv[e];
        }
#pragma unroll
        for (int i = 0; i < (has_w ? N : 0); ++i) {
          float gv[8];
          unpack8x(gr[i], gv);
#pragma unroll
          for (int e = 0; e < 8; ++e) sums[i * N + j] += gv[e] * xv[e];
        }
      }
#pragma unroll
      for (int i = 0; i < (has_w ? N : 0); ++i) {
        float gv[8];
        unpack8x(gr[i], gv);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          dyv[e] += bt[i] * gv[e];
          sums[N * N + i] += gv[e] * yv[e];
        }
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
          for (int e = 0; e < 8; ++e) o[j][e] += rc[i][j] * gv[e];
      }
      if (has_w) st8(dy + static_cast<size_t>(t) * C + c, dyv);
      if (dX != nullptr) {
#pragma unroll
        for (int j = 0; j < N; ++j) st8(dX + (static_cast<size_t>(t) * N + j) * C + c, o[j]);
      }
    }
    // every lane takes part in the reduction; lane l ends up with the total of sums[l]
    const float total = warp_transpose_sum<N * N + 2 * N>(sums, lane);
    if (lane < N * N) {
      if (has_w) dR[t * N * N + lane] = total;
    } else if (lane < N * N + N) {
      if (has_w) dbeta[t * N + (lane - N * N)] = total;
    } else if (lane < N * N + 2 * N) {
      if (has_r) dalpha[t * N + (lane - N * N - N)] = total;
    }
  }
}

// z[t][:] = (1/n) sum_i X[t][i][:]   (what the coefficient network of a site sees)
__global__ void __launch_bounds__(256)
mhc_mean_kernel(const __nv_bfloat16* __restrict__ X, __nv_bfloat16* __restrict__ z, int T, int n, int C) {
  grid_chain();
  const int vec = C >> 3;
  const long long total = static_cast<long long>(T) * vec;
  const float inv = 1.f / static_cast<float>(n);
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(idx / vec);
    const int c = static_cast<int>(idx % vec) * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < n; ++i) {
      float xv[8];
      ld8(X + (static_cast<size_t>(t) * n + i) * C + c, xv);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += xv[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] *= inv;
    st8(z + static_cast<size_t>(t) * C + c, acc);
  }
}

// Gradient of the streams entering a site, all three consumers in one pass:
//   dX[t][j][:] = g[t][j][:] (from the write, may be null) + alpha[t][j] dh[t][:] (read, may be null)
//                 + dz[t][:] / n (stream mean, may be null)
__global__ void __launch_bounds__(256)
mhc_dx_combine_kernel(const __nv_bfloat16* __restrict__ g, const float* __restrict__ alpha,
                      const __nv_bfloat16* __restrict__ dh, const __nv_bfloat16* __restrict__ dz,
                      __nv_bfloat16* __restrict__ dX, int T, int n, int C) {
  grid_chain();
  const int vec = C >> 3;
  const long long total = static_cast<long long>(T) * vec;
  const float inv = 1.f / static_cast<float>(n);
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(idx / vec);
    const int c = static_cast<int>(idx % vec) * 8;
    float hv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, zv[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (dh != nullptr) ld8(dh + static_cast<size_t>(t) * C + c, hv);
    if (dz != nullptr) {
      ld8(dz + static_cast<size_t>(t) * C + c, zv);
#pragma unroll
      for (int e = 0; e < 8; ++e) zv[e] *= inv;
    }
    for (int j = 0; j < n; ++j) {
      float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (g != nullptr) ld8(g + (static_cast<size_t>(t) * n + j) * C + c, o);
      const float a = (dh != nullptr) ? alpha[t * n + j] : 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] += a * hv[e] + zv[e];
      st8(dX + (static_cast<size_t>(t) * n + j) * C + c, o);
    }
  }
}

static int grid_for(long long work, int threads) {
  long long b = (work + threads - 1) / threads;
  if (b > 148LL * 16) b = 148LL * 16;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace nplm

using namespace nplm;

extern "C" int nplm_dwconv(const void* x, const void* w, const void* bias, const int* s_start,
                           const int* s_end, void* y, int T, int C, int KS, int flip, int skip, cudaStream_t st) {
  if (T <= 0) return 0;
  if ((C % 8) || KS < 1 || KS > MAX_KS || !(KS & 1)) return -3;
  if ((KS == 3 || KS == 5 || KS == 7 || KS == 9) &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 7) == 0) {
    const int run = dw_run(T, C);
    const dim3 grid((T + 8 * run - 1) / (8 * run), (C + 127) / 128);
#define NPLM_DWCONV(KS_)                                                                                   \
  launch_chained(dwconv_run_kernel<KS_>, grid, 256, 0, st, reinterpret_cast<const __nv_bfloat16*>(x),      \
                 reinterpret_cast<const __nv_bfloat16*>(w), reinterpret_cast<const __nv_bfloat16*>(bias),   \
                 s_start, s_end, reinterpret_cast<__nv_bfloat16*>(y), T, C, flip, skip, run)
    switch (KS) {
      case 3: NPLM_DWCONV(3); break;
      case 5: NPLM_DWCONV(5); break;
      case 7: NPLM_DWCONV(7); break;
      default: NPLM_DWCONV(9); break;
    }
#undef NPLM_DWCONV
    return static_cast<int>(cudaGetLastError());
  }
  launch_when(static_cast<long long>(T) * C <= CHAIN_ELEMENTS, dwconv_kernel,
      grid_for(static_cast<long long>(T) * (C / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(w),
      reinterpret_cast<const __nv_bfloat16*>(bias), s_start, s_end, reinterpret_cast<__nv_bfloat16*>(y), T, C,
      KS, flip, skip);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_dwconv_bwd_w(const void* x, const void* dy, const int* s_start, const int* s_end,
                                 float* dw, float* dbias, int T, int C, int KS, cudaStream_t st) {
  if (T <= 0) return 0;
  if (KS < 1 || KS > MAX_KS || !(KS & 1)) return -3;
  if ((KS == 3 || KS == 5 || KS == 7 || KS == 9) && C % DW_CH == 0 &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy)) & 7) == 0) {
    const int run = dw_run(T, C);
    const dim3 grid((T + 8 * run - 1) / (8 * run), (C + 127) / 128);
#define NPLM_DWCONV_W(KS_)                                                                                   \
  launch_chained(dwconv_bwd_w_run_kernel<KS_>, grid, 256, 0, st, reinterpret_cast<const __nv_bfloat16*>(x),  \
                 reinterpret_cast<const __nv_bfloat16*>(dy), s_start, s_end, dw, dbias, T, C, run)
    switch (KS) {
      case 3: NPLM_DWCONV_W(3); break;
      case 5: NPLM_DWCONV_W(5); break;
      case 7: NPLM_DWCONV_W(7); break;
      default: NPLM_DWCONV_W(9); break;
    }
#undef NPLM_DWCONV_W
    return static_cast<int>(cudaGetLastError());
  }
  const int tokens_per_block = 512;
  const dim3 grid((T + tokens_per_block - 1) / tokens_per_block, (C + 31) / 32);
  launch_chained(dwconv_bwd_w_kernel, grid, 256, 0, st, reinterpret_cast<const __nv_bfloat16*>(x),
      reinterpret_cast<const __nv_bfloat16*>(dy), s_start, s_end, dw, dbias, T, C, KS, tokens_per_block);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_mhc_read(const void* X, const float* alpha, void* h, int T, int n, int C, cudaStream_t st) {
  if (T <= 0) return 0;
  if ((C % 8) || n < 1 || n > MAX_STREAMS) return -3;
  launch_when(static_cast<long long>(T) * n * C <= CHAIN_ELEMENTS, mhc_read_kernel,
      grid_for(static_cast<long long>(T) * (C / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(X), alpha, reinterpret_cast<__nv_bfloat16*>(h), T, n, C);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_mhc_mean(const void* X, void* z, int T, int n, int C, cudaStream_t st) {
  if (T <= 0) return 0;
  if ((C % 8) || n < 1 || n > MAX_STREAMS) return -3;
  launch_when(static_cast<long long>(T) * n * C <= CHAIN_ELEMENTS, mhc_mean_kernel,
      grid_for(static_cast<long long>(T) * (C / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(X), reinterpret_cast<__nv_bfloat16*>(z), T, n, C);
  return static_cast<int>(cudaGetLastError());
}

extern "C" int nplm_mhc_dx_combine(const void* g, const float* alpha, const void* dh, const void* dz, void* dX,
                                   int T, int n, int C, cudaStream_t st) {
  if (T <= 0) return 0;
  if ((C % 8) || n < 1 || n > MAX_STREAMS || (dh != nullptr && alpha == nullptr)) return -3;
  launch_when(static_cast<long long>(T) * n * C <= CHAIN_ELEMENTS, mhc_dx_combine_kernel,
      grid_for(static_cast<long long>(T) * (C / 8), 256), 256, 0, st,
      reinterpret_cast<const __nv_bfloat16*>(g), alpha, reinterpret_cast<const __nv_bfloat16*>(dh),
      reinterpret_cast<const __nv_bfloat16*>(dz), reinterpret_cast<__nv_bfloat16*>(dX), T, n, C);
  return static_cast<int>(cudaGetLastError());
}

// z (bf16 [T][C], may be null): the stream mean of what is written.
extern "C" int nplm_mhc_write(const void* X, const void* y, const float* R, const float* beta, void* Xn, void* z,
                              int T, int n, int C, cudaStream_t st) {
  if (T <= 0) return 0;
  if ((C % 8) || n < 1 || n > 4) return -3;
  const int grid = grid_for(static_cast<long long>(T) * (C / 8), 256);
#define NPLM_MHC_WRITE(N_)                                                                              \
  launch_when(static_cast<long long>(T) * n * C <= CHAIN_ELEMENTS,                                              \
              z != nullptr ? mhc_write_kernel<N_, true> : mhc_write_kernel<N_, false>, grid, 256, 0, st,        \
              reinterpret_cast<const __nv_bfloat16*>(X), reinterpret_cast<const __nv_bfloat16*>(y), R, beta,    \
              reinterpret_cast<__nv_bfloat16*>(Xn), reinterpret_cast<__nv_bfloat16*>(z), T, C)
  switch (n) {
    case 1: NPLM_MHC_WRITE(1); break;
    case 2: NPLM_MHC_WRITE(2); break;
    case 3: NPLM_MHC_WRITE(3); break;
    default: NPLM_MHC_WRITE(4); break;
  }
#undef NPLM_MHC_WRITE
  return static_cast<int>(cudaGetLastError());
}

// With dz (and dXn, alpha, dh) the joined form: dXn, alpha, dh and dz are the parts of the next site's gradient.
extern "C" int nplm_mhc_bwd(const void* X, const void* y, const float* R, const float* alpha,
                            const float* beta, const void* dXn, const void* dh, const void* dz, void* dX, void* dy,
                            float* dR, float* dalpha, float* dbeta, int T, int n, int C, cudaStream_t st) {
  if (T <= 0) return 0;
  if ((C % 8) || n < 1 || n > 4) return -3;
  if (dz != nullptr && (dXn == nullptr || dh == nullptr || alpha == nullptr)) return -3;
  if (dXn == nullptr && dh == nullptr) return 0;
  int blocks = (T + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const auto go = [&](auto kern) {
    launch_when(static_cast<long long>(T) * n * C <= CHAIN_ELEMENTS, kern, blocks, 256, 0, st,
                reinterpret_cast<const __nv_bfloat16*>(X), reinterpret_cast<const __nv_bfloat16*>(y), R, alpha, beta,
                reinterpret_cast<const __nv_bfloat16*>(dXn), reinterpret_cast<const __nv_bfloat16*>(dh),
                reinterpret_cast<const __nv_bfloat16*>(dz), reinterpret_cast<__nv_bfloat16*>(dX),
                reinterpret_cast<__nv_bfloat16*>(dy), dR, dalpha, dbeta, T, C);
  };
#define NPLM_MHC_BWD(N_)                                         \
  dz != nullptr    ? go(mhc_bwd_kernel<N_, true, false, true>)   \
  : dXn == nullptr ? go(mhc_bwd_kernel<N_, false, true>)         \
  : dh != nullptr  ? go(mhc_bwd_kernel<N_, true, true>)          \
                   : go(mhc_bwd_kernel<N_, true, false>)
  switch (n) {
    case 1: NPLM_MHC_BWD(1); break;
    case 2: NPLM_MHC_BWD(2); break;
    case 3: NPLM_MHC_BWD(3); break;
    default: NPLM_MHC_BWD(4); break;
  }
#undef NPLM_MHC_BWD
  return static_cast<int>(cudaGetLastError());
}

// ---------------------------------------------------------------------------- device-side MLM masking
// Counter-based (Philox4x32-10) masking of packed token ids, the semantics of the host collator
// (src/nanoplm/pretraining/collator.py:333-382): a position is selected with probability p_sel
// unless its id is special (bit set in special_mask) or it lies at / beyond n_real; selected
// positions keep their id as label and become <mask> with probability p_mask, a random id from
// pool[0..pool_n) with probability p_rand, or stay unchanged. The stream depends only on
// (seed, step, position), so a batch is reproducible whatever the launch geometry.
#include <curand_kernel.h>

namespace nplm {

__global__ void __launch_bounds__(256)
mlm_mask_kernel(const long long* __restrict__ ids_in, long long* __restrict__ ids_out,
                long long* __restrict__ labels, int n, int n_real, unsigned long long special_mask,
                int mask_id, const int* __restrict__ pool, int pool_n, float p_sel, float p_mask,
                float p_rand, unsigned long long seed, unsigned long long step) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    curandStatePhilox4_32_10_t st;
    curand_init(seed, static_cast<unsigned long long>(i), step * 4ULL, &st);
    const float4 u = curand_uniform4(&st);
    const long long id = ids_in[i];
    const bool special = id < 0 || id >= 64 || ((special_mask >> id) & 1ULL) || i >= n_real;
    long long out = id, lab = -100;
    if (!special && u.x <= p_sel) {        // curand_uniform is (0, 1]
      lab = id;
      if (u.y <= p_mask) {
        out = mask_id;
      } else if (u.y <= p_mask + p_rand) {
        int k = static_cast<int>(u.z * pool_n);
        if (k >= pool_n) k = pool_n - 1;
        out = pool[k];
      }
    }
    ids_out[i] = out;
    labels[i] = lab;
  }
}

}  // namespace nplm

extern "C" int nplm_mlm_mask(const long long* ids_in, long long* ids_out, long long* labels, int n, int n_real,
                             unsigned long long special_mask, int mask_id, const int* pool, int pool_n,
                             float p_sel, float p_mask, float p_rand, unsigned long long seed,
                             unsigned long long step, cudaStream_t st) {
  if (n <= 0) return 0;
  if (pool_n <= 0) return -3;
  int blocks = (n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  nplm::mlm_mask_kernel<<<blocks, 256, 0, st>>>(ids_in, ids_out, labels, n, n_real, special_mask, mask_id, pool,
                                                pool_n, p_sel, p_mask, p_rand, seed, step);
  return static_cast<int>(cudaGetLastError());
}

// ---------------------------------------------------------------------------- mHC coefficients
// One thread per token turns the raw outputs of the coefficient projection (before tanh) into the
// mixing coefficients of one hyper-connection site:
//   d      = tanh(pre[t, :])                                   [2N + N*N]
//   alpha  = softmax(a + s0 * d[0:N])
//   beta   = 2 * sigmoid(b + s1 * d[N:2N])
//   R      = exp(sinkhorn_log(r + s2 * d[2N:], iters))         (rows, then columns, `iters` times)
// The backward kernel recomputes the forward, keeps the value after every Sinkhorn half-step
// (for y = x - logsumexp(x): dx = dy - exp(y) * sum(dy)), and returns the gradient w.r.t. pre
// (bf16) plus block-reduced atomics for the static parameters a, b, r and the three scales.
// The reference has no hyper-connections.
namespace nplm {

constexpr int MHC_MAX_ITERS = 8;

// The static parts a [N], b [N], r [N*N] and scales s [3] of a site as fp32, read from fp32 or bf16 parameters.
template <int N, typename P>
struct MhcStatic {
  float a[N], b[N], r[N * N], s[3];
  __device__ __forceinline__ MhcStatic(const P* pa, const P* pb, const P* pr, const P* ps) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      a[i] = static_cast<float>(pa[i]);
      b[i] = static_cast<float>(pb[i]);
    }
#pragma unroll
    for (int i = 0; i < N * N; ++i) r[i] = static_cast<float>(pr[i]);
#pragma unroll
    for (int i = 0; i < 3; ++i) s[i] = static_cast<float>(ps[i]);
  }
};

template <int N>
__device__ __forceinline__ void mhc_coef_forward(const float (&d)[2 * N + N * N], const float* a, const float* b,
                                                 const float* r, const float* s, int iters,
                                                 float (&alpha)[N], float (&beta)[N], float (&x)[N * N],
                                                 float* hist) {
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    alpha[i] = a[i] + s[0] * d[i];
    mx = fmaxf(mx, alpha[i]);
  }
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    alpha[i] = __expf(alpha[i] - mx);
    sum += alpha[i];
  }
#pragma unroll
  for (int i = 0; i < N; ++i) alpha[i] /= sum;
#pragma unroll
  for (int i = 0; i < N; ++i) beta[i] = 2.f / (1.f + __expf(-(b[i] + s[1] * d[N + i])));
#pragma unroll
  for (int i = 0; i < N * N; ++i) x[i] = r[i] + s[2] * d[2 * N + i];
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int i = 0; i < N; ++i) {   // rows
      float m = -INFINITY, se = 0.f;
#pragma unroll
      for (int j = 0; j < N; ++j) m = fmaxf(m, x[i * N + j]);
#pragma unroll
      for (int j = 0; j < N; ++j) se += __expf(x[i * N + j] - m);
      const float lse = m + __logf(se);
#pragma unroll
      for (int j = 0; j < N; ++j) x[i * N + j] -= lse;
    }
    if (hist != nullptr) {
#pragma unroll
      for (int i = 0; i < N * N; ++i) hist[(2 * it) * N * N + i] = x[i];
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {   // columns
      float m = -INFINITY, se = 0.f;
#pragma unroll
      for (int i = 0; i < N; ++i) m = fmaxf(m, x[i * N + j]);
#pragma unroll
      for (int i = 0; i < N; ++i) se += __expf(x[i * N + j] - m);
      const float lse = m + __logf(se);
#pragma unroll
      for (int i = 0; i < N; ++i) x[i * N + j] -= lse;
    }
    if (hist != nullptr) {
#pragma unroll
      for (int i = 0; i < N * N; ++i) hist[(2 * it + 1) * N * N + i] = x[i];
    }
  }
}

template <int N, typename P>
__global__ void __launch_bounds__(128)
mhc_coef_fwd_kernel(const __nv_bfloat16* __restrict__ pre, const P* __restrict__ pa, const P* __restrict__ pb,
                    const P* __restrict__ pr, const P* __restrict__ ps, int iters, int T, float* __restrict__ alpha_out, float* __restrict__ beta_out,
                    float* __restrict__ R_out) {
  grid_chain();
  constexpr int M = 2 * N + N * N;
  const MhcStatic<N, P> st(pa, pb, pr, ps);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
    float d[M];
#pragma unroll
    for (int i = 0; i < M; ++i) d[i] = tanhf(__bfloat162float(pre[static_cast<size_t>(t) * M + i]));
    float alpha[N], beta[N], x[N * N];
    mhc_coef_forward<N>(d, st.a, st.b, st.r, st.s, iters, alpha, beta, x, nullptr);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      alpha_out[t * N + i] = alpha[i];
      beta_out[t * N + i] = beta[i];
    }
#pragma unroll
    for (int i = 0; i < N * N; ++i) R_out[static_cast<size_t>(t) * N * N + i] = __expf(x[i]);
  }
}

template <int N, typename P>
__global__ void __launch_bounds__(128)
mhc_coef_bwd_kernel(const __nv_bfloat16* __restrict__ pre, const P* __restrict__ pa, const P* __restrict__ pb,
                    const P* __restrict__ pr, const P* __restrict__ ps, int iters, int T, const float* __restrict__ dalpha, const float* __restrict__ dbeta,
                    const float* __restrict__ dR, __nv_bfloat16* __restrict__ dpre,
                    float* __restrict__ da, float* __restrict__ db, float* __restrict__ dr,
                    float* __restrict__ ds) {
  grid_chain();
  constexpr int M = 2 * N + N * N;
  static_assert(M + 3 <= 32, "parameter gradients are reduced with one value per lane");
  const MhcStatic<N, P> st(pa, pb, pr, ps);
  // per-thread sums of the parameter gradients: [da (N) | db (N) | dr (N*N) | ds (3)]
  float acc[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = 0.f;
  const int lane = threadIdx.x & 31;
  // every warp runs the same number of iterations (the reduction below is warp-wide)
  const int per_pass = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < T; base += per_pass) {
    const int t = base + threadIdx.x;
    if (t < T) {
      float d[M];
#pragma unroll
      for (int i = 0; i < M; ++i) d[i] = tanhf(__bfloat162float(pre[static_cast<size_t>(t) * M + i]));
      float alpha[N], beta[N], x[N * N];
      float hist[2 * MHC_MAX_ITERS * N * N];
      mhc_coef_forward<N>(d, st.a, st.b, st.r, st.s, iters, alpha, beta, x, hist);
      float gd[M];   // gradient w.r.t. d (tanh output)
      // alpha = softmax(u): du = alpha * (dalpha - sum alpha * dalpha)
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < N; ++i) dot += alpha[i] * dalpha[t * N + i];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float du = alpha[i] * (dalpha[t * N + i] - dot);
        acc[i] += du;
        acc[2 * N + N * N] += du * d[i];
        gd[i] = du * st.s[0];
      }
      // beta = 2 sigmoid(v): dv = dbeta * beta * (1 - beta / 2)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float dv = dbeta[t * N + i] * beta[i] * (1.f - 0.5f * beta[i]);
        acc[N + i] += dv;
        acc[2 * N + N * N + 1] += dv * d[N + i];
        gd[N + i] = dv * st.s[1];
      }
      // R = exp(x_final): dx = dR * R, then back through the half-steps
      float g[N * N];
#pragma unroll
      for (int i = 0; i < N * N; ++i) g[i] = dR[static_cast<size_t>(t) * N * N + i] * __expf(x[i]);
      for (int it = iters - 1; it >= 0; --it) {
        const float* yc = hist + (2 * it + 1) * N * N;   // after the column step
#pragma unroll
        for (int j = 0; j < N; ++j) {
          float sg = 0.f;
#pragma unroll
          for (int i = 0; i < N; ++i) sg += g[i * N + j];
#pragma unroll
          for (int i = 0; i < N; ++i) g[i * N + j] -= __expf(yc[i * N + j]) * sg;
        }
        const float* yr = hist + (2 * it) * N * N;       // after the row step
#pragma unroll
        for (int i = 0; i < N; ++i) {
          float sg = 0.f;
#pragma unroll
          for (int j = 0; j < N; ++j) sg += g[i * N + j];
#pragma unroll
          for (int j = 0; j < N; ++j) g[i * N + j] -= __expf(yr[i * N + j]) * sg;
        }
      }
#pragma unroll
      for (int i = 0; i < N * N; ++i) {
        acc[2 * N + i] += g[i];
        acc[2 * N + N * N + 2] += g[i] * d[2 * N + i];
        gd[2 * N + i] = g[i] * st.s[2];
      }
#pragma unroll
      for (int i = 0; i < M; ++i)
        dpre[static_cast<size_t>(t) * M + i] = __float2bfloat16(gd[i] * (1.f - d[i] * d[i]));
    }
  }
  // warp-wide sums (lane l receives the total of acc[l]), one atomic per value and warp
  const float total = warp_transpose_sum<M + 3>(acc, lane);
  if (lane < N) atomicAdd(&da[lane], total);
  else if (lane < 2 * N) atomicAdd(&db[lane - N], total);
  else if (lane < 2 * N + N * N) atomicAdd(&dr[lane - 2 * N], total);
  else if (lane < M + 3) atomicAdd(&ds[lane - M], total);
}

}  // namespace nplm

namespace nplm {
template <int N, typename P>
static void mhc_coef_fwd_launch(const __nv_bfloat16* pre, const void* a, const void* b, const void* r, const void* s,
                                int iters, int T, float* alpha, float* beta, float* R, int blocks, cudaStream_t st) {
  launch_chained(mhc_coef_fwd_kernel<N, P>, blocks, 128, 0, st, pre, reinterpret_cast<const P*>(a),
      reinterpret_cast<const P*>(b), reinterpret_cast<const P*>(r), reinterpret_cast<const P*>(s), iters, T, alpha, beta,
      R);
}
template <int N, typename P>
static void mhc_coef_bwd_launch(const __nv_bfloat16* pre, const void* a, const void* b, const void* r, const void* s,
                                int iters, int T, const float* dalpha, const float* dbeta, const float* dR,
                                __nv_bfloat16* dpre, float* da, float* db, float* dr, float* ds, int blocks,
                                cudaStream_t st) {
  launch_chained(mhc_coef_bwd_kernel<N, P>, blocks, 128, 0, st, pre, reinterpret_cast<const P*>(a),
      reinterpret_cast<const P*>(b), reinterpret_cast<const P*>(r), reinterpret_cast<const P*>(s), iters, T, dalpha,
      dbeta, dR, dpre, da, db, dr, ds);
}
}  // namespace nplm

// a, b, r, s: the site's parameters, all fp32 (param_bf16 = 0) or all bf16 (1).
extern "C" int nplm_mhc_coef_fwd(const void* pre, const void* a, const void* b, const void* r, const void* s,
                                 int param_bf16, int iters, int T, int n, float* alpha, float* beta, float* R,
                                 cudaStream_t st) {
  if (T <= 0) return 0;
  if (n != 4 && n != 2) return -3;
  if (iters < 1 || iters > nplm::MHC_MAX_ITERS) return -3;
  int blocks = (T + 127) / 128;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(pre);
  auto go = n == 4 ? (param_bf16 ? nplm::mhc_coef_fwd_launch<4, __nv_bfloat16> : nplm::mhc_coef_fwd_launch<4, float>)
                   : (param_bf16 ? nplm::mhc_coef_fwd_launch<2, __nv_bfloat16> : nplm::mhc_coef_fwd_launch<2, float>);
  go(p, a, b, r, s, iters, T, alpha, beta, R, blocks, st);
  return static_cast<int>(cudaGetLastError());
}

// da / db / dr / ds (fp32) are accumulated: callers pass zeroed or running buffers.
extern "C" int nplm_mhc_coef_bwd(const void* pre, const void* a, const void* b, const void* r, const void* s,
                                 int param_bf16, int iters, int T, int n, const float* dalpha, const float* dbeta,
                                 const float* dR, void* dpre, float* da, float* db, float* dr, float* ds,
                                 cudaStream_t st) {
  if (T <= 0) return 0;
  if (n != 4 && n != 2) return -3;
  if (iters < 1 || iters > nplm::MHC_MAX_ITERS) return -3;
  int blocks = (T + 127) / 128;
  if (blocks > 148 * 4) blocks = 148 * 4;
  const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(pre);
  auto go = n == 4 ? (param_bf16 ? nplm::mhc_coef_bwd_launch<4, __nv_bfloat16> : nplm::mhc_coef_bwd_launch<4, float>)
                   : (param_bf16 ? nplm::mhc_coef_bwd_launch<2, __nv_bfloat16> : nplm::mhc_coef_bwd_launch<2, float>);
  go(p, a, b, r, s, iters, T, dalpha, dbeta, dR, reinterpret_cast<__nv_bfloat16*>(dpre), da, db, dr, ds, blocks, st);
  return static_cast<int>(cudaGetLastError());
}
