// Inference attention with an additive relative-position bias for the T5-style teacher
// (head_dim 64 or 128, non-causal, key-padding mask through per-token key ranges), sm_100a.
//
//   out[t, h, :] = softmax_k( scale * q_t . k_k + bias[h][k - t + S - 1] ) v_k,   k in [seq_start[t], seq_end[t])
//
// Replaces the eager attention of the HF T5 encoder the reference uses as its distillation teacher
// (src/nanoplm/distillation/models/teacher/prott5.py:24-52 loads T5EncoderModel; the bias is T5's
// bucketed relative_attention_bias, shared by all layers). bias is a per-head table indexed by
// the relative position (key - query), built once per forward on the host side of the model.
//
// Persistent and warp-specialised: a CTA per SM walks (256-query pair of tiles, head) items. Two softmax warpgroups, one per
// 128-query tile, a thread per query row; one MMA-issuing warp per tile; one loader warp. The flat token axis (batch
// x padded length) is tiled regardless of sequence boundaries, every row masks keys outside its own range. Keys
// are consumed 64 at a time: the two tiles' scores (2 x 64 columns), bf16 probabilities (2 x 32) and outputs (2 x 128 for
// head_dim 128) then all have their own tensor-memory columns, so the score product of a step runs while the previous
// step's softmax and output product do, and a tile's chain hides behind the other's. The bias row of a thread is
// read from a per-item table in shared memory (neighbouring lanes read neighbouring words).
//
// The kernel it replaces ran one chain of MMA -> softmax -> MMA per CTA with the output in registers and two passes over the
// scores, two CTAs an SM: 703 us for 21 700 tokens and 32 heads of 128 in sequences of 21 - 512, 349 us now; 25 000
// tokens in sequences of 21 - 1 001 1 553 and 687 us. Relative distance from fp64 over lengths of 20 - 2000 and score deviations
// of 1 - 16: 0.985 - 0.999 times that kernel's (head dimension 128).
#include "common.cuh"

namespace nplm {

constexpr int AB_T = 128;
constexpr int AB_TILE = AB_T * 64 * 2;  // one [128][64] bf16 tile, 16 KB
constexpr float AB_LOG2E = 1.4426950408889634f;

__device__ __forceinline__ uint32_t ab_swz(int r, int chunk) {
  return static_cast<uint32_t>(r * 128 + ((chunk ^ (r & 7)) << 4));
}

struct AbArgs {
  const int* seq_start;  // [T]
  const int* seq_end;    // [T]
  const float* bias;     // [H][2*S-1], index = key - query + S - 1
  int T, H, S;
  float scale;
  int* status;
};

constexpr int AB_KC = 64;                       // keys per step
constexpr int AB_THREADS = 384;                 // warps 0-3, 4-7: softmax of tile 0 / 1; 8: loader; 9, 10: MMA; 11: idle
constexpr int AB_LOADER_WARP = 8, AB_MMA_WARP = 9;
constexpr int AB_TAB = 2304;                    // floats of a tile's bias table: key ranges up to 2 176 keys

template <int D>
struct AbCfg {
  static constexpr int NA = D / 64;                       // 64-column atoms per operand tile
  static constexpr int Q_TILE = NA * AB_TILE;             // [atom][128 rows][128 B]
  static constexpr int KA = AB_KC * 128;                  // bytes of one K / V atom
  static constexpr int KV_TILE = NA * KA;                 // [atom][64 rows][128 B]
  static constexpr int STAGES = D == 128 ? 2 : 4;
  static constexpr int OFF_Q = 0;                         // [2 buffers][2 tiles]; a tile's buffer stages its output
  static constexpr int OFF_K = OFF_Q + 4 * Q_TILE;
  static constexpr int OFF_V = OFF_K + STAGES * KV_TILE;
  static constexpr int OFF_TAB = OFF_V + STAGES * KV_TILE;
  static constexpr int OFF_BAR = OFF_TAB + 2 * AB_TAB * 4;
  static constexpr int SMEM = OFF_BAR + 512;
};

// Key range of an item and the steps [a, b) in which each tile takes part; lo / hi: union over the tile's rows.
struct AbGeo {
  int kv_lo, n;
  int a[2], b[2];
};

// Computed by a whole warp: 16 coalesced loads, four warp reductions.
__device__ __forceinline__ AbGeo ab_geometry(const AbArgs& args, int pair, int lane) {
  const int t0 = pair * 2 * AB_T, T = args.T;
  int lo[2], hi[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    lo[i] = 0x7fffffff;
    hi[i] = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int row = t0 + i * AB_T + k * 32 + lane;
      if (row < T) {
        const int s = __ldg(args.seq_start + row), e = __ldg(args.seq_end + row);
        if (e > s) {
          lo[i] = min(lo[i], s);
          hi[i] = max(hi[i], e);
        }
      }
    }
    lo[i] = __reduce_min_sync(0xffffffffu, lo[i]);
    hi[i] = __reduce_max_sync(0xffffffffu, hi[i]);
  }
  AbGeo g;
  g.kv_lo = min(lo[0], lo[1]);
  const int kv_hi = max(hi[0], hi[1]);
  g.n = kv_hi > g.kv_lo ? (kv_hi - g.kv_lo + AB_KC - 1) / AB_KC : 0;
  if (g.n == 0) g.kv_lo = 0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    g.a[i] = g.b[i] = 0;
    if (hi[i] > lo[i]) {
      g.a[i] = (lo[i] - g.kv_lo) / AB_KC;
      g.b[i] = (hi[i] - g.kv_lo + AB_KC - 1) / AB_KC;
    }
  }
  return g;
}

// barrier over one softmax warpgroup with an AND over everybody's predicate
__device__ __forceinline__ bool ab_barrier_and(int id, bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t"
      ".reg .pred q, o;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "bar.red.and.pred o, %1, 128, q;\n\t"
      "selp.u32 %0, 1, 0, o;\n\t"
      "}"
      : "=r"(r)
      : "r"(id), "r"(static_cast<uint32_t>(p))
      : "memory");
  return r != 0;
}

template <int D>
__global__ void __launch_bounds__(AB_THREADS, 1)
fa_bias_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV,
                   const __grid_constant__ CUtensorMap tmO, const AbArgs args) {
  using C = AbCfg<D>;
  constexpr int NA = C::NA, STAGES = C::STAGES;
  extern __shared__ __align__(1024) uint8_t smem[];
  if (smem_u32(smem) & 1023u) {
    grid_wait();
    if (threadIdx.x == 0) atomicExch(args.status, ST_BAD_ARG);
    return;
  }
  uint8_t* sQ = smem + C::OFF_Q;
  uint8_t* sK = smem + C::OFF_K;
  uint8_t* sV = smem + C::OFF_V;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t* q_full = bars;                  // [2]
  // [2] every consumer (both warpgroups, whose output leaves through the buffer, and both MMA issuers) gives a buffer
  // back once per item, and only after it has seen that item's q_full: nobody can be two items behind or ahead
  uint64_t* q_empty = q_full + 2;
  uint64_t* k_full = q_empty + 2;           // [STAGES]
  uint64_t* k_empty = k_full + STAGES;      // both MMA issuers
  uint64_t* v_full = k_empty + STAGES;
  uint64_t* v_empty = v_full + STAGES;
  uint64_t* s_full = v_empty + STAGES;      // [2] per tile: scores of a step are in TMEM
  uint64_t* s_free = s_full + 2;            // the warpgroup holds them in registers
  uint64_t* p_ready = s_free + 2;           // probabilities are in TMEM
  uint64_t* pv_done = p_ready + 2;          // the step's output product has finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int T = args.T, H = args.H, HD = H * D;
  const int n_items = ((T + 2 * AB_T - 1) / (2 * AB_T)) * H;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 4);
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 4);
      mbar_init(&p_ready[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 2);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 2);
    }
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKV);
    tma_prefetch_desc(&tmO);
  }
  grid_wait();
  if (warp == AB_MMA_WARP) {
    __syncwarp();
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_release();
  // columns: S0 [0,64), S1 [64,128), P0 [128,160), P1 [160,192), O0 [256,256+D), O1 [384,384+D)

  if (warp == AB_LOADER_WARP) {
    // ------------------------------------------------------------------ loader
    uint32_t qc = 0, kc = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++qc) {
      const int h = item % H, pair = item / H;
      const AbGeo g = ab_geometry(args, pair, lane);
      if (elect_one()) {
        const int colQ = h * D, colK = HD + h * D, colV = 2 * HD + h * D;
        const uint32_t qb = qc & 1u;
        const int t0 = pair * 2 * AB_T;
        if (!mbar_wait(&q_empty[qb], ((qc >> 1) & 1u) ^ 1u)) ok = false;
        if (ok) {
          const int nq = t0 + AB_T < T ? 2 : 1;
          mbar_arrive_expect_tx(&q_full[qb], nq * C::Q_TILE);
          for (int i = 0; i < nq; ++i)
#pragma unroll
            for (int x = 0; x < NA; ++x)
              tma_load_2d(sQ + (qb * 2 + i) * C::Q_TILE + x * AB_TILE, &tmQ, &q_full[qb], colQ + x * 64, t0 + i * AB_T);
        }
        uint32_t k = kc;
        for (int j = 0; j < g.n && ok; ++j, ++k) {
          const uint32_t st = k % STAGES, ph = (k / STAGES) & 1u;
          const int kv0 = g.kv_lo + j * AB_KC;
          if (!mbar_wait(&k_empty[st], ph ^ 1u)) { ok = false; break; }
          mbar_arrive_expect_tx(&k_full[st], C::KV_TILE);
#pragma unroll
          for (int x = 0; x < NA; ++x)
            tma_load_2d(sK + st * C::KV_TILE + x * C::KA, &tmKV, &k_full[st], colK + x * 64, kv0);
          if (!mbar_wait(&v_empty[st], ph ^ 1u)) { ok = false; break; }
          mbar_arrive_expect_tx(&v_full[st], C::KV_TILE);
#pragma unroll
          for (int x = 0; x < NA; ++x)
            tma_load_2d(sV + st * C::KV_TILE + x * C::KA, &tmKV, &v_full[st], colV + x * 64, kv0);
        }
        if (!ok && *abort_flag == 0) {
          atomicExch(args.status, ST_TIMEOUT_EMPTY);
          *abort_flag = 1;
        }
        if (*abort_flag) ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      kc += g.n;
    }
  } else if (warp == AB_MMA_WARP || warp == AB_MMA_WARP + 1) {
    // ------------------------------------------------------------------ MMA issuers, one per query tile
    const int i = warp - AB_MMA_WARP;
    constexpr uint32_t idesc_s = make_idesc_bf16(128, AB_KC, 0, 0);
    constexpr uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);
    const uint32_t tS = tmem_base + i * 64, tP = tmem_base + 128 + i * 32, tO = tmem_base + 256 + i * 128;
    uint32_t qc = 0, kc = 0, s_cnt = 0, p_cnt = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++qc) {
      const AbGeo g = ab_geometry(args, item / H, lane);
      const int ja = i ? g.a[1] : g.a[0], jb = i ? g.b[1] : g.b[0];
      if (elect_one()) {
        int why = ST_TIMEOUT_FULL;
        uint32_t sc = s_cnt, pc = p_cnt;
        const uint32_t qb = qc & 1u;
        if (!mbar_wait(&q_full[qb], (qc >> 1) & 1u)) ok = false;
        const uint32_t qa = smem_u32(sQ + (qb * 2 + i) * C::Q_TILE);
        for (int j = 0; j <= g.n && ok; ++j) {
          if (j < g.n) {   // scores of step j
            const uint32_t st = (kc + j) % STAGES, ph = ((kc + j) / STAGES) & 1u;
            if (!mbar_wait(&k_full[st], ph)) { ok = false; break; }
            if (j >= ja && j < jb) {
              if (!mbar_wait(&s_free[i], (sc & 1u) ^ 1u)) { ok = false; why = ST_TIMEOUT_TMEM_EMPTY; break; }
              tc_fence_after();
              const uint32_t ka = smem_u32(sK + st * C::KV_TILE);
#pragma unroll
              for (int k = 0; k < D / 16; ++k)
                umma_bf16(tS, make_smem_desc(qa + (k >> 2) * AB_TILE + (k & 3) * 32, 16, 1024),
                          make_smem_desc(ka + (k >> 2) * C::KA + (k & 3) * 32, 16, 1024), idesc_s, k > 0 ? 1u : 0u);
              umma_commit(&s_full[i]);
              ++sc;
            }
            umma_commit(&k_empty[st]);     // by both issuers
          }
          if (j >= 1) {    // output product of step j - 1
            const int jj = j - 1;
            const uint32_t st = (kc + jj) % STAGES, ph = ((kc + jj) / STAGES) & 1u;
            if (!mbar_wait(&v_full[st], ph)) { ok = false; break; }
            if (jj >= ja && jj < jb) {
              if (!mbar_wait(&p_ready[i], pc & 1u)) { ok = false; why = ST_TIMEOUT_MISC; break; }
              tc_fence_after();
              const uint32_t va = smem_u32(sV + st * C::KV_TILE);
#pragma unroll
              for (int k = 0; k < AB_KC / 16; ++k)   // P: 8 columns per 16 keys; V (MN-major): 16 key rows = 2048 bytes
                umma_bf16_ts(tO, tP + k * 8, make_smem_desc(va + k * 2048, C::KA, 1024), idesc_o,
                             (jj > ja || k > 0) ? 1u : 0u);
              umma_commit(&pv_done[i]);
              ++pc;
            }
            umma_commit(&v_empty[st]);
          }
        }
        if (ok) mbar_arrive(&q_empty[qb]);   // (the warpgroup waits for the products that read the buffer)
        if (!ok && *abort_flag == 0) {
          atomicExch(args.status, why);
          *abort_flag = 1;
        }
        if (*abort_flag) ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      kc += g.n;
      s_cnt += jb - ja;
      p_cnt += jb - ja;
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ softmax warpgroups
    const int i = warp >> 2;
    const int quarter = warp & 3;
    const int rl = quarter * 32 + lane;                // row inside the tile
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tS = tmem_base + i * 64 + lane_addr, tP = tmem_base + 128 + i * 32 + lane_addr;
    const uint32_t tO = tmem_base + 256 + i * 128 + lane_addr;
    float* tab = reinterpret_cast<float*>(smem + C::OFF_TAB) + i * AB_TAB;
    const float sl2 = args.scale * AB_LOG2E;
    const int S = args.S;
    uint32_t qc = 0, s_cnt = 0, pv_cnt = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++qc) {
      const int h = item % H, pair = item / H;
      const AbGeo g = ab_geometry(args, pair, lane);
      const int ja = i ? g.a[1] : g.a[0], jb = i ? g.b[1] : g.b[0];
      const int row0 = pair * 2 * AB_T + i * AB_T;
      const int row = row0 + rl;
      int lo = 0, hi = 0;
      if (row < T) {
        lo = __ldg(args.seq_start + row);
        hi = __ldg(args.seq_end + row);
      }
      const float* gb = args.bias + static_cast<size_t>(h) * (2 * S - 1);
      // tab[t] = bias of (key - row) = kbase - (row0 + 127) + t: thread rl finds key kbase + u at tab[u + 127 - rl].
      // Entries outside the table belong to keys of other sequences and are masked.
      const int kbase = g.kv_lo + ja * AB_KC;
      const int len = (jb - ja) * AB_KC + 127;
      const bool in_smem = len <= AB_TAB;
      if (in_smem) {
        const int first = kbase - row0 - 127 + S - 1;
        for (int t = rl; t < len; t += 128) {
          const int x = first + t;
          tab[t] = (x >= 0 && x < 2 * S - 1) ? __ldg(gb + x) * AB_LOG2E : 0.f;
        }
      }
      ok = ab_barrier_and(1 + i, *abort_flag == 0);
      if (!ok) break;
      float m_used = -1e30f, l_run = 0.f;
      for (int j = ja; j < jb; ++j) {
        const int kv0 = g.kv_lo + j * AB_KC;
        ok = mbar_wait(&s_full[i], s_cnt & 1u);
        ++s_cnt;
        ok = __all_sync(0xffffffffu, ok && *abort_flag == 0);
        if (!ok) break;
        tc_fence_after();
        const bool none = __all_sync(0xffffffffu, kv0 >= hi || kv0 + AB_KC <= lo);   // no row of the warp sees the block
        uint32_t r[AB_KC];
        if (!none) {
          tmem_ld32(tS, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
          tmem_ld32(tS + 32, *reinterpret_cast<uint32_t(*)[32]>(&r[32]));
          tmem_ld_wait();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_free[i]);   // the score tile may be overwritten
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        if (!none) {
          const bool inside = kv0 >= lo && kv0 + AB_KC <= hi;
          uint64_t bits = ~0ull;                  // bit e: key kv0 + e lies inside the row's range
          if (!inside) {
            const int x = max(lo - kv0, 0), y = min(hi - kv0, AB_KC);
            bits = y > x ? (~0ull >> (64 - (y - x))) << x : 0ull;
          }
          if (in_smem) {
            const float* tb = tab + (j - ja) * AB_KC + 127 - rl;
#pragma unroll
            for (int e = 0; e < AB_KC; ++e) r[e] = __float_as_uint(fmaf(__uint_as_float(r[e]), sl2, tb[e]));
          } else {
            const float* tb = gb + (kv0 - row + S - 1);
#pragma unroll
            for (int e = 0; e < AB_KC; ++e)
              if ((bits >> e) & 1ull) r[e] = __float_as_uint(fmaf(__uint_as_float(r[e]), sl2, __ldg(tb + e) * AB_LOG2E));
          }
          if (!__all_sync(0xffffffffu, inside)) {
#pragma unroll
            for (int e = 0; e < AB_KC; ++e)
              if (!((bits >> e) & 1ull)) r[e] = 0xff800000u;
          }
#pragma unroll
          for (int e = 0; e < AB_KC; ++e) mx[e & 3] = fmaxf(mx[e & 3], __uint_as_float(r[e]));
        }
        const float m_new = fmaxf(m_used, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
        // The running maximum follows every growth, so that a row's largest probability is 1 and free of rounding. (Left
        // behind by up to 2^8 the output accumulator needed fewer rescalings, 300 against 334 us for 21 700 tokens and 32
        // heads of 128, but the outputs were up to 1.23 times as far from fp64.)
        const bool grow = __any_sync(0xffffffffu, m_new > m_used);
        float alpha = 1.f;
        if (grow) {
          alpha = exp2f(m_used - m_new);
          m_used = m_new;
        }
        if (j > ja) {
          // the previous output product has finished: P may be overwritten and O rescaled
          ok = mbar_wait(&pv_done[i], pv_cnt & 1u);
          ++pv_cnt;
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          if (grow) {
#pragma unroll
            for (int c = 0; c < D; c += 32) {
              uint32_t o[32];
              tmem_ld32(tO + c, o);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
              tmem_st32(tO + c, o);
            }
            tmem_st_wait();
          }
        }
        // the sum of what enters the product, i.e. of the rounded probabilities: their errors then partly cancel
        float2 ps[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        uint32_t pk[32];
        if (!none) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const float p0 = exp2f(__uint_as_float(r[2 * c]) - m_used), p1 = exp2f(__uint_as_float(r[2 * c + 1]) - m_used);
            pk[c] = pack_bf16x2(p0, p1);
            ps[c & 3] = add2(ps[c & 3], unpack_bf16x2(pk[c]));
          }
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) pk[c] = 0u;
        }
        tmem_st32(tP, pk);
        tmem_st_wait();
        const float2 ps2 = add2(add2(ps[0], ps[1]), add2(ps[2], ps[3]));
        l_run = l_run * alpha + (ps2.x + ps2.y);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[i]);
      }
      if (ok && jb > ja) {
        ok = mbar_wait(&pv_done[i], pv_cnt & 1u);   // the item's last output product
        ++pv_cnt;
      }
      // The output leaves through this tile's Q buffer, which the finished score products no longer read. A tile without
      // keys or rows has waited for no product: the loads of Q have to have landed before the buffer is written, and
      // before it is given back (an early arrival would count for the item that the buffer still holds)
      const uint32_t qb = qc & 1u;
      ok = ok && mbar_wait(&q_full[qb], (qc >> 1) & 1u);
      ok = ab_barrier_and(1 + i, ok && *abort_flag == 0);
      if (!ok) break;
      tc_fence_after();
      if (row0 < T) {
        uint8_t* so = sQ + (qb * 2 + i) * C::Q_TILE;
        const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
#pragma unroll
        for (int c = 0; c < D; c += 32) {
          uint32_t o[32];
          if (jb > ja) {
            tmem_ld32(tO + c, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = 0u;   // no key for any row of the tile
          }
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint4 u;
            uint32_t* p = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
            for (int q = 0; q < 4; ++q)
              p[q] = pack_bf16x2(__uint_as_float(o[e + 2 * q]) * inv, __uint_as_float(o[e + 2 * q + 1]) * inv);
            *reinterpret_cast<uint4*>(so + (c >> 6) * AB_TILE + ab_swz(rl, ((c & 63) + e) >> 3)) = u;
          }
        }
        tc_fence_before();
        fence_proxy_async_smem();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + i) : "memory");
        if (quarter == 0 && elect_one()) {            // rows past the end of the batch are clipped
#pragma unroll
          for (int x = 0; x < NA; ++x) tma_store_2d(&tmO, so + x * AB_TILE, h * D + x * 64, row0);
          tma_store_commit();
          tma_store_wait_read<0>();
        }
      }
      if (quarter == 0 && elect_one()) mbar_arrive(&q_empty[qb]);
    }
    if (quarter == 0 && elect_one()) tma_store_wait<0>();
    __syncwarp();
    if (!ok && lane == 0 && *abort_flag == 0) {
      atomicExch(args.status, ST_TIMEOUT_TMEM_FULL);
      *abort_flag = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == AB_MMA_WARP) {
    tc_fence_after();
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

typedef CUresult (*AbEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                               CUtensorMapFloatOOBfill);

static AbEncodeFn ab_encode_fn() {
  static AbEncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<AbEncodeFn>(p);
  }
  return fn;
}

template <int D>
static int ab_launch(const CUtensorMap& tmQ, const CUtensorMap& tmKV, const CUtensorMap& tmO, const AbArgs& a,
                     cudaStream_t st) {
  constexpr int smem = AbCfg<D>::SMEM;
  static bool configured_on[nplm::MAX_DEVICES];
  const int dev_slot = nplm::current_device_slot();
  if (dev_slot < 0) return -4;
  bool& configured = configured_on[dev_slot];
  if (!configured) {
    NPLM_CUDA_CHECK(cudaFuncSetAttribute(fa_bias_fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_slot);
  const int n_items = ((a.T + 2 * AB_T - 1) / (2 * AB_T)) * a.H;
  launch_chained(fa_bias_fwd_kernel<D>, n_items < sms ? n_items : sms, AB_THREADS, smem, st, tmQ, tmKV, tmO, a);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace nplm

using namespace nplm;

// qkv bf16 [T][3][H][D]; out bf16 [T][H*D]; bias fp32 [H][2*S-1] with S >= the longest key range.
extern "C" int nplm_fa_bias_fwd(const void* qkv, void* out, const int* seq_start, const int* seq_end,
                                const float* bias, int T, int H, int D, int S, float scale, int* status,
                                cudaStream_t st) {
  if (T <= 0) return 0;
  if ((D != 64 && D != 128) || S < 1 || (reinterpret_cast<uintptr_t>(qkv) & 15)) return -3;
  if ((reinterpret_cast<uintptr_t>(out) & 15) || H <= 0) return -3;
  AbEncodeFn fn = ab_encode_fn();
  if (fn == nullptr) return -1;
  auto make = [&](CUtensorMap* map, const void* base, uint64_t cols, uint32_t rows) {
    cuuint64_t dims[2] = {cols, static_cast<cuuint64_t>(T)};
    cuuint64_t strides[1] = {cols * 2};
    cuuint32_t estr[2] = {1, 1};
    cuuint32_t box[2] = {64, rows};
    return nplm::with_context([&] {
             return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
           }) == CUDA_SUCCESS;
  };
  CUtensorMap tmQ, tmKV, tmO;
  const uint64_t cols = static_cast<uint64_t>(H) * D;
  if (!make(&tmQ, qkv, 3 * cols, AB_T) || !make(&tmKV, qkv, 3 * cols, AB_KC) || !make(&tmO, out, cols, AB_T)) return -2;
  AbArgs a;
  a.seq_start = seq_start;
  a.seq_end = seq_end;
  a.bias = bias;
  a.T = T;
  a.H = H;
  a.S = S;
  a.scale = scale;
  a.status = status;
  return D == 64 ? ab_launch<64>(tmQ, tmKV, tmO, a, st) : ab_launch<128>(tmQ, tmKV, tmO, a, st);
}
