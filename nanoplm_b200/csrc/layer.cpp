// Host-side launch sequences of plain encoder layers (pre-norm, rotary attention, SwiGLU MLP, no biases): all
// kernels of a forward pass from one call, and all of its backward pass from another, for one layer or a run of layers.
//
// The kernels and their order are those of the op-by-op path (nanoplm_b200/models/encoder.py: EncoderLayer); what
// this saves is the interpreter between them: a launch from Python costs 15 - 20 us (wrapper, checks, allocation, autograd
// node), the same launch from here 4. A layer has 7 launches forward and 14 backward, so calls whose kernels take
// less than that (single proteins, small batches, small models) were bound by the interpreter.
//
// The kernels live in other shared objects; nplm_layer_init receives their entry points once. Every function
// returns 0, or the first non-zero code of a launch.
#include <cstddef>
#include <cstdint>

#include "entry_points.h"

namespace {

using namespace nplm;

struct Entry {   // in the order of `_native` in ops/layer.py
  decltype(&nplm_gemm_bf16) gemm;
  decltype(&nplm_gemm_bf16_pair) pair;
  decltype(&nplm_gemm_bf16_delta) delta;
  decltype(&nplm_norm_fwd) norm_fwd;
  decltype(&nplm_norm_bwd) norm_bwd;
  decltype(&nplm_fa_fwd_ws) fa_fwd;
  decltype(&nplm_fa_bwd_ws_zeroed) fa_bwd;
};
Entry fn;

// Positions in the argument arrays that ops/layer.py fills; BWD_ ones follow those of the forward call.
enum Arg {
  A_T, A_C, A_I, A_H, A_WINDOW, A_NORM1, A_RMS, A_TRAIN,
  A_X, A_W_QKV, A_W_O, A_W_IN, A_W_OUT, A_N1, A_N2,
  A_SEQ_START, A_SEQ_END, A_POS, A_COS, A_SIN,
  A_BUF, A_Y, A_STATUS, A_STREAM,
  BWD_DX, BWD_SCRATCH, BWD_G_QKV, BWD_G_O, BWD_G_IN, BWD_G_OUT, BWD_G_N1, BWD_G_N2,
  BWD_SPLITS_QKV, BWD_SPLITS_O, BWD_SPLITS_IN, BWD_SPLITS_OUT, BWD_ATTENTION_MODE,
  BWD_ARGS, FWD_ARGS = BWD_DX
};

typedef unsigned char u8;

struct Cut {   // consecutive 256-byte aligned parts of one allocation
  u8* base;
  size_t at = 0;
  explicit Cut(void* p) : base(static_cast<u8*>(p)) {}
  u8* take(size_t bytes) {
    u8* p = base + at;
    at += (bytes + 255) & ~static_cast<size_t>(255);
    return p;
  }
};

// The tensors of a forward pass, in one allocation. With a backward pass to come everything has a place of its own;
// without one a tensor takes the place of those that no later kernel reads: o that of h1 (its last reader is the QKV
// product), and the MLP's h2 and hs those of h1 / o and qkv (last read by the attention and its output product).
struct Saved {
  void *h1, *qkv, *o, *x1, *h2, *pre, *hs;
  float *mean1, *rstd1, *lse, *mean2, *rstd2;
  size_t bytes;
  Saved(void* buf, long long T, long long C, long long I, long long H, bool norm1, bool train) {
    Cut c(buf);
    const size_t t = static_cast<size_t>(T);
    if (!train) {
      mean1 = rstd1 = mean2 = rstd2 = nullptr;
      pre = nullptr;
      x1 = c.take(t * C * 2);
      const size_t first = c.at;
      o = c.take(t * (norm1 && C > H * 64 ? C : H * 64) * 2);
      h1 = norm1 ? o : nullptr;
      qkv = c.take(t * 3 * H * 64 * 2);
      lse = reinterpret_cast<float*>(c.take(t * H * 4));
      Cut m(buf);
      m.at = first;
      h2 = m.take(t * C * 2);
      hs = m.take(t * I * 2);
      bytes = c.at > m.at ? c.at : m.at;
      return;
    }
    h1 = norm1 ? c.take(t * C * 2) : nullptr;
    mean1 = norm1 ? reinterpret_cast<float*>(c.take(t * 4)) : nullptr;
    rstd1 = norm1 ? reinterpret_cast<float*>(c.take(t * 4)) : nullptr;
    qkv = c.take(t * 3 * H * 64 * 2);
    o = c.take(t * H * 64 * 2);
    lse = reinterpret_cast<float*>(c.take(t * H * 4));
    x1 = c.take(t * C * 2);
    mean2 = reinterpret_cast<float*>(c.take(t * 4));
    rstd2 = reinterpret_cast<float*>(c.take(t * 4));
    h2 = c.take(t * C * 2);
    pre = c.take(t * 2 * I * 2);
    hs = c.take(t * I * 2);
    bytes = c.at;
  }
};

// Scratch of a backward pass. The pre-activation gradients are dead once the MLP's part is done and the attention's
// tensors take their place.
struct Scratch {
  void *dpre, *dh, *dx1, *d_o, *dqkv;
  float *delta, *dq;
  size_t bytes;
  Scratch(void* buf, long long T, long long C, long long I, long long H) {
    const size_t t = static_cast<size_t>(T);
    Cut c(buf);
    dh = c.take(t * C * 2);
    dx1 = c.take(t * C * 2);
    const size_t shared = c.at;
    dpre = c.take(t * 2 * I * 2);
    Cut a(buf);
    a.at = shared;
    d_o = a.take(t * H * 64 * 2);
    delta = reinterpret_cast<float*>(a.take(t * H * 4));
    dq = reinterpret_cast<float*>(a.take(t * H * 64 * 4));
    dqkv = a.take(t * 3 * H * 64 * 2);
    bytes = c.at > a.at ? c.at : a.at;
  }
};

struct Call {
  int* status;
  cudaStream_t stream;
  // bf16 output: tiles and CTA pairs as ops.kernels.gemm chooses by default
  int out(const void* A, const void* B, void* Cp, const void* R, int M, int N, int K, int ldb, int ldc, int ldr, int b_mn,
          int epi, const int* pos = nullptr, const float* cosp = nullptr, const float* sinp = nullptr,
          int rope_cols = 0) const {
    const int bn = gemm_tile_width(M, N, epi);
    if (bn == 256 && gemm_pair_pays(M, N, K, epi))
      return fn.pair(A, B, Cp, R, M, N, K, K, ldb, ldc, ldr, 0, b_mn, epi, 1, 0, pos, cosp, sinp, rope_cols, status, stream);
    return fn.gemm(A, B, Cp, R, M, N, K, K, ldb, ldc, ldr, 0, b_mn, epi, 1, bn, 0, 0, pos, cosp, sinp, rope_cols, status,
                   stream);
  }
  // fp32 C[N][K] += dy[T][N]^T x[T][K]
  int wgrad(const void* dy, const void* x, float* g, int T, int N, int K, int splits) const {
    return fn.gemm(dy, x, g, nullptr, N, K, T, N, K, K, 0, 1, 1, EPI_ATOMIC_F32, splits, K >= 256 ? 256 : 128, 0, 0, nullptr,
                   nullptr, nullptr, 0, status, stream);
  }
};

template <typename P>
P* ptr(const long long* a, int i) {
  return reinterpret_cast<P*>(static_cast<intptr_t>(a[i]));
}

#define TRY(call)              \
  do {                         \
    const int rc_ = (call);    \
    if (rc_ != 0) return rc_;  \
  } while (0)

}  // namespace

extern "C" void nplm_layer_init(void* const* f) {
  fn.gemm = reinterpret_cast<decltype(fn.gemm)>(f[0]);
  fn.pair = reinterpret_cast<decltype(fn.pair)>(f[1]);
  fn.delta = reinterpret_cast<decltype(fn.delta)>(f[2]);
  fn.norm_fwd = reinterpret_cast<decltype(fn.norm_fwd)>(f[3]);
  fn.norm_bwd = reinterpret_cast<decltype(fn.norm_bwd)>(f[4]);
  fn.fa_fwd = reinterpret_cast<decltype(fn.fa_fwd)>(f[5]);
  fn.fa_bwd = reinterpret_cast<decltype(fn.fa_bwd)>(f[6]);
}

extern "C" int nplm_gemm_tile_width(long long M, long long N, int epi) { return gemm_tile_width(M, N, epi); }
extern "C" int nplm_gemm_pair_pays(long long M, long long N, long long K, int epi) { return gemm_pair_pays(M, N, K, epi); }

// Length of the argument array of a forward (0) or backward (1) call.
extern "C" int nplm_layer_args(int backward) { return backward ? BWD_ARGS : FWD_ARGS; }

// Bytes of the forward pass's buffer (backward = 0) or of the backward pass's scratch (1).
extern "C" long long nplm_layer_bytes(long long T, long long C, long long I, long long H, int norm1, int train,
                                      int backward) {
  return static_cast<long long>(backward ? Scratch(nullptr, T, C, I, H).bytes
                                         : Saved(nullptr, T, C, I, H, norm1 != 0, train != 0).bytes);
}

// a: see Arg
extern "C" int nplm_layer_fwd(const long long* a, double eps1, double eps2, double scale) {
  const int T = static_cast<int>(a[A_T]), C = static_cast<int>(a[A_C]), I = static_cast<int>(a[A_I]), H = static_cast<int>(a[A_H]);
  const int window = static_cast<int>(a[A_WINDOW]), rms = static_cast<int>(a[A_RMS]);
  const bool norm1 = a[A_NORM1] != 0, train = a[A_TRAIN] != 0;
  const int HD = H * 64;
  if (T <= 0) return 0;
  const void *x = ptr<void>(a, A_X), *wqkv = ptr<void>(a, A_W_QKV), *wo = ptr<void>(a, A_W_O), *win = ptr<void>(a, A_W_IN),
             *wout = ptr<void>(a, A_W_OUT), *n1 = ptr<void>(a, A_N1), *n2 = ptr<void>(a, A_N2);
  const int *ss = ptr<int>(a, A_SEQ_START), *se = ptr<int>(a, A_SEQ_END), *pos = ptr<int>(a, A_POS);
  const float *cosp = ptr<float>(a, A_COS), *sinp = ptr<float>(a, A_SIN);
  const Saved s(ptr<void>(a, A_BUF), T, C, I, H, norm1, train);
  void* y = ptr<void>(a, A_Y);
  const Call k{ptr<int>(a, A_STATUS), ptr<CUstream_st>(a, A_STREAM)};
  if (norm1)
    TRY(fn.norm_fwd(x, nullptr, n1, s.h1, rms ? nullptr : s.mean1, s.rstd1, T, C, static_cast<float>(eps1), rms, k.stream));
  const void* h1 = norm1 ? s.h1 : x;
  TRY(k.out(h1, wqkv, s.qkv, nullptr, T, 3 * HD, C, C, 3 * HD, 0, 0, EPI_ROPE, pos, cosp, sinp, 2 * HD));
  TRY(fn.fa_fwd(s.qkv, s.o, s.lse, ss, se, T, H, 64, window, static_cast<float>(scale), 0, k.status, k.stream));
  TRY(k.out(s.o, wo, s.x1, x, T, C, HD, HD, C, C, 0, EPI_ADD));
  TRY(fn.norm_fwd(s.x1, nullptr, n2, s.h2, rms ? nullptr : s.mean2, s.rstd2, T, C, static_cast<float>(eps2), rms, k.stream));
  TRY(k.out(s.h2, win, s.hs, s.pre, T, 2 * I, C, C, I, s.pre != nullptr ? 2 * I : 0, 0, EPI_SWIGLU));
  return k.out(s.hs, wout, y, s.x1, T, C, I, I, C, C, 0, EPI_ADD);
}

// a: see Arg, with A_Y = the incoming gradient dy. The fp32 gradients are added to; attention mode -1 is the default, 3 the
// reproducible one.
extern "C" int nplm_layer_bwd(const long long* a, double scale) {
  const int T = static_cast<int>(a[A_T]), C = static_cast<int>(a[A_C]), I = static_cast<int>(a[A_I]), H = static_cast<int>(a[A_H]);
  const int window = static_cast<int>(a[A_WINDOW]), rms = static_cast<int>(a[A_RMS]);
  const bool norm1 = a[A_NORM1] != 0;
  const int HD = H * 64;
  if (T <= 0) return 0;
  const void *x = ptr<void>(a, A_X), *wqkv = ptr<void>(a, A_W_QKV), *wo = ptr<void>(a, A_W_O), *win = ptr<void>(a, A_W_IN),
             *wout = ptr<void>(a, A_W_OUT), *n1 = ptr<void>(a, A_N1), *n2 = ptr<void>(a, A_N2);
  const int *ss = ptr<int>(a, A_SEQ_START), *se = ptr<int>(a, A_SEQ_END), *pos = ptr<int>(a, A_POS);
  const float *cosp = ptr<float>(a, A_COS), *sinp = ptr<float>(a, A_SIN);
  const Saved s(ptr<void>(a, A_BUF), T, C, I, H, norm1, true);
  const void* dy = ptr<void>(a, A_Y);
  const Call k{ptr<int>(a, A_STATUS), ptr<CUstream_st>(a, A_STREAM)};
  void* dx = ptr<void>(a, BWD_DX);
  const Scratch d(ptr<void>(a, BWD_SCRATCH), T, C, I, H);
  float *g_qkv = ptr<float>(a, BWD_G_QKV), *g_o = ptr<float>(a, BWD_G_O), *g_in = ptr<float>(a, BWD_G_IN), *g_out = ptr<float>(a, BWD_G_OUT),
        *g_n1 = ptr<float>(a, BWD_G_N1), *g_n2 = ptr<float>(a, BWD_G_N2);
  const int mode = static_cast<int>(a[BWD_ATTENTION_MODE]);
  // MLP
  TRY(k.out(dy, wout, d.dpre, s.pre, T, I, C, I, 2 * I, 2 * I, 1, EPI_SWIGLU_BWD));
  TRY(k.wgrad(dy, s.hs, g_out, T, C, I, static_cast<int>(a[BWD_SPLITS_OUT])));
  TRY(k.wgrad(d.dpre, s.h2, g_in, T, 2 * I, C, static_cast<int>(a[BWD_SPLITS_IN])));
  TRY(k.out(d.dpre, win, d.dh, nullptr, T, C, 2 * I, C, C, 0, 1, EPI_STORE));
  TRY(fn.norm_bwd(d.dh, s.x1, nullptr, n2, rms ? nullptr : s.mean2, s.rstd2, dy, d.dx1, g_n2, nullptr, T, C, 0, rms,
                  k.stream));
  // attention
  float* dq = mode == 3 ? nullptr : d.dq;
  TRY(fn.delta(d.dx1, wo, d.d_o, s.o, d.delta, dq, T, HD, C, C, HD, HD, HD, 1, k.status, k.stream));
  TRY(k.wgrad(d.dx1, s.o, g_o, T, C, HD, static_cast<int>(a[BWD_SPLITS_O])));
  TRY(fn.fa_bwd(s.qkv, nullptr, d.d_o, s.lse, d.dqkv, dq, d.delta, ss, se, T, H, 64, window,
                static_cast<float>(scale), pos, cosp, sinp, 0, mode, k.status, k.stream));
  TRY(k.wgrad(d.dqkv, norm1 ? s.h1 : x, g_qkv, T, 3 * HD, C, static_cast<int>(a[BWD_SPLITS_QKV])));
  if (!norm1)   // the layer input enters the projection and the residual: both gradients in one epilogue
    return k.out(d.dqkv, wqkv, dx, d.dx1, T, C, 3 * HD, C, C, C, 1, EPI_ADD);
  TRY(k.out(d.dqkv, wqkv, d.dh, nullptr, T, C, 3 * HD, C, C, 0, 1, EPI_STORE));
  return fn.norm_bwd(d.dh, x, nullptr, n1, rms ? nullptr : s.mean1, s.rstd1, d.dx1, dx, g_n1, nullptr, T, C, 0, rms, k.stream);
}

// `layers` consecutive layers: their argument arrays and (eps1, eps2, scale) triples one after the other. Backward calls go from
// the last array to the first.
extern "C" int nplm_layers_fwd(const long long* a, const double* d, int layers) {
  for (int l = 0; l < layers; ++l) TRY(nplm_layer_fwd(a + l * FWD_ARGS, d[3 * l], d[3 * l + 1], d[3 * l + 2]));
  return 0;
}

extern "C" int nplm_layers_bwd(const long long* a, const double* d, int layers) {
  for (int l = layers - 1; l >= 0; --l) TRY(nplm_layer_bwd(a + l * BWD_ARGS, d[3 * l + 2]));
  return 0;
}
