// C entry points that host code of this package calls directly (layer.cpp): declared once, for the files that define
// them and for the one that calls them, so that a change of a signature on one side does not compile on the other.
#pragma once

typedef struct CUstream_st* cudaStream_t;   // (as the CUDA runtime declares it; host-only files do without its headers)

namespace nplm {
// Epilogue forms of the bf16 GEMM.
enum : int {
  EPI_STORE = 0,       // C(bf16) = acc
  EPI_ADD = 1,         // C(bf16) = acc + R(bf16)
  EPI_ATOMIC_F32 = 2,  // C(fp32) += acc   (split-K capable; used for weight gradients)
  EPI_GELU = 3,        // C(bf16) = gelu(acc) (erf form); also writes the pre-activation to R when R != null
  EPI_RELU = 7,        // as EPI_GELU with ReLU. A form of its own: chosen at run time inside EPI_GELU it kept that
                       // epilogue's code and registers (55 424 x 4096 x 1024: 488 -> 350 us)
  EPI_STORE_F32 = 4,   // C(fp32) = acc
  EPI_SWIGLU = 5,      // B tile = [value rows | gate rows]; C(bf16, N/2 wide) = silu(gate)*value,
                       // pre-activations (bf16, N wide) written to R when R != null
  EPI_ROPE = 6,        // C(bf16) = acc with rotary embedding applied to every 64-wide head whose
                       // first column is < rope_cols (the q and k parts of a fused QKV projection)
  EPI_STORE_DELTA = 9, // C(bf16) = acc, and delta[col / 64][row] = sum over each 64-column head of
                       // bf16(acc) * R (the attention backward's rowsum(dO * O), R = O)
  EPI_AXPBY = 10,      // C(bf16) = alpha * acc + beta * R(bf16, may be null); stacks of equal problems only
  EPI_SWIGLU_BWD = 8,  // acc = gradient of the SwiGLU output h = silu(gate) * value, N wide;
                       // R = the pre-activations [value | gate] (bf16, 2N wide); C (bf16, 2N wide) =
                       // [acc * silu(gate) | acc * value * silu'(gate)], the gradient of R
};

// Whether a bf16-output GEMM on 256-wide tiles runs on CTA pairs by default (ops/kernels.py has the same rule, and a test
// compares the two). A pair's tile takes a third less operand traffic per FLOP but costs about 0.6 us more from launch
// to store and moves 256 rows at a time, so it pays once the tiles fill more than one wave of 148, or several where the
// contraction is short. Graph-timed single / pair, us:
//   store, add, GELU, ReLU: 1024 columns of K = 1024, 3 072 rows (96 tiles) 12.4 / 12.8, 4 864 (152) 17.8 / 17.3, 55 424
//     102 / 91; K = 512, 32 768 x 512 (512 tiles) 25.0 / 25.6, 55 424 x 512 (866) 37.2 / 36.9
//   SwiGLU: 4096 of 1024, 1 024 rows (128) 12.1 / 13.0, 1 536 (192) 17.8 / 17.3, 55 424 332 / 288; 2048 of 512, 4 864 rows
//     (304) 15.7 / 15.9, 6 144 (384) 16.4 / 16.3
//   RoPE (whose pair form has eight epilogue warps, and a stage less): 3072 of 1024, 6 144 rows (576) 31.7 / 32.8, 8 704
//     (816) 44.7 / 44.3, 55 424 270 / 249; 2304 of 768, 32 768 rows (2 304) 97.1 / 97.7, 55 424 (3 897) 162 / 162; 1536 of
//     512, 236 rows 9.3 / 12.2, 55 424 82.6 / 88.6
//   SwiGLU backward (eight epilogue warps): 1 row 12.5 / 11.0, 8 704 x 2048 of 1024 57 / 46, 55 424 292 / 237
inline bool gemm_pair_pays(long long M, long long N, long long K, int epi) {
  const long long tiles = (M + 127) / 128 * ((N + 255) / 256);
  if (epi == EPI_SWIGLU_BWD || epi == EPI_STORE_DELTA) return true;
  if (epi == EPI_ROPE) return K >= 1024 ? tiles > 740 : K >= 768 && tiles > 2600;
  return K >= 768 ? tiles > 148 : tiles * K > (epi == EPI_SWIGLU ? 190000 : 400000);
}

// Tile width (columns) of a bf16-output GEMM by default (ops/kernels.py has the same rule, and a test compares the two): the
// narrowest tiles that one wave of 148 CTAs covers. Below a wave a GEMM takes as long as one tile, i.e. launch, first
// loads, K / 64 steps and the epilogue of a tile's columns one 64-column chunk after the other; a narrow tile has fewer of
// those and loads less a step, and the idle multiprocessors take the other columns. Past a wave the wide tiles'
// lower operand traffic wins. Graph-timed us, 64 / 128 / 256 columns:
//   add, 512 columns of K = 512: 236 rows 5.1 / 5.8 / 8.1, 2 050 (136 tiles of 64) 5.4 / 6.1 / 8.5, 4 600 (144 of 128) 7.8 /
//     6.5 / 8.6, 8 160 (128 of 256) 12.0 / 8.9 / 9.1; of K = 1024: 236 rows 6.8 / 7.5 / 10.3
//   RoPE, 1536 of 512: 236 rows 6.6 / 7.0 / 8.5, 1 000 (96 of 128) 9.1 / 7.2 / 8.7, 2 050 (102 of 256) 11.8 / 10.2 / 9.0
//   SwiGLU (a tile's columns are value and gate, so 128 at least), 2048 of 512: 236 rows - / 6.0 / 7.7, 1 000 (128 of 128)
//     - / 6.8 / 8.1, 2 050 (136 of 256) - / 9.1 / 8.8
//   GELU, 512 of 512: 236 rows 7.5 / 8.9 / 12.5; data gradient, 512 of 2048: 236 rows 9.7 / 10.1 / 13.0
inline int gemm_tile_width(long long M, long long N, int epi) {
  if (epi == EPI_SWIGLU_BWD || epi == EPI_STORE_DELTA || epi == EPI_ATOMIC_F32 || epi == EPI_STORE_F32)
    return N >= 256 || epi == EPI_SWIGLU_BWD || epi == EPI_STORE_DELTA ? 256 : 128;
  const long long rows = (M + 127) / 128;
  if (epi != EPI_SWIGLU && rows * ((N + 63) / 64) <= 148) return 64;
  return (N < 256 && epi != EPI_SWIGLU) || rows * ((N + 127) / 128) <= 148 ? 128 : 256;
}
}  // namespace nplm

extern "C" {
int nplm_gemm_bf16(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb, int ldc,
                   int ldr, int a_mn, int b_mn, int epi, int splits, int bn, int max_ctas, int direct_epilogue,
                   const int* rope_pos, const float* rope_cos, const float* rope_sin, int rope_cols, int* status,
                   cudaStream_t stream);
int nplm_gemm_bf16_pair(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb,
                        int ldc, int ldr, int a_mn, int b_mn, int epi, int splits, int direct_epilogue,
                        const int* rope_pos, const float* rope_cos, const float* rope_sin, int rope_cols, int* status,
                        cudaStream_t stream);
// clear (fp32 [M][N], may be null) is set to zero.
int nplm_gemm_bf16_delta(const void* A, const void* B, void* C, const void* R, float* delta, float* clear, int M, int N, int K,
                         int lda, int ldb, int ldc, int ldr, int b_mn, int* status, cudaStream_t stream);
int nplm_norm_fwd(const void* x, const int* ids, const void* w, void* y, float* mean, float* rstd, int T, int C, float eps,
                  int rms, cudaStream_t st);
int nplm_norm_bwd(const void* dy, const void* x, const int* ids, const void* w, const float* mean, const float* rstd,
                  const void* dres, void* dx, float* dw, float* dtable, int T, int C, int V, int rms, cudaStream_t st);
int nplm_fa_fwd_ws(const void* qkv, void* out, float* lse, const int* seq_start, const int* seq_end, int T, int H, int D,
                   int window, float scale, int max_ctas, int* status, cudaStream_t st);
int nplm_fa_bwd_ws_zeroed(const void* qkv, const void* out, const void* dout, const float* lse, void* dqkv, float* dq_acc,
                          float* delta, const int* seq_start, const int* seq_end, int T, int H, int D, int window,
                          float scale, const int* rope_pos, const float* rope_cos, const float* rope_sin, int max_ctas,
                          int mode, int* status, cudaStream_t st);
}
