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
  EPI_SWIGLU_BWD = 8,  // acc = gradient of the SwiGLU output h = silu(gate) * value, N wide;
                       // R = the pre-activations [value | gate] (bf16, 2N wide); C (bf16, 2N wide) =
                       // [acc * silu(gate) | acc * value * silu'(gate)], the gradient of R
};
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
int nplm_gemm_bf16_delta(const void* A, const void* B, void* C, const void* R, float* delta, int M, int N, int K, int lda,
                         int ldb, int ldc, int ldr, int b_mn, int* status, cudaStream_t stream);
int nplm_norm_fwd(const void* x, const int* ids, const void* w, void* y, float* mean, float* rstd, int T, int C, float eps,
                  int rms, cudaStream_t st);
int nplm_norm_bwd(const void* dy, const void* x, const int* ids, const void* w, const float* mean, const float* rstd,
                  const void* dres, void* dx, float* dw, float* dtable, int T, int C, int V, int rms, cudaStream_t st);
int nplm_fa_fwd_ws(const void* qkv, void* out, float* lse, const int* seq_start, const int* seq_end, int T, int H, int D,
                   int window, float scale, int max_ctas, int* status, cudaStream_t st);
int nplm_fa_bwd_ws_mode(const void* qkv, const void* out, const void* dout, const float* lse, void* dqkv, float* dq_acc,
                        float* delta, const int* seq_start, const int* seq_end, int T, int H, int D, int window,
                        float scale, const int* rope_pos, const float* rope_cos, const float* rope_sin, int max_ctas,
                        int mode, int* status, cudaStream_t st);
}
