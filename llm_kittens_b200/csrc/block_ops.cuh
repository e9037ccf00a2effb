// Entry points that are called from another file of the library (forward.cu). The files that define them include this too, so
// that a signature that is changed in one place only does not compile.
#pragma once
#include "common.cuh"

LLMK_API int llmk_layernorm_fwd(void* normed, void* mean, void* rstd, const void* inp, const void* weight, const void* bias, int N, int C,
                                void* stream);
LLMK_API int llmk_rmsnorm_fwd(void* normed, void* rstd, const void* inp, const void* weight, int N, int C, float eps, void* stream);
LLMK_API int llmk_gemm(int mode, int epi, const void* A, const void* B, void* C, void* C2, const void* bias, const void* aux, int M, int N,
                       int K, void* workspace, long workspace_bytes, int* status, int max_ctas, void* stream);
LLMK_API int llmk_gemm_qkv_rope(const void* A, const void* B, void* C, int M, int N, int K, const void* rope, int T, int rope_cols, int HS,
                                int* status, int max_ctas, const void* b_ready, long b_chunk, int b_tick, long limit_ns, void* stream);
LLMK_API int llmk_gemm_swiglu(const void* A, const void* Wup, const void* Wgate, void* act, void* up, void* gate, int M, int H, int K,
                              int* status, int max_ctas, const void* up_ready, const void* gate_ready, long b_chunk, int b_tick,
                              long limit_ns, void* stream);
LLMK_API int llmk_rope_qk(void* qkv, const void* freqs, int B, int T, int NH, int NKVH, int HS, int interleaved, int inverse, void* stream);
LLMK_API int llmk_attention_fwd(void* out, void* lse, const void* qkv, int B, int T, int NH, int NKVH, int HS, void* stream);
LLMK_API int llmk_attention_fwd_tc(void* out, void* lse, const void* qkv, int B, int T, int NH, int NKVH, int HS, int* status, void* stream);
