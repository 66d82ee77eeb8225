// C interface of the model kernels (libpiccl_ops.so) that the native training step calls; each returns 0 or an error code.
#pragma once
#include <stddef.h>
#ifdef __cplusplus
extern "C" {
#endif
int piccl_ops_embed_fwd(const long long* idx, const void* wte, const void* wpe, void* out, int rows, int S, int C, void* stream);
int piccl_ops_ln_fwd(const void* x, const void* res, const void* gamma, const void* beta, void* sum_out, void* y, float* mean, float* rstd, int rows, int C, float eps, void* stream);
int piccl_ops_ln_bwd_parts(int rows, int C);
int piccl_ops_ln_bwd(const void* dy, const void* xin, const void* gamma, const float* mean, const float* rstd, const void* dres, void* dx, float* part, int with_dsum, int rows, int C, void* stream);
int piccl_ops_gemm(int layout, int epi, const void* A, const void* B, void* C, void* pre, const void* bias, const void* aux, float* part, void* ws, size_t ws_bytes, int M, int N, int K, void* stream);
int piccl_ops_bias_gelu_fwd(const void* h, const void* bias, void* h_out, void* g, long long rows, int C, void* stream);
int piccl_ops_gelu_bwd(const void* dg, const void* h, void* dh, float* part, long long rows, int C, void* stream);
int piccl_ops_colsum(const void* x, void* out, float* workspace, int rows, int C, int rows_per_block, int accumulate, void* stream);
int piccl_ops_col_parts(long long rows, int C);
int piccl_ops_qkv_grad(const void* const* g, const long long* strides, void* dqkv, float* part, int B, int S, int H, int D, void* stream);
struct piccl_finish_job { const float* part; void* out; int nparts, C, accumulate, pad; };
int piccl_ops_finish_parts(const void* jobs, int n, void* stream);
int piccl_ops_ce(void* logits, const long long* targets, float* loss, int rows, int V, int Vp, float gscale, int grad, void* stream);
int piccl_ops_mean(const float* x, float* out, int n, void* stream);
int piccl_ops_pass_loss(const float* rows, float* loss, int n, void* stream);
int piccl_ops_wpe_bwd(const void* dx, void* dwpe, int B, int S, int rows, int C, int accumulate, void* stream);
int piccl_ops_wte_bwd_rows(const long long* idx, const void* dx, float* stage, int* owner, void* dwte, int rows, int C, void* stream);
int piccl_ops_attn_pays(int backward, int B, int S, int H, int sms);
int piccl_ops_attn_rows(int S);
int piccl_ops_attn_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, void* stream);
int piccl_ops_attn_parts(int B, int S);
int piccl_ops_attn_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* scratch, void* dqkv, float* part, int B, int S, int H, void* stream);
#ifdef __cplusplus
}
#endif
