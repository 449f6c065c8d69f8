// The C entry points that the C++ autograd functions call (autograd_native.cpp), declared once: the kernel sources that define them and the
// module that looks them up both include this file, so a changed argument list is a compile error on either side, and both rebuild.
#pragma once
#include <cuda_runtime_api.h>

extern "C" {
// gemm_sm100.cu
int sb_gemm_bf16(const void* A, const void* B, void* C, const void* bias, const void* residual, int M, int N, int K, int lda, int ldb,
                 int ldc, int ldr, int a_mn, int b_mn, int beta, unsigned int* status, int max_ctas, cudaStream_t stream);
int sb_gemm_last_error_detail();
// attn_sm100.cu
int sb_attn_last_encode_result();
// elementwise.cu
int sb_colsum(const void* x, float* out, int T, int N, cudaStream_t st);
int sb_rmsnorm_fwd(const void* x, const void* w, void* y, float* a_out, int T, int D, float eps, int form, cudaStream_t st);
int sb_rmsnorm_bwd_blocks(int T, int D);
int sb_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* a_in, const void* gres, void* dx, void* dw, float* partial,
                   int T, int D, float eps, int form, cudaStream_t st);
int sb_glu_fwd(const void* ab, void* h, long long T, int F, int act, cudaStream_t st);
int sb_glu_bwd(const void* ab, const void* dh, void* dab, long long T, int F, int act, cudaStream_t st);
int sb_ce_fwd(const void* logits, const long long* labels, float* loss, float* lse, long long T, int V, cudaStream_t st);
int sb_ce_bwd(const void* logits, const long long* labels, const float* lse, const float* g, void* dlogits, long long T, int V,
              cudaStream_t st);
// conv.cu
int sb_dwconv_fwd(const void* x, const void* halo, const float* w, void* y, int B, int L, int C, int K, cudaStream_t st);
int sb_dwconv_fwd_taps(const void* x, const void* halo, const void* w, int w_bf16, float* wf, void* y, int B, int L, int C, int K,
                       cudaStream_t st);
int sb_dwconv_bwd(const void* x, const void* halo, const float* w, const void* dy, void* dx, void* dhalo, float* dw, int B, int L, int C,
                  int K, cudaStream_t st);
int sb_se_fwd(const void* feat, const void* halo, const float* w, void* z, int B, int L, int D, int G, int K, int pregate, int postgate,
              cudaStream_t st);
int sb_se_fwd_taps(const void* feat, const void* halo, const void* w, int w_bf16, float* wf, void* z, int B, int L, int D, int G, int K,
                   int pregate, int postgate, cudaStream_t st);
int sb_se_bwd(const void* feat, const void* halo, const float* w, const void* dz, void* dfeat, void* dhalo, float* dw, int B, int L, int D,
              int G, int K, int pregate, int postgate, cudaStream_t st);
// mr_conv.cu
int sb_mr_fwd(const void* feat, const void* halo, const float* h, const float* bias, void* z, void* ysave, int B, int L, int D, int G,
              int K, cudaStream_t st);
int sb_mr_bwd(const void* feat, const void* halo, const float* h, const float* bias, const void* dz, const void* ysave, void* dfeat,
              void* dhalo, float* dh, float* dbias, int B, int L, int D, int G, int K, cudaStream_t st);
// mr_conv_tc.cu
int sb_mr_tc_fwd(const void* feat, const void* halo, const float* h, const float* bias, void* z, int B, int L, int D, int G, int K,
                 cudaStream_t st);
int sb_mr_tc_bwd(const void* feat, const void* halo, const float* h, const float* bias, const void* dz, void* dfeat, void* dhalo, float* dh,
                 float* dbias, int B, int L, int D, int G, int K, cudaStream_t st);
// mr_conv_umma.cu
int sb_mr_umma_fwd(const void* feat, const float* h, const float* bias, void* z, int B, int L, int D, int G, int K, unsigned int* status,
                   cudaStream_t st);
int sb_mr_umma_bwd(const void* feat, const float* h, const float* bias, const void* dz, void* dfeat, float* dh, float* dbias, int B, int L,
                   int D, int G, int K, unsigned int* status, cudaStream_t st);
// li_scan.cu
int sb_li_fwd_tiled(const void* feat, const float* gamma, const float* p, const float* R, const float* bias, const float* state_in,
                    float* state_out, float* modal, float* S, void* z, int B, int L, int D, int O, int TC, cudaStream_t st);
int sb_li_bwd_tiled_chunk();
int sb_li_bwd_tiled(const void* feat, const void* dz, const float* modal, const float* bias, const float* state_in, const float* dstate_out,
                    float* S, float* A, float* dRp, float* dBp, void* dfeat, float* dR, float* dll, float* db, float* dstate_in, int B,
                    int L, int D, int O, cudaStream_t st);
// attn_sm100.cu
int sb_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int H, int Lq, int Lk, const long long* q_str,
                const long long* k_str, const long long* v_str, const long long* o_str, int causal, float scale, unsigned int* status,
                cudaStream_t stream);
int sb_attn_bwd(const void* go, const void* q, const void* k, const void* v, const void* out, const float* lse, const float* glse,
                float* stats, float* dq_acc, void* dq, void* dk, int B, int H, int Lq, int Lk, void* dv, const long long* g_str,
                const long long* q_str, const long long* k_str, const long long* v_str, const long long* o_str, const long long* dq_str,
                const long long* dk_str, const long long* dv_str, int causal, float scale, unsigned int* status, cudaStream_t stream);
int sb_attn_rope(const void* const* src, void* const* dst, const long long* src_str, const long long* dst_str, const int* src_f32, int n,
                 const float* cs, const float* sn, int B, int L, int H, int rd, int inverse, cudaStream_t stream);
}
