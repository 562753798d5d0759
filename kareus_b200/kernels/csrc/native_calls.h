// Entry points of libkareus_b200.so that the extension module calls (torch/fastcall.cpp).  The sources that define them include
// this too, so that a changed signature does not compile until both sides have it.
#pragma once
#include <cuda_runtime.h>

extern "C" {
int kb_gemm_work_bf16(const void* A, const void* B, void* C, int M, int N, int K, int a_mn, int lda, int b_mn, int ldb, int ldc,
                      int num_sms, float* work, int* status, cudaStream_t stream);
long kb_gemm_scratch_floats(int M, int N, int K, int b_mn, int num_sms);
int kb_gemm_accum_bf16(const void* A, const void* B, float* C, int M, int N, int K, int a_mn, int lda, int b_mn, int ldb,
                       int ldc, int num_sms, float* work, int* status, cudaStream_t stream);
long kb_gemm_accum_scratch_floats(int M, int N, int K, int num_sms);
int kb_flash_attn_fwd(const void* q, long qs_s, long qs_b, long qs_g, long qs_r, const void* k, long ks_s, long ks_b,
                      long ks_g, const void* v, long vs_s, long vs_b, long vs_g, void* out, float* lse, int sq, int skv, int b,
                      int g, int rep, int d, float scale, int causal, int q_offset, int* status, cudaStream_t stream);
long kb_flash_attn_bwd_scratch_floats(int sq, int skv, int b, int g, int rep, int d);
int kb_flash_attn_bwd(const void* q, long qs_s, long qs_b, long qs_g, long qs_r, const void* k, long ks_s, long ks_b,
                      long ks_g, const void* v, long vs_s, long vs_b, long vs_g, const void* o, const void* dO,
                      const float* lse, void* dq, long dqs_s, long dqs_b, long dqs_g, long dqs_r, void* dk, long dks_s,
                      long dks_b, long dks_g, void* dv, long dvs_s, long dvs_b, long dvs_g, float* work, int sq, int skv,
                      int b, int g, int rep, int d, float scale, int causal, int q_offset, int* status, cudaStream_t stream);
}
