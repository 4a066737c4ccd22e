// GEMMs of a few tokens (gemm_skinny_sm100.cu), called by the entry points of gemm_sm100.cu and gemm_wq_sm100.cu.
// `*_applies` says whether sizes and alignment allow the kernel and make it the faster one; the calls return the entry
// points' codes.  `settled`: W, its scales and the bias are not written by the launch that precedes the call on the stream; they
// may then be read while that one still runs.
#pragma once
#include <cuda_runtime_api.h>

namespace tgi {

bool skinny_bf16_applies(const void* X, const void* W, int M, int N, int K, int ldx, int max_ctas);
int skinny_bf16(const void* X, int ldx, const void* W, void* C, const void* bias, int M, int N, int K, int max_ctas, int settled,
                int* status, cudaStream_t stream);

bool skinny_fp8_applies(const void* X, const float* xs_t, const void* W, int M, int K);
int skinny_fp8(const void* X, const float* xs_t, int xs_pitch, const void* W, const float* wscale, void* C, const void* bias,
               int M, int N, int K, int max_ctas, int settled, int* status, cudaStream_t stream);

bool skinny_int4_applies(const void* X, const void* W, const void* scale, const void* zp, int M, int N, int K, int group);
int skinny_int4(const void* X, const void* W, const void* scale, const void* zp, int group, void* C, const void* bias, int M, int N,
                int K, int max_ctas, int settled, int* status, cudaStream_t stream);

}  // namespace tgi
