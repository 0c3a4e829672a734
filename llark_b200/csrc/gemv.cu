// Skinny linear layer for the single-token decode step of the generation path:
//   C[M, N] = A[M, K] . W[N, K]^T (+ bias[N]) (+ R[M, N]),  M <= 8 rows, bf16 in / out, fp32 accumulation.
// With M = batch (1 for the reference's inference scripts) the op is a pure stream of the weight matrix (N * K * 2 bytes,
// 13.5 GB per token over a 7B model): the few-rows product of skinny.cu. The engines reach it through llark_gemm_ex; this entry is kept for
// programs that call the C interface.
#include "skinny.cuh"

namespace llark {
extern thread_local int g_last_cuda_error;
}

using namespace llark;

extern "C" int llark_gemv(const void* A, long long lda, const void* W, long long ldw, void* C, long long ldc,
                          const void* bias, const void* R, long long ldr, int M, int N, int K, cudaStream_t st) {
    if (M <= 0 || M > 8 || N <= 0 || K <= 0 || (K & 7) || (lda & 7) || (ldw & 7) || lda < K || ldw < K || ldc < N ||
        (R && ldr < N))
        return LLARK_EINVAL;
    if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) return LLARK_EINVAL;
    skinny::Args a = {};
    a.A = (const __nv_bfloat16*)A, a.lda = lda, a.W = (const __nv_bfloat16*)W, a.ldw = ldw;
    a.C = C, a.ldc = ldc, a.bias = bias, a.R = R, a.ldr = ldr;
    a.M = M, a.N = N, a.K = K;
    cudaError_t e = skinny::launch(a, st);
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}
