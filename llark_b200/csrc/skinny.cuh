// Products with few rows: C[M, N] = f(A[M, K] W[N, K]^T), M <= 64, bf16 operands, fp32 sums (skinny.cu). The decode steps'
// linears (gemv.cu, seq_ops.cu, gemm_tcgen05.cu) and routed experts (seq_moe.cu) launch it.
#pragma once
#include "common.cuh"

namespace llark {
namespace skinny {

constexpr int kMaxRows = 64;

enum { kActNone = 0, kActRelu2, kActReluGlu, kActClampGlu, kActSiluGlu, kActRope, kActSwiglu };

struct Args {
    const __nv_bfloat16 *A, *W;
    long long lda, ldw;
    void* C;
    long long ldc;
    int c_fp32;
    const void* bias;  // [N] or NULL; float if bias_fp32
    int bias_fp32;
    const void* R;     // residual of C's type, or NULL
    long long ldr;
    int M, N, K;       // N: rows of W (kActSiluGlu, kActSwiglu: gate rows, then as many up rows: N counts both)
    int act;
    float limit, slope;
    // kActRope: columns below rope_cols are rotated per 128-wide head, position = (first + row) % rope_S
    const __nv_bfloat16 *rope_cos, *rope_sin;
    int rope_S, rope_cols, first;
    // Routed experts: tile list of (expert, first sorted row, rows <= 64), its length in meta[0] (at most max_tiles); rows of A
    // are perm[sorted row] / top (NULL: the sorted row itself), W holds one [N, K] block per expert, sums are multiplied by
    // in_wts[perm[sorted row]] when given. M is not used.
    const int *tiles, *meta, *perm;
    int max_tiles, top;
    const float* in_wts;
    // The weights were there before the kernel in front of this one began (launches of one call behind each other): they are
    // fetched before that kernel has ended. Otherwise they are only asked for in L2, which a later write does no harm to.
    int weights_there;
};

// Whether launch() takes these operands: 16-byte pieces of A and W
inline bool fits(const void* A, long long lda, const void* W, long long ldw, int K) {
    return K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0 &&
           ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
}
cudaError_t launch(const Args& a, cudaStream_t st);

}  // namespace skinny
}  // namespace llark
