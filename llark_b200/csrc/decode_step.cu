// A decode step's layers in one call: the launches of the Llama decoder layer for up to 64 rows (one token per request), layer after
// layer on the caller's stream. The kernels and their order are those of the single entry points; what it saves is the host's part of seven
// calls a layer (380 us of a step of two layers, 247 us of kernels). The first kernel begins when all before it on the stream has
// ended; the others begin early and fetch weights (what lies there is then no longer written) while those before them end.
#include "skinny.cuh"

#include <math.h>

namespace llark {
extern thread_local int g_last_cuda_error;
}
using namespace llark;

extern "C" long long llark_decode_scratch(int B, int H, int I) {  // normed rows | q k v | attention | middle | gate times up, bf16
    return (long long)B * (6LL * H + I) * 2 + 5 * 256;
}

extern "C" int llark_decode_layers(const LlarkDecodeLayer* layers, int n_layers, void* x, void* scratch, const void* cos_row,
                                   const void* sin_row, int pos, int B, int s_max, int H, int I, int n_heads, float eps, float* rstd,
                                   cudaStream_t st) {
    if (!layers || n_layers <= 0 || !x || !scratch || !cos_row || !sin_row || !rstd || B <= 0 || B > 64 || H <= 0 || I <= 0 || H % 8 || I % 8 ||
        n_heads <= 0 || H != n_heads * 128 || ((reinterpret_cast<uintptr_t>(cos_row) | reinterpret_cast<uintptr_t>(sin_row)) & 15))
        return LLARK_EINVAL;
    char* at = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~uintptr_t(255));
    auto take = [&](long long cols) {
        void* p = at;
        at += (B * cols * 2 + 255) / 256 * 256;
        return p;
    };
    void *xn = take(H), *qkv = take(3LL * H), *attn = take(H), *mid = take(H), *act = take(I);
    const float scale = (float)(1.0 / sqrt(128.0));
    // C[B, N] = f(A[B, K] W[N, K]^T) (+ R)
    auto product = [&](const void* A, const void* W, void* C, long long ldc, const void* R, int N, int K, int act) {
        if (!skinny::fits(A, K, W, K, K) || ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(R)) & 15)) return (int)LLARK_EINVAL;
        skinny::Args a = {};
        a.A = (const __nv_bfloat16*)A, a.lda = K, a.W = (const __nv_bfloat16*)W, a.ldw = K;
        a.C = C, a.ldc = ldc, a.R = R, a.ldr = ldc;
        a.M = B, a.N = N, a.K = K, a.act = act;
        a.rope_cos = (const __nv_bfloat16*)cos_row, a.rope_sin = (const __nv_bfloat16*)sin_row;
        a.rope_S = 1, a.rope_cols = 2 * H;  // every row at the tables' first position
        a.weights_there = 1;
        const cudaError_t e = skinny::launch(a, st);
        if (e != cudaSuccess) g_last_cuda_error = (int)e;
        return (int)(e == cudaSuccess ? LLARK_OK : LLARK_ECUDA);
    };
    for (int l = 0; l < n_layers; ++l) {
        const LlarkDecodeLayer& w = layers[l];
        int rc = rmsnorm_rows(x, w.norm1, xn, rstd, B, H, eps, l > 0, st);
        if (!rc) rc = product(xn, w.qkv, qkv, 3LL * H, nullptr, 3 * H, H, skinny::kActRope);
        if (!rc) rc = llark_attn_decode_packed(qkv, 3LL * H, w.k, w.v, pos, attn, B, s_max, n_heads, 128, scale, st);
        if (!rc) rc = product(attn, w.o, mid, H, x, H, H, skinny::kActNone);
        if (!rc) rc = rmsnorm_rows(mid, w.norm2, xn, rstd, B, H, eps, true, st);
        if (!rc) rc = product(xn, w.gate_up, act, I, nullptr, 2 * I, H, skinny::kActSwiglu);
        if (!rc) rc = product(act, w.down, x, H, mid, H, I, skinny::kActNone);  // x has been read
        if (rc) return rc;
    }
    return LLARK_OK;
}
