// A decode step's layers in one call: the launches of the Llama decoder layer for up to 64 rows (one token per request), layer after
// layer on the caller's stream. The kernels, their order and their arguments are those of the single entry points; what it saves is the
// host's part of seven calls a layer (380 us of a step of two layers, 247 us of kernels).
#include "common.cuh"

#include <math.h>

extern "C" long long llark_decode_scratch(int B, int H, int I) {  // normed rows | q k v | attention | middle | gate times up, bf16
    return (long long)B * (6LL * H + I) * 2 + 5 * 256;
}

extern "C" int llark_decode_layers(const LlarkDecodeLayer* layers, int n_layers, void* x, void* scratch, const void* cos_row,
                                   const void* sin_row, int pos, int B, int s_max, int H, int I, int n_heads, float eps, float* rstd,
                                   cudaStream_t st) {
    if (!layers || n_layers <= 0 || !x || !scratch || !cos_row || !sin_row || !rstd || B <= 0 || B > 64 || H <= 0 || I <= 0 || H % 8 || I % 8 ||
        n_heads <= 0 || H != n_heads * 128)
        return LLARK_EINVAL;
    char* at = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~uintptr_t(255));
    auto take = [&](long long cols) {
        void* p = at;
        at += (B * cols * 2 + 255) / 256 * 256;
        return p;
    };
    void *xn = take(H), *qkv = take(3LL * H), *attn = take(H), *mid = take(H), *act = take(I);
    const LlarkGemmEpilogue rope = {LLARK_EPI_ROPE, cos_row, sin_row, 0, 1, 2 * H, 0.f, 0.f};  // every row at the tables' first position
    const LlarkGemmEpilogue swiglu = {LLARK_EPI_SWIGLU, nullptr, nullptr, 0, 0, 0, 0.f, 0.f};
    const float scale = (float)(1.0 / sqrt(128.0));
    for (int l = 0; l < n_layers; ++l) {
        const LlarkDecodeLayer& w = layers[l];
        int rc = llark_rmsnorm_fwd(x, w.norm1, xn, rstd, B, H, eps, st);
        if (!rc) rc = llark_gemm_ex(xn, 0, H, w.qkv, 0, H, qkv, 3LL * H, 0, nullptr, 0, nullptr, 0, B, 3 * H, H, 0, 0, &rope, st);
        if (!rc) rc = llark_attn_decode_packed(qkv, 3LL * H, w.k, w.v, pos, attn, B, s_max, n_heads, 128, scale, st);
        if (!rc) rc = llark_gemm(attn, 0, H, w.o, 0, H, mid, H, 0, nullptr, 0, x, H, B, H, H, 0, 0, st);
        if (!rc) rc = llark_rmsnorm_fwd(mid, w.norm2, xn, rstd, B, H, eps, st);
        if (!rc) rc = llark_gemm_ex(xn, 0, H, w.gate_up, 0, H, act, I, 0, nullptr, 0, nullptr, 0, B, 2 * I, H, 0, 0, &swiglu, st);
        if (!rc) rc = llark_gemm(act, 0, I, w.down, 0, I, x, H, 0, nullptr, 0, mid, H, B, H, I, 0, 0, st);  // x has been read
        if (rc) return rc;
    }
    return LLARK_OK;
}
