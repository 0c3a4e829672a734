// Attention of single-token steps: one query per request against the keys and values of its store (attn_step.cu).
#pragma once
#include "common.cuh"

namespace llark {
namespace attnstep {

struct Args {
    const __nv_bfloat16 *q, *k, *v;  // q [B, H * D]; k, v: entry e of a store at (e * G + g) * D
    __nv_bfloat16* out;              // [B, out_ld]
    long long out_ld;
    int B, H, G, D;
    // Which keys row b sees. lens given: entries b * cap + (0 .. min(lens[b], cap) - 1). Otherwise the row is a token of request
    // r = tok_seq[b] at position p = pos0[r] + b - cu[r], sees lo .. p with lo = max(0, p - window + 1), or the start of p's block
    // of `chunk` positions, and position j is entry slot[r] * cap + j % cap.
    const int *lens, *tok_seq, *cu, *pos0, *slot;
    // packed given (with neither lens nor tok_seq; G = H): row b of packed [B, packed_ld] holds q | k | v of the new token, which is
    // entry n_keys - 1 of every row's cap entries: its key and value are stored there (k_new, v_new are k and v, to be written)
    // before they are read. q is then not used.
    const __nv_bfloat16* packed;
    long long packed_ld;
    __nv_bfloat16 *k_new, *v_new;
    int n_keys;
    int cap, window, chunk;
    const float* scale_h;  // [H], or NULL: scale
    float scale, softcap, out_scale;
    const float* sink;     // [H] or NULL
    const float* gate;     // [B, gate_ld] or NULL
    long long gate_ld;
    int gate_per_head;
    const float* vfreq;    // [D / 2] or NULL: outputs are turned back by the query's position
    int v_interleaved;
    int one_wave;          // set by launch()
};

// Whether launch() takes these operands: head sizes it is built for, rows in 16-byte pieces
inline bool fits(int rows, int H, int G, int D, const void* q, const void* k, const void* v) {
    return rows <= 65535 && G > 0 && H % G == 0 && (D == 64 || D == 128 || D == 256) &&
           ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v)) & 15) == 0;
}
cudaError_t launch(const Args& a, cudaStream_t st);

}  // namespace attnstep
}  // namespace llark
