// Jukebox front end kernels (everything of the 5b VQ-VAE encoder + prior that is not a GEMM).
// Reference call sites: jukebox/main.py:54-68 (get_z -> vqvae.encode), :101-110 (prior.forward, only_encode),
// :113-130 (windowed_average). Arithmetic follows openai/jukebox@08efbbc
// (the upstream source is not vendored; oracle/jukebox_oracle.py is the CPU restatement these are tested against).
//
// All activations fp32 (the reference runs the prior with fp16=False). The conv stack is written time-tiled with
// all channels of a tile resident in shared memory, so each ResConv1DBlock is ONE pass over HBM
// (read x, write x'), 1.42 GB a clip in all where each is fused by itself.
#include "common.cuh"
#include <math.h>
#include <stdlib.h>

namespace llark {
namespace jbconv {  // jb_conv_tc.cu
bool takes_resblock(int dil);
int resblock(const float* x, const float* w1, const float* b1, const float* w2, const float* b2, float* y, int N, int T, int dil,
             cudaStream_t st);
int chain_length(const int* dil, int n);  // jb_chain_tc.cu
int chain(const float* x, const float* w0, const float* b0, const float* const* w, const int* dil, int n, float* y, int N, int T, cudaStream_t st);
bool takes_down(int c_in, int c_out);
int down(const float* x, const float* w, const float* b, float* y, int N, int c_in, int T, cudaStream_t st);
bool takes_k3(int c_in, int c_out);
int k3(const float* x, const float* w, const float* b, float* y, int N, int T, cudaStream_t st);
}  // namespace jbconv
namespace jbvq {  // jb_vq_tc.cu
int encode(const float* x, const float* cb, long long* codes, int N, int T, int n_codes, cudaStream_t st);
}

extern thread_local int g_last_cuda_error;
static inline int jb_check() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

// Register-tiled direct convolution from a shared-memory input tile. 256 threads = 8 warps; warp w owns the channel
// group cg = w % NCG (CPT = COUT / NCG output channels) and the time group tg = w / NCG; lane l of it computes the
// TPT output positions tg*32*TPT + l + 32*k. Weights sit in shared memory transposed to [ci][tap][co] so a thread
// fetches its CPT channels with CPT/4 broadcast LDS.128 per tap: per input channel that is TPT*KT scalar LDS +
// KT*CPT/4 LDS.128 against TPT*KT*CPT FMAs (>= 4 FMAs per shared-memory wavefront; the first version issued one
// LDS per FMA and was MIO-bound at 29 % FMA utilisation). The accumulation order
// (bias, then ci ascending, taps ascending) is unchanged, so results are bit-identical to that version.
template <int COUT, int KT, int STRIDE, int NCG, int TPT>
struct ConvTile {
    static constexpr int CPT = COUT / NCG;
    static constexpr int TGROUPS = 8 / NCG;
    static constexpr int TILE_T = TGROUPS * 32 * TPT;  // output positions per CTA
    static_assert(CPT % 4 == 0 && 8 % NCG == 0, "tile shape");

    // sx: [c_in][in_w] input tile whose column j holds the input needed by output position 0 tap 0 at j = 0.
    // swT: [c_in][KT][COUT].
    __device__ static __forceinline__ void run(const float* __restrict__ sx, int in_w, int dil,
                                               const float* __restrict__ swT, int c_in,
                                               const float* __restrict__ bias, float (&acc)[TPT][CPT], int& cg,
                                               int& tl0) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        cg = warp % NCG;
        tl0 = (warp / NCG) * (32 * TPT) + lane;
#pragma unroll
        for (int k = 0; k < TPT; ++k)
#pragma unroll
            for (int c = 0; c < CPT; ++c) acc[k][c] = bias[cg * CPT + c];
        for (int ci = 0; ci < c_in; ++ci) {
            float xv[TPT][KT];
#pragma unroll
            for (int k = 0; k < TPT; ++k)
#pragma unroll
                for (int j = 0; j < KT; ++j) xv[k][j] = sx[ci * in_w + (tl0 + 32 * k) * STRIDE + j * dil];
#pragma unroll
            for (int j = 0; j < KT; ++j) {
                const float4* wp = reinterpret_cast<const float4*>(swT + (ci * KT + j) * COUT + cg * CPT);
#pragma unroll
                for (int c4 = 0; c4 < CPT / 4; ++c4) {
                    const float4 w = wp[c4];
#pragma unroll
                    for (int k = 0; k < TPT; ++k) {
                        acc[k][4 * c4 + 0] = fmaf(w.x, xv[k][j], acc[k][4 * c4 + 0]);
                        acc[k][4 * c4 + 1] = fmaf(w.y, xv[k][j], acc[k][4 * c4 + 1]);
                        acc[k][4 * c4 + 2] = fmaf(w.z, xv[k][j], acc[k][4 * c4 + 2]);
                        acc[k][4 * c4 + 3] = fmaf(w.w, xv[k][j], acc[k][4 * c4 + 3]);
                    }
                }
            }
        }
    }
};
// Input tile [c_in][in_w] <- x[n, :, t_first + j] (zero outside [0, T)), optionally through ReLU. Eight independent
// global loads are issued per thread before the first is consumed: the original one-load-then-store loop (with an
// integer division per element) left a single load in flight per thread and was 36 % of the res-block's stall samples.
template <bool RELU>
__device__ __forceinline__ void load_x_tile(float* sx, const float* __restrict__ xn, int c_in, int T, int in_w,
                                            int t_first) {
    for (int j = threadIdx.x; j < in_w; j += blockDim.x) {
        const int ti = t_first + j;
        const bool ok = ti >= 0 && ti < T;
        const float* src = xn + (ok ? ti : 0);
        int ci = 0;
        for (; ci + 8 <= c_in; ci += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = ok ? src[(long long)(ci + u) * T] : 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u) sx[(ci + u) * in_w + j] = RELU ? fmaxf(v[u], 0.f) : v[u];
        }
        for (; ci < c_in; ++ci) {
            const float v = ok ? src[(long long)ci * T] : 0.f;
            sx[ci * in_w + j] = RELU ? fmaxf(v, 0.f) : v;
        }
    }
}
// global w [COUT][c_in][KT] -> shared [c_in][KT][COUT]
template <int COUT, int KT>
__device__ __forceinline__ void load_weights_T(float* swT, const float* __restrict__ w, int c_in) {
    // consecutive threads write consecutive shared-memory words (conflict-free) and gather from global/L1: the
    // transposing direction must be the read, a strided smem store is a COUT-way bank conflict
    for (int i = threadIdx.x; i < COUT * c_in * KT; i += blockDim.x) {
        const int r = i / COUT, co = i % COUT;  // r = ci*KT + k
        swT[i] = w[co * (c_in * KT) + r];
    }
}

// ---------------------------------------------------------------------------------------------- down conv k4 s2 p1
// y[n,co,t] = b[co] + sum_ci sum_k w[co,ci,k] * x[n,ci,2t-1+k].
template <int COUT>
struct DownCfg {
    using Tile = ConvTile<COUT, 4, 2, COUT / 16, 2>;
};
template <int COUT>
__global__ void __launch_bounds__(256)
conv_down_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                 float* __restrict__ y, int c_in, int T) {
    using Tile = typename DownCfg<COUT>::Tile;
    extern __shared__ __align__(16) float sm[];
    const int To = T / 2;
    const int n = blockIdx.y;
    const int t0 = blockIdx.x * Tile::TILE_T;
    const int in_w = 2 * Tile::TILE_T + 2;
    float* swT = sm;                         // [c_in][4][COUT]  (first: keeps it 16-byte aligned)
    float* sx = sm + COUT * c_in * 4;        // [c_in][in_w]
    load_x_tile<false>(sx, x + (long long)n * c_in * T, c_in, T, in_w, 2 * t0 - 1);
    load_weights_T<COUT, 4>(swT, w, c_in);
    __syncthreads();
    float acc[2][Tile::CPT];
    int cg, tl0;
    Tile::run(sx, in_w, 1, swT, c_in, bias, acc, cg, tl0);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int t = t0 + tl0 + 32 * k;
        if (t < To) {
#pragma unroll
            for (int c = 0; c < Tile::CPT; ++c) y[((long long)n * COUT + cg * Tile::CPT + c) * To + t] = acc[k][c];
        }
    }
}

// ---------------------------------------------------------------------------------------------- fused res block
// y = x + W2 * relu(W1 (*dilation d, k=3) relu(x) + b1) + b2,   32 channels.
using ResTile1 = ConvTile<32, 3, 1, 2, 2>;  // 256 output positions per CTA
using ResTile2 = ConvTile<32, 1, 1, 2, 2>;
constexpr int RES_TT = ResTile1::TILE_T;
__global__ void __launch_bounds__(256)
resblock_kernel(const float* __restrict__ x, const float* __restrict__ w1, const float* __restrict__ b1,
                const float* __restrict__ w2, const float* __restrict__ b2, float* __restrict__ y, int T, int d) {
    extern __shared__ __align__(16) float sm[];
    constexpr int C = 32;
    const int n = blockIdx.y;
    const int t0 = blockIdx.x * RES_TT;
    const int in_w = RES_TT + 2 * d;
    float* sw1T = sm;                  // [C][3][C]
    float* sw2T = sw1T + C * C * 3;    // [C][C]
    float* sh = sw2T + C * C;          // relu(h) tile [C][RES_TT]
    float* sx = sh + C * RES_TT;       // relu(x) tile [C][in_w]
    load_x_tile<true>(sx, x + (long long)n * C * T, C, T, in_w, t0 - d);
    load_weights_T<C, 3>(sw1T, w1, C);
    load_weights_T<C, 1>(sw2T, w2, C);
    __syncthreads();
    float acc[2][ResTile1::CPT];
    int cg, tl0;
    ResTile1::run(sx, in_w, d, sw1T, C, b1, acc, cg, tl0);
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int c = 0; c < ResTile1::CPT; ++c) sh[(cg * ResTile1::CPT + c) * RES_TT + tl0 + 32 * k] = fmaxf(acc[k][c], 0.f);
    __syncthreads();
    ResTile2::run(sh, RES_TT, 1, sw2T, C, b2, acc, cg, tl0);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int t = t0 + tl0 + 32 * k;
        if (t < T) {
#pragma unroll
            for (int c = 0; c < ResTile2::CPT; ++c) {
                const long long off = ((long long)n * C + cg * ResTile2::CPT + c) * T + t;
                y[off] = x[off] + acc[k][c];
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------- conv k3 s1 p1
template <int COUT>
struct K3Cfg {
    using Tile = ConvTile<COUT, 3, 1, COUT / 16, 2>;
};
template <int COUT>
__global__ void __launch_bounds__(256)
conv_k3_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
               float* __restrict__ y, int c_in, int T) {
    using Tile = typename K3Cfg<COUT>::Tile;
    extern __shared__ __align__(16) float sm[];
    const int n = blockIdx.y;
    const int t0 = blockIdx.x * Tile::TILE_T;
    const int in_w = Tile::TILE_T + 2;
    float* swT = sm;                       // [c_in][3][COUT]
    float* sx = sm + COUT * c_in * 3;      // [c_in][in_w]
    load_x_tile<false>(sx, x + (long long)n * c_in * T, c_in, T, in_w, t0 - 1);
    load_weights_T<COUT, 3>(swT, w, c_in);
    __syncthreads();
    float acc[2][Tile::CPT];
    int cg, tl0;
    Tile::run(sx, in_w, 1, swT, c_in, bias, acc, cg, tl0);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int t = t0 + tl0 + 32 * k;
        if (t < T) {
#pragma unroll
            for (int c = 0; c < Tile::CPT; ++c) y[((long long)n * COUT + cg * Tile::CPT + c) * T + t] = acc[k][c];
        }
    }
}

// ---------------------------------------------------------------------------------------------- LayerNorm
// A CTA per row. VPT > 0: the row stays in registers, VPT * 4 values a thread, and is read once; VPT = 0 (rows of more than
// LN_VPT * 1024 values) reads it three times. Sums and results are the same in both. Memory-bound: 16384 rows of 4800 values to bf16
// 92 us on a B200 (71 at the copy rate), 117 when every row was read three times behind five barriers.
constexpr int LN_VPT = 5;
template <int VPT>
__global__ void __launch_bounds__(256)
layernorm_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                 void* __restrict__ y, int y_bf16, int W, float eps) {
    __shared__ float red[2][8];
    const long long row = blockIdx.x;
    const float* xr = x + row * W;
    float4 kept[VPT > 0 ? VPT : 1];
    auto walk = [&](bool first, auto&& f) {  // f(values, index) over this thread's pieces of the row
        if constexpr (VPT > 0) {
            if (first)
#pragma unroll
                for (int k = 0; k < VPT; ++k) {
                    const int i = (threadIdx.x + k * 256) * 4;
                    if (i < W) kept[k] = *reinterpret_cast<const float4*>(xr + i);
                }
#pragma unroll
            for (int k = 0; k < VPT; ++k) {
                const int i = (threadIdx.x + k * 256) * 4;
                if (i < W) f(kept[k], i);
            }
        } else {
            for (int i = threadIdx.x * 4; i < W; i += 1024) f(*reinterpret_cast<const float4*>(xr + i), i);
        }
    };
    auto total = [&](float s, float* part) {
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
        __syncthreads();
        return warp_sum((threadIdx.x & 31) < 8 ? part[threadIdx.x & 31] : 0.f);
    };
    float s = 0.f;
    walk(true, [&](const float4 v, int) { s += v.x + v.y + v.z + v.w; });
    const float mean = total(s, red[0]) / (float)W;
    float q = 0.f;
    walk(false, [&](const float4 v, int) {
        const float a = v.x - mean, b = v.y - mean, c = v.z - mean, d = v.w - mean;
        q += a * a + b * b + c * c + d * d;
    });
    const float rstd = rsqrtf(total(q, red[1]) / (float)W + eps);
    walk(false, [&](const float4 v, int i) {
        const float4 g = *reinterpret_cast<const float4*>(gamma + i);
        const float4 b = *reinterpret_cast<const float4*>(beta + i);
        const float o0 = (v.x - mean) * rstd * g.x + b.x, o1 = (v.y - mean) * rstd * g.y + b.y,
                    o2 = (v.z - mean) * rstd * g.z + b.z, o3 = (v.w - mean) * rstd * g.w + b.w;
        if (y_bf16) {
            uint2 o;
            o.x = pack_bf16x2(o0, o1);
            o.y = pack_bf16x2(o2, o3);
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(y) + row * W + i) = o;
        } else {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(y) + row * W + i) = make_float4(o0, o1, o2, o3);
        }
    });
}

// ---------------------------------------------------------------------------------------------- prior input embedding
// A block has a time step of up to K clips: its two additive rows are read once for them, and their token rows are under way together. Bound
// by memory: 2 clips x 8192 steps x 4800 (two additive tables of 157 MB, 315 MB written) 124 us with K = 2, 166 with K = 1. K = 1 for one
// clip, and where the tables stay in L2 anyway and blocks matter more: 64 clips x 16 steps 9 us (43 with all clips in a block).
template <int K>
__global__ void __launch_bounds__(256)
jb_embed_kernel(const long long* __restrict__ codes, const float* __restrict__ emb,
                                const float* __restrict__ y_cond, const float* __restrict__ pos_emb,
                                const float* __restrict__ x_cond, float* __restrict__ out, int N, int T, int W) {
    const int t = blockIdx.x, n0 = blockIdx.y * K;
    const float* pe = pos_emb + (long long)t * W;
    const float* xc = x_cond + (long long)t * W;
    const float* src[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int n = min(n0 + k, N - 1);
        src[k] = t == 0 ? y_cond : emb + codes[(long long)n * T + t - 1] * W;
    }
    for (int i = threadIdx.x * 4; i < W; i += blockDim.x * 4) {
        const float4 b = *reinterpret_cast<const float4*>(pe + i);
        const float4 c = *reinterpret_cast<const float4*>(xc + i);
        float4 a[K];
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (K == 1 || n0 + k < N) a[k] = *reinterpret_cast<const float4*>(src[k] + i);
        // reference order: (x_emb + pos_emb) + x_cond
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (K == 1 || n0 + k < N)
                *reinterpret_cast<float4*>(out + ((long long)(n0 + k) * T + t) * W + i) = make_float4(
                    (a[k].x + b.x) + c.x, (a[k].y + b.y) + c.y, (a[k].z + b.z) + c.z, (a[k].w + b.w) + c.w);
    }
}

// ---------------------------------------------------------------------------------------------- factored attention
// One CTA per (group, head, n). A group is <= 128 queries and <= 128 keys gathered with a stride:
//   pattern 0 (block):            group g = block g; queries = keys = positions g*blk + i;           causal
//   pattern 1 (transposed block): group g = offset g; queries = keys = positions i*blk + g;          causal in i
//   pattern 2 (previous block):   group g = block g; queries g*blk + i, keys (g-1)*blk + i (none for g=0); full
// Each warp processes one query at a time: lanes over keys for QK^T, lanes over channels for PV (fp32 SIMT).
__global__ void __launch_bounds__(256)
jb_sparse_attn_kernel(const float* __restrict__ qkv, float* __restrict__ out, int T, int heads, int dh, int blk,
                      int pattern, float scale) {
    extern __shared__ float sm[];
    const int g = blockIdx.x, h = blockIdx.y, n = blockIdx.z;
    const int nblk = T / blk;
    int nq, nk, qstride, q0, k0;
    bool causal;
    if (pattern == 0) { nq = nk = blk; qstride = 1; q0 = k0 = g * blk; causal = true; }
    else if (pattern == 1) { nq = nk = nblk; qstride = blk; q0 = k0 = g; causal = true; }
    else { nq = blk; nk = (g == 0) ? 0 : blk; qstride = 1; q0 = g * blk; k0 = (g - 1) * blk; causal = false; }
    const int ldk = dh + 1;
    float* sK = sm;               // [nk][ldk]
    float* sV = sK + 128 * ldk;   // [nk][ldk]
    float* sQ = sV + 128 * ldk;   // [8 warps][dh]
    float* sP = sQ + 8 * dh;      // [8 warps][128]
    const long long rs = 3LL * heads * dh;
    const float* base = qkv + (long long)n * T * rs;
    for (int i = threadIdx.x; i < nk * dh; i += blockDim.x) {
        const int r = i / dh, c = i % dh;
        const long long pos = k0 + (long long)r * qstride;
        sK[r * ldk + c] = base[pos * rs + (long long)heads * dh + h * dh + c];
        sV[r * ldk + c] = base[pos * rs + 2LL * heads * dh + h * dh + c];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* myq = sQ + warp * dh;
    float* myp = sP + warp * 128;
    for (int qi = warp; qi < nq; qi += 8) {
        const long long qpos = q0 + (long long)qi * qstride;
        for (int c = lane; c < dh; c += 32) myq[c] = base[qpos * rs + h * dh + c];
        __syncwarp();
        const int kmax = causal ? qi + 1 : nk;  // keys [0, kmax)
        float sc[4];
        float mx = -INFINITY;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int kj = lane + r * 32;
            float dot = -INFINITY;
            if (kj < kmax) {
                dot = 0.f;
                const float* kr = sK + kj * ldk;
                for (int c = 0; c < dh; ++c) dot = fmaf(myq[c], kr[c], dot);
                dot *= scale;
            }
            sc[r] = dot;
            mx = fmaxf(mx, dot);
        }
        mx = warp_max(mx);
        float sum = 0.f;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float p = (sc[r] == -INFINITY) ? 0.f : __expf(sc[r] - mx);
            sc[r] = p;
            sum += p;
        }
        sum = warp_sum(sum);
        const float inv = sum > 0.f ? 1.f / sum : 0.f;
#pragma unroll
        for (int r = 0; r < 4; ++r) myp[lane + r * 32] = sc[r] * inv;
        __syncwarp();
        float* orow = out + ((long long)n * T + qpos) * ((long long)heads * dh) + h * dh;
        for (int c = lane; c < dh; c += 32) {
            float acc = 0.f;
            for (int kj = 0; kj < kmax; ++kj) acc = fmaf(myp[kj], sV[kj * ldk + c], acc);
            orow[c] = acc;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------------- factored attention, tensor cores
// Same contract as jb_sparse_attn_kernel, on mma.sync m16n8k8 TF32 (fp32 accumulate): the SIMT kernel above issues one
// shared-memory load per FMA and runs at ~6 TFLOP/s (4.7 ms per prior layer at batch 8, a third of the front end); here one CTA = one (group, head, n), each warp owns 16 query rows:
//   S = Q K^T  (Q fragments in registers, K from shared memory, 19 k-steps of 8 over the 150(+2 zero) channels),
//   softmax in registers on the accumulator fragments (quad shuffles),
//   O = P V    with P taken straight from the S accumulators: the m16n8k8 A fragment wants key slots (t, t+4) where the
//              accumulator holds keys (2t, 2t+1), so the k index of the P.V product is permuted consistently -- slot t
//              reads V row 8j+2t, slot t+4 reads V row 8j+2t+1 -- and no shuffle is needed.
// K and V rows are gathered (stride 1 or `blk`) into shared memory by cp.async, all of them under way at once, and Q goes to its
// fragments; S waits for K alone. It is bound by these loads: with eight granules of 8 bytes a thread in flight through registers, and V
// after Q in one buffer, 16384 tokens x 8 heads took 239 us (64 rows) and 302 us (128 rows); now 119
// and 179. Operands are rounded to TF32 (cvt.rna) when the fragments are formed. Causal key tiles
// above the diagonal are skipped. Output fp32 or bf16 (fused cast for the bf16 prior).
constexpr int JA_LD = 156;   // shared-memory row pitch (floats): 156 mod 32 = 28 -> conflict-free fragment loads
constexpr int JA_KS = 19;    // k-steps of 8 covering head channels (<= 152)
__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// rows x dh floats gathered from global (row r at base + (pos0 + r*stride)*rs) into smem [rows][JA_LD], pad columns zero: every granule of
// 8 bytes (dh is even, rows are 8-byte aligned) is asked for at once, none passes through a register
__device__ __forceinline__ void ja_ask_rows(float* dst, const float* __restrict__ base, long long pos0, int stride,
                                            long long rs, int rows, int dh) {
    const int lane = threadIdx.x & 31;
    const float* src = base + (pos0 + (long long)(threadIdx.x >> 5) * stride) * rs;
    const long long step = (long long)(blockDim.x >> 5) * stride * rs;
    for (int r = threadIdx.x >> 5; r < rows; r += blockDim.x >> 5, src += step) {  // a warp per row
#pragma unroll
        for (int k = 0; k < (JA_LD / 2 + 31) / 32; ++k) {
            const int c = 2 * (lane + 32 * k);
            float* to = dst + r * JA_LD + c;
            if (c < dh)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(to)), "l"(src + c) : "memory");
            else if (c < JA_LD)
                *reinterpret_cast<float2*>(to) = make_float2(0.f, 0.f);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int NKT>  // key tiles of 8 (8 -> 64 keys, 16 -> 128 keys)
__global__ void __launch_bounds__(256)
jb_sparse_attn_tc_kernel(const float* __restrict__ qkv, void* __restrict__ out, int out_bf16, int T, int heads, int dh,
                         int blk, int pattern, float scale) {
    extern __shared__ __align__(16) float sm[];
    constexpr int NK = NKT * 8;
    float* sK = sm;                 // [NK][JA_LD]
    float* sV = sm + NK * JA_LD;    // [NK][JA_LD]
    const int g = blockIdx.x, h = blockIdx.y, n = blockIdx.z;
    int qstride, q0, k0;
    bool causal, has_keys = true;
    if (pattern == 0) { qstride = 1; q0 = k0 = g * blk; causal = true; }
    else if (pattern == 1) { qstride = blk; q0 = k0 = g; causal = true; }
    else { qstride = 1; q0 = g * blk; k0 = (g - 1) * blk; causal = false; has_keys = g > 0; }
    const long long rs = 3LL * heads * dh;
    const long long ow = (long long)heads * dh;
    const float* base = qkv + (long long)n * T * rs + (long long)h * dh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gq = lane >> 2, t4 = lane & 3;
    const int r0 = warp * 16 + gq;  // this thread's rows inside the group: r0 and r0 + 8
    if (!has_keys) {  // previous-block pattern, first block: no keys -> zeros (the SIMT kernel and the reference agree)
        for (int i = threadIdx.x; i < NK * dh; i += blockDim.x) {
            const long long pos = q0 + (long long)(i / dh) * qstride;
            const long long o = ((long long)n * T + pos) * ow + (long long)h * dh + i % dh;
            if (out_bf16) reinterpret_cast<__nv_bfloat16*>(out)[o] = __float2bfloat16_rn(0.f);
            else reinterpret_cast<float*>(out)[o] = 0.f;
        }
        return;
    }
    ja_ask_rows(sK, base + (long long)heads * dh, k0, qstride, rs, NK, dh);
    ja_ask_rows(sV, base + 2LL * heads * dh, k0, qstride, rs, NK, dh);
    uint32_t qa[JA_KS][4];
    {
        const float* q = base + (q0 + (long long)r0 * qstride) * rs;
        const float* q8 = q + 8LL * qstride * rs;
#pragma unroll
        for (int ks = 0; ks < JA_KS; ++ks) {
            const int c = ks * 8 + t4;
            qa[ks][0] = to_tf32(c < dh ? q[c] : 0.f);
            qa[ks][1] = to_tf32(c < dh ? q8[c] : 0.f);
            qa[ks][2] = to_tf32(c + 4 < dh ? q[c + 4] : 0.f);
            qa[ks][3] = to_tf32(c + 4 < dh ? q8[c + 4] : 0.f);
        }
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // K is there
    // key tiles this warp needs: causal rows 16w .. 16w+15 see keys <= 16w+15
    const int nt_end = causal ? min(NKT, 2 * warp + 2) : NKT;
    float sc[NKT][4];
#pragma unroll
    for (int nt = 0; nt < NKT; ++nt) {
        sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
        if (nt < nt_end) {
            const float* kr = sK + (nt * 8 + gq) * JA_LD + t4;
#pragma unroll
            for (int ks = 0; ks < JA_KS; ++ks) mma_tf32(sc[nt], qa[ks], to_tf32(kr[ks * 8]), to_tf32(kr[ks * 8 + 4]));
        }
    }
    // softmax over the keys of rows r0 (elements 0,1) and r0+8 (elements 2,3)
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < NKT; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int key = nt * 8 + 2 * t4 + (e & 1);
            const int row = r0 + (e >> 1) * 8;
            const bool ok = nt < nt_end && (!causal || key <= row);
            const float v = ok ? sc[nt][e] * scale : -INFINITY;
            sc[nt][e] = v;
            mx[e >> 1] = fmaxf(mx[e >> 1], v);
        }
    }
    float sum[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
        mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    }
#pragma unroll
    for (int nt = 0; nt < NKT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float p = (sc[nt][e] == -INFINITY) ? 0.f : __expf(sc[nt][e] - mx[e >> 1]);
            sc[nt][e] = p;
            sum[e >> 1] += p;
        }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // V is there
    float oacc[JA_KS][4];
#pragma unroll
    for (int nn = 0; nn < JA_KS; ++nn) oacc[nn][0] = oacc[nn][1] = oacc[nn][2] = oacc[nn][3] = 0.f;
#pragma unroll
    for (int j = 0; j < NKT; ++j) {
        if (j < nt_end) {
            uint32_t pa[4];
            pa[0] = to_tf32(sc[j][0]);  // (row r0,   key 8j+2t)   -> k slot t
            pa[1] = to_tf32(sc[j][2]);  // (row r0+8, key 8j+2t)
            pa[2] = to_tf32(sc[j][1]);  // (row r0,   key 8j+2t+1) -> k slot t+4
            pa[3] = to_tf32(sc[j][3]);
            const float* v0 = sV + (j * 8 + 2 * t4) * JA_LD + gq;
#pragma unroll
            for (int nn = 0; nn < JA_KS; ++nn) mma_tf32(oacc[nn], pa, to_tf32(v0[nn * 8]), to_tf32(v0[JA_LD + nn * 8]));
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float inv = sum[r] > 0.f ? 1.f / sum[r] : 0.f;
        const long long pos = q0 + (long long)(r0 + r * 8) * qstride;
        const long long o = ((long long)n * T + pos) * ow + (long long)h * dh;
#pragma unroll
        for (int nn = 0; nn < JA_KS; ++nn) {
            const int col = nn * 8 + 2 * t4;
            if (col < dh) {
                const float a = oacc[nn][2 * r] * inv, b = oacc[nn][2 * r + 1] * inv;
                if (out_bf16)
                    *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(out) + o + col) = pack_bf16x2(a, b);
                else
                    *reinterpret_cast<float2*>(reinterpret_cast<float*>(out) + o + col) = make_float2(a, b);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------- elementwise
__global__ void quick_gelu_kernel(const float* __restrict__ x, float* __restrict__ y, long long n) {
    long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    const long long stride = (long long)gridDim.x * blockDim.x * 4;
    for (; i + 4 <= n; i += stride) {
        float4 v = *reinterpret_cast<const float4*>(x + i);
        v.x = v.x / (1.f + __expf(-1.702f * v.x));
        v.y = v.y / (1.f + __expf(-1.702f * v.y));
        v.z = v.z / (1.f + __expf(-1.702f * v.z));
        v.w = v.w / (1.f + __expf(-1.702f * v.w));
        *reinterpret_cast<float4*>(y + i) = v;
    }
    if (i < n)
        for (long long j = i; j < n; ++j) y[j] = x[j] / (1.f + __expf(-1.702f * x[j]));
}
__global__ void add3_kernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ c,
                            float* __restrict__ out, long long n) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (; i < n; i += stride) out[i] = c ? (a[i] + b[i]) + c[i] : a[i] + b[i];
}
// out[n, f, c] = mean_{j<frame} acts[n, f*frame + j, c]; grid (frames, N, ceil(W/4/blockDim)), 4 columns per thread,
// the `frame` row loads of a thread are independent (two accumulators) so a warp keeps ~frame x 512 B in flight.
__global__ void jb_pool_kernel(const float* __restrict__ acts, float* __restrict__ out, long long clip_stride, int frames,
                               int W, int frame) {
    const int f = blockIdx.x;
    const int c = (blockIdx.z * blockDim.x + threadIdx.x) * 4;
    if (c >= W) return;
    const float* src = acts + (long long)blockIdx.y * clip_stride + (long long)f * frame * W + c;
    float* dst = out + ((long long)blockIdx.y * frames + f) * W + c;
    if (c + 4 <= W && (W & 3) == 0) {
        float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
        int j = 0;
        for (; j + 1 < frame; j += 2) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(src + (long long)j * W));
            const float4 b = __ldg(reinterpret_cast<const float4*>(src + (long long)(j + 1) * W));
            s0.x += a.x; s0.y += a.y; s0.z += a.z; s0.w += a.w;
            s1.x += b.x; s1.y += b.y; s1.z += b.z; s1.w += b.w;
        }
        if (j < frame) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(src + (long long)j * W));
            s0.x += a.x; s0.y += a.y; s0.z += a.z; s0.w += a.w;
        }
        const float inv = 1.f / (float)frame;
        *reinterpret_cast<float4*>(dst) =
            make_float4((s0.x + s1.x) * inv, (s0.y + s1.y) * inv, (s0.z + s1.z) * inv, (s0.w + s1.w) * inv);
    } else {
        for (int k = 0; k < 4 && c + k < W; ++k) {
            float sum = 0.f;
            for (int j = 0; j < frame; ++j) sum += src[(long long)j * W + k];
            dst[k] = sum / (float)frame;
        }
    }
}
// Timing conditioning of the top-level prior (LabelConditioner.forward -> pos_emb, jukebox/main.py:93):
// out[t, :] = (total_row + abs_table[abs_bins[t], :]) + rel_table[rel_bins[t], :] -- the reference's order of additions.
__global__ void jb_label_cond_kernel(const float* __restrict__ total_row, const float* __restrict__ abs_table,
                                     const float* __restrict__ rel_table, const int* __restrict__ abs_bins,
                                     const int* __restrict__ rel_bins, float* __restrict__ out, int W) {
    const int t = blockIdx.x;
    const float* a = abs_table + (long long)abs_bins[t] * W;
    const float* r = rel_table + (long long)rel_bins[t] * W;
    float* o = out + (long long)t * W;
    for (int c = threadIdx.x; c < W; c += blockDim.x) o[c] = (total_row[c] + a[c]) + r[c];
}
// colsum over rows of a bf16 [rows, H] matrix -> bf16 [H] (bias gradient), fp32 accumulate. Memory-bound: 32 columns per CTA, a lane each;
// the 16 warps take every 16th row, eight loads on their way, and their sums meet in shared memory. One thread walking all rows of a
// column waited for one load after another: 8192 rows of 4096 columns, not in L2, 578 us; now 55.
constexpr int kColsumWarps = 16;
__global__ void __launch_bounds__(kColsumWarps * 32)
colsum_bf16_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ out, long long rows, int H, int accumulate) {
    __shared__ float part[kColsumWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (c < H)
#pragma unroll 8
        for (long long r = warp; r < rows; r += kColsumWarps) s += __bfloat162float(x[r * H + c]);
    part[warp][lane] = s;
    __syncthreads();
    if (warp || c >= H) return;
    for (int w = 1; w < kColsumWarps; ++w) s += part[w][lane];
    if (accumulate) s += __bfloat162float(out[c]);
    out[c] = __float2bfloat16_rn(s);
}

static int set_dyn_smem(const void* fn, int bytes) {
    if (bytes <= 48 * 1024) return LLARK_OK;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

}  // namespace llark

using namespace llark;

// LLARK_JB_CONV_TC=0 selects the fp32 FMA kernels for every convolution of the encoder (read per call: tests toggle it)
static bool use_conv_tc() {
    const char* e = getenv("LLARK_JB_CONV_TC");
    return !(e && e[0] == '0');
}

extern "C" int llark_jb_conv_down(const float* x, const float* w, const float* bias, float* y, int N, int c_in,
                                  int c_out, int T, cudaStream_t st) {
    if (N <= 0 || T <= 0 || (T & 1) || c_in <= 0 || (c_out != 32 && c_out != 64)) return LLARK_EINVAL;
    if (use_conv_tc() && jbconv::takes_down(c_in, c_out)) return jbconv::down(x, w, bias, y, N, c_in, T, st);
    int rc;  // one channel in (the waveform), or other widths: memory-bound or small
    if (c_out == 32) {
        constexpr int TILE = DownCfg<32>::Tile::TILE_T;
        const int smem = (c_in * (2 * TILE + 2) + c_out * c_in * 4) * (int)sizeof(float);
        dim3 grid((T / 2 + TILE - 1) / TILE, N);
        rc = set_dyn_smem((const void*)conv_down_kernel<32>, smem);
        if (rc) return rc;
        conv_down_kernel<32><<<grid, 256, smem, st>>>(x, w, bias, y, c_in, T);
    } else {
        constexpr int TILE = DownCfg<64>::Tile::TILE_T;
        const int smem = (c_in * (2 * TILE + 2) + c_out * c_in * 4) * (int)sizeof(float);
        dim3 grid((T / 2 + TILE - 1) / TILE, N);
        rc = set_dyn_smem((const void*)conv_down_kernel<64>, smem);
        if (rc) return rc;
        conv_down_kernel<64><<<grid, 256, smem, st>>>(x, w, bias, y, c_in, T);
    }
    return jb_check();
}

extern "C" int llark_jb_resblock(const float* x, const float* w1, const float* b1, const float* w2, const float* b2,
                                 float* y, int N, int T, int dilation, cudaStream_t st) {
    if (N <= 0 || T <= 0 || dilation < 1 || dilation > 243) return LLARK_EINVAL;
    if (use_conv_tc() && jbconv::chain_length(&dilation, 1) == 1) {  // up to dilation 32; 201 us against 257 at 27
        const float* const w[4] = {w1, b1, w2, b2};
        return jbconv::chain(x, nullptr, nullptr, w, &dilation, 1, y, N, T, st);
    }
    if (use_conv_tc() && jbconv::takes_resblock(dilation)) return jbconv::resblock(x, w1, b1, w2, b2, y, N, T, dilation, st);
    const int smem = (32 * (RES_TT + 2 * dilation) + 32 * RES_TT + 32 * 32 * 3 + 32 * 32) * (int)sizeof(float);
    int rc = set_dyn_smem((const void*)resblock_kernel, smem);
    if (rc) return rc;
    dim3 grid((T + RES_TT - 1) / RES_TT, N);
    resblock_kernel<<<grid, 256, smem, st>>>(x, w1, b1, w2, b2, y, T, dilation);
    return jb_check();
}

extern "C" int llark_jb_resblocks_length(const int* dilations, int n) {
    return use_conv_tc() && dilations ? jbconv::chain_length(dilations, n) : 0;
}

extern "C" int llark_jb_resblocks(const float* x, const float* const* weights, const int* dilations, int n, float* y, int N, int T,
                                  cudaStream_t st) {
    if (N <= 0 || T <= 0 || n <= 0 || !x || !weights || !dilations || !y || jbconv::chain_length(dilations, n) != n) return LLARK_EINVAL;
    return jbconv::chain(x, nullptr, nullptr, weights, dilations, n, y, N, T, st);
}

extern "C" int llark_jb_wave_resblocks(const float* wave, const float* w, const float* bias, const float* const* weights, const int* dilations,
                                       int n, float* y, int N, int T, cudaStream_t st) {
    if (N <= 0 || T <= 0 || (T & 1) || n <= 0 || !wave || !w || !bias || !weights || !dilations || !y || jbconv::chain_length(dilations, n) != n)
        return LLARK_EINVAL;
    return jbconv::chain(wave, w, bias, weights, dilations, n, y, N, T / 2, st);
}

extern "C" int llark_jb_conv_k3(const float* x, const float* w, const float* bias, float* y, int N, int c_in, int c_out,
                                int T, cudaStream_t st) {
    if (N <= 0 || T <= 0 || c_in <= 0 || (c_out != 32 && c_out != 64)) return LLARK_EINVAL;
    if (use_conv_tc() && jbconv::takes_k3(c_in, c_out)) return jbconv::k3(x, w, bias, y, N, T, st);
    int rc;
    if (c_out == 64) {
        constexpr int TILE = K3Cfg<64>::Tile::TILE_T;
        const int smem = (c_in * (TILE + 2) + c_out * c_in * 3) * (int)sizeof(float);
        dim3 grid((T + TILE - 1) / TILE, N);
        rc = set_dyn_smem((const void*)conv_k3_kernel<64>, smem);
        if (rc) return rc;
        conv_k3_kernel<64><<<grid, 256, smem, st>>>(x, w, bias, y, c_in, T);
    } else {
        constexpr int TILE = K3Cfg<32>::Tile::TILE_T;
        const int smem = (c_in * (TILE + 2) + c_out * c_in * 3) * (int)sizeof(float);
        dim3 grid((T + TILE - 1) / TILE, N);
        rc = set_dyn_smem((const void*)conv_k3_kernel<32>, smem);
        if (rc) return rc;
        conv_k3_kernel<32><<<grid, 256, smem, st>>>(x, w, bias, y, c_in, T);
    }
    return jb_check();
}

extern "C" int llark_jb_vq_encode(const float* x, const float* codebook, long long* codes, int N, int T, int n_codes,
                                  cudaStream_t st) {
    if (N <= 0 || T <= 0 || n_codes <= 0) return LLARK_EINVAL;
    return jbvq::encode(x, codebook, codes, N, T, n_codes, st);
}

extern "C" int llark_layernorm_fwd(const float* x, const float* gamma, const float* beta, void* y, int y_bf16,
                                   long long rows, int W, float eps, cudaStream_t st) {
    if (rows <= 0 || W <= 0 || (W & 3)) return LLARK_EINVAL;
    if (W <= LN_VPT * 1024)
        layernorm_kernel<LN_VPT><<<(unsigned)rows, 256, 0, st>>>(x, gamma, beta, y, y_bf16, W, eps);
    else
        layernorm_kernel<0><<<(unsigned)rows, 256, 0, st>>>(x, gamma, beta, y, y_bf16, W, eps);
    return jb_check();
}

extern "C" int llark_jb_embed_tokens(const long long* codes, const float* emb, const float* y_cond,
                                     const float* pos_emb, const float* x_cond, float* out, int N, int T, int W,
                                     cudaStream_t st) {
    if (N <= 0 || T <= 0 || (W & 3)) return LLARK_EINVAL;
    const bool in_l2 = (long long)T * W * 8 <= 64LL << 20;
    const int k = N == 1 || in_l2 ? 1 : N == 2 ? 2 : 4;
    const dim3 grid(T, (N + k - 1) / k);
    auto* kernel = k == 1 ? jb_embed_kernel<1> : k == 2 ? jb_embed_kernel<2> : jb_embed_kernel<4>;
    kernel<<<grid, 256, 0, st>>>(codes, emb, y_cond, pos_emb, x_cond, out, N, T, W);
    return jb_check();
}

extern "C" int llark_jb_sparse_attn(const float* qkv, float* out, int N, int T, int heads, int dh, int block,
                                    int pattern, cudaStream_t st) {
    if (N <= 0 || T <= 0 || block <= 0 || T % block || pattern < 0 || pattern > 2) return LLARK_EINVAL;
    const int nblk = T / block;
    if (block > 128 || nblk > 128 || dh > 256) return LLARK_EINVAL;
    const int groups = (pattern == 1) ? block : nblk;
    const int smem = (2 * 128 * (dh + 1) + 8 * dh + 8 * 128) * (int)sizeof(float);
    int rc = set_dyn_smem((const void*)jb_sparse_attn_kernel, smem);
    if (rc) return rc;
    dim3 grid(groups, heads, N);
    jb_sparse_attn_kernel<<<grid, 256, smem, st>>>(qkv, out, T, heads, dh, block, pattern, 1.f / sqrtf((float)dh));
    return jb_check();
}

// Tensor-core variant (TF32 operands, fp32 accumulate); out fp32 or bf16. LLARK_EINVAL when the geometry is outside
// its envelope (64- or 128-row groups, even head width <= 152): callers then use llark_jb_sparse_attn.
extern "C" int llark_jb_sparse_attn_tc(const float* qkv, void* out, int out_bf16, int N, int T, int heads, int dh,
                                       int block, int pattern, cudaStream_t st) {
    if (N <= 0 || T <= 0 || block <= 0 || T % block || pattern < 0 || pattern > 2) return LLARK_EINVAL;
    const int nblk = T / block;
    const int rows = (pattern == 1) ? nblk : block;  // queries (= keys) per group
    if ((rows != 64 && rows != 128) || dh > 8 * JA_KS || (dh & 1)) return LLARK_EINVAL;
    const int groups = (pattern == 1) ? block : nblk;
    const int smem = 2 * rows * JA_LD * (int)sizeof(float);
    dim3 grid(groups, heads, N);
    const float scale = 1.f / sqrtf((float)dh);
    int rc;
    if (rows == 64) {
        rc = set_dyn_smem((const void*)jb_sparse_attn_tc_kernel<8>, smem);
        if (rc) return rc;
        jb_sparse_attn_tc_kernel<8><<<grid, 128, smem, st>>>(qkv, out, out_bf16, T, heads, dh, block, pattern, scale);
    } else {
        rc = set_dyn_smem((const void*)jb_sparse_attn_tc_kernel<16>, smem);
        if (rc) return rc;
        jb_sparse_attn_tc_kernel<16><<<grid, 256, smem, st>>>(qkv, out, out_bf16, T, heads, dh, block, pattern, scale);
    }
    return jb_check();
}

static inline int ew_grid(long long n, int per_thread) {
    long long b = (n / per_thread + 255) / 256;
    if (b < 1) b = 1;
    if (b > 148 * 16) b = 148 * 16;
    return (int)b;
}
extern "C" int llark_quick_gelu(const float* x, float* y, long long n, cudaStream_t st) {
    if (n <= 0) return LLARK_OK;
    quick_gelu_kernel<<<ew_grid(n, 4), 256, 0, st>>>(x, y, n);
    return jb_check();
}
extern "C" int llark_add3(const float* a, const float* b, const float* c, float* out, long long n, cudaStream_t st) {
    if (n <= 0) return LLARK_OK;
    add3_kernel<<<ew_grid(n, 1), 256, 0, st>>>(a, b, c, out, n);
    return jb_check();
}
extern "C" int llark_jb_pool_batched(const float* acts, float* out, int N, long long clip_stride, int T_valid, int W,
                                     int frame, cudaStream_t st) {
    if (frame <= 0 || W <= 0 || N <= 0) return LLARK_EINVAL;
    const int frames = T_valid / frame;
    if (frames <= 0) return LLARK_OK;
    dim3 grid(frames, N, (W + 1023) / 1024);
    jb_pool_kernel<<<grid, 256, 0, st>>>(acts, out, clip_stride, frames, W, frame);
    return jb_check();
}
extern "C" int llark_jb_pool(const float* acts, float* out, int T_valid, int W, int frame, cudaStream_t st) {
    return llark_jb_pool_batched(acts, out, 1, 0, T_valid, W, frame, st);
}
extern "C" int llark_jb_label_cond(const float* total_row, const float* abs_table, const float* rel_table,
                                   const int* abs_bins, const int* rel_bins, float* out, int T, int W, cudaStream_t st) {
    if (T <= 0 || W <= 0) return LLARK_EINVAL;
    jb_label_cond_kernel<<<T, 256, 0, st>>>(total_row, abs_table, rel_table, abs_bins, rel_bins, out, W);
    return jb_check();
}
extern "C" int llark_colsum(const void* x, void* out, long long rows, int H, int accumulate, cudaStream_t st) {
    if (rows <= 0 || H <= 0) return LLARK_EINVAL;
    colsum_bf16_kernel<<<(H + 31) / 32, kColsumWarps * 32, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)out, rows, H, accumulate);
    return jb_check();
}
