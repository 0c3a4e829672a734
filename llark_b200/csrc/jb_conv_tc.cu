// The Jukebox encoder's convolutions on tcgen05: fp32 in and out, every product as three TF32 products of split operands.
//
// A convolution over time with few channels is a product with the time steps as rows: D[t, co] = sum over taps and channels of
// x[ci, t * stride + tap * dilation - pad] w[co, ci, tap]. A thread owns a time step: it reads the 32 channels of a tap (coalesced over
// the threads), splits them (x = hi + lo, hi what TF32 holds) and writes them as one 128-byte row of the A operand (128-byte swizzle),
// and later finds its sums in its own TMEM lane, so that neither the layout change nor the epilogue needs another pass through shared
// memory. Sums: hi hi in one accumulator, hi lo + lo hi in another (the tensor cores cut instead of rounding: short chains, 4e-7 of the
// terms' norm). A CTA walks tiles of 128 time steps with the weights resident (split once); the next tap's values are on their way
// while a tap's products run, and two CTAs share an SM.
//
//   res block   y = x + W2 relu(W1 (*dilation d, 3 taps) relu(x) + b1) + b2, both convolutions of a tile in one visit: the second's A
//               operand is the first's result, written by the thread that owns the row
//   others      taps 4 stride 2 (32 or 64 channels in, 32 out), taps 3 (32 in, 64 out)
//
// What bounds it: the instructions that split and write the operands, then memory (a res block reads and writes every value once).
// Measured on a B200, 4 clips x 524288 steps x 32 channels: see the launchers.
#include "common.cuh"

namespace llark {
extern thread_local int g_last_cuda_error;
namespace jbconv {

constexpr int TT = 128;                 // time steps per tile = threads = TMEM lanes
constexpr int kHalf = TT * 128;         // hi or lo part of a 32-channel slice of A: 16 KB
constexpr int kBuf = 2 * kHalf;

struct Args {
    const float *x, *w1, *b1, *w2, *b2;
    float* y;
    int T, To, dil, tiles_per_clip, tiles;  // input and output steps per clip
};

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {  // 128-byte rows, 8-row groups of 1024 bytes, 128-byte swizzle
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ uint32_t idesc_tf32(int n) {  // fp32 sums, both operands TF32 and K-major, M = 128
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TT >> 4) << 24);
}
__device__ __forceinline__ void split(float v, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u);  // rounded to nearest: |v - hi| <= 2^-12 |v|
    lo = __uint_as_float(__float_as_uint(v - hi) & 0xffffe000u);         // the difference is exact; cut at 2^-22 |v|
}
// 32 values as row r of a slice, split into its two parts
template <bool RELU>
__device__ __forceinline__ void put_row(unsigned char* buf, int r, const float (&v)[32]) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        float hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split(RELU ? fmaxf(v[4 * q + e], 0.f) : v[4 * q + e], hi[e], lo[e]);
        unsigned char* p = buf + r * 128 + ((q ^ (r & 7)) << 4);
        *reinterpret_cast<float4*>(p) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4*>(p + kHalf) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
}
// weights [COUT][NCI * 32][TAPS] -> per (tap, 32 channels): hi rows [COUT][32], then lo rows
template <int TAPS, int NCI, int COUT>
__device__ __forceinline__ void put_weights(unsigned char* dst, const float* __restrict__ w) {
    for (int i = threadIdx.x; i < TAPS * NCI * COUT * 32; i += TT) {
        const int ci = i & 31, co = (i >> 5) % COUT, kb = i / (32 * COUT), tap = kb / NCI, cb = kb % NCI;
        float hi, lo;
        split(w[((long long)co * (NCI * 32) + cb * 32 + ci) * TAPS + tap], hi, lo);
        unsigned char* p = dst + kb * (2 * COUT * 128) + co * 128 + (((ci >> 2) ^ (co & 7)) << 4) + (ci & 3) * 4;
        *reinterpret_cast<float*>(p) = hi;
        *reinterpret_cast<float*>(p + COUT * 128) = lo;
    }
}
// one slice of 32 channels: hi hi into column d_hh, the two mixed products into column d_x
template <int COUT>
__device__ __forceinline__ void products(uint32_t a, uint32_t w, uint32_t d_hh, uint32_t d_x, bool first) {
    const uint32_t id = idesc_tf32(COUT);
    const uint64_t ah = smem_desc(a), al = smem_desc(a + kHalf), wh = smem_desc(w), wl = smem_desc(w + COUT * 128);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint64_t o = (uint64_t)(2 * k);  // 8 channels = 32 bytes
        umma_tf32(d_hh, ah + o, wh + o, id, !(first && k == 0));
        umma_tf32(d_x, al + o, wh + o, id, !(first && k == 0));
        umma_tf32(d_x, ah + o, wl + o, id, 1);
    }
}

// shared memory: two slices of A | W1 | W2 (res block); 1024-byte aligned
template <int TAPS, int NCI, int COUT, bool RES> constexpr int smem_bytes() {
    return 2 * kBuf + TAPS * NCI * 2 * COUT * 128 + (RES ? 2 * 32 * 128 : 0) + 1024;
}

template <int TAPS, int STRIDE, int NCI, int COUT, bool RES>
__global__ void __launch_bounds__(TT, 2)
conv_kernel(const Args p) {
    extern __shared__ unsigned char raw[];
    __shared__ uint64_t bar[2];
    __shared__ uint32_t tmem_base;
    __shared__ float sb[COUT + 32];
    constexpr int KB = TAPS * NCI, CIN = NCI * 32;
    unsigned char* sm = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    unsigned char* sw1 = sm + 2 * kBuf;
    unsigned char* sw2 = sw1 + KB * 2 * COUT * 128;
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_base, 128);
        tmem_relinquish();
    }
    put_weights<TAPS, NCI, COUT>(sw1, p.w1);
    if (RES) put_weights<1, 1, 32>(sw2, p.w2);
    for (int i = tid; i < COUT; i += TT) sb[i] = p.b1[i];
    if (RES && tid < 32) sb[COUT + tid] = p.b2[tid];
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base, lane0 = tmem + ((uint32_t)(warp * 32) << 16);
    // columns: first convolution hi hi at 0, mixed at 64; second at 32 and 96
    float v[32], xc[RES ? 32 : 1];
    auto load = [&](int tile, int kb) {
        const int clip = tile / p.tiles_per_clip, t = (tile - clip * p.tiles_per_clip) * TT + tid;
        const int tap = kb / NCI, cb = kb % NCI;
        const int at = STRIDE == 1 ? t + (tap - TAPS / 2) * p.dil : STRIDE * t + tap - 1;
        const float* src = p.x + ((long long)clip * CIN + cb * 32) * p.T + at;
        const bool in = at >= 0 && at < p.T && t < p.To;
#pragma unroll
        for (int c = 0; c < 32; ++c) v[c] = in ? src[(long long)c * p.T] : 0.f;
    };
    int g = 0;  // groups of products so far: group g works on slice g & 1 and reports on barrier g & 1
    auto wait_group = [&](int n) { mbar_wait(&bar[n & 1], (uint32_t)((n >> 1) & 1)); };
    if ((int)blockIdx.x < p.tiles) load(blockIdx.x, 0);
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
#pragma unroll
        for (int kb = 0; kb < KB; ++kb) {
            unsigned char* buf = sm + (g & 1) * kBuf;
            if (g >= 2) wait_group(g - 2);
            put_row<RES>(buf, tid, v);
            if (RES && kb == 1)
#pragma unroll
                for (int c = 0; c < 32; ++c) xc[RES ? c : 0] = v[c];  // the residual: this thread's own step
            if (kb + 1 < KB)
                load(tile, kb + 1);
            else if (tile + (int)gridDim.x < p.tiles)
                load(tile + gridDim.x, 0);
            fence_proxy_async_smem();
            tc_fence_before();
            __syncthreads();  // the slice is written, and (first of a tile) the sums of the tile before have been read
            if (tid == 0) {
                tc_fence_after();
                products<COUT>(smem_u32(buf), smem_u32(sw1) + kb * 2 * COUT * 128, tmem, tmem + 64, kb == 0);
                umma_commit(&bar[g & 1]);
            }
            ++g;
        }
        const int clip = tile / p.tiles_per_clip, t = (tile - clip * p.tiles_per_clip) * TT + tid;
        wait_group(g - 1);
        tc_fence_after();
        float* out = p.y + (long long)clip * COUT * p.To + t;
        if constexpr (RES) {
            uint32_t a[32], b[32];
            tmem_ld_32x32b_x32(lane0, a);
            tmem_ld_32x32b_x32(lane0 + 64, b);
            tmem_ld_wait();
            float h[32];
#pragma unroll
            for (int c = 0; c < 32; ++c) h[c] = (__uint_as_float(a[c]) + __uint_as_float(b[c])) + sb[c];
            unsigned char* buf = sm + (g & 1) * kBuf;  // free: group g - 1 and all before it are done
            put_row<true>(buf, tid, h);
            fence_proxy_async_smem();
            tc_fence_before();
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
                products<32>(smem_u32(buf), smem_u32(sw2), tmem + 32, tmem + 96, true);
                umma_commit(&bar[g & 1]);
            }
            ++g;
            wait_group(g - 1);
            tc_fence_after();
            tmem_ld_32x32b_x32(lane0 + 32, a);
            tmem_ld_32x32b_x32(lane0 + 96, b);
            tmem_ld_wait();
            if (t < p.To)
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    out[(long long)c * p.To] = xc[c] + ((__uint_as_float(a[c]) + __uint_as_float(b[c])) + sb[COUT + c]);
        } else {
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 32) {
                uint32_t a[32], b[32];
                tmem_ld_32x32b_x32(lane0 + c0, a);
                tmem_ld_32x32b_x32(lane0 + 64 + c0, b);
                tmem_ld_wait();
                if (t < p.To)
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        out[(long long)(c0 + c) * p.To] = (__uint_as_float(a[c]) + __uint_as_float(b[c])) + sb[c0 + c];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 128);
}

template <int TAPS, int STRIDE, int NCI, int COUT, bool RES>
static int launch(Args a, int N, cudaStream_t st) {
    constexpr int smem = smem_bytes<TAPS, NCI, COUT, RES>();
    a.tiles_per_clip = (a.To + TT - 1) / TT;
    if ((long long)a.tiles_per_clip * N > 0x7fffffff) return LLARK_EINVAL;
    a.tiles = a.tiles_per_clip * N;
    const int grid = a.tiles < 296 ? a.tiles : 296;  // two CTAs on each of the 148 SMs
    cudaError_t e = cudaFuncSetAttribute(conv_kernel<TAPS, STRIDE, NCI, COUT, RES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) {
        conv_kernel<TAPS, STRIDE, NCI, COUT, RES><<<grid, TT, smem, st>>>(a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

int resblock(const float* x, const float* w1, const float* b1, const float* w2, const float* b2, float* y, int N, int T, int dil,
             cudaStream_t st) {
    return launch<3, 1, 1, 32, true>(Args{x, w1, b1, w2, b2, y, T, T, dil, 0, 0}, N, st);
}
bool takes_down(int c_in, int c_out) { return (c_in == 32 || c_in == 64) && c_out == 32; }
int down(const float* x, const float* w, const float* b, float* y, int N, int c_in, int T, cudaStream_t st) {
    const Args a{x, w, b, nullptr, nullptr, y, T, T / 2, 1, 0, 0};
    return c_in == 32 ? launch<4, 2, 1, 32, false>(a, N, st) : launch<4, 2, 2, 32, false>(a, N, st);
}
bool takes_k3(int c_in, int c_out) { return c_in == 32 && c_out == 64; }
int k3(const float* x, const float* w, const float* b, float* y, int N, int T, cudaStream_t st) {
    return launch<3, 1, 1, 64, false>(Args{x, w, b, nullptr, nullptr, y, T, T, 1, 0, 0}, N, st);
}

}  // namespace jbconv
}  // namespace llark
