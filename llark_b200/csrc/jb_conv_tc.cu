// The Jukebox encoder's convolutions on tcgen05: fp32 in and out, every product as three TF32 products of split operands.
//
// A convolution over time with few channels is a product with the time steps as rows: D[t, co] = sum over taps and channels of
// x[ci, t * stride + tap * dilation - pad] w[co, ci, tap]. A thread owns a time step: it reads its 32 channels (coalesced over the
// threads), splits them once (x = hi + lo, hi what TF32 holds) and writes them as one 128-byte row of the A operand (128-byte swizzle);
// a tap is the same rows read from another first row, stride 2 keeps even and odd steps apart. The thread later finds its sums in its
// own TMEM lane, so that neither the layout change nor the epilogue needs another pass through shared memory. The weights stay in
// shared memory, split once, hi rows and lo rows behind one another: one product of the hi part with both (hi hi and hi lo side by side
// in TMEM), one of the lo part with the hi rows. hi hi has accumulators of its own, one for the even taps, one for the odd ones: the
// tensor cores cut instead of rounding, so chains are kept short (error of a res block against 64 bits 8e-8 of its second product;
// 64 channels in, stride 2: 2.8e-7, with one chain 5.2e-7).
//
// A CTA is two or three groups of four warps, each with tiles of 128 steps, rows of A, accumulators and a barrier of its own; the next
// tile's values are requested as soon as this one's rows are written.
//
//   res block   y = x + W2 relu(W1 (*dilation d, 3 taps) relu(x) + b1) + b2, both convolutions of a tile in one visit: the second's A
//               operand is the first's result, written by the thread that owns the row. For dilations from 33 on: up to 32
//               jb_chain_tc.cu is ahead (158 to 171 us at the size below)
//   others      taps 4 stride 2 (32 or 64 channels in, 32 out), taps 3 (32 in, 64 out)
//
// What bounds it: the latency of load, split, product and read-back of a tile, hidden only by the other groups (a res block reads and
// writes every value once; the tensor pipe works less than a fifth of the time). Measured on a B200, 4 clips x 524288 steps x 32 channels, a
// res block: 232 us for dilations up to 64 and 323 at 81 (products issued by one lane 257 and 346), with mma.sync 413 and 685. Three groups of four warps and not more: 168
// registers a thread hold a step's 32 channels, the next step's and the sums (20 of them spilled); two groups with the input staged by cp.async: 325.
#include "common.cuh"

namespace llark {
extern thread_local int g_last_cuda_error;
namespace jbconv {

constexpr int TT = 128;        // time steps per tile = threads of a group = TMEM lanes
constexpr int kMaxDil = 81;    // two groups: the largest power of three whose halo rows (at most 256) two passes of 128 threads cover
constexpr int kMaxDil3 = 64;   // three groups: halo rows one for every thread, and the end of shared memory

struct Args {
    const float *x, *w1, *b1, *w2, *b2;
    float* y;
    int T, To, dil, rows, tiles_per_clip, tiles;  // input and output steps per clip; rows of A in a region
};

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {  // 128-byte rows, 8-row groups of 1024 bytes, 128-byte swizzle
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ uint32_t idesc_tf32(int n) {  // fp32 sums, both operands TF32 and K-major, M = 128
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TT >> 4) << 24);
}
// The leading part is rounded on its bits. The NaN of the GPU's own arithmetic (0x7fffffff) becomes -0 there, so the other part has to
// keep it, and is not rounded on its bits: the tensor cores cut the 13 bits that TF32 lacks, and times 1 + 2^-11.5 before that cut an
// error is 0.65 units of the last place at most and 0 on average (cvt.rna.tf32 for both parts is as exact and 6 % slower: 3471 us for the
// encoder of 4 clips against 3263).
__device__ __forceinline__ void split(float v, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u);  // |v - hi| <= 2^-11 |v|
    lo = (v - hi) * 1.00034527f;                                          // the difference is exact: |v - hi - lo| < 2^-21 |v|
}
// 32 values as row r of a region, split into its two parts, lo_at bytes apart
template <bool RELU>
__device__ __forceinline__ void put_row(unsigned char* region, int lo_at, int r, const float (&v)[32]) {
    unsigned char* row = region + r * 128;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        float hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split(RELU ? fmaxf(v[4 * q + e], 0.f) : v[4 * q + e], hi[e], lo[e]);
        unsigned char* p = row + ((q ^ (r & 7)) << 4);
        *reinterpret_cast<float4*>(p) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<float4*>(p + lo_at) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
}
// weights [COUT][NCI * 32][TAPS] -> per (32 channels, tap): hi rows [COUT][32], then lo rows; odd taps the other way round
template <int TAPS, int NCI, int COUT>
__device__ __forceinline__ bool put_weights(unsigned char* dst, const float* __restrict__ w) {  // true: one is 2^60 or more, or NaN
    bool large = false;
    for (int i = threadIdx.x; i < TAPS * NCI * COUT * 32; i += blockDim.x) {
        const int ci = i & 31, co = (i >> 5) % COUT, kb = i / (32 * COUT), tap = kb % TAPS, cb = kb / TAPS;
        float hi, lo;
        const float v = w[((long long)co * (NCI * 32) + cb * 32 + ci) * TAPS + tap];
        large |= !(fabsf(v) < 1152921504606846976.f);
        split(v, hi, lo);
        unsigned char* p = dst + kb * (2 * COUT * 128) + co * 128 + (((ci >> 2) ^ (co & 7)) << 4) + (ci & 3) * 4;
        *reinterpret_cast<float*>(p) = tap & 1 ? lo : hi;
        *reinterpret_cast<float*>(p + COUT * 128) = tap & 1 ? hi : lo;
    }
    return large;
}
// 32 channels of a tap. SIDE 0: hi hi into COUT columns from d on, hi lo + lo hi into the COUT columns behind them; SIDE 1: the weights'
// lo rows come first, hi hi goes into the COUT columns behind the shared ones. first: hi hi begins a chain; first_lo: the shared one.
template <int COUT, int SIDE>
__device__ __forceinline__ void products(uint32_t a, int lo_at, uint32_t w, uint32_t d, bool first, bool first_lo) {
    const uint64_t ah = smem_desc(a), al = smem_desc(a + lo_at), wd = smem_desc(w), wh = smem_desc(w + (SIDE ? COUT * 128 : 0)),
                   wl = smem_desc(w + (SIDE ? 0 : COUT * 128));
    const uint32_t both = d + (SIDE ? COUT : 0), hh = d + (SIDE ? 2 * COUT : 0), mid = d + COUT;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint64_t o = (uint64_t)(2 * k);  // 8 channels = 32 bytes
        const bool f = first && k == 0, fl = first_lo && k == 0;
        if (f == fl) {
            warp_umma_tf32(both, ah + o, wd + o, idesc_tf32(2 * COUT), !f);
        } else {
            warp_umma_tf32(hh, ah + o, wh + o, idesc_tf32(COUT), !f);
            warp_umma_tf32(mid, ah + o, wl + o, idesc_tf32(COUT), !fl);
        }
        warp_umma_tf32(mid, al + o, wh + o, idesc_tf32(COUT), 1);
    }
}

// One step's sums of 32 output channels by FMAs, bias first, channels outside, taps inside: for steps whose split products are not
// finite. An infinite value, or one that rounds to infinity, has a low part that is NaN, and infinity times a low part is another
// infinity or NaN: what belongs there is what the FMAs give. Nothing but such values gets here.
template <int TAPS, int STRIDE, int CIN>
__device__ __noinline__ void step_by_fma(const float* x, const float* w, const float* b, int T, int t, float (&h)[32]) {
#pragma unroll 1
    for (int c = 0; c < 32; ++c) {
        float acc = b[c];
#pragma unroll 1
        for (int i = 0; i < CIN * TAPS; ++i) {
            const int ci = i / TAPS, at = STRIDE * t + (i % TAPS) - 1;
            acc = fmaf(w[(long long)c * CIN * TAPS + i], at >= 0 && at < T ? x[(long long)ci * T + at] : 0.f, acc);
        }
        h[c] = acc;
    }
}

// The same for a res block's step, all of it: relu(NaN) = 0 as everywhere in them.
__device__ __noinline__ void res_step_by_fma(const Args& p, const float* x, int t, float (&o)[32]) {
    float h[32];
#pragma unroll 1
    for (int c = 0; c < 32; ++c) {
        float acc = p.b1[c];
#pragma unroll 1
        for (int i = 0; i < 96; ++i) {
            const int at = t + (i % 3 - 1) * p.dil;
            acc = fmaf(p.w1[c * 96 + i], at >= 0 && at < p.T ? fmaxf(x[(long long)(i / 3) * p.T + at], 0.f) : 0.f, acc);
        }
        h[c] = fmaxf(acc, 0.f);
    }
#pragma unroll 1
    for (int c = 0; c < 32; ++c) {
        float acc = p.b2[c];
#pragma unroll 1
        for (int i = 0; i < 32; ++i) acc = fmaf(p.w2[c * 32 + i], h[i], acc);
        o[c] = x[(long long)c * p.T + t] + acc;
    }
}

// A tile's input rows: stride 1: one region, row r is step t0 - dil + r; stride 2: even steps (row r is step 2 (t0 + r)), then odd ones
// (row r is step 2 (t0 + r) - 1). Shared memory, 1024-byte aligned: W1 | W2 (res block) | per group: the regions, hi rows then lo rows.
template <int TAPS, int STRIDE, int NCI, int COUT, bool RES, int NG>
__global__ void __launch_bounds__(NG * TT, 1)
conv_kernel(const Args p) {
    extern __shared__ unsigned char raw[];
    __shared__ uint64_t bars[NG];
    __shared__ uint32_t tmem_base;
    __shared__ float sb[COUT + 32];
    constexpr int CIN = NCI * 32, kGroup = RES ? 160 : 3 * COUT, kCols = NG * kGroup > 256 ? 512 : 256;
    const int grp = __shfl_sync(0xffffffffu, threadIdx.x >> 7, 0), tid = threadIdx.x & 127, warp = __shfl_sync(0xffffffffu, (threadIdx.x >> 5) & 3, 0);
    const int lo_at = p.rows * 128, region = 2 * lo_at;
    unsigned char* sw1 = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    unsigned char* sw2 = sw1 + TAPS * NCI * 2 * COUT * 128;
    unsigned char* sa = sw2 + (RES ? 2 * 32 * 128 : 0) + grp * (STRIDE * region);
    uint64_t* bar = &bars[grp];
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    if (threadIdx.x < 32) {
        tmem_alloc(&tmem_base, kCols);
        tmem_relinquish();
    }
    bool every = put_weights<TAPS, NCI, COUT>(sw1, p.w1);  // res block: all steps by FMAs
    if (RES) every |= put_weights<1, 1, 32>(sw2, p.w2);
    for (int i = threadIdx.x; i < COUT; i += NG * TT) sb[i] = p.b1[i];
    if (RES && threadIdx.x < 32) sb[COUT + threadIdx.x] = p.b2[threadIdx.x];
    fence_proxy_async_smem();
    tc_fence_before();
    if (RES)
        every = __syncthreads_or(every);
    else
        __syncthreads();
    tc_fence_after();
    // a group's columns: hi hi of the even taps, the mixed products, hi hi of the odd taps; the second convolution's (res block) from 96 on
    const uint32_t tmem = tmem_base + grp * kGroup, lane0 = tmem + ((uint32_t)(warp * 32) << 16);
    auto group_sync = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + grp) : "memory"); };
    auto where = [&](int tile, int& clip, int& t0) {
        clip = tile / p.tiles_per_clip;
        t0 = (tile - clip * p.tiles_per_clip) * TT;
    };
    const int n_halo = STRIDE == 1 ? 2 * p.dil : 2;
    const bool pairs = STRIDE == 2 && (reinterpret_cast<uintptr_t>(p.x) & 7) == 0;  // T is even
    float v[STRIDE][32], hv[32], xc[RES ? 32 : 1];
    auto load_halo = [&](int tile, int cb, int i) {
        int clip, t0;
        where(tile, clip, t0);
        const float* base = p.x + ((long long)clip * CIN + cb * 32) * p.T;
        const int at = STRIDE == 1 ? (i < p.dil ? t0 - p.dil + i : t0 + TT + i - p.dil) : (i == 0 ? 2 * t0 - 1 : 2 * (t0 + TT));
        const bool in = at >= 0 && at < p.T;
#pragma unroll
        for (int c = 0; c < 32; ++c) hv[c] = in ? base[(long long)c * p.T + at] : 0.f;
    };
    auto load = [&](int tile, int cb) {
        int clip, t0;
        where(tile, clip, t0);
        const float* base = p.x + ((long long)clip * CIN + cb * 32) * p.T;
        const float* src = base + STRIDE * (t0 + tid);
        const bool in = t0 + tid < p.To;
        if (STRIDE == 2 && pairs) {
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                const float2 f = in ? *reinterpret_cast<const float2*>(src + (long long)c * p.T) : make_float2(0.f, 0.f);
                v[0][c] = f.x;
                v[STRIDE - 1][c] = f.y;
            }
        } else {
#pragma unroll
            for (int s = 0; s < STRIDE; ++s)
#pragma unroll
                for (int c = 0; c < 32; ++c) v[s][c] = in ? src[(long long)c * p.T + s] : 0.f;
        }
        if (tid < n_halo) load_halo(tile, cb, tid);
    };
    int n = 0;  // product groups issued so far, each waited for before its rows are written again
    auto wait_last = [&]() { mbar_wait(bar, (uint32_t)((n - 1) & 1)); };
    auto read_sums = [&](int c0, float (&h)[32]) {  // 32 channels of the first convolution's three sums
        uint32_t a[32], b[32];
        tmem_ld_32x32b_x32(lane0 + c0, a);
        tmem_ld_32x32b_x32(lane0 + 2 * COUT + c0, b);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; ++c) h[c] = __uint_as_float(a[c]) + __uint_as_float(b[c]);
        tmem_ld_32x32b_x32(lane0 + COUT + c0, a);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; ++c) h[c] += __uint_as_float(a[c]);
    };
    const int first = blockIdx.x * NG + grp, step = gridDim.x * NG;
    if (first < p.tiles) load(first, 0);
    for (int tile = first; tile < p.tiles; tile += step) {
#pragma unroll
        for (int cb = 0; cb < NCI; ++cb) {
            if (cb) wait_last();
            if (STRIDE == 1) {
                put_row<RES>(sa, lo_at, tid + p.dil, v[0]);
                if (tid < n_halo) put_row<RES>(sa, lo_at, tid < p.dil ? tid : TT + tid, hv);
                if (RES && NG == 2 && tid + TT < n_halo) {  // more than 128 halo rows: the rest is read now
                    load_halo(tile, cb, tid + TT);
                    put_row<RES>(sa, lo_at, TT + TT + tid, hv);
                }
            } else {
                put_row<RES>(sa, lo_at, tid, v[0]);
                put_row<RES>(sa + region, lo_at, tid + 1, v[STRIDE - 1]);
                if (tid < 2) put_row<RES>(sa + (tid == 0 ? region : 0), lo_at, tid == 0 ? 0 : TT, hv);
            }
            if (RES)
#pragma unroll
                for (int c = 0; c < 32; ++c) xc[RES ? c : 0] = v[0][c];  // the residual: this thread's own step
            if (cb + 1 < NCI)
                load(tile, cb + 1);
            else if (tile + step < p.tiles)
                load(tile + step, 0);
            fence_proxy_async_smem();
            tc_fence_before();
            group_sync();  // the rows are written, and the sums of the tile before have been read
            if (warp == 0) {  // of the group, together
                tc_fence_after();
                const uint32_t a = smem_u32(sa), w = smem_u32(sw1) + cb * TAPS * 2 * COUT * 128;
#pragma unroll
                for (int tap = 0; tap < TAPS; ++tap) {
                    const uint32_t rows = STRIDE == 1 ? a + tap * p.dil * 128 : a + (tap & 1 ? 0 : region) + (tap >> 1) * 128;
                    if (tap & 1)
                        products<COUT, 1>(rows, lo_at, w + tap * 2 * COUT * 128, tmem, cb == 0 && tap == 1, false);
                    else
                        products<COUT, 0>(rows, lo_at, w + tap * 2 * COUT * 128, tmem, cb == 0 && tap == 0, cb == 0 && tap == 0);
                }
                warp_umma_commit(bar);
            }
            ++n;
        }
        int clip, t0;
        where(tile, clip, t0);
        const int t = t0 + tid;
        wait_last();
        tc_fence_after();
        float* out = p.y + (long long)clip * COUT * p.To + t;
        if constexpr (RES) {
            float h[32];
            read_sums(0, h);
#pragma unroll
            for (int c = 0; c < 32; ++c) h[c] += sb[c];
            const float first = h[0];  // a row that does not split leaves NaN in all channels, so one tells
            put_row<true>(sa, lo_at, tid, h);
            fence_proxy_async_smem();
            tc_fence_before();
            group_sync();
            if (warp == 0) {  // of the group, together
                tc_fence_after();
                products<32, 0>(smem_u32(sa), lo_at, smem_u32(sw2), tmem + 96, true, true);
                warp_umma_commit(bar);
            }
            ++n;
            wait_last();
            tc_fence_after();
            uint32_t a[32], b[32];
            tmem_ld_32x32b_x32(lane0 + 96, a);
            tmem_ld_32x32b_x32(lane0 + 128, b);
            tmem_ld_wait();
            const float second = __uint_as_float(a[0]) + __uint_as_float(b[0]);
            if (!(fabsf(first) <= 3.402823466e38f) || !(fabsf(second) <= 3.402823466e38f) || every) {
                if (t < p.To) {
                    float f[32];
                    res_step_by_fma(p, p.x + (long long)clip * CIN * p.T, t, f);
#pragma unroll
                    for (int c = 0; c < 32; ++c) out[(long long)c * p.To] = f[c];
                }
            } else if (t < p.To) {
#pragma unroll
                for (int c = 0; c < 32; ++c)
                    out[(long long)c * p.To] = xc[c] + ((__uint_as_float(a[c]) + __uint_as_float(b[c])) + sb[COUT + c]);
            }
        } else {
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 32) {
                float h[32], odd = 0.f;
                read_sums(c0, h);
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    h[c] += sb[c0 + c];
                    odd = fmaf(h[c], 0.f, odd);  // NaN as soon as one of them is not finite
                }
                if (odd != 0.f && t < p.To) {
                    float f[32];
                    step_by_fma<TAPS, STRIDE, CIN>(p.x + (long long)clip * CIN * p.T, p.w1 + c0 * CIN * TAPS, p.b1 + c0, p.T, t, f);
#pragma unroll
                    for (int c = 0; c < 32; ++c) h[c] = f[c];
                }
                if (t < p.To)
#pragma unroll
                    for (int c = 0; c < 32; ++c) out[(long long)(c0 + c) * p.To] = h[c];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) tmem_dealloc(tmem_base, kCols);
}

template <int TAPS, int STRIDE, int NCI, int COUT, bool RES, int NG>
static int launch(Args a, int N, cudaStream_t st) {
    a.rows = STRIDE == 1 ? (TT + 2 * a.dil + 7) & ~7 : TT + 8;
    const int smem = 1024 + TAPS * NCI * 2 * COUT * 128 + (RES ? 2 * 32 * 128 : 0) + NG * STRIDE * 2 * a.rows * 128;
    a.tiles_per_clip = (a.To + TT - 1) / TT;
    if ((long long)a.tiles_per_clip * N > 0x7fffffff) return LLARK_EINVAL;
    a.tiles = a.tiles_per_clip * N;
    const int grid = a.tiles < 148 * NG ? (a.tiles + NG - 1) / NG : 148;
    auto kernel = conv_kernel<TAPS, STRIDE, NCI, COUT, RES, NG>;
    // the limit is the function's, and another thread may launch it with another dilation: always the largest size
    const int most_rows = RES ? (TT + 2 * (NG == 3 ? kMaxDil3 : kMaxDil) + 7) & ~7 : a.rows;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem + NG * STRIDE * 2 * (most_rows - a.rows) * 128);
    if (e == cudaSuccess) {
        kernel<<<grid, NG * TT, smem, st>>>(a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

bool takes_resblock(int dil) { return dil <= kMaxDil; }
int resblock(const float* x, const float* w1, const float* b1, const float* w2, const float* b2, float* y, int N, int T, int dil,
             cudaStream_t st) {
    const Args a{x, w1, b1, w2, b2, y, T, T, dil, 0, 0, 0};
    return dil <= kMaxDil3 ? launch<3, 1, 1, 32, true, 3>(a, N, st) : launch<3, 1, 1, 32, true, 2>(a, N, st);
}
bool takes_down(int c_in, int c_out) { return (c_in == 32 || c_in == 64) && c_out == 32; }
int down(const float* x, const float* w, const float* b, float* y, int N, int c_in, int T, cudaStream_t st) {
    const Args a{x, w, b, nullptr, nullptr, y, T, T / 2, 1, 0, 0, 0};
    return c_in == 32 ? launch<4, 2, 1, 32, false, 2>(a, N, st) : launch<4, 2, 2, 32, false, 2>(a, N, st);
}
bool takes_k3(int c_in, int c_out) { return c_in == 32 && c_out == 64; }
int k3(const float* x, const float* w, const float* b, float* y, int N, int T, cudaStream_t st) {
    return launch<3, 1, 1, 64, false, 2>(Args{x, w, b, nullptr, nullptr, y, T, T, 1, 0, 0, 0}, N, st);
}

}  // namespace jbconv
}  // namespace llark
