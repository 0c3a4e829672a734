// Res blocks of the Jukebox encoder, up to four in one visit: y = x + W2 relu(W1 (*dilation d, 3 taps) relu(x) + b1) + b2, 32 channels,
// fp32 in and out, on tcgen05.
//
// One block alone (jb_conv_tc.cu) reads and writes every value once and waits for its tile's load, split, product and read-back. Here a
// CTA has a window of 512 steps of a clip and takes it through all blocks: a thread owns a step and keeps its 32 channels in registers,
// memory is read once and written once for the four, and a row is split once per convolution (no halo rows to split again). The steps
// that a block cannot know (dilation d takes d on either side) are lost: after dilations 1, 3, 9, 27 the inner 432 of 512 are results,
// and windows overlap by 80.
//
// A value is the sum of three bf16 numbers (24 bits), a product of two the six partial products down to 2^-16 of the first:
//   first convolution    A: rows of 64 bytes (32 channels, 64-byte swizzle) in shared memory, a region for each part, 32 spare rows at
//                        both ends; a tap is the same rows read from another first row. B: per tap the rows of the weights' first,
//                        second and third parts behind one another, kept in shared memory for all blocks. Sums: c0 = a1 b1,
//                        c1 = a1 b2 + a2 b1, c2 = a1 b3 + a2 b2 + a3 b1: a1 times all three (N = 96), a2 times the first two into the
//                        columns from c1 on, a3 times the first into c2
//   second convolution   A: the hidden rows, which need no shift, in TMEM, written by the thread that owns the step; c2 added to c1
// (Three TF32 products of two parts, as in jb_conv_tc.cu, take 256 bytes a row, for which there is no room beside four blocks' weights,
// and a third more passes of the A operand.)
//
// The four groups of four warps (128 rows each) meet only where they need one another: a group's products wait for its neighbours' rows,
// new rows for the neighbours' products, and the groups' first products are issued one group after another, so that the first reads its
// sums back and splits while the others' products run.
//
// An infinite number, or one whose first part rounds to infinity, leaves NaN in its other parts and so in all 32 sums of the rows that see it: the
// first channel's sums of either convolution tell; weights and biases from 2^60 on are told by their staging. The windows that had some
// are walked again in the end, block after block by FMAs in the order of the FMA kernel (relu(NaN) is 0 as there). Nothing but such numbers
// gets there. What it cannot tell: single products beyond the largest number, of both signs in one sum, are NaN and not the first one's
// infinity. (A look at all 32 channels for large numbers: 678 us where this takes 633.)
//
// What bounds it: 28 products a group and block, one behind another, and some 800 instructions a warp and block between them; 6500 cycles a
// block and window. Measured on a B200, 4 clips x 524288 steps, dilations 1, 3, 9, 27: 477 us where four launches of one block took 1075;
// one block alone 158 to 171 (257). Issued by one lane instead of a warp together a product took 50 to 85 cycles whatever its N, and the
// four blocks 634 us. Error of the encoder against 64 bits 2.2e-6 (2.9e-6). Tried: both convolutions from shared memory, all groups in step: 820;
// hidden rows in TMEM, all groups in step: 772; two windows of 256 steps side by side: 999; parts cut instead of rounded: 669.
#include "common.cuh"

namespace llark {
extern thread_local int g_last_cuda_error;
namespace jbconv {

constexpr int kMost = 4;                          // blocks per visit
constexpr int kWin = 512, kSpare = 32;            // steps of a window; spare rows on either side = the largest dilation
constexpr int kPart = (kWin + 2 * kSpare) * 64;   // bytes of a region: one part of every row
constexpr int kTapBytes = 96 * 64;                // a tap's weights: 32 rows for each part
constexpr int kBlockBytes = 4 * kTapBytes;        // three taps and the second convolution
constexpr int kHidden = 80;                       // a group's columns (128): c0, c1, c2; the hidden rows' parts from 80 on
constexpr int kMostHalo = 128;                    // dilations of a visit in all: at least half of a window is results
constexpr int kSmemChain = 1024 + 3 * kPart + kMost * kBlockBytes + kMost * 64 * 4;

struct ChainArgs {
    const float *x, *w1[kMost], *b1[kMost], *w2[kMost], *b2[kMost];
    float* y;
    int dil[kMost], blocks, halo;  // halo: sum of the dilations
    int T, windows_per_clip, windows;
    // WAVE: the blocks' input is the strided convolution of a waveform x [clips, 2 T] (one channel, taps 4, pad 1), made where it is needed:
    const float *w0, *b0;
};

// Channel by channel, bias first and the taps in order, as the FMA kernel of that convolution sums: v are samples 2 t - 1 .. 2 t + 2.
struct Samples { float v[4]; };
__device__ __forceinline__ Samples samples(const ChainArgs& p, int clip, int t) {
    const float* wave = p.x + (long long)clip * 2 * p.T;
    Samples s;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int i = 2 * t - 1 + k;
        s.v[k] = i >= 0 && i < 2 * p.T ? wave[i] : 0.f;
    }
    return s;
}
__device__ __forceinline__ float strided(const Samples& s, float4 w, float b) {
    return fmaf(w.w, s.v[3], fmaf(w.z, s.v[2], fmaf(w.y, s.v[1], fmaf(w.x, s.v[0], b))));
}

__device__ __forceinline__ uint64_t desc64(uint32_t addr) {  // 64-byte rows, 8-row groups of 512 bytes, 64-byte swizzle
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
__device__ __forceinline__ uint32_t idesc_bf16(int n) {  // fp32 sums, both operands bf16 and K-major, M = 128
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// two numbers as bf16, and what is left of them (exact: the difference of a number and its rounding to 8 bits)
__device__ __forceinline__ uint32_t part2(float& a, float& b) {
    const uint32_t u = pack_bf16x2(a, b);
    a -= __uint_as_float(u << 16);
    b -= __uint_as_float(u & 0xffff0000u);
    return u;
}
// the next part of eight numbers, and what is left of them
__device__ __forceinline__ uint4 part8(float (&v)[8]) {
    return make_uint4(part2(v[0], v[1]), part2(v[2], v[3]), part2(v[4], v[5]), part2(v[6], v[7]));
}
__device__ __forceinline__ bool too_large(float v) { return !(fabsf(v) < 1152921504606846976.f); }  // 2^60, or NaN
// eight channels (q: which eight) of row r
__device__ __forceinline__ void put8(unsigned char* region, int r, int q, float (&v)[8]) {
    unsigned char* p = region + r * 64 + ((q ^ ((r >> 1) & 3)) << 4);
#pragma unroll
    for (int part = 0; part < 3; ++part) *reinterpret_cast<uint4*>(p + part * kPart) = part8(v);
}
// weights [32][32][TAPS] -> per tap 96 rows: first parts, second parts, third parts
template <int TAPS>
__device__ __forceinline__ bool put_taps(unsigned char* dst, const float* __restrict__ w) {  // true: one is too large
    bool odd = false;
    for (int i = threadIdx.x; i < TAPS * 32 * 32; i += blockDim.x) {
        const int ci = i & 31, co = (i >> 5) & 31, tap = i >> 10;
        float v = w[(co * 32 + ci) * TAPS + tap];
        odd |= too_large(v);
#pragma unroll
        for (int part = 0; part < 3; ++part) {
            const __nv_bfloat16 h = __float2bfloat16_rn(v);
            v -= __bfloat162float(h);
            const int row = part * 32 + co;
            *reinterpret_cast<__nv_bfloat16*>(dst + tap * kTapBytes + row * 64 + (((ci >> 3) ^ ((row >> 1) & 3)) << 4) + (ci & 7) * 2) = h;
        }
    }
    return odd;
}
// one tap: A rows from byte address a on (first part), weights at w, sums at d
__device__ __forceinline__ void tap_products(uint32_t a, uint32_t w, uint32_t d, bool first) {
    const uint64_t a1 = desc64(a), a2 = desc64(a + kPart), a3 = desc64(a + 2 * kPart), b = desc64(w);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint64_t o = (uint64_t)(2 * k);  // 16 channels = 32 bytes
        warp_umma_f16(d, a1 + o, b + o, idesc_bf16(96), !(first && k == 0));
        warp_umma_f16(d + 32, a2 + o, b + o, idesc_bf16(64), 1);
        warp_umma_f16(d + 64, a3 + o, b + o, idesc_bf16(32), 1);
    }
}
// the second convolution: A is this group's own rows, so they stay in TMEM (16 columns for each part from a on); c2's products go to c1
__device__ __forceinline__ void second_products(uint32_t a, uint32_t w, uint32_t d) {
    const uint64_t b1 = desc64(w), b2 = desc64(w + 32 * 64), b3 = desc64(w + 64 * 64);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint64_t o = (uint64_t)(2 * k);
        const uint32_t a1 = a + 8 * k;  // 16 channels = 8 columns
        warp_umma_f16_ts(d, a1, b1 + o, idesc_bf16(64), k != 0);
        warp_umma_f16_ts(d + 32, a1, b3 + o, idesc_bf16(32), 1);
        warp_umma_f16_ts(d + 32, a1 + 16, b1 + o, idesc_bf16(32), 1);
        warp_umma_f16_ts(d + 32, a1 + 16, b2 + o, idesc_bf16(32), 1);
        warp_umma_f16_ts(d + 32, a1 + 32, b1 + o, idesc_bf16(32), 1);
    }
}
__device__ __forceinline__ void tmem_st_x4(uint32_t taddr, uint4 u) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w) : "memory");
}
__device__ __forceinline__ void tmem_ld_x8(uint32_t taddr, float (&v)[8]) {
    uint32_t u[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ void bias8(const float* b, float (&u)[8]) {
    const float4 u0 = *reinterpret_cast<const float4*>(b), u1 = *reinterpret_cast<const float4*>(b + 4);
    u[0] = u0.x, u[1] = u0.y, u[2] = u0.z, u[3] = u0.w, u[4] = u1.x, u[5] = u1.y, u[6] = u1.z, u[7] = u1.w;
}

// A window by FMAs: bias first, channels outside, taps inside. A thread has a step, rows: [32][kWin].
template <bool WAVE>
__device__ __noinline__ void window_by_fma(const ChainArgs& p, float* rows, int win) {
    const int clip = win / p.windows_per_clip, i = threadIdx.x;
    const int t = (win - clip * p.windows_per_clip) * (kWin - 2 * p.halo) - p.halo + i;
    const bool in = t >= 0 && t < p.T;
    const long long at = (long long)clip * 32 * p.T + t;
    __syncthreads();  // the window before has been read
    if (WAVE) {
        const Samples s = in ? samples(p, clip, t) : Samples{};
        for (int c = 0; c < 32; ++c)
            rows[c * kWin + i] = in ? strided(s, make_float4(p.w0[4 * c], p.w0[4 * c + 1], p.w0[4 * c + 2], p.w0[4 * c + 3]), p.b0[c]) : 0.f;
    } else {
        for (int c = 0; c < 32; ++c) rows[c * kWin + i] = in ? p.x[at + (long long)c * p.T] : 0.f;
    }
#pragma unroll 1
    for (int b = 0; b < p.blocks; ++b) {
        __syncthreads();
        float h[32], o[32];
        for (int c = 0; c < 32; ++c) {
            float acc = p.b1[b][c];
            for (int k = 0; k < 96; ++k) {
                const int j = i + (k % 3 - 1) * p.dil[b];
                acc = fmaf(p.w1[b][c * 96 + k], j >= 0 && j < kWin ? fmaxf(rows[k / 3 * kWin + j], 0.f) : 0.f, acc);
            }
            h[c] = fmaxf(acc, 0.f);
        }
        for (int c = 0; c < 32; ++c) {
            float acc = p.b2[b][c];
            for (int k = 0; k < 32; ++k) acc = fmaf(p.w2[b][c * 32 + k], h[k], acc);
            o[c] = rows[c * kWin + i] + acc;
        }
        __syncthreads();  // the neighbours have read this row
        for (int c = 0; c < 32; ++c) rows[c * kWin + i] = in ? o[c] : 0.f;
    }
    if (in && i >= p.halo && i < kWin - p.halo)
        for (int c = 0; c < 32; ++c) p.y[at + (long long)c * p.T] = rows[c * kWin + i];
}

// Which of a CTA's windows are walked again: a bit each, the last bit for all from there on.
__device__ __forceinline__ int bit_of(int win) { return min((win - (int)blockIdx.x) / (int)gridDim.x, 32 * 32 - 1); }
__device__ __forceinline__ void again(uint32_t* odd, int win) { atomicOr(&odd[bit_of(win) >> 5], 1u << (bit_of(win) & 31)); }

template <bool WAVE>
__global__ void __launch_bounds__(kWin, 1)
chain_kernel(const __grid_constant__ ChainArgs p) {
    extern __shared__ unsigned char raw[];
    __shared__ uint64_t ready[4], done1[4], done2[4], turn[4];  // per group: rows written; first products done; second products done; first products on their way
    __shared__ uint32_t tmem_base;
    __shared__ uint32_t odd[32];
    __shared__ float4 sw0[WAVE ? 32 : 1];
    __shared__ float sb0[WAVE ? 32 : 1];
    unsigned char* sa = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    unsigned char* sw = sa + 3 * kPart;
    float* sb = reinterpret_cast<float*>(sw + kMost * kBlockBytes);  // [block][b1 | b2]
    const int g = __shfl_sync(0xffffffffu, threadIdx.x >> 7, 0), warp = __shfl_sync(0xffffffffu, (threadIdx.x >> 5) & 3, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i) {
            mbar_init(&ready[i], 4);
            mbar_init(&done1[i], 1);
            mbar_init(&done2[i], 1);
            mbar_init(&turn[i], 1);
        }
        mbar_fence_init();
    }
    if (threadIdx.x < 32) {
        tmem_alloc(&tmem_base, 512);
        tmem_relinquish();
    }
    if (WAVE && threadIdx.x < 32) {
        const float* w = p.w0 + 4 * threadIdx.x;
        sw0[threadIdx.x] = make_float4(w[0], w[1], w[2], w[3]);
        sb0[threadIdx.x] = p.b0[threadIdx.x];
    }
    bool every = false;
    for (int b = 0; b < p.blocks; ++b) {
        every |= put_taps<3>(sw + b * kBlockBytes, p.w1[b]);
        every |= put_taps<1>(sw + b * kBlockBytes + 3 * kTapBytes, p.w2[b]);
        if (threadIdx.x < 32) {
            const float u1 = p.b1[b][threadIdx.x], u2 = p.b2[b][threadIdx.x];
            sb[b * 64 + threadIdx.x] = u1;
            sb[b * 64 + 32 + threadIdx.x] = u2;
            every |= too_large(u1) || too_large(u2);
        }
    }
    for (int i = threadIdx.x; i < 3 * kPart / 16; i += kWin) reinterpret_cast<uint4*>(sa)[i] = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async_smem();
    tc_fence_before();
    const uint32_t odd_from_the_start = __syncthreads_or(every) ? 0xffffffffu : 0u;
    tc_fence_after();
    if (threadIdx.x < 32) odd[threadIdx.x] = odd_from_the_start;
    __syncthreads();
    const uint32_t tmem = tmem_base + g * 128, lane0 = tmem + ((uint32_t)(warp * 32) << 16);
    const int row = kSpare + threadIdx.x, stride = kWin - 2 * p.halo;
    auto where = [&](int win, int& clip, int& t) {
        clip = win / p.windows_per_clip;
        t = (win - clip * p.windows_per_clip) * stride - p.halo + (int)threadIdx.x;
    };
    uint32_t par = 0;  // every barrier completes once per block
    for (int win = blockIdx.x; win < p.windows; win += gridDim.x) {
        int clip, t;
        where(win, clip, t);
        const bool in = t >= 0 && t < p.T;  // outside: zeros for every convolution
        float x[32];
        if (WAVE) {
            const Samples s = in ? samples(p, clip, t) : Samples{};
#pragma unroll
            for (int c = 0; c < 32; ++c) x[c] = in ? strided(s, sw0[c], sb0[c]) : 0.f;
        } else {
            const float* src = p.x + (long long)clip * 32 * p.T + t;
#pragma unroll
            for (int c = 0; c < 32; ++c) x[c] = in ? src[(long long)c * p.T] : 0.f;
        }
        if (win + (int)gridDim.x < p.windows) {  // the next window on its way to L2
            int nclip, nt;
            where(win + gridDim.x, nclip, nt);
            if (WAVE) {
                if (nt >= 0 && nt < p.T && (lane & 15) == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.x + (long long)nclip * 2 * p.T + 2 * nt));
            } else if (nt >= 0 && nt < p.T && (lane & 7) == 0) {
                const float* next = p.x + (long long)nclip * 32 * p.T + nt;
#pragma unroll 4
                for (int c = 0; c < 32; ++c) asm volatile("prefetch.global.L2 [%0];" ::"l"(next + (long long)c * p.T));
            }
        }
#pragma unroll 1
        for (int b = 0; b < p.blocks; ++b, par ^= 1) {
            const float* bias = sb + b * 64;
            // the neighbours' products of the block before have read these rows (the first time nothing is waited for)
            if (g > 0) mbar_wait(&done1[g - 1], par ^ 1);
            if (g < 3) mbar_wait(&done1[g + 1], par ^ 1);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = in ? fmaxf(x[8 * q + e], 0.f) : 0.f;
                put8(sa, row, q, v);
            }
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[g]);
            if (warp == 0) {  // of the group, together
                if (g > 0) mbar_wait(&ready[g - 1], par);
                mbar_wait(&ready[g], par);
                if (g < 3) mbar_wait(&ready[g + 1], par);
                if (g > 0) mbar_wait(&turn[g - 1], par);  // one group's products after another's: the first's sums can be read early
                tc_fence_after();
                const uint32_t a = smem_u32(sa) + (kSpare + g * 128) * 64, w = smem_u32(sw) + b * kBlockBytes;
                const int d = p.dil[b] * 64;
#pragma unroll
                for (int tap = 0; tap < 3; ++tap) tap_products(a + (tap - 1) * d, w + tap * kTapBytes, tmem, tap == 0);
                warp_umma_commit(&done1[g]);
                __syncwarp();
                if (lane == 0) mbar_arrive(&turn[g]);
            }
            __syncwarp();
            mbar_wait(&done1[g], par);
            tc_fence_after();
            float s[32];
#pragma unroll
            for (int q = 0; q < 4; ++q) {  // all of c1 and c2 first: the hidden rows' parts take c2's last columns
                float c1[8], c2[8];
                tmem_ld_x8(lane0 + 32 + 8 * q, c1);
                tmem_ld_x8(lane0 + 64 + 8 * q, c2);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) s[8 * q + e] = c1[e] + c2[e];
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float v[8], u[8];
                tmem_ld_x8(lane0 + 8 * q, v);
                bias8(bias + 8 * q, u);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    v[e] = (v[e] + s[8 * q + e]) + u[e];
                    if (q == 0 && e == 0 && !(fabsf(v[0]) <= 3.402823466e38f)) again(odd, win);
                    v[e] = fmaxf(v[e], 0.f);
                }
#pragma unroll
                for (int part = 0; part < 3; ++part) tmem_st_x4(lane0 + kHidden + 16 * part + 4 * q, part8(v));
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
            if (warp == 0) {  // of the group, together
                tc_fence_after();
                second_products(tmem + kHidden, smem_u32(sw) + b * kBlockBytes + 3 * kTapBytes, tmem);
                warp_umma_commit(&done2[g]);
            }
            __syncwarp();
            mbar_wait(&done2[g], par);
            tc_fence_after();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float c0[8], c1[8], u[8];
                tmem_ld_x8(lane0 + 8 * q, c0);
                tmem_ld_x8(lane0 + 32 + 8 * q, c1);
                bias8(bias + 32 + 8 * q, u);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float o = (c0[e] + c1[e]) + u[e];
                    if (q == 0 && e == 0 && !(fabsf(o) <= 3.402823466e38f)) again(odd, win);
                    x[8 * q + e] += o;
                }
            }
        }
        if (in && (int)threadIdx.x >= p.halo && (int)threadIdx.x < kWin - p.halo) {
            float* dst = p.y + (long long)clip * 32 * p.T + t;
#pragma unroll
            for (int c = 0; c < 32; ++c) dst[(long long)c * p.T] = x[c];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) tmem_dealloc(tmem_base, 512);
    for (int win = blockIdx.x; win < p.windows; win += gridDim.x)
        if (odd[bit_of(win) >> 5] >> (bit_of(win) & 31) & 1u) window_by_fma<WAVE>(p, reinterpret_cast<float*>(sa), win);
}

int chain_length(const int* dil, int n) {
    int k = 0, halo = 0;
    while (k < n && k < kMost && dil[k] >= 1 && dil[k] <= kSpare && halo + dil[k] <= kMostHalo) halo += dil[k++];
    return k;
}

// w0, b0: of the strided convolution in front, or NULL
int chain(const float* x, const float* w0, const float* b0, const float* const* w, const int* dil, int n, float* y, int N, int T, cudaStream_t st) {
    ChainArgs a = {};
    a.w0 = w0, a.b0 = b0;
    a.x = x, a.y = y, a.T = T, a.blocks = n;
    for (int b = 0; b < n; ++b) {
        a.w1[b] = w[4 * b], a.b1[b] = w[4 * b + 1], a.w2[b] = w[4 * b + 2], a.b2[b] = w[4 * b + 3];
        a.dil[b] = dil[b];
        a.halo += dil[b];
    }
    const int stride = kWin - 2 * a.halo;
    a.windows_per_clip = (T + stride - 1) / stride;
    if ((long long)a.windows_per_clip * N > 0x7fffffff - 148) return LLARK_EINVAL;
    a.windows = a.windows_per_clip * N;
    auto kernel = w0 ? chain_kernel<true> : chain_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemChain);
    if (e == cudaSuccess) {
        kernel<<<a.windows < 148 ? a.windows : 148, kWin, kSmemChain, st>>>(a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

}  // namespace jbconv
}  // namespace llark
