// Nearest code of the Jukebox bottleneck: x [N, 64, T] channels-first against a codebook [n_codes, 64], fp32.
//
// The result is the first minimum of dist = (|x|^2 - 2 x.k) + |k|^2 in fp32, every sum in the order of the channels, as one walk over all
// codes gives it. Walking them all is 64 FMAs a pair; here tensor cores say which codes can be it at all, and only those are walked:
//   s_j = |k_j|^2 - 2 (x1 k1 + x1 k2 + x2 k1) with x = x1 + x2, k = k1 + k2 in bf16 parts (tcgen05, fp32 sums) is off from dist_j - |x|^2 by
//   at most eps = 2^-13 |x| |k| + 2^-21 (|x| + |k|)^2, |k| the largest of the codes so far: two parts leave 2^-18 of a number, so
//   that the product lacks three times 2^-18 |x| |k| (Cauchy-Schwarz), the sum of 192 products on the tensor cores is off by less than
//   2^-16 |x| |k|, the walk's sum of 64 by 2^-18, and the three fp32 roundings of dist by 2^-24 (|x| + |k|)^2 each.
//   Every code whose s - eps is not above the least s + eps is walked.
// From 1e18 on (|x| or a code's |k|) sums may pass the largest number, and the bound says nothing: all codes are walked.
// Codes whose |k|^2 is not finite have a dist that is not below anything, and are no candidates; a vector whose |x|^2 is not finite has
// none below infinity and keeps code 0. Candidates are noted in runs of 32 codes, twelve runs a thread.
//
// A CTA has 256 vectors (two row tiles of A), or 128 where there are then no more CTAs than SMs, and goes through the codebook in tiles of 128
// codes: four threads make one row of B of the next tile while the tensor cores multiply; two or four threads share a vector's sums. As
// soon as a list overflows even after runs have been struck off, or where in the end a vector has more candidates than one in sixteen codes
// (each costs its thread a microsecond, alone), the CTA walks all codes for its vectors (walk_all): with codes that are close or equal that is
// what has to be done anyway. Vectors are counted through, whatever their clips' lengths.
//
// With no more than a CTA of 64 vectors an SM, or up to 256 codes, walk_all is all there is (walk_kernel): no slower than a walk of one lane per
// two vectors for any data, where candidates would be faster for codes apart and slower for codes together.
//
// What bounds it: a tile's chain of conversion, products and sums' reading, and the candidates' walks at the end; walk_all: shared memory, 64
// FMAs for four 16-byte reads. Measured on a B200, 2048 codes, us, codes apart / a third of them equal; in brackets the walk of one lane per two
// vectors: 64 to 8192 vectors 84 / 84 (107), 16384 62 / 175 (210), 24576 89 / 260 (312), 32768 91 / 260 (415); 512 codes, 16384 vectors 23 / 51
// (55), 32768 31 / 82 (100). The walk of 8192 vectors by CTAs of 128: 62 / 165. Of 64 codes and less the walk's staging is seen: 10 (8).
#include "common.cuh"
#include <math.h>

namespace llark {
extern thread_local int g_last_cuda_error;
namespace jbvq {

// x [N, 64, T] and the codes in shared memory, channel by channel; a thread has 8 vectors x 8 codes of a tile
template <int ROWS, int THREADS>
struct Walk {
    static constexpr int kGroups = ROWS / 8, kShares = THREADS / kGroups, kCodes = 8 * kShares, kPitch = kCodes + 4;
    static constexpr int kTileFloats = 64 * kPitch;
    static constexpr int kBytes = (64 * ROWS + 2 * kTileFloats) * 4;
    static_assert(kShares >= 8 && kGroups % 4 == 0 && 2 * kTileFloats >= 2 * ROWS * kShares, "");
};
// All codes for ROWS vectors from number v0 on (of N T): dist as above, every sum in the order of the channels. The thread's vectors and codes are two
// runs of four each, half a tile apart: a quarter-warp reads 128 bytes side by side.
template <int ROWS, int THREADS>
__device__ __forceinline__ void walk_all(float* sx, float* sk, float* skk, float* sxx, const float* __restrict__ x,
                         const float* __restrict__ cb, long long* __restrict__ codes, int v0, int vectors, int T, int n_codes) {
    using W = Walk<ROWS, THREADS>;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int vg = (warp % (W::kGroups / 4)) * 4 + (lane >> 3), cg = (warp / (W::kGroups / 4)) * 8 + (lane & 7);
    auto ask = [&](int tile) {  // 4 codes x 8 channels a warp: sectors of 32 bytes there, all banks here
        float* dst = sk + (tile & 1) * W::kTileFloats;
        for (int i = warp; i < 8 * (W::kCodes / 4); i += THREADS / 32) {
            const int e = (i & 7) * 8 + (lane >> 2), r = (i >> 3) * 4 + (lane & 3), j = tile * W::kCodes + r;
            if (j < n_codes)  // what lies behind the last code is multiplied and never taken
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst + e * W::kPitch + r)), "l"(cb + (long long)j * 64 + e)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    {
        static_assert(THREADS % ROWS == 0, "");
        const int v = v0 + tid % ROWS, n = v / T;
        const float* src = x + (long long)n * 64 * T + (v - n * T);
        for (int e = tid / ROWS; e < 64; e += THREADS / ROWS) {
            float* to = sx + e * ROWS + tid % ROWS;
            if (v < vectors)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(to)), "l"(src + (long long)e * T) : "memory");
            else
                *to = 0.f;
        }
    }
    ask(0);
    float best[8];
    int code[8];
#pragma unroll
    for (int v = 0; v < 8; ++v) best[v] = INFINITY, code[v] = 0;
    const int tiles = (n_codes + W::kCodes - 1) / W::kCodes;
    for (int tile = 0; tile < tiles; ++tile) {
        const float* k0 = sk + (tile & 1) * W::kTileFloats;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // this tile is there, and the one before has been read
        if (tile + 1 < tiles) ask(tile + 1);
        if (tid < W::kCodes) {
            float kk = 0.f;
#pragma unroll 16
            for (int e = 0; e < 64; ++e) kk = fmaf(k0[e * W::kPitch + tid], k0[e * W::kPitch + tid], kk);
            skk[(tile & 1) * W::kCodes + tid] = kk;
        }
        if (tile == 0 && tid >= THREADS - ROWS) {
            const int v = tid - (THREADS - ROWS);
            float xx = 0.f;
#pragma unroll 16
            for (int e = 0; e < 64; ++e) xx = fmaf(sx[e * ROWS + v], sx[e * ROWS + v], xx);
            sxx[v] = xx;
        }
        float dot[8][8];
#pragma unroll
        for (int v = 0; v < 8; ++v)
#pragma unroll
            for (int c = 0; c < 8; ++c) dot[v][c] = 0.f;
        const float *px = sx + vg * 4, *pk = k0 + cg * 4;
        const int left = n_codes - tile * W::kCodes;
        if ((cg & ~7) * 4 < left)  // the warp's first code
#pragma unroll 2
        for (int e = 0; e < 64; ++e, px += ROWS, pk += W::kPitch) {
            const float4 xa = *reinterpret_cast<const float4*>(px), xb = *reinterpret_cast<const float4*>(px + ROWS / 2);
            const float4 ka = *reinterpret_cast<const float4*>(pk), kb = *reinterpret_cast<const float4*>(pk + W::kCodes / 2);
            const float xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w}, kv[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
#pragma unroll
            for (int v = 0; v < 8; ++v)
#pragma unroll
                for (int c = 0; c < 8; ++c) dot[v][c] = fmaf(xv[v], kv[c], dot[v][c]);
        }
        __syncthreads();  // |k|^2 of this tile, |x|^2
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int r = (c >> 2) * (W::kCodes / 2) + cg * 4 + (c & 3), j = tile * W::kCodes + r;
            const float kk = skk[(tile & 1) * W::kCodes + r];
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const float dist = (sxx[(v >> 2) * (ROWS / 2) + vg * 4 + (v & 3)] - 2.f * dot[v][c]) + kk;
                if (j < n_codes && dist < best[v]) {
                    best[v] = dist;
                    code[v] = j;
                }
            }
        }
    }
    __syncthreads();
    float* sd = sk;  // [share][vector]
    int* sj = reinterpret_cast<int*>(sk + ROWS * W::kShares);
#pragma unroll
    for (int v = 0; v < 8; ++v) {
        const int at = cg * ROWS + (v >> 2) * (ROWS / 2) + vg * 4 + (v & 3);
        sd[at] = best[v];
        sj[at] = code[v];
    }
    __syncthreads();
    if (tid < ROWS && v0 + tid < vectors) {
        float d = INFINITY;
        int j = 0;
        for (int c = 0; c < W::kShares; ++c) {  // the shares' codes are not in order: equal ones, the first
            const float dc = sd[c * ROWS + tid];
            const int jc = sj[c * ROWS + tid];
            if (dc < d || (dc == d && d < INFINITY && jc < j)) d = dc, j = jc;
        }
        codes[v0 + tid] = j;
    }
}

constexpr int kWalkRows = 64, kWalkThreads = 128;
__global__ void __launch_bounds__(kWalkThreads, 3)
walk_kernel(const float* __restrict__ x, const float* __restrict__ cb, long long* __restrict__ codes, int vectors, int T, int n_codes) {
    using W = Walk<kWalkRows, kWalkThreads>;
    extern __shared__ __align__(16) unsigned char raw[];
    __shared__ float skk[2 * W::kCodes], sxx[kWalkRows];
    float* sx = reinterpret_cast<float*>(raw);
    walk_all<kWalkRows, kWalkThreads>(sx, sx + 64 * kWalkRows, skk, sxx, x, cb, codes, blockIdx.x * kWalkRows, vectors, T, n_codes);
}

// in vq_kernel: called, so that its registers are not the sums' and candidates'
template <int ROWS, int THREADS>
__device__ __noinline__ void walk_all_called(float* sx, float* sk, float* skk, float* sxx,
                                             const float* __restrict__ x, const float* __restrict__ cb, long long* __restrict__ codes,
                                             int v0, int vectors, int T, int n_codes) {
    walk_all<ROWS, THREADS>(sx, sk, skk, sxx, x, cb, codes, v0, vectors, T, n_codes);
}

constexpr int kE = 64, kThreads = 512, kTile = 128, kList = 12;
constexpr int kPartB = kTile * 128;                // bytes of a part: 64 bf16 a row
constexpr int kListBytes = kList * kThreads * 12;  // per run: s - eps of its least, which of the 32, number of the run
template <int ROWS>  // 128 or 256 vectors, 4 or 2 threads each
struct Shape {
    static constexpr int kPartA = ROWS * 128, kParts = kThreads / ROWS, kCols = kTile / kParts;
    static constexpr int kLists = 1024 + 2 * kPartA + 2 * 2 * kPartB + kListBytes, kWalk = 1024 + Walk<ROWS, kThreads>::kBytes;
    static constexpr int kSmem = kLists > kWalk ? kLists : kWalk;  // walk_all takes the place of rows and lists
};

__device__ __forceinline__ uint64_t desc(uint32_t addr) {  // 128-byte rows, 8-row groups of 1024 bytes, 128-byte swizzle
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTile >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

__device__ __forceinline__ void load8(const float* __restrict__ src, bool vec, float (&v)[8]) {
    if (vec) {
        const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = src[e];
    }
}
// eight channels (q: which eight) of row r, both parts
__device__ __forceinline__ void put8(unsigned char* rows, int part_bytes, int r, int q, const float (&v)[8]) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        hi[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
        lo[i] = pack_bf16x2(v[2 * i] - __uint_as_float(hi[i] << 16), v[2 * i + 1] - __uint_as_float(hi[i] & 0xffff0000u));
    }
    unsigned char* p = rows + r * 128 + ((q ^ (r & 7)) << 4);
    *reinterpret_cast<uint4*>(p) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(p + part_bytes) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

struct Runs {  // a thread's noted runs, ascending
    float* low;
    uint32_t* mask;
    int* run;
    int n;
    bool all;  // too many: all codes are walked
};
__device__ __noinline__ void note(Runs& r, float low, uint32_t mask, int run, float least) {
    if (r.all) return;
    if (r.n == kList) {
        int k = 0;
        for (int i = 0; i < kList; ++i) {
            const float l = r.low[i * kThreads];
            if (l <= least) {
                r.low[k * kThreads] = l;
                r.mask[k * kThreads] = r.mask[i * kThreads];
                r.run[k * kThreads] = r.run[i * kThreads];
                ++k;
            }
        }
        r.n = k;
        if (k == kList) {
            r.all = true;
            return;
        }
    }
    r.low[r.n * kThreads] = low;
    r.mask[r.n * kThreads] = mask;
    r.run[r.n * kThreads] = run;
    ++r.n;
}

template <int ROWS>
__global__ void __launch_bounds__(kThreads, 1)
vq_kernel(const float* __restrict__ x, const float* __restrict__ cb, long long* __restrict__ codes, int vectors, int T, int n_codes) {
    using S = Shape<ROWS>;
    constexpr int kPartA = S::kPartA, kParts = S::kParts, kCols = S::kCols;
    extern __shared__ unsigned char raw[];
    __shared__ __align__(16) float skk[2 * Walk<ROWS, kThreads>::kCodes];  // of two tiles; read four at a time
    __shared__ uint64_t bar[2];
    __shared__ uint32_t tmem_base, most_kk;  // most_kk: bits of the largest finite |k|^2 of the tiles made so far
    __shared__ float s_least[kParts][ROWS], s_dist[kParts][ROWS];
    __shared__ int s_code[kParts][ROWS];
    unsigned char* sa = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    unsigned char* sb = sa + 2 * kPartA;
    unsigned char* sl = sb + 2 * 2 * kPartB;
    const int tid = threadIdx.x, row = tid & (ROWS - 1), part = tid / ROWS, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int v0 = blockIdx.x * ROWS, number = v0 + row, n = number / T;  // this thread's vector
    const bool vec = (reinterpret_cast<uintptr_t>(cb) & 15) == 0, in = number < vectors;
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
        most_kk = 0u;
    }
    if (warp == 0) {
        tmem_alloc(&tmem_base, 512);
        tmem_relinquish();
    }
    const float* const xs = x + (long long)n * kE * T + (number - n * T);
    float xx = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = in ? xs[(long long)(8 * q + e) * T] : 0.f;
            xx = fmaf(v[e], v[e], xx);
        }
        if (q * kParts / 8 == part) put8(sa, kPartA, row, q, v);  // the threads of a vector write a share of its row each
    }
    const float xn = sqrtf(xx) * 1.0001f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base, lane0 = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (row >> 7) * kTile + part * kCols;
    const int tiles = (n_codes + kTile - 1) / kTile;

    auto make_tile = [&](int tile) {  // a quarter of a code: 16 channels
        const int r = tid >> 2, seg = tid & 3, j = tile * kTile + r, buf = tile & 1;
        const bool real = j < n_codes;
        const float* src = cb + (long long)(real ? j : 0) * kE + 16 * seg;
        float v[2][8];
        load8(src, vec, v[0]);
        load8(src + 8, vec, v[1]);
        float kk = real ? 0.f : INFINITY;
#pragma unroll
        for (int s = 0; s < 4; ++s) {  // in the order of the channels, handed from quarter to quarter
            float sum = kk;
#pragma unroll
            for (int i = 0; i < 16; ++i) sum = fmaf(v[i >> 3][i & 7], v[i >> 3][i & 7], sum);
            kk = __shfl_sync(0xffffffffu, sum, (lane & ~3) + s);
        }
        put8(sb + buf * 2 * kPartB, kPartB, r, 2 * seg, v[0]);
        put8(sb + buf * 2 * kPartB, kPartB, r, 2 * seg + 1, v[1]);
        if (!real) kk = INFINITY;
        if (seg == 0) skk[buf * kTile + r] = kk;
        const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(kk < INFINITY ? kk : 0.f));
        if (lane == 0) atomicMax(&most_kk, most);
        fence_proxy_async_smem();
    };
    auto multiply = [&](int tile) {  // one warp
        const uint32_t b = smem_u32(sb) + (tile & 1) * 2 * kPartB;
#pragma unroll
        for (int rt = 0; rt < ROWS / 128; ++rt) {
            const uint32_t a = smem_u32(sa) + rt * 128 * 128, d = tmem + (tile & 1) * 256 + rt * kTile;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                warp_umma_f16(d, desc(a) + 2 * k, desc(b) + 2 * k, kIdesc, k != 0);
                warp_umma_f16(d, desc(a) + 2 * k, desc(b + kPartB) + 2 * k, kIdesc, 1);
                warp_umma_f16(d, desc(a + kPartA) + 2 * k, desc(b) + 2 * k, kIdesc, 1);
            }
        }
        warp_umma_commit(&bar[tile & 1]);
    };

    float least = INFINITY;  // smallest s + eps so far
    const bool live = in && xx < INFINITY;
    float* const list = reinterpret_cast<float*>(sl);
    Runs runs = {list + tid, reinterpret_cast<uint32_t*>(list + kList * kThreads) + tid,
                 reinterpret_cast<int*>(list + 2 * kList * kThreads) + tid, 0, false};
    make_tile(0);
    __syncthreads();
    bool many = false;
    for (int tile = 0; tile < tiles; ++tile) {
        const int buf = tile & 1;
        if (warp == 0) {
            tc_fence_after();
            multiply(tile);
        }
        __syncwarp();
        // the other buffer's last readers were the products of tile - 1, which were waited for, and the sums' readers, who are past the barrier
        const float kn = sqrtf(__uint_as_float(*const_cast<volatile uint32_t*>(&most_kk))) * 1.0001f;
        if (tile + 1 < tiles) make_tile(tile + 1);
        const float eps = 1.220703125e-4f * xn * kn + 4.76837158203125e-7f * (xn + kn) * (xn + kn) + 1e-30f;
        if (!(xn < 1e18f && kn < 1e18f)) runs.all = true;
        mbar_wait(&bar[buf], (tile >> 1) & 1);
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < kCols; c += 32) {
            uint32_t u[32];
            tmem_ld_32x32b_x32(lane0 + buf * 256 + c, u);
            tmem_ld_wait();
            float s[32], m = INFINITY;
            const float4* kk = reinterpret_cast<const float4*>(&skk[buf * kTile + part * kCols + c]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 k4 = kk[i];
                s[4 * i] = fmaf(-2.f, __uint_as_float(u[4 * i]), k4.x), s[4 * i + 1] = fmaf(-2.f, __uint_as_float(u[4 * i + 1]), k4.y);
                s[4 * i + 2] = fmaf(-2.f, __uint_as_float(u[4 * i + 2]), k4.z), s[4 * i + 3] = fmaf(-2.f, __uint_as_float(u[4 * i + 3]), k4.w);
                m = fminf(m, fminf(fminf(s[4 * i], s[4 * i + 1]), fminf(s[4 * i + 2], s[4 * i + 3])));
            }
            least = fminf(least, m + eps);
            if (live && m - eps <= least && m < INFINITY) {
                uint32_t mask = 0u;
#pragma unroll
                for (int i = 0; i < 32; ++i) mask |= s[i] - eps <= least ? 1u << i : 0u;
                const int run = tile * 4 + ((part * kCols + c) >> 5), real = n_codes - 32 * run;  // behind the last code: none
                if (real < 32) mask &= (1u << max(real, 0)) - 1u;
                note(runs, m - eps, mask, run, least);
            }
        }
        tc_fence_before();
        if (__syncthreads_or(live && runs.all)) {  // sums read, next tile's rows written
            many = true;
            break;
        }
    }
    s_least[part][row] = least;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kParts; ++i) least = fminf(least, s_least[i][row]);
    int candidates = 0;
    for (int i = 0; i < runs.n; ++i)
        if (runs.low[i * kThreads] <= least) candidates += __popc(runs.mask[i * kThreads]);
    if (__syncthreads_or(many || (live && candidates > n_codes / 16 + 4))) {
        if (warp == 0) tmem_dealloc(tmem, 512);
        float* sx = reinterpret_cast<float*>(sa);
        walk_all_called<ROWS, kThreads>(sx, sx + kE * ROWS, skk, s_dist[0], x, cb, codes, v0, vectors, T, n_codes);
        return;
    }
    float best = INFINITY;
    int code = 0;
    if (live) {
        float xv[kE];
#pragma unroll
        for (int e = 0; e < kE; ++e) xv[e] = xs[(long long)e * T];
        auto walk = [&](int j) {
            const float* src = cb + (long long)j * kE;
            float dot = 0.f, kk = 0.f;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                float k[8];
                load8(src + 8 * q, vec, k);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    dot = fmaf(xv[8 * q + e], k[e], dot);
                    kk = fmaf(k[e], k[e], kk);
                }
            }
            const float dist = (xx - 2.f * dot) + kk;
            if (dist < best) {
                best = dist;
                code = j;
            }
        };
        int i = 0, base = 0;
        uint32_t mask = 0u;
        for (;;) {  // one place that walks, whichever run the next candidate is of
            while (mask == 0u && i < runs.n) {
                if (runs.low[i * kThreads] <= least) mask = runs.mask[i * kThreads], base = 32 * runs.run[i * kThreads];
                ++i;
            }
            if (mask == 0u) break;
            walk(base + __ffs(mask) - 1);
            mask &= mask - 1u;
        }
    }
    if (part) {
        s_dist[part][row] = best;
        s_code[part][row] = code;
    }
    __syncthreads();
    if (part == 0 && in) {
#pragma unroll
        for (int i = 1; i < kParts; ++i) {
            const float d = s_dist[i][row];
            const int j = s_code[i][row];
            if (d < best || (d == best && d < INFINITY && j < code)) best = d, code = j;
        }
        codes[number] = code;
    }
    if (warp == 0) tmem_dealloc(tmem, 512);
}

template <int ROWS>
static cudaError_t launch(const float* x, const float* cb, long long* codes, int vectors, int T, int n_codes, cudaStream_t st) {
    const cudaError_t e = cudaFuncSetAttribute(vq_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<ROWS>::kSmem);
    if (e != cudaSuccess) return e;
    vq_kernel<ROWS><<<(vectors + ROWS - 1) / ROWS, kThreads, Shape<ROWS>::kSmem, st>>>(x, cb, codes, vectors, T, n_codes);
    return cudaGetLastError();
}

int encode(const float* x, const float* cb, long long* codes, int N, int T, int n_codes, cudaStream_t st) {
    if ((long long)N * T > 0x7fffffff - 256) return LLARK_EINVAL;  // 550 GB of vectors
    const int vectors = N * T;
    using W = Walk<kWalkRows, kWalkThreads>;
    cudaError_t e;
    if (vectors <= 148 * kWalkRows || n_codes <= 256) {
        e = cudaFuncSetAttribute(walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, W::kBytes);
        if (e == cudaSuccess) {
            const int smem = n_codes > W::kCodes ? W::kBytes : W::kBytes - W::kTileFloats * 4;  // one tile has no next
            walk_kernel<<<(vectors + kWalkRows - 1) / kWalkRows, kWalkThreads, smem, st>>>(x, cb, codes, vectors, T, n_codes);
            e = cudaGetLastError();
        }
    } else {
        e = vectors <= 148 * 128 ? launch<128>(x, cb, codes, vectors, T, n_codes, st) : launch<256>(x, cb, codes, vectors, T, n_codes, st);
    }
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

}  // namespace jbvq
}  // namespace llark
