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
// none below infinity and keeps code 0. Candidates are noted in runs of 32 codes, twelve runs a thread; if that overflows even after runs have
// been struck off, the thread walks all codes of its half.
//
// A CTA has 256 vectors (two row tiles of A) and goes through the codebook in tiles of 128 codes: four threads make one row of B of the
// next tile while the tensor cores multiply; two threads share a vector's sums, 64 columns each.
//
// What bounds it: a tile's chain of conversion, products and sums' reading, and the candidates' walks at the end. Measured on a B200, 32768
// vectors, us, walk over all codes / here: 2048 codes 425 / 97, a hundred times closer together 420 / 90, 512 codes 103 / 32. With one
// bf16 part each (bound 2^-7 |x| |k|, so that more is walked) 169, and 949 where codes are close.
#include "common.cuh"
#include <math.h>

namespace llark {
extern thread_local int g_last_cuda_error;
namespace jbvq {

constexpr int kE = 64, kRows = 256, kThreads = 2 * kRows, kTile = 128, kList = 12;
constexpr int kPartA = kRows * 128, kPartB = kTile * 128;  // bytes of a part: 64 bf16 a row
constexpr int kListBytes = kList * kThreads * 12;          // per run: s - eps of its least, which of the 32, number of the run
constexpr int kSmem = 1024 + 2 * kPartA + 2 * 2 * kPartB + kListBytes;

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
    bool all;  // too many: walk everything
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

__global__ void __launch_bounds__(kThreads, 1)
vq_kernel(const float* __restrict__ x, const float* __restrict__ cb, long long* __restrict__ codes, int T, int n_codes) {
    extern __shared__ unsigned char raw[];
    __shared__ __align__(16) float skk[2][kTile];  // read four at a time
    __shared__ uint64_t bar[2];
    __shared__ uint32_t tmem_base, most_kk;  // most_kk: bits of the largest finite |k|^2 of the tiles made so far
    __shared__ float s_least[2][kRows], s_dist[kRows];
    __shared__ int s_code[kRows];
    unsigned char* sa = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    unsigned char* sb = sa + 2 * kPartA;
    unsigned char* sl = sb + 2 * 2 * kPartB;
    const int tid = threadIdx.x, row = tid & (kRows - 1), half = tid / kRows, warp = tid >> 5, lane = tid & 31;
    const int n = blockIdx.y, t = blockIdx.x * kRows + row;
    const bool vec = (reinterpret_cast<uintptr_t>(cb) & 15) == 0, in = t < T;
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
    const float* const xs = x + (long long)n * kE * T + t;
    float xx = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            v[e] = in ? xs[(long long)(8 * q + e) * T] : 0.f;
            xx = fmaf(v[e], v[e], xx);
        }
        if ((q >> 2) == half) put8(sa, kPartA, row, q, v);  // the two threads of a vector write half of its row each
    }
    const float xn = sqrtf(xx) * 1.0001f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base, lane0 = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (row >> 7) * kTile + half * 64;
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
        if (seg == 0) skk[buf][r] = kk;
        const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(kk < INFINITY ? kk : 0.f));
        if (lane == 0) atomicMax(&most_kk, most);
        fence_proxy_async_smem();
    };
    auto multiply = [&](int tile) {  // one thread
        const uint32_t b = smem_u32(sb) + (tile & 1) * 2 * kPartB;
#pragma unroll
        for (int rt = 0; rt < 2; ++rt) {
            const uint32_t a = smem_u32(sa) + rt * 128 * 128, d = tmem + (tile & 1) * 256 + rt * kTile;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                umma_f16(d, desc(a) + 2 * k, desc(b) + 2 * k, kIdesc, k != 0);
                umma_f16(d, desc(a) + 2 * k, desc(b + kPartB) + 2 * k, kIdesc, 1);
                umma_f16(d, desc(a + kPartA) + 2 * k, desc(b) + 2 * k, kIdesc, 1);
            }
        }
        umma_commit(&bar[tile & 1]);
    };

    float least = INFINITY;  // smallest s + eps so far
    const bool live = in && xx < INFINITY;
    float* const list = reinterpret_cast<float*>(sl);
    Runs runs = {list + tid, reinterpret_cast<uint32_t*>(list + kList * kThreads) + tid,
                 reinterpret_cast<int*>(list + 2 * kList * kThreads) + tid, 0, false};
    make_tile(0);
    __syncthreads();
    for (int tile = 0; tile < tiles; ++tile) {
        const int buf = tile & 1;
        if (tid == 0) {
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
        for (int c = 0; c < 64; c += 32) {
            uint32_t u[32];
            tmem_ld_32x32b_x32(lane0 + buf * 256 + c, u);
            tmem_ld_wait();
            float s[32], m = INFINITY;
            const float4* kk = reinterpret_cast<const float4*>(&skk[buf][half * 64 + c]);
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
                const int run = tile * 4 + half * 2 + (c >> 5), real = n_codes - 32 * run;  // behind the last code: none
                if (real < 32) mask &= (1u << max(real, 0)) - 1u;
                note(runs, m - eps, mask, run, least);
            }
        }
        tc_fence_before();
        __syncthreads();  // sums read, next tile's rows written
    }
    s_least[half][row] = least;
    __syncthreads();
    least = fminf(least, s_least[half ^ 1][row]);
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
        int i = 0, next = half * 64;  // runs noted: the next one; all codes: the next one of this half of every tile
        uint32_t mask = 0u;
        int base = 0;
        for (;;) {  // one place that walks, however the next code is found
            int j;
            if (runs.all) {
                if (next >= n_codes) break;
                j = next;
                next += (next & 63) == 63 ? 65 : 1;
            } else {
                while (mask == 0u && i < runs.n) {
                    if (runs.low[i * kThreads] <= least) mask = runs.mask[i * kThreads], base = 32 * runs.run[i * kThreads];
                    ++i;
                }
                if (mask == 0u) break;
                j = base + __ffs(mask) - 1;
                mask &= mask - 1u;
            }
            walk(j);
        }
    }
    if (half) {
        s_dist[row] = best;
        s_code[row] = code;
    }
    __syncthreads();
    if (!half && in) {
        const float d = s_dist[row];
        const int j = s_code[row];
        if (d < best || (d == best && d < INFINITY && j < code)) code = j;
        codes[(long long)n * T + t] = code;
    }
    if (warp == 0) tmem_dealloc(tmem, 512);
}

int encode(const float* x, const float* cb, long long* codes, int N, int T, int n_codes, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(vq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e == cudaSuccess) {
        vq_kernel<<<dim3((T + kRows - 1) / kRows, N), kThreads, kSmem, st>>>(x, cb, codes, T, n_codes);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

}  // namespace jbvq
}  // namespace llark
