// Sliding-window attention of prompts on tcgen05, heads of 128: the case of seq_swa_mma.cu (packed steps, keys from the step's own rows
// or from the request's ring, window or chunk, sinks, gates) without the soft cap and without rotated values.
//
// CTA = 128 queries of one (request, head), 64 keys at a time from the first key that any of its queries sees; two CTAs share an SM, so
// that the softmax of one runs beside the products of the other. Seven warps:
//   0, 1   bring Q, then K0 K1 V0 K2 V1 ... through three 16 KB slots by cp.async (rows of the step or of the ring: no tensor map covers
//          both), written in the 128-byte swizzle that the products read
//   2      S = Q K^T into one of two TMEM tiles (the next tile's while the softmax works), O += P V
//   3 - 6  softmax, a query row per thread: scores from TMEM, fp32 scale, mask, maximum and sum; P as bf16 rows in shared memory. O is
//          rescaled in TMEM when a row's maximum has grown, and not only when it has by 2^8: with the true maximum the largest
//          probability is 1, which bf16 holds exactly (error against 64 bits 0.002033 like mma.sync's, with the late maximum
//          0.002096 at 204 us instead of 224)
//
// What bounds it: the exponentials (16 per SM and clock) and the softmax around them; V and K are read from L2 by every head of a group.
// Measured on a B200, 32 heads over 8, us: 4 prompts of 2048 tokens, window 1024, 184 (559 TFLOP/s of visible pairs; 224 at first; seq_swa_mma.cu 722), window
// 128 90 (253); 32 portions of 96 tokens behind 2000 236 (498); 4 prompts of 2048, 1757, 1465 and 1173 tokens, window 1024, 148, which took 184 before the
// products were issued by the warp together (see warp_umma_f16) and the softmax took two numbers per instruction and a mask word for 32 keys.
#include "common.cuh"

namespace llark {
extern thread_local int g_last_cuda_error;
namespace swatc {

typedef __nv_bfloat16 bf16_t;
constexpr int HD = 128, BQ = 128, BK = 64, kThreads = 224, kSlots = 3;
constexpr int kSlotBytes = BK * HD * 2;
constexpr int kOffKV = BQ * HD * 2, kOffP = kOffKV + kSlots * kSlotBytes, kSmem = kOffP + BQ * BK * 2 + 1024;

struct Args {
    const bf16_t *qn, *kn, *vv, *kring, *vring;
    const float *gate, *scale_h, *sink;
    bf16_t* out;
    const int *cu, *pos0, *slot;
    long long gate_ld, out_ld;
    int H, G, window, cap, gate_per_head, chunk;
    float out_scale;
};

__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lbo) {  // 128-byte swizzle, groups of eight rows 1024 bytes apart
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, int bytes) {  // bytes 0: zeros, src is not read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A query's weighted sum of values by FMAs, four channels a lane, over the keys lo .. hi that it sees (counted as in the kernel; m: its
// largest score): for rows in whose key tiles a value is infinite or NaN, since the products multiply what a row does not see by 0, and
// that is NaN. Only rows whose own scores are finite get here, a warp at a time: a lane scores a key, then all take its value.
__device__ __noinline__ float4 sum_by_fma(const Args& a, const bf16_t* q, int row0, int n_ring, int ring0, long long ring_base, int g, int lo,
                                          int hi, float sc, float m) {
    const int lane = threadIdx.x & 31;
    auto row = [&](const bf16_t* own, const bf16_t* ring, int k) {
        const bool old = k < n_ring;
        const int e = ring0 + k;
        return (old ? ring : own) + ((old ? ring_base + (e >= a.cap ? e - a.cap : e) : (long long)row0 + k - n_ring) * a.G + g) * HD;
    };
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int k0 = lo; k0 <= hi; k0 += 32) {
        float p = 0.f;
        if (k0 + lane <= hi) {
            const uint4 *qr = reinterpret_cast<const uint4*>(q), *kr = reinterpret_cast<const uint4*>(row(a.kn, a.kring, k0 + lane));
            float s = 0.f;
#pragma unroll 4
            for (int c = 0; c < HD / 8; ++c) {
                const uint4 x = qr[c], y = kr[c];
                const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 u = unpack_bf16x2(xs[e]), v = unpack_bf16x2(ys[e]);
                    s = fmaf(u.y, v.y, fmaf(u.x, v.x, s));
                }
            }
            p = ex2(s * sc - m);
        }
#pragma unroll 4
        for (int j = 0; j < 32; ++j) {
            if (k0 + j > hi) break;  // the same for the whole warp
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const uint2 v = *reinterpret_cast<const uint2*>(row(a.vv, a.vring, k0 + j) + 4 * lane);
            const float2 v0 = unpack_bf16x2(v.x), v1 = unpack_bf16x2(v.y);
            o = make_float4(fmaf(pj, v0.x, o.x), fmaf(pj, v0.y, o.y), fmaf(pj, v1.x, o.z), fmaf(pj, v1.y, o.w));
        }
    }
    return o;
}

__global__ void __launch_bounds__(kThreads, 2)
swa_tc_kernel(const __grid_constant__ Args a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bars[2 * kSlots + 6];
    __shared__ uint32_t tmem_slot;
    const int b = blockIdx.z, h = blockIdx.y, g = h / (a.H / a.G);
    const int row0 = a.cu[b], n = a.cu[b + 1] - row0, qt0 = blockIdx.x * BQ;
    if (qt0 >= n) return;
    unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t *kv_full = bars, *kv_empty = kv_full + kSlots, *s_full = kv_empty + kSlots, *s_empty = s_full + 2, *p_full = s_empty + 2,
             *pv_done = p_full + 1;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kSlots; ++i) {
            mbar_init(&kv_full[i], 2);
            mbar_init(&kv_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_empty[i], 4);
        }
        mbar_init(p_full, 4);
        mbar_init(pv_done, 1);
        mbar_fence_init();
    }
    if (warp == 2) {
        tmem_alloc(&tmem_slot, 256);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot, tmem_o = tmem + 128;
    // Keys are counted from the first one that any query of the tile sees, at position k_lo; the first n_ring of them come from the ring.
    const long long p0 = a.pos0[b], pq_lo = p0 + qt0, pq_hi = p0 + min(qt0 + BQ, n) - 1;
    const long long k_lo = a.chunk > 0 ? (pq_lo / a.chunk) * a.chunk : (pq_lo - a.window + 1 > 0 ? pq_lo - a.window + 1 : 0);
    const int n_keys = (int)(pq_hi - k_lo) + 1, n_ring = (int)(p0 - k_lo), tiles = (n_keys + BK - 1) / BK;

    if (warp < 2) {
        const int c = threadIdx.x & 15, r0 = threadIdx.x >> 4;  // this thread's 16 bytes of the rows r0, r0 + 4, ...
        const uint32_t sq = smem_u32(smem), skv = sq + kOffKV;
        const long long ring_base = (long long)a.slot[b] * a.cap;
        const int ring0 = (int)(k_lo % a.cap);
        auto at = [&](uint32_t base, int rows, int r) { return base + (c >> 3) * (rows * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4); };
#pragma unroll 8
        for (int r = r0; r < BQ; r += 4) {
            const bool in = qt0 + r < n;
            cp16(at(sq, BQ, r), a.qn + ((long long)(row0 + (in ? qt0 + r : 0)) * a.H + h) * HD + c * 8, in ? 16 : 0);
        }
        int issued = 0;
        auto item = [&](const bf16_t* own, const bf16_t* ring, int tile) {
            const int slot = issued % kSlots;
            mbar_wait(&kv_empty[slot], (uint32_t)((issued / kSlots) & 1) ^ 1);
            const uint32_t dst = skv + slot * kSlotBytes;
            const int k0 = tile * BK;
            if (k0 >= n_ring && k0 + BK <= n_keys) {
                const bf16_t* src = own + ((long long)(row0 + k0 - n_ring + r0) * a.G + g) * HD + c * 8;
                const long long ld = (long long)4 * a.G * HD;
#pragma unroll
                for (int i = 0; i < BK / 4; ++i) cp16(at(dst, BK, r0 + 4 * i), src + i * ld, 16);
            } else {
#pragma unroll 4
                for (int i = 0; i < BK / 4; ++i) {
                    const int r = r0 + 4 * i, k = k0 + r;
                    const bf16_t* base = own;
                    long long row = row0 + k - n_ring;
                    if (k < n_ring) {
                        const int e = ring0 + k;  // fewer than cap keys behind k_lo
                        base = ring;
                        row = ring_base + (e >= a.cap ? e - a.cap : e);
                    }
                    const bool in = k < n_keys;
                    cp16(at(dst, BK, r), in ? base + (row * a.G + g) * HD + c * 8 : own, in ? 16 : 0);
                }
            }
            cp_commit();
            if (issued) {
                cp_wait<1>();
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&kv_full[(issued - 1) % kSlots]);
            }
            ++issued;
        };
        item(a.kn, a.kring, 0);  // its arrival covers Q's too
        for (int j = 0; j < tiles; ++j) {
            if (j + 1 < tiles) item(a.kn, a.kring, j + 1);
            item(a.vv, a.vring, j);
        }
        cp_wait<0>();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&kv_full[(issued - 1) % kSlots]);
    } else if (warp == 2) {  // together
        {
            constexpr uint32_t kBase = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BQ >> 4) << 24);  // fp32 sums, bf16 operands
            const uint32_t idesc_s = kBase | ((uint32_t)(BK >> 3) << 17), idesc_pv = kBase | (1u << 16) | ((uint32_t)(HD >> 3) << 17);
            const uint64_t q = make_desc(smem_u32(smem), 0), pd = make_desc(smem_u32(smem + kOffP), 0);
            int used = 0;
            auto issue_s = [&](int j) {
                const int sb = j & 1, slot = used % kSlots;
                mbar_wait(&s_empty[sb], ((uint32_t)(j >> 1) & 1) ^ 1);
                mbar_wait(&kv_full[slot], (uint32_t)(used / kSlots) & 1);
                tc_fence_after();
                const uint64_t k = make_desc(smem_u32(smem + kOffKV + slot * kSlotBytes), 0);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    warp_umma_f16(tmem + sb * BK, q + (i >> 2) * (BQ * 128 >> 4) + (i & 3) * 2, k + (i >> 2) * (BK * 128 >> 4) + (i & 3) * 2,
                             idesc_s, i != 0);
                warp_umma_commit(&kv_empty[slot]);
                warp_umma_commit(&s_full[sb]);
                ++used;
            };
            issue_s(0);
            for (int j = 0; j < tiles; ++j) {
                if (j + 1 < tiles) issue_s(j + 1);
                const int slot = used % kSlots;
                mbar_wait(&kv_full[slot], (uint32_t)(used / kSlots) & 1);
                mbar_wait(p_full, (uint32_t)j & 1);
                tc_fence_after();
                const uint64_t v = make_desc(smem_u32(smem + kOffKV + slot * kSlotBytes), BK * 128);  // [key][channel]: MN-major
#pragma unroll
                for (int i = 0; i < 4; ++i) warp_umma_f16(tmem_o, pd + i * 2, v + i * 128, idesc_pv, (j | i) != 0);
                warp_umma_commit(&kv_empty[slot]);
                warp_umma_commit(pv_done);
                ++used;
            }
        }
    } else {
        const int quad = warp & 3, r = quad * 32 + lane;  // the TMEM lanes that this warp may read; the row
        const uint32_t lane0 = tmem + ((uint32_t)(quad * 32) << 16);
        constexpr float kLog2e = 1.4426950408889634f;
        const float sc = a.scale_h[h] * kLog2e;  // softmax through exp2
        // the row sees the keys lo .. hi (none behind the prompt's end); the warp sees key tiles in full between lo of its last row and hi
        // of its first
        const long long pq = pq_lo + r;
        const long long first = a.chunk > 0 ? (pq / a.chunk) * a.chunk : pq - a.window + 1;
        const int lo = first > k_lo ? (int)(first - k_lo) : 0, hi = qt0 + r < n ? (int)(pq - k_lo) : -1;
        const int lo_all = __reduce_max_sync(0xffffffffu, lo), hi_all = __reduce_min_sync(0xffffffffu, hi);
        float m = -INFINITY, l = 0.f;
        for (int j = 0; j < tiles; ++j) {
            const int sb = j & 1, k0 = j * BK;
            mbar_wait(&s_full[sb], (uint32_t)(j >> 1) & 1);
            tc_fence_after();
            uint32_t s[2][32];
            tmem_ld_32x32b_x32(lane0 + sb * BK, s[0]);
            tmem_ld_32x32b_x32(lane0 + sb * BK + 32, s[1]);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_empty[sb]);
            const bool whole = k0 >= lo_all && k0 + BK - 1 <= hi_all;
            const uint64_t sc2 = two(sc, sc);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    float x, y;
                    apart(mul2(two(__uint_as_float(s[e][c]), __uint_as_float(s[e][c + 1])), sc2), x, y);
                    s[e][c] = __float_as_uint(x);
                    s[e][c + 1] = __float_as_uint(y);
                }
                if (!whole) {
                    const int from = lo - (k0 + e * 32), to = hi - (k0 + e * 32);  // the row sees these of the 32 keys
                    uint32_t seen = to < 0 || from > 31 ? 0u : to >= 31 ? 0xffffffffu : (2u << to) - 1u;
                    if (from > 0 && from < 32) seen &= 0xffffffffu << from;
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (!((seen >> c) & 1u)) s[e][c] = __float_as_uint(-INFINITY);
                }
            }
            float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int c = 0; c < 32; c += 2)
                    top[(c >> 1) & 3] = max3(top[(c >> 1) & 3], __uint_as_float(s[e][c]), __uint_as_float(s[e][c + 1]));
            const float cand = fmaxf(m, fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])));
            const float use = cand == -INFINITY ? 0.f : cand;
            const float alpha = ex2(m - use);
            m = cand;
            uint64_t sum[2] = {0, 0};
            const uint64_t less = two(-use, -use);
            uint32_t pk[32];
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int c = 0; c < 32; c += 2) {
                    float x, y;
                    apart(add2(two(__uint_as_float(s[e][c]), __uint_as_float(s[e][c + 1])), less), x, y);
                    x = ex2(x);
                    y = ex2(y);
                    sum[(c >> 1) & 1] = add2(sum[(c >> 1) & 1], two(x, y));
                    pk[e * 16 + (c >> 1)] = pack_bf16x2(x, y);
                }
            float s0, s1;
            apart(add2(sum[0], sum[1]), s0, s1);
            l = l * alpha + (s0 + s1);
            if (j > 0) {
                mbar_wait(pv_done, (uint32_t)(j - 1) & 1);  // P's rows are free, O holds the tiles before
                tc_fence_after();
                if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
                    for (int c = 0; c < HD / 32; ++c) {
                        uint32_t o[32];
                        tmem_ld_32x32b_x32(lane0 + 128 + c * 32, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
                        tmem_st_32x32b_x32(lane0 + 128 + c * 32, o);
                    }
                    tmem_st_wait();
                }
            }
            unsigned char* prow = smem + kOffP + r * 128;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                *reinterpret_cast<uint4*>(prow + ((u ^ (r & 7)) << 4)) = make_uint4(pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        mbar_wait(pv_done, (uint32_t)(tiles - 1) & 1);
        tc_fence_after();
        const bool ok = qt0 + r < n;
        const long long trow = row0 + (ok ? qt0 + r : 0);
        // a sink adds exp(sink_h) to the denominator; a row of the prompt has seen its own key: m is finite
        float inv = a.out_scale / (a.sink ? l + exp2f(a.sink[h] * kLog2e - m) : l);
        if (a.gate && a.gate_per_head) inv *= 1.0f / (1.0f + expf(-a.gate[trow * a.gate_ld + h]));
        float odd = 0.f;  // NaN as soon as a sum is not finite
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(lane0 + 128 + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) odd = fmaf(__uint_as_float(o[e]), 0.f, odd);
            if (ok) {
                if (a.gate && !a.gate_per_head) {
                    const float* gp = a.gate + trow * a.gate_ld + h * HD + c * 32;
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * (1.0f / (1.0f + expf(-gp[e]))));
                }
                bf16_t* dst = a.out + trow * a.out_ld + h * HD + c * 32;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        w[e] = pack_bf16x2(__uint_as_float(o[8 * u + 2 * e]) * inv, __uint_as_float(o[8 * u + 2 * e + 1]) * inv);
                    *reinterpret_cast<uint4*>(dst + 8 * u) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
            __syncwarp();
        }
        tc_fence_before();
        for (uint32_t rows = __ballot_sync(0xffffffffu, ok && odd != 0.f && l < INFINITY); rows; rows &= rows - 1) {
            const int from = __ffs(rows) - 1;
            const long long t = row0 + qt0 + quad * 32 + from;
            const float4 s = sum_by_fma(a, a.qn + (t * a.H + h) * HD, row0, n_ring, (int)(k_lo % a.cap), (long long)a.slot[b] * a.cap, g,
                                        __shfl_sync(0xffffffffu, lo, from), __shfl_sync(0xffffffffu, hi, from), sc,
                                        __shfl_sync(0xffffffffu, m, from));
            const float f = __shfl_sync(0xffffffffu, inv, from);
            float r[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (a.gate && !a.gate_per_head) r[e] *= 1.0f / (1.0f + expf(-a.gate[t * a.gate_ld + h * HD + 4 * lane + e]));
                r[e] *= f;
            }
            *reinterpret_cast<uint2*>(a.out + t * a.out_ld + h * HD + 4 * lane) = make_uint2(pack_bf16x2(r[0], r[1]), pack_bf16x2(r[2], r[3]));
        }
    }
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
}

// From 32 tokens of the longest request on: 16 heads, 64 prompts of 16 / 24 / 32 / 64 tokens 30.4 / 30.2 / 29.6 / 24.3 us here and 28.3 /
// 29.2 / 30.0 / 34.3 there; with 1024 keys in the ring it is ahead from 16 on (250 against 267). Output rows must take 16-byte stores.
bool takes(int D, int max_len, float softcap, const float* vfreq, const void* out, long long out_ld) {
    return D == HD && max_len >= 32 && softcap == 0.f && !vfreq && out_ld % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
}
int launch(const void* qn, const void* kn, const void* vv, const void* kring, const void* vring, const float* gate, long long gate_ld,
           const float* scale_h, void* out, const int* cu, const int* pos0, const int* slot, int n_seq, int max_len, int H, int G,
           int window, int cap, const float* sink, int gate_per_head, int chunk, long long out_ld, float out_scale, cudaStream_t st) {
    const Args a{(const bf16_t*)qn, (const bf16_t*)kn, (const bf16_t*)vv, (const bf16_t*)kring, (const bf16_t*)vring, gate, scale_h, sink,
                 (bf16_t*)out, cu, pos0, slot, gate_ld, out_ld, H, G, window, cap, gate_per_head, chunk, out_scale};
    cudaError_t e = cudaFuncSetAttribute(swa_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e == cudaSuccess) {
        swa_tc_kernel<<<dim3((max_len + BQ - 1) / BQ, H, n_seq), kThreads, kSmem, st>>>(a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

}  // namespace swatc
}  // namespace llark
