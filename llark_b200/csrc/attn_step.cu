// Attention of single-token steps (see attn_step.cuh): a stream of the keys and values, read once for all the query heads of a
// key head.
//
// A CTA of four warps takes HG query heads of one key head of one request; a warp takes 16 keys at a time. Scores come from
// mma.sync.m16n8k16 with the keys as the M side (bf16 operands, exact products, fp32 sums): summing over d may take the entries
// of 32 in any order, so every thread reads 16-byte pieces of two key rows straight into fragments, and the values' pieces are
// requested at the same time: 8 KB per warp are on their way at D = 128, and there is no barrier in the loop. Softmax, its
// running maximum and sum, the probabilities and the weighted sum are fp32 (the latter on the FMA units: a probability never
// becomes 16 bits). What bounds it is memory, or for few requests the number of CTAs: those are cut along the keys over a
// cluster of up to eight CTAs, which meet in distributed shared memory.
//
// Measured on a B200: 32 requests x 32 heads x 1500 keys, D = 128: 126 us (342 with a block per head that scored a key per thread;
// floor 118 us at 6.65 TB/s); one request, 1024 keys: 11 us (33).
#include "attn_step.cuh"

namespace llark {
namespace attnstep {

typedef __nv_bfloat16 bf16_t;
constexpr int kWarps = 4, kThreads = kWarps * 32;
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ void mma16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

template <int D, int HG>
__global__ void __launch_bounds__(kThreads, D < 256 && HG <= 4 ? 4 : 2)
attn_step_kernel(const Args p, int cs) {
    constexpr int NC = D / 32;        // 32-wide pieces of a head
    constexpr int LPK = D / 8;        // lanes that share a value row, eight channels each
    constexpr int KPI = 32 / LPK;     // value rows per load of a warp
    constexpr int NV = 16 / KPI;      // such loads per 16 keys
    constexpr int VB = NV > 8 ? 8 : NV;
    __shared__ float sp[kWarps][HG][16], sa[kWarps][HG];
    __shared__ float sacc[kWarps][HG][D];
    __shared__ float sm_m[kWarps][HG], sm_l[kWarps][HG];
    __shared__ float tot[HG][D], tot_m[HG], tot_l[HG];  // of the CTA
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int rank = cs > 1 ? (int)(blockIdx.x % cs) : 0;
    const int h0 = ((int)blockIdx.x / cs) * HG, b = blockIdx.y;  // HG divides H / G
    const int kvh = h0 / (p.H / p.G);
    long long pos = 0, base;
    int nkeys, ring0 = 0;
    if (p.one_wave) let_next_begin();
    if (p.lens) {
        nkeys = p.lens[b] < p.cap ? p.lens[b] : p.cap;
        base = (long long)b * p.cap;
    } else if (p.packed) {
        nkeys = p.n_keys;
        base = (long long)b * p.cap;
    } else {
        const int r = p.tok_seq[b];
        pos = (long long)p.pos0[r] + (b - p.cu[r]);
        const long long lo = p.chunk > 0 ? (pos / p.chunk) * p.chunk : (pos - p.window + 1 > 0 ? pos - p.window + 1 : 0);
        nkeys = (int)(pos - lo + 1);
        ring0 = (int)(lo % p.cap);  // keys in sight never outnumber the store's entries
        base = (long long)p.slot[r] * p.cap;
    }
    const long long ld = (long long)p.G * D;
    const bf16_t* kb = p.k + base * ld + kvh * D;
    const bf16_t* vb = p.v + base * ld + kvh * D;
    const bf16_t* qrow = p.packed ? p.packed + b * p.packed_ld + h0 * D : p.q + ((long long)b * p.H + h0) * D;
    if (p.packed && rank == cs - 1) {  // the CTA that reads the last key stores the new one first (every query head has a key head)
        if (threadIdx.x < D / 4) {
            const int i = threadIdx.x % (D / 8) * 8;
            const bool second = threadIdx.x >= D / 8;
            *reinterpret_cast<uint4*>((second ? p.v_new : p.k_new) + (base + nkeys - 1) * ld + kvh * D + i) =
                *reinterpret_cast<const uint4*>(qrow + (second ? 2 : 1) * p.H * D + i);
        }
        __syncthreads();
    }
    // ---- queries: head g of the group, the pieces that this thread's key pieces meet
    uint4 qf[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        qf[c] = make_uint4(0, 0, 0, 0);
        if (g < HG) qf[c] = *reinterpret_cast<const uint4*>(qrow + g * D + c * 32 + t * 8);
    }
    // this thread's two heads (columns 2 t, 2 t + 1 of the scores)
    float sc[2] = {0.f, 0.f};
#pragma unroll
    for (int x = 0; x < 2; ++x)
        if (2 * t + x < HG) sc[x] = p.scale_h ? p.scale_h[h0 + 2 * t + x] : p.scale;
    const float cap2 = p.softcap * kLog2e;
#pragma unroll
    for (int x = 0; x < 2; ++x) sc[x] = p.softcap > 0.f ? sc[x] / p.softcap : sc[x] * kLog2e;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    float acc[HG][8];
#pragma unroll
    for (int h = 0; h < HG; ++h)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[h][e] = 0.f;

    const int ntiles = (nkeys + 15) >> 4;
    const int t_hi = (int)((long long)(rank + 1) * ntiles / cs);
    auto entry = [&](int jj) {
        int e = ring0 + jj;
        if (e >= p.cap) e -= p.cap;
        return (long long)e * ld;
    };
    for (int tile = (int)((long long)rank * ntiles / cs) + warp; tile < t_hi; tile += kWarps) {
        const int j0 = tile * 16;
        const bool in0 = j0 + g < nkeys, in1 = j0 + g + 8 < nkeys;
        uint4 k0[NC], k1[NC], vf[VB];
        const bf16_t* r0 = kb + (in0 ? entry(j0 + g) : 0) + t * 8;
        const bf16_t* r1 = kb + (in1 ? entry(j0 + g + 8) : 0) + t * 8;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            k0[c] = k1[c] = make_uint4(0, 0, 0, 0);
            if (in0) k0[c] = *reinterpret_cast<const uint4*>(r0 + c * 32);
            if (in1) k1[c] = *reinterpret_cast<const uint4*>(r1 + c * 32);
        }
        auto load_v = [&](int i0) {
#pragma unroll
            for (int i = 0; i < VB; ++i) {
                const int j = j0 + (i0 + i) * KPI + lane / LPK;
                vf[i] = make_uint4(0, 0, 0, 0);
                if (j < nkeys) vf[i] = *reinterpret_cast<const uint4*>(vb + entry(j) + (lane % LPK) * 8);
            }
        };
        load_v(0);
        float s[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            mma16(s, k0[c].x, k1[c].x, k0[c].y, k1[c].y, qf[c].x, qf[c].y);
            mma16(s2, k0[c].z, k1[c].z, k0[c].w, k1[c].w, qf[c].z, qf[c].w);
        }
        // ---- rows g, g + 8 (keys) x columns 2 t, 2 t + 1 (heads)
        float mt[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float v = (s[e] + s2[e]) * sc[e & 1];
            if (p.softcap > 0.f) v = cap2 * tanhf(v);
            s[e] = (e < 2 ? in0 : in1) ? v : -INFINITY;
            mt[e & 1] = fmaxf(mt[e & 1], s[e]);
        }
        float alpha[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            mt[x] = fmaxf(mt[x], __shfl_xor_sync(0xffffffffu, mt[x], 4));
            mt[x] = fmaxf(mt[x], __shfl_xor_sync(0xffffffffu, mt[x], 8));
            mt[x] = fmaxf(mt[x], __shfl_xor_sync(0xffffffffu, mt[x], 16));
            const float mn = fmaxf(m[x], mt[x]);
            alpha[x] = mn == -INFINITY ? 1.f : exp2f(m[x] - mn);
            m[x] = mn;
            l[x] *= alpha[x];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int x = e & 1;
            const float pr = exp2f(s[e] - (m[x] == -INFINITY ? 0.f : m[x]));  // 0 for -inf, NaN stays
            l[x] += pr;
            if (2 * t + x < HG) sp[warp][2 * t + x][g + (e >> 1) * 8] = pr;
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
            if (g == 0 && 2 * t + x < HG) sa[warp][2 * t + x] = alpha[x];
        __syncwarp();
#pragma unroll
        for (int h = 0; h < HG; ++h) {
            const float a = sa[warp][h];
            if (a != 1.f) {  // the same for the whole warp
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[h][e] *= a;
            }
        }
#pragma unroll
        for (int i0 = 0; i0 < NV; i0 += VB) {
            if (i0) load_v(i0);
#pragma unroll
            for (int i = 0; i < VB; ++i) {
                const int row = (i0 + i) * KPI + lane / LPK;
                const float2 f0 = unpack_bf16x2(vf[i].x), f1 = unpack_bf16x2(vf[i].y), f2 = unpack_bf16x2(vf[i].z),
                             f3 = unpack_bf16x2(vf[i].w);
                const float f[8] = {f0.x, f0.y, f1.x, f1.y, f2.x, f2.y, f3.x, f3.y};
#pragma unroll
                for (int h = 0; h < HG; ++h) {
                    const float pr = sp[warp][h][row];
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[h][e] = fmaf(pr, f[e], acc[h][e]);
                }
            }
        }
        __syncwarp();  // the probabilities are read before the next 16 keys' take their place
    }
    // ---- the warp's sums: over its keys' lanes, then to shared memory
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        l[x] += __shfl_xor_sync(0xffffffffu, l[x], 4);
        l[x] += __shfl_xor_sync(0xffffffffu, l[x], 8);
        l[x] += __shfl_xor_sync(0xffffffffu, l[x], 16);
        if (g == 0 && 2 * t + x < HG) {
            sm_m[warp][2 * t + x] = m[x];
            sm_l[warp][2 * t + x] = l[x];
        }
    }
#pragma unroll
    for (int h = 0; h < HG; ++h)
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            float v = acc[h][e];
#pragma unroll
            for (int o = LPK; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane < LPK) sacc[warp][h][lane * 8 + e] = v;
        }
    __syncthreads();
    for (int i = threadIdx.x; i < HG * D; i += kThreads) {
        const int h = i / D, e = i % D;
        float mm = -INFINITY, lt = 0.f, o = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, sm_m[w][h]);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float f = sm_m[w][h] == -INFINITY ? 0.f : exp2f(sm_m[w][h] - mm);
            lt = fmaf(sm_l[w][h], f, lt);
            o = fmaf(sacc[w][h][e], f, o);
        }
        tot[h][e] = o;
        if (e == 0) {
            tot_m[h] = mm;
            tot_l[h] = lt;
        }
    }
    if (cs > 1)
        cluster_sync_all();
    else
        __syncthreads();
    // ---- this CTA's share of the outputs
    auto value = [&](int h, int e) {
        float mm = p.sink ? p.sink[h0 + h] * kLog2e : -INFINITY, lt = 0.f, o = 0.f;
        if (cs == 1) {
            mm = fmaxf(mm, tot_m[h]);
            const float f = tot_m[h] == -INFINITY ? 0.f : exp2f(tot_m[h] - mm);
            lt = tot_l[h] * f;
            o = tot[h][e] * f;
        } else {
            const uint32_t am = smem_u32(&tot_m[h]), al = smem_u32(&tot_l[h]), ao = smem_u32(&tot[h][e]);
            for (int r = 0; r < cs; ++r) mm = fmaxf(mm, ld_cluster(mapa_shared(am, (uint32_t)r)));
            for (int r = 0; r < cs; ++r) {
                const float mr = ld_cluster(mapa_shared(am, (uint32_t)r));
                const float f = mr == -INFINITY ? 0.f : exp2f(mr - mm);
                lt = fmaf(ld_cluster(mapa_shared(al, (uint32_t)r)), f, lt);
                o = fmaf(ld_cluster(mapa_shared(ao, (uint32_t)r)), f, o);
            }
        }
        if (p.sink) lt += exp2f(p.sink[h0 + h] * kLog2e - mm);
        return nkeys > 0 ? o / lt * p.out_scale : 0.f;
    };
    const int share = (HG * D) / cs;  // cs <= 8 divides it
    for (int i = rank * share + (int)threadIdx.x; i < (rank + 1) * share; i += kThreads) {
        const int h = i / D, e = i % D;
        float o = value(h, e);
        if (p.vfreq) {  // pair mp turned by -pos * vfreq[mp]: (2 mp, 2 mp + 1), or (mp, mp + D / 2)
            const bool second = p.v_interleaved ? (e & 1) : e >= D / 2;
            const int mp = p.v_interleaved ? e >> 1 : (second ? e - D / 2 : e);
            const float w = value(h, p.v_interleaved ? e ^ 1 : (second ? mp : mp + D / 2));
            float si, co;
            sincosf((float)pos * p.vfreq[mp], &si, &co);
            o = second ? o * co - w * si : o * co + w * si;
        }
        if (p.gate) o *= 1.0f / (1.0f + expf(-p.gate[(long long)b * p.gate_ld + (p.gate_per_head ? h0 + h : (h0 + h) * D + e)]));
        p.out[(long long)b * p.out_ld + (h0 + h) * D + e] = __float2bfloat16_rn(o);
    }
    if (cs > 1) cluster_sync_all();  // nobody leaves while its sums may still be read
}

template <int D, int HG>
static cudaError_t go(Args a, cudaStream_t st) {
    const long long ctas = (long long)(a.H / HG) * a.B;
    int cs = 1;  // cut along the keys until there are about four CTAs for each of the 148 SMs
    while (cs < 8 && ctas * cs * 2 <= 592) cs *= 2;
    // Where all CTAs are resident at once the next kernel may come in while they end (a step of one row 242 -> 239 us); it would take room
    // from CTAs that are still to come (32 rows 525 -> 545). Launched early itself, 1024 CTAs became slower, 540 -> 660.
    a.one_wave = ctas * cs <= 592;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.H / HG * cs), (unsigned)a.B);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cs > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, attn_step_kernel<D, HG>, a, cs);
}

cudaError_t launch(const Args& a, cudaStream_t st) {
    // query heads per CTA: as many of a key head's as divide them, up to eight (four at D = 256, for the registers)
    const int rep = a.H / a.G;
#define LLARK_STEP(D_)                                                    \
    if (D_ < 256 && rep % 8 == 0) return go<D_, D_ < 256 ? 8 : 4>(a, st); \
    if (rep % 4 == 0) return go<D_, 4>(a, st);                            \
    if (rep % 2 == 0) return go<D_, 2>(a, st);                            \
    return go<D_, 1>(a, st);
    if (a.D == 64) { LLARK_STEP(64) }
    if (a.D == 128) { LLARK_STEP(128) }
    LLARK_STEP(256)
#undef LLARK_STEP
}

}  // namespace attnstep
}  // namespace llark
