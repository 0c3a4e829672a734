// Products with few rows (decode steps, routed experts of a few tokens): a stream of the weight matrix. See skinny.cuh.
//
// What bounds it is how many bytes of the weights are on their way. A CTA of four warps takes a tile of weight rows; its operands
// come by cp.async through a ring of 64-wide slices of K (54 to 108 KB of it per CTA, four or two CTAs per SM), and matrices with
// few rows are also cut along K over a cluster of up to eight CTAs, whose partial sums meet in distributed shared memory in a
// fixed order (no atomics, no workspace). The weights are the M side of the products and the tokens the N side, so that up to 64
// tokens ride on one read of a weight. A slice is kept as 128-byte rows whose 16-byte pieces are XORed with the row number: the
// copies and ldmatrix are free of bank conflicts, and it is the 128-byte swizzle of tcgen05 operands.
//
// A decode step is a row of such products with short kernels between them, and each of them filled an empty chip and drained it again:
// 202 us of products for 163 us of bytes in a step of two layers and the head, one row, and 268 us for the whole step. So a CTA starts
// while the kernel in front of it ends (launch_early): its weights are under way, or on their way to L2, before the tokens are there.
// The next kernel is let in at once: after half of the slices or with the last ones asked for the step took 2 to 3 us longer.
// Measured, a step of 1 / 8 / 32 rows: 269 -> 236, 297 -> 270, 560 -> 525 us.
//
// Measured on a B200, launches in a row on rotating weights (floor = the weights at 6.55 TB/s), against the 256-row tiles of the
// tcgen05 GEMM core: N 4096 K 4096, 32 tokens 10.7 us (core 28.7, floor 5.1); N 22016 K 4096 39.4 (54.9, 27.5); N 4096 K 11008
// 19.3 (61.0, 13.8); N 32004 K 4096 45.9 (56.3, 40.0); 64 tokens 13.2 / 45.2 / 22.0 / 49.7; one token 7.7 / 30.2 / 16.3 / 41.6.
#include "skinny.cuh"

#include <atomic>

namespace llark {
namespace skinny {

typedef __nv_bfloat16 bf16_t;
constexpr int BN = 64, BK = 64, kThreads = 128;
constexpr int kStageMma = BN * 128 + 8 * 128, kStagesMma = 6;  // 54 KB: four CTAs per SM
constexpr int RP = BN + 4;  // row pitch of the partial sums [token][row] (16-byte pieces)

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(p)
                 : "memory");
}
__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// gate rows in the first half of W, up rows in the second
__host__ __device__ __forceinline__ bool gate_up(const Args& p) { return p.act == kActSiluGlu || p.act == kActSwiglu; }

// byte offset of 16-byte piece c of row r in a slice
__device__ __forceinline__ uint32_t piece(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }

template <typename TC> __device__ __forceinline__ float ldc_(const void* p, long long i);
template <> __device__ __forceinline__ float ldc_<float>(const void* p, long long i) { return static_cast<const float*>(p)[i]; }
template <> __device__ __forceinline__ float ldc_<bf16_t>(const void* p, long long i) {
    return __bfloat162float(static_cast<const bf16_t*>(p)[i]);
}

// Four neighbouring sums, added up over the cluster's CTAs in their order
__device__ __forceinline__ void total4(const float* red, int at, int cs, float (&x)[4]) {
    if (cs == 1) {
        const float4 v = *reinterpret_cast<const float4*>(red + at);
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
        return;
    }
    const uint32_t addr = smem_u32(red + at);
#pragma unroll
    for (int r0 = 0; r0 < 8; r0 += 4) {
        if (r0 >= cs) break;
        float v[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)  // four requested before the first is used
            if (r0 + r < cs)
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v[r][0]), "=f"(v[r][1]), "=f"(v[r][2]), "=f"(v[r][3])
                             : "r"(mapa_shared(addr, (uint32_t)(r0 + r)))
                             : "memory");
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (r0 + r < cs)
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = r0 + r == 0 ? v[r][e] : x[e] + v[r][e];
    }
}
__device__ __forceinline__ void store4(float* C, const float (&v)[4], bool vec, int n) {
    if (vec && n >= 4)
        *reinterpret_cast<float4*>(C) = make_float4(v[0], v[1], v[2], v[3]);
    else
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (e < n) C[e] = v[e];
}
__device__ __forceinline__ void store4(bf16_t* C, const float (&v)[4], bool vec, int n) {
    if (vec && n >= 4)
        *reinterpret_cast<uint2*>(C) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    else
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (e < n) C[e] = __float2bfloat16_rn(v[e]);
}

// A tile's columns from the partial sums red [token][row] (ROWS weight rows, PITCH apart) of the cluster's CTAs; this CTA does its
// share of them, four results at a time. The two rows that a paired activation or a rotation needs are 2 u and 2 u + 1, or u and
// u + ROWS / 2.
template <typename TC, bool GROUPED, int ROWS, int PITCH>
__device__ __forceinline__ void epilogue(const Args& p, const float* red, int M, int row0, int base, int cs, int rank) {
    const bool adjacent = p.act == kActReluGlu || p.act == kActClampGlu, halves = gate_up(p), rope = p.act == kActRope;
    const bool two = adjacent || halves || rope;
    const int quads = (two ? ROWS / 8 : ROWS / 4) / cs, q0 = rank * quads;
    const int n_out = adjacent || halves ? p.N >> 1 : p.N;
    TC* C = static_cast<TC*>(p.C);
    const bool vec = p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & (4 * sizeof(TC) - 1)) == 0;
    auto bias_at = [&](int c) { return p.bias_fp32 ? ldc_<float>(p.bias, c) : ldc_<bf16_t>(p.bias, c); };
    for (int i = threadIdx.x; i < M * quads; i += kThreads) {
        const int m = i / quads, u = 4 * (q0 + i % quads);
        const int col = adjacent ? (base >> 1) + u : base + u, n = n_out - col;
        if (n <= 0) continue;
        TC* c = C + (long long)(GROUPED ? row0 + m : m) * p.ldc + col;
        float x[4], y[4];
        if (!two) {
            total4(red, m * PITCH + u, cs, x);
            if (p.bias)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < n) x[e] += bias_at(col + e);
            if (GROUPED && p.in_wts) {
                const float f = p.in_wts[p.perm[row0 + m]];
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] *= f;
            }
            if (p.act == kActRelu2)
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = fmaxf(x[e], 0.f) * fmaxf(x[e], 0.f);
            if (p.R)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < n) x[e] += ldc_<TC>(p.R, (long long)m * p.ldr + col + e);
            store4(c, x, vec, n);
            continue;
        }
        if (adjacent) {
            float a[4], b[4];
            total4(red, m * PITCH + 2 * u, cs, a);
            total4(red, m * PITCH + 2 * u + 4, cs, b);
            x[0] = a[0], y[0] = a[1], x[1] = a[2], y[1] = a[3], x[2] = b[0], y[2] = b[1], x[3] = b[2], y[3] = b[3];
            if (p.bias)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (e < n) {
                        x[e] += bias_at(2 * (col + e));
                        y[e] += bias_at(2 * (col + e) + 1);
                    }
        } else {
            total4(red, m * PITCH + u, cs, x);
            total4(red, m * PITCH + u + ROWS / 2, cs, y);
        }
        if (rope) {  // out = bf16(bf16(x cos) + bf16(rotate_half(x) sin)), as the fused GEMM epilogue rounds
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] = bf16_round(x[e]);
                y[e] = bf16_round(y[e]);
            }
            if (col < p.rope_cols) {  // the same for all four: whole heads are rotated
                const long long at = (long long)(m % p.rope_S) * 128 + (col & 127);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float c1 = __bfloat162float(p.rope_cos[at + e]), s1 = __bfloat162float(p.rope_sin[at + e]);
                    const float c2 = __bfloat162float(p.rope_cos[at + e + 64]), s2 = __bfloat162float(p.rope_sin[at + e + 64]);
                    const float o = bf16_round(x[e] * c1) + bf16_round(-y[e] * s1);
                    y[e] = bf16_round(y[e] * c2) + bf16_round(x[e] * s2);
                    x[e] = o;
                }
            }
            store4(c, x, vec, n);
            store4(c + 64, y, vec, n);
            continue;
        }
        if (GROUPED && p.in_wts) {
            const float f = p.in_wts[p.perm[row0 + m]];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] *= f;
                y[e] *= f;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (p.act == kActReluGlu) {
                x[e] = fmaxf(x[e], 0.f) * y[e];
            } else if (p.act == kActSwiglu) {  // the rounding steps of the product and of the op behind it
                const float gr = bf16_round(x[e]);
                x[e] = bf16_round(__fdividef(gr, 1.f + __expf(-gr))) * bf16_round(y[e]);
            } else if (p.act == kActSiluGlu) {
                x[e] = x[e] * (1.0f / (1.0f + expf(-x[e]))) * y[e];
            } else {
                x[e] = fminf(x[e], p.limit);
                x[e] = x[e] / (1.0f + expf(-p.slope * x[e])) * (fminf(fmaxf(y[e], -p.limit), p.limit) + 1.0f);
            }
        }
        store4(c, x, vec, n);
    }
}

// Where a tile's weight rows begin, and what is added to a row's number from the middle of the tile on: pairs that meet in the
// epilogue are then half a tile apart (gate and up halves; a rotated head's two halves, when the tile is smaller than a head).
template <int ROWS>
__device__ __forceinline__ void tile_rows(const Args& p, int tile, int& base, int& gap) {
    base = tile * ROWS;
    gap = 0;
    if (gate_up(p)) {
        base = tile * (ROWS / 2);
        gap = (p.N >> 1) - ROWS / 2;
    } else if (p.act == kActRope && ROWS == 64) {
        base = (tile >> 1) * 128 + (tile & 1) * 32;
        gap = 32;
    }
}
template <int ROWS>
__device__ __forceinline__ bool row_live(const Args& p, int base, int gap, int i) {
    return gate_up(p) ? base + (i & (ROWS / 2 - 1)) < (p.N >> 1) : base + i + (i >= ROWS / 2 ? gap : 0) < p.N;
}

// The first SLICES slices of this CTA's weights, asked for in L2
template <int ROWS, int SLICES>
__device__ __forceinline__ void ahead(const Args& p, const bf16_t* W, int base, int gap, int c_lo, int n) {
    for (int i = threadIdx.x; i < ROWS * SLICES; i += kThreads) {
        const int r = i / SLICES, s = i % SLICES;
        if (s < n && row_live<ROWS>(p, base, gap, r))
            prefetch_l2(W + (long long)(base + r + (r >= ROWS / 2 ? gap : 0)) * p.ldw + (c_lo + s) * BK);
    }
}

// ------------------------------------------------------------------------------------------------ up to eight tokens
template <typename TC>
__global__ void __launch_bounds__(kThreads, 4)
skinny_kernel(const Args p, int cs) {
    extern __shared__ __align__(128) unsigned char smraw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = cs > 1 ? (int)(blockIdx.x % cs) : 0, tile = (int)blockIdx.x / cs;
    int base, gap;
    tile_rows<BN>(p, tile, base, gap);
    const uint32_t sm = smem_u32(smraw);
    const int nch = (p.K + BK - 1) / BK;
    const int c_lo = rank * nch / cs, n = (rank + 1) * nch / cs - c_lo;

    // ---- what this thread copies: four pieces of the weights' slice, and the first half of the threads one of the tokens'
    const int pc = threadIdx.x & 7, pr = threadIdx.x >> 3;
    const bf16_t* wsrc[4];
    bool wlive[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int i = pr + 16 * j;
        wlive[j] = row_live<BN>(p, base, gap, i);
        wsrc[j] = p.W + (wlive[j] ? (long long)(base + i + (i >= BN / 2 ? gap : 0)) * p.ldw : 0) + pc * 8;
    }
    const bool alive = pr < p.M;
    const bf16_t* asrc = p.A + (alive ? pr * p.lda : 0) + pc * 8;
    auto issue_w = [&](int c, int stage) {
        const int k = (c_lo + c) * BK;
        const bool in = k + pc * 8 < p.K;
        const uint32_t w = sm + stage * kStageMma;
#pragma unroll
        for (int j = 0; j < 4; ++j) copy16(w + piece(pr + 16 * j, pc), wlive[j] && in ? wsrc[j] + k : p.W, wlive[j] && in);
    };
    auto issue_a = [&](int c, int stage) {
        const int k = (c_lo + c) * BK;
        const bool in = alive && k + pc * 8 < p.K;
        if (pr < 8) copy16(sm + stage * kStageMma + BN * 128 + piece(pr, pc), in ? asrc + k : p.A, in);
    };
    // The tensor cores cut what does not fit their accumulators instead of rounding it, so the products of a slice start from
    // zero and its sums are added up in registers: the error over K = 4096 is that of fp32 FMAs (1.2e-7; 1.0e-6 in one chain).
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    let_next_begin();
    if (!p.weights_there) {
        ahead<BN, kStagesMma - 1>(p, p.W, base, gap, c_lo, n);
        wait_for_previous();
    }
#pragma unroll
    for (int s = 0; s < kStagesMma - 1; ++s) {
        if (s < n) issue_w(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (p.weights_there) wait_for_previous();
    if (pr < 8) {  // the tokens of the first slices, by loads: a copy of theirs would be done after all of the weights before it
        uint4 v[kStagesMma - 1];
#pragma unroll
        for (int s = 0; s < kStagesMma - 1; ++s) {
            const int k = (c_lo + s) * BK;
            v[s] = make_uint4(0, 0, 0, 0);
            if (s < n && alive && k + pc * 8 < p.K) v[s] = *reinterpret_cast<const uint4*>(asrc + k);
        }
#pragma unroll
        for (int s = 0; s < kStagesMma - 1; ++s)
            *reinterpret_cast<uint4*>(smraw + s * kStageMma + BN * 128 + piece(pr, pc)) = v[s];
    }
    int st = 0, st_in = kStagesMma - 1;
    for (int it = 0; it < n; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStagesMma - 2) : "memory");
        __syncthreads();  // slice `it` is there for everybody, and everybody is done with the one before
        if (it + kStagesMma - 1 < n) {
            issue_w(it + kStagesMma - 1, st_in);
            issue_a(it + kStagesMma - 1, st_in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const uint32_t w = sm + st * kStageMma, a = w + BN * 128;
        const int wr = warp * 16 + (lane & 15);
        float acc[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ks += 2) {
            uint32_t w0[4], w1[4], b[4];
            ldsm4(w0, w + piece(wr, ks * 2 + (lane >> 4)));
            ldsm4(w1, w + piece(wr, ks * 2 + 2 + (lane >> 4)));
            ldsm4(b, a + piece(lane & 7, ks * 2 + (lane >> 3)));
            mma16(acc[0], w0, b[0], b[1]);
            mma16(acc[1], w1, b[2], b[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] += acc[0][e] + acc[1][e];
        if (++st == kStagesMma) st = 0;
        if (++st_in == kStagesMma) st_in = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // ---- partial sums to shared memory, [token][row]
    float* red = reinterpret_cast<float*>(smraw);
#pragma unroll
    for (int e = 0; e < 4; ++e)
        red[(2 * (lane & 3) + (e & 1)) * RP + warp * 16 + (lane >> 2) + (e >> 1) * 8] = sum[e];
    if (cs > 1)
        cluster_sync_all();
    else
        __syncthreads();
    epilogue<TC, false, BN, RP>(p, red, p.M, 0, base, cs, rank);
    if (cs > 1) cluster_sync_all();  // nobody leaves while its partial sums may still be read
}

// ------------------------------------------------------------------------------------------------ more tokens
// From nine tokens on the fragments of A that every warp of the kernel above reads again fill the shared-memory pipe (64 tokens:
// 2.3x the memory time). Here the same slices go to tcgen05.mma: 128 weight rows are its M side, up to NTOK tokens its N side, the
// sums lie in NTOK columns of TMEM. CH: every CH slices the products start from zero, in one of two sets of columns, and are added up
// in registers while the next ones are multiplied (CH 0: one chain over K, 2 to 9e-6 of the result where fp32 FMAs give 1e-7).
constexpr int TN = 128, TRP = TN + 4;
template <int NTOK> constexpr int kStages = NTOK <= 16 ? 6 : NTOK <= 32 ? 5 : 4;  // 108, 100, 96 KB: two CTAs per SM

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {  // 8-row groups of 1024 bytes, 128-byte swizzle
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

template <int NTOK, typename TC, bool GROUPED, int CH>
__global__ void __launch_bounds__(kThreads)
skinny_tc_kernel(const Args p, int cs) {
    extern __shared__ unsigned char smraw_[];
    constexpr int kStage = TN * 128 + NTOK * 128, S = kStages<NTOK>;
    constexpr int kCols = CH ? 2 * NTOK : NTOK < 32 ? 32 : NTOK;
    __shared__ uint64_t done[S];
    __shared__ uint32_t tmem_base;
    unsigned char* smraw = smraw_ + ((1024u - (smem_u32(smraw_) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = cs > 1 ? (int)(blockIdx.x % cs) : 0, tile = (int)blockIdx.x / cs;
    int M = p.M, row0 = 0;
    const bf16_t* W = p.W;
    if (GROUPED) {
        wait_for_previous();
        if ((int)blockIdx.y >= p.meta[0]) return;  // the whole cluster
        const int* t = p.tiles + 3 * blockIdx.y;
        W += (long long)t[0] * p.N * p.K;
        row0 = t[1];
        M = t[2];
    }
    int base, gap;
    tile_rows<TN>(p, tile, base, gap);
    if (threadIdx.x == 0) {
        for (int i = 0; i < S; ++i) mbar_init(&done[i], 1);
        mbar_fence_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_base, kCols);
        tmem_relinquish();
    }
    const uint32_t sm = smem_u32(smraw);
    const int nch = (p.K + BK - 1) / BK;
    const int c_lo = rank * nch / cs, n = (rank + 1) * nch / cs - c_lo;
    const int pc = threadIdx.x & 7, pr = threadIdx.x >> 3;
    const bf16_t* wsrc[8];
    bool wlive[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int i = pr + 16 * j;
        wlive[j] = row_live<TN>(p, base, gap, i);
        wsrc[j] = W + (wlive[j] ? (long long)(base + i + (i >= TN / 2 ? gap : 0)) * p.ldw : 0) + pc * 8;
    }
    constexpr int NA = NTOK / 16;
    const bf16_t* asrc[NA];
    bool alive[NA];
#pragma unroll
    for (int j = 0; j < NA; ++j) {
        const int m = pr + 16 * j;
        alive[j] = m < M;
        long long r = 0;
        if (alive[j]) r = GROUPED ? (p.perm ? p.perm[row0 + m] / p.top : row0 + m) : m;
        asrc[j] = p.A + r * p.lda + pc * 8;
    }
    const int m_pad = (M + 15) & ~15;  // tokens that are multiplied
    auto issue_w = [&](int c, int stage) {
        const int k = (c_lo + c) * BK;
        const bool in = k + pc * 8 < p.K;
        const uint32_t w = sm + stage * kStage;
#pragma unroll
        for (int j = 0; j < 8; ++j) copy16(w + piece(pr + 16 * j, pc), wlive[j] && in ? wsrc[j] + k : p.W, wlive[j] && in);
    };
    auto issue_a = [&](int c, int stage) {
        const int k = (c_lo + c) * BK;
        const uint32_t a = sm + stage * kStage + TN * 128;
#pragma unroll
        for (int j = 0; j < NA; ++j) {
            const bool in = alive[j] && k + pc * 8 < p.K;
            if (pr + 16 * j < m_pad) copy16(a + piece(pr + 16 * j, pc), in ? asrc[j] + k : p.A, in);
        }
    };
    const bool early = !GROUPED && p.weights_there;
    if (!GROUPED && !early) ahead<TN, S - 1>(p, W, base, gap, c_lo, n);
    tc_fence_before();
    __syncthreads();  // TMEM is allocated
    tc_fence_after();
    let_next_begin();
    if (!GROUPED && !early) wait_for_previous();
#pragma unroll
    for (int s = 0; s < S - 1; ++s) {
        if (s < n) issue_w(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (early) wait_for_previous();
    {  // the tokens of the first slices, by loads: a copy of theirs would be done after all of the weights before it
        uint4 v[S - 1][NA];
#pragma unroll
        for (int s = 0; s < S - 1; ++s)
#pragma unroll
            for (int j = 0; j < NA; ++j) {
                const int k = (c_lo + s) * BK;
                v[s][j] = make_uint4(0, 0, 0, 0);
                if (s < n && alive[j] && k + pc * 8 < p.K) v[s][j] = *reinterpret_cast<const uint4*>(asrc[j] + k);
            }
#pragma unroll
        for (int s = 0; s < S - 1; ++s)
#pragma unroll
            for (int j = 0; j < NA; ++j)
                *reinterpret_cast<uint4*>(smraw + s * kStage + TN * 128 + piece(pr + 16 * j, pc)) = v[s][j];
    }
    const uint32_t tmem = tmem_base;
    // fp32 sums, bf16 operands, both K-major, M = 128, N = m_pad
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(m_pad >> 3) << 17) | ((uint32_t)(TN >> 4) << 24);
    auto set = [](int it) { return CH ? it / (CH ? CH : 1) % 2 * NTOK : 0; };  // the columns of a slice's products
    float sum[NTOK];  // of weight row warp * 32 + lane
#pragma unroll
    for (int j = 0; j < NTOK; ++j) sum[j] = 0.f;
    auto add = [&](int it) {  // the sums up to slice `it`, whose products have been waited for
        tc_fence_after();
        constexpr int NL = NTOK < 32 ? NTOK : 32;
#pragma unroll
        for (int c0 = 0; c0 < NTOK; c0 += NL) {
            if (c0 >= m_pad) break;  // the same for everybody
            uint32_t v[NL];
            const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16) + set(it) + c0;
            if constexpr (NL == 16)
                tmem_ld_32x32b_x16(at, v);
            else
                tmem_ld_32x32b_x32(at, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < NL; ++j) sum[c0 + j] += __uint_as_float(v[j]);  // columns from m_pad on hold nothing and are not used
        }
        tc_fence_before();
    };
    int st = 0, st_in = S - 1;
    for (int it = 0; it < n; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        fence_proxy_async_smem();
        __syncthreads();  // slice `it` is there, written by everybody; everybody has taken the sums before those of slice it - 1
        if (threadIdx.x == 0) {
            tc_fence_after();
            const uint64_t wd = smem_desc(sm + st * kStage), ad = smem_desc(sm + st * kStage + TN * 128);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                umma_f16(tmem + set(it), wd + (uint64_t)(k * 2), ad + (uint64_t)(k * 2), idesc, (CH ? it % (CH ? CH : 1) : it) != 0 || k != 0);
            umma_commit(&done[st]);
        }
        if (it) mbar_wait(&done[st_in], (uint32_t)(((it - 1) / S) & 1));  // the slice before: its place is free, its sums are there
        if (it + S - 1 < n) {
            issue_w(it + S - 1, st_in);
            issue_a(it + S - 1, st_in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (CH && it && it % (CH ? CH : 1) == 0) add(it - 1);
        if (++st == S) st = 0;
        if (++st_in == S) st_in = 0;
    }
    mbar_wait(&done[(n - 1) % S], (uint32_t)(((n - 1) / S) & 1));
    add(n - 1);
    // ---- partial sums to shared memory, [token][row]: the slices are no longer read
    float* red = reinterpret_cast<float*>(smraw);
#pragma unroll
    for (int j = 0; j < NTOK; ++j)
        if (j < m_pad) red[j * TRP + warp * 32 + lane] = sum[j];
    if (cs > 1)
        cluster_sync_all();
    else
        __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kCols);
    epilogue<TC, GROUPED, TN, TRP>(p, red, M, row0, base, cs, rank);
    if (cs > 1) cluster_sync_all();  // nobody leaves while its partial sums may still be read
}

// ------------------------------------------------------------------------------------------------ host
template <typename F>
static cudaError_t go(F kernel, std::atomic<unsigned long long>& allowed, int smem, const Args& a, int cs, int tiles,
                      cudaStream_t st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(allowed.load(std::memory_order_relaxed) >> dev & 1)) {  // once per device
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev < 64) allowed.fetch_or(1ull << dev, std::memory_order_relaxed);
    }
    return launch_early(kernel, dim3((unsigned)(tiles * cs), a.tiles ? (unsigned)a.max_tiles : 1u), dim3(kThreads), (size_t)smem, cs, st, a, cs);
}
template <typename TC>
static cudaError_t go_mma(const Args& a, int cs, int tiles, cudaStream_t st) {
    static std::atomic<unsigned long long> allowed{0};
    return go(skinny_kernel<TC>, allowed, kStagesMma * kStageMma, a, cs, tiles, st);
}
template <int NTOK, typename TC, bool GROUPED, int CH>
static cudaError_t go_tc(const Args& a, int cs, int tiles, cudaStream_t st) {
    static std::atomic<unsigned long long> allowed{0};
    return go(skinny_tc_kernel<NTOK, TC, GROUPED, CH>, allowed, kStages<NTOK> * (TN * 128 + NTOK * 128) + 1024, a, cs, tiles, st);
}

cudaError_t launch(const Args& a, cudaStream_t st) {
    const bool grouped = a.tiles != nullptr;
    // Up to eight tokens the mma.sync kernel: as fast as the other or faster (K = 2048, N = 2048: 5.4 against 6.7 us), and ten
    // times as exact. Routed experts have 0 to 64 tokens per tile, known only on the device.
    const bool tc = grouped || a.M > 8;
    const int rows = tc ? TN : BN;
    const int tiles = gate_up(a) ? (a.N / 2 + rows / 2 - 1) / (rows / 2) : (a.N + rows - 1) / rows;
    // Cut along K until the grid holds as many CTAs as are resident at once (four or two for each of the 148 SMs), as long as a
    // CTA keeps four slices of K.
    const int nch = (a.K + BK - 1) / BK;
    const long long most = tc ? 296 : 592;
    int cs = 1;
    while (cs < 8 && (long long)tiles * (grouped ? a.max_tiles : 1) * cs * 2 <= most && nch / (cs * 2) >= 4) cs *= 2;
#define LLARK_SKINNY(N_, GR_, CH_) (a.c_fp32 ? go_tc<N_, float, GR_, CH_>(a, cs, tiles, st) : go_tc<N_, bf16_t, GR_, CH_>(a, cs, tiles, st))
    if (!tc) return a.c_fp32 ? go_mma<float>(a, cs, tiles, st) : go_mma<bf16_t>(a, cs, tiles, st);
    if (grouped) return LLARK_SKINNY(64, true, 1);
    // Short chains for what fp32 FMAs computed before: narrow products, paired activations with an fp32 result and results off 16-byte
    // boundaries. The others took the tcgen05 core, whose one chain over K errs by 4 to 12e-6; cut over a cluster theirs are shorter (0.5 to 1.4e-6), and 6 % faster than
    // short ones (a decode step of 32 rows 549 us against 582).
    if (a.N < 64 || (a.c_fp32 && (a.act == kActReluGlu || a.act == kActClampGlu)) || a.ldc % (a.c_fp32 ? 4 : 8) ||
        (reinterpret_cast<uintptr_t>(a.C) & 15)) {
        if (a.M <= 16) return LLARK_SKINNY(16, false, 1);
        if (a.M <= 32) return LLARK_SKINNY(32, false, 1);
        return LLARK_SKINNY(64, false, 1);
    }
    if (a.M <= 16) return LLARK_SKINNY(16, false, 0);
    if (a.M <= 32) return LLARK_SKINNY(32, false, 0);
    return LLARK_SKINNY(64, false, 0);
#undef LLARK_SKINNY
}

}  // namespace skinny
}  // namespace llark
