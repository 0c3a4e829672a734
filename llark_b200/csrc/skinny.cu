// Products with few rows (decode steps, routed experts of a few tokens): a stream of the weight matrix. See skinny.cuh.
//
// What bounds it is how many bytes of the weights are on their way. A CTA takes a tile of weight rows; its operands come through a ring of
// 64-wide slices of K (54 or 112 KB of it per CTA, four or two CTAs per SM), and matrices with few rows are also cut along K over a
// cluster of up to eight CTAs, whose partial sums meet in distributed shared memory in a fixed order (no atomics, no workspace). The
// weights are the M side of the products and the tokens the N side, so that up to 64 tokens ride on one read of a weight. A slice is kept
// as 128-byte rows whose 16-byte pieces are XORed with the row number: cp.async and ldmatrix are free of bank conflicts, and it is the
// 128-byte swizzle of TMA boxes and tcgen05 operands.
//
// A decode step is a row of such products with short kernels between them, and each of them filled an empty chip and drained it again:
// 202 us of products for 163 us of bytes in a step of two layers and the head, one row, and 268 us for the whole step. So a CTA starts
// while the kernel in front of it ends (launch_early): its weights are under way, or on their way to L2, before the tokens are there.
// The next kernel is let in at once: after half of the slices or with the last ones asked for the step took 2 to 3 us longer.
// Measured, a step of 1 / 8 / 32 rows behind 1024 / 1024 / 1500 positions: 269 -> 236, 306 -> 280, 547 -> 485 us (the last with weights through TMA; 510
// without).
//
// Measured on a B200, launches in a row on rotating weights (floor = the weights at 6.55 TB/s), against the 256-row tiles of the
// tcgen05 GEMM core: N 4096 K 4096, 32 tokens 11.1 us (core 28.7, floor 5.1); N 22016 K 4096 33.0 (54.9, 27.5); N 4096 K 11008
// 19.3 (61.0, 13.8); N 32004 K 4096 43.3 (56.3, 40.0); 64 tokens 12.8 / 34.2 / 21.0 / 46.0; one token 7.7 / 30.2 / 16.3 / 41.6.
#include "skinny.cuh"

#include <cuda.h>

#include <atomic>

namespace llark {
int tensor_map_2d(CUtensorMap* out, const void* ptr, long long inner, long long outer, long long ld, int box_inner, int box_outer,
                  int elem_bytes);  // gemm_tcgen05.cu
int tensor_map_batches(CUtensorMap* out, const void* ptr, long long inner, long long outer, long long ld, int batches, int box_inner,
                       int box_outer, int elem_bytes);

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

// A unit is a row of W, or the two rows that meet in the epilogue.
__host__ __device__ __forceinline__ bool adjacent_rows(const Args& p) { return p.act == kActReluGlu || p.act == kActClampGlu; }
__host__ __device__ __forceinline__ bool paired(const Args& p) { return adjacent_rows(p) || gate_up(p) || p.act == kActRope; }

// The results of the `units` units from u0 on (both multiples of four), from the partial sums red [token][row] (rows PITCH apart) of the
// cluster's CTAs; this CTA does its share of them, four at a time. The two rows of a unit are rows 2 u and 2 u + 1 of the tile, or u and
// u + units.
template <typename TC, bool GROUPED, int PITCH>
__device__ __forceinline__ void epilogue(const Args& p, const float* red, int M, int row0, int u0, int units, int cs, int rank) {
    const bool adjacent = adjacent_rows(p), rope = p.act == kActRope, two = paired(p);
    const int quads = units >> 2, q0 = rank * quads / cs, nq = (rank + 1) * quads / cs - q0;
    const int all = two ? p.N >> 1 : p.N;
    TC* C = static_cast<TC*>(p.C);
    const bool vec = p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & (4 * sizeof(TC) - 1)) == 0;
    auto bias_at = [&](int c) { return p.bias_fp32 ? ldc_<float>(p.bias, c) : ldc_<bf16_t>(p.bias, c); };
    for (int i = threadIdx.x; i < M * nq; i += kThreads) {
        const int m = i / nq, u = 4 * (q0 + i % nq);
        const int n = all - (u0 + u), col = rope ? ((u0 + u) >> 6) * 128 + ((u0 + u) & 63) : u0 + u;
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
            total4(red, m * PITCH + u + units, cs, y);
        }
        if (rope) {  // out = bf16(bf16(x cos) + bf16(rotate_half(x) sin)), as the fused GEMM epilogue rounds
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] = bf16_round(x[e]);
                y[e] = bf16_round(y[e]);
            }
            if (col < p.rope_cols) {  // the same for all four: whole heads are rotated
                const long long at = (long long)((p.first + m) % p.rope_S) * 128 + (col & 127);
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
    epilogue<TC, false, RP>(p, red, p.M, 0, tile * (paired(p) ? BN / 2 : BN), paired(p) ? BN / 2 : BN, cs, rank);
    if (cs > 1) cluster_sync_all();  // nobody leaves while its partial sums may still be read
}

// ------------------------------------------------------------------------------------------------ more tokens
// From nine tokens on the fragments of A that every warp of the kernel above reads again fill the shared-memory pipe (64 tokens:
// 2.3x the memory time). Here the same slices go to tcgen05.mma: 128 weight rows are its M side, up to NTOK tokens its N side, the
// sums lie in NTOK columns of TMEM. CH: every CH slices the products start from zero, in one of two sets of columns, and are added up
// in registers while the next ones are multiplied (CH 0: one chain over K, 2 to 9e-6 of the result where fp32 FMAs give 1e-7).
//
// The weights come as TMA boxes that one thread requests. With cp.async a slice took 0.6 us of every warp's instructions and of waiting
// for the products of the slice before, whatever its bytes, and two slices less were under way: N 22016 K 4096 39.4 -> 33.0 us with 32
// tokens, 45.2 -> 34.2 with 64; N 12288 K 4096 23.6 -> 20.4, 27.0 -> 22.9; routed experts of 32 tokens 114 -> 111. Issued by the warp
// together (see warp_umma_f16) instead of by one lane: 33.8 -> 32.9, 34.4 -> 32.9, 20.7 -> 19.6, 23.1 -> 22.1; experts 112 -> 104.
constexpr int TN = 128, TRP = TN + 4;
constexpr int kTcSmem = 112 * 1024, kMaxStages = 12;  // two CTAs per SM
constexpr int kGroupedSmem = kTcSmem - 1024;
// How W is cut: a tile of `units` units, `rows` rows of W (a multiple of eight), for the cs CTAs of a cluster
struct Cut {
    int units, rows, cs, stages;
};

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

// Four warps for the sums and results, one that requests, one that multiplies, and two that copy tokens: where they are gathered, and up to
// 32 of them, where the same few lines asked for by every CTA at once hold up the weights' boxes in the TMA (N 32004: 43.2 us, by boxes 44.6);
// 64 tokens come as boxes, of which more slices are under way (N 22016: 41.6 us by copies, 37.5).
__host__ __device__ constexpr bool copied(int ntok, bool grouped) { return grouped || ntok <= 32; }
__host__ __device__ constexpr int tc_threads(bool copies) { return copies ? 256 : 192; }
constexpr int kTokenLag = 3;     // slices of tokens on their way while the next is requested

template <int NTOK, typename TC, bool GROUPED, int CH>
__global__ void __launch_bounds__(tc_threads(copied(NTOK, GROUPED)), 2)
skinny_tc_kernel(const Args p, const Cut cut, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap amap) {
    extern __shared__ unsigned char smraw_[];
    constexpr bool COPIES = copied(NTOK, GROUPED);
    const int cs = cut.cs;
    constexpr int kCols = CH ? 2 * NTOK : NTOK < 32 ? 32 : NTOK;
    __shared__ uint64_t full[kMaxStages], empty[kMaxStages], ready[2], drained[2];
    __shared__ uint32_t tmem_base;
    unsigned char* smraw = smraw_ + ((1024u - (smem_u32(smraw_) & 1023u)) & 1023u);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = cs > 1 ? (int)(blockIdx.x % cs) : 0, tile = (int)blockIdx.x / cs;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kMaxStages; ++i) {
            mbar_init(&full[i], COPIES ? 3 : 1);  // the request, and both warps of the tokens
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ready[i], 1);
            mbar_init(&drained[i], 4);
        }
        mbar_fence_init();
    }
    if (warp == 5) {
        tmem_alloc(&tmem_base, kCols);
        tmem_relinquish();
    }
    const uint32_t sm = smem_u32(smraw);
    const int nch = (p.K + BK - 1) / BK;
    const int c_lo = rank * nch / cs, n = (rank + 1) * nch / cs - c_lo;
    tc_fence_before();
    __syncthreads();  // TMEM is allocated
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    let_next_begin();
    int M = p.M, row0 = 0, expert = 0;
    if (GROUPED) {
        wait_for_previous();
        if ((int)blockIdx.y >= p.meta[0]) {  // the whole cluster
            if (warp == 5) tmem_dealloc(tmem, kCols);
            return;
        }
        const int* t = p.tiles + 3 * blockIdx.y;
        expert = t[0];
        row0 = t[1];
        M = t[2];
    }
    const int u0 = tile * cut.units;
    const int wrow = p.act == kActRope ? (u0 >> 6) * 128 + (u0 & 63) : adjacent_rows(p) ? 2 * u0 : u0;
    const int m_pad = (M + 15) & ~15;  // tokens that are multiplied
    // of a stage, in bytes; with few tokens a routed tile has room for more stages than the worst case
    const int kWeights = (GROUPED ? TN : cut.rows) * 128, kStage = kWeights + (GROUPED ? m_pad : NTOK) * 128;
    const int S = GROUPED ? kGroupedSmem / kStage : cut.stages;
    auto set = [](int it) { return CH ? it / (CH ? CH : 1) % 2 * NTOK : 0; };  // the columns of a slice's products
    float sum[NTOK];  // of weight row warp * 32 + lane
    if (warp < 4) {
        wait_for_previous();  // for the residual, and before anything is written
#pragma unroll
        for (int j = 0; j < NTOK; ++j) sum[j] = 0.f;
        const int chains = CH ? (n + (CH ? CH : 1) - 1) / (CH ? CH : 1) : 1;
        for (int c = 0; c < chains; ++c) {
            mbar_wait(&ready[c & 1], (uint32_t)((c >> 1) & 1));
            tc_fence_after();
            constexpr int NL = NTOK < 32 ? NTOK : 32;
#pragma unroll
            for (int c0 = 0; c0 < NTOK; c0 += NL) {
                if (c0 >= m_pad) break;  // the same for everybody
                uint32_t v[NL];
                const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16) + (CH ? (c & 1) * NTOK : 0) + c0;
                if constexpr (NL == 16)
                    tmem_ld_32x32b_x16(at, v);
                else
                    tmem_ld_32x32b_x32(at, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < NL; ++j) sum[c0 + j] += __uint_as_float(v[j]);  // columns from m_pad on hold nothing and are not used
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&drained[c & 1]);
        }
    } else if (warp == 4) {
        if (lane == 0) {
            const int other = gate_up(p) ? p.N >> 1 : p.act == kActRope && cut.units < 64 ? 64 : 0;  // where the units' other rows are
            auto each = [&](int it, auto use) {  // the boxes of a slice
                const int k = (c_lo + it) * BK;
                use(k, wrow, 0);
                if (other) use(k, wrow + other, kWeights / 2);
            };
            auto request = [&](int it, int st) {
                mbar_arrive_expect_tx(&full[st], COPIES ? kWeights : kStage);
                each(it, [&](int k, int row, int at) {
                    if (GROUPED)
                        tma_load_3d(smraw + st * kStage + at, &wmap, &full[st], k, row, expert);
                    else
                        tma_load_2d(smraw + st * kStage + at, &wmap, &full[st], k, row);
                });
            };
            if (!GROUPED && !p.weights_there) {
                for (int it = 0; it < S && it < n; ++it) each(it, [&](int k, int row, int) { tma_prefetch_2d(&wmap, k, row); });
                wait_for_previous();
            }
            const int first = n < S ? n : S;
            for (int it = 0; it < first; ++it) request(it, it);
            auto tokens = [&](int it, int st) {
                if (!COPIES) tma_load_2d(smraw + st * kStage + kWeights, &amap, &full[st], (c_lo + it) * BK, 0);
            };
            if (!COPIES) {
                if (p.weights_there) wait_for_previous();
                for (int it = 0; it < first; ++it) tokens(it, it);
            }
            for (int it = S, st = 0, ph = 0; it < n; ++it) {
                mbar_wait(&empty[st], ph);
                request(it, st);
                tokens(it, st);
                if (++st == S) st = 0, ph ^= 1;
            }
        }
    } else if (warp == 5) {
        {
            // fp32 sums, bf16 operands, both K-major, M = 128, N = m_pad
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(m_pad >> 3) << 17) | ((uint32_t)(TN >> 4) << 24);
            for (int it = 0, st = 0, ph = 0; it < n; ++it) {
                const int c = CH ? it / (CH ? CH : 1) : 0;
                if (CH && c >= 2 && it % (CH ? CH : 1) == 0) mbar_wait(&drained[c & 1], (uint32_t)(((c >> 1) - 1) & 1));
                mbar_wait(&full[st], ph);
                tc_fence_after();
                const uint64_t wd = smem_desc(sm + st * kStage), ad = smem_desc(sm + st * kStage + kWeights);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    warp_umma_f16(tmem + set(it), wd + (uint64_t)(k * 2), ad + (uint64_t)(k * 2), idesc, (CH ? it % (CH ? CH : 1) : it) != 0 || k != 0);
                warp_umma_commit(&empty[st]);
                if (it == n - 1 || (CH && (it + 1) % (CH ? CH : 1) == 0)) warp_umma_commit(&ready[c & 1]);
                if (++st == S) st = 0, ph ^= 1;
            }
        }
    } else if (COPIES) {
        wait_for_previous();
        const int pc = threadIdx.x & 7, pr = (threadIdx.x - 192) >> 3;
        constexpr int NA = NTOK / 8;
        const bf16_t* asrc[NA];
        bool alive[NA];
#pragma unroll
        for (int j = 0; j < NA; ++j) {
            const int m = pr + 8 * j;
            alive[j] = m < M;
            long long r = 0;
            if (alive[j]) r = !GROUPED ? m : p.perm ? p.perm[row0 + m] / p.top : row0 + m;
            asrc[j] = p.A + r * p.lda + pc * 8;
        }
        int st = 0, ph = 1, st_out = 0;
        for (int it = 0; it < n + kTokenLag; ++it) {
            if (it < n) {
                if (it >= S) mbar_wait(&empty[st], ph);
                const int k = (c_lo + it) * BK;
                const uint32_t a = sm + st * kStage + kWeights;
#pragma unroll
                for (int j = 0; j < NA; ++j) {
                    const bool in = alive[j] && k + pc * 8 < p.K;
                    if (pr + 8 * j < m_pad) copy16(a + piece(pr + 8 * j, pc), in ? asrc[j] + k : p.A, in);
                }
                if (++st == S) st = 0, ph ^= 1;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (it >= kTokenLag) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kTokenLag) : "memory");
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[st_out]);
                if (++st_out == S) st_out = 0;
            }
        }
    }
    __syncwarp();
    // ---- partial sums to shared memory, [token][row]: the slices are no longer read
    float* red = reinterpret_cast<float*>(smraw);
    if (warp < 4) {
#pragma unroll
        for (int j = 0; j < NTOK; ++j)
            if (j < m_pad) red[j * TRP + warp * 32 + lane] = sum[j];
    }
    if (cs > 1)
        cluster_sync_all();
    else
        __syncthreads();
    if (warp == 5) tmem_dealloc(tmem, kCols);
    if (warp < 4) epilogue<TC, GROUPED, TRP>(p, red, M, row0, u0, cut.units, cs, rank);
    if (cs > 1) cluster_sync_all();  // nobody leaves while its partial sums may still be read
}

// ------------------------------------------------------------------------------------------------ host
template <typename F, typename... X>
static cudaError_t go(F kernel, std::atomic<unsigned long long>& allowed, int most, int smem, int threads, int tiles, int cs, cudaStream_t st,
                      const Args& a, const X&... more) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(allowed.load(std::memory_order_relaxed) >> dev & 1)) {  // once per device
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return e;
        if (dev < 64) allowed.fetch_or(1ull << dev, std::memory_order_relaxed);
    }
    return launch_early(kernel, dim3((unsigned)(tiles * cs), a.tiles ? (unsigned)a.max_tiles : 1u), dim3(threads), (size_t)smem, cs, st, a, more...);
}
template <typename TC>
static cudaError_t go_mma(const Args& a, int cs, int tiles, cudaStream_t st) {
    static std::atomic<unsigned long long> allowed{0};
    return go(skinny_kernel<TC>, allowed, kStagesMma * kStageMma, kStagesMma * kStageMma, kThreads, tiles, cs, st, a, cs);
}
static int units_of(const Args& a) { return paired(a) ? a.N / 2 : a.N; }

// Stages that fit beside what the products read behind the last one: they take 128 rows whatever the tile has
static int stages(int rows, int ntok, int& smem) {
    const int stage = (rows + ntok) * 128, tail = stage < TN * 128 ? TN * 128 - stage : 0;
    int s = (kTcSmem - 1024 - tail) / stage;
    if (s > kMaxStages) s = kMaxStages;
    smem = s * stage + tail + 1024;
    if (smem < ntok * TRP * 4 + 1024) smem = ntok * TRP * 4 + 1024;  // the partial sums
    return s;
}
// The weights as their tensor map has them: K by rows of W by experts. What a box reaches past an expert's last row is zeros and not read, the
// last expert's as well; a tile's expert is one that there is, so the third extent need not be their number.
struct Boxes {
    long long inner, outer;
    int experts, rows;  // rows of a box
};
static Boxes boxes_of(const Args& a, const Cut& cut) {
    const bool halves = gate_up(a) || (a.act == kActRope && cut.units < 64);  // two boxes for a slice
    return {a.K, a.N, a.tiles ? 65536 : 0, halves ? cut.units : cut.rows};
}
template <int NTOK, typename TC, bool GROUPED, int CH>
static cudaError_t go_tc(const Args& a, Cut cut, cudaStream_t st) {
    static std::atomic<unsigned long long> allowed{0};
    int smem;
    cut.stages = stages(cut.rows, NTOK, smem);
    if (GROUPED) smem = kTcSmem;
    const Boxes b = boxes_of(a, cut);
    CUtensorMap wmap;
    if (b.experts ? tensor_map_batches(&wmap, a.W, b.inner, b.outer, a.ldw, b.experts, BK, b.rows, 2)
                  : tensor_map_2d(&wmap, a.W, b.inner, b.outer, a.ldw, BK, b.rows, 2))
        return cudaErrorInvalidValue;
    CUtensorMap amap = wmap;
    if (!copied(NTOK, GROUPED) && tensor_map_2d(&amap, a.A, a.K, a.M, a.lda, BK, NTOK, 2)) return cudaErrorInvalidValue;
    return go(skinny_tc_kernel<NTOK, TC, GROUPED, CH>, allowed, kTcSmem, smem, tc_threads(copied(NTOK, GROUPED)), (units_of(a) + cut.units - 1) / cut.units, cut.cs, st, a,
              cut, wmap, amap);
}

// Whether the products of every slice of K start from zero (CH = 1 of skinny_tc_kernel): what fp32 FMAs computed before the tensor cores did, narrow
// products, paired activations with an fp32 result and results off 16-byte boundaries, and routed experts. The others are a chain over a CTA's
// part of K, in adders that cut what does not fit, and 6 % faster (a decode step of 32 rows 549 us against 582).
static bool short_chains(const Args& a) {
    return a.tiles || a.N < 64 || (a.c_fp32 && (a.act == kActReluGlu || a.act == kActClampGlu)) || a.ldc % (a.c_fp32 ? 4 : 8) ||
           (reinterpret_cast<uintptr_t>(a.C) & 15);
}

// How the products of more than eight rows and of routed experts are cut
static Cut cut_of(const Args& a) {
    const bool grouped = a.tiles != nullptr, two = paired(a);
    const int nch = (a.K + BK - 1) / BK, all = units_of(a), most = two ? TN / 2 : TN;
    // Tiles of 128 rows, cut along K until the grid holds two CTAs for each of the 148 SMs, as long as a CTA keeps four slices of K
    Cut cut = {most, TN, 1, 0};
    const int tiles = (all + most - 1) / most;
    while (cut.cs < 8 && (long long)tiles * (grouped ? a.max_tiles : 1) * cut.cs * 2 <= 296 && nch / (cut.cs * 2) >= 4) cut.cs *= 2;
    if (!grouped) {
        const int ntok = a.M <= 16 ? 16 : a.M <= 32 ? 32 : 64;
        // The tiles and clusters with most of the weights under way, of those that are all resident at once (two CTAs for each of the 148 SMs; of
        // clusters of four and eight 71 and 33 fit), as long as a CTA keeps four slices of K; larger tiles and smaller clusters unless others have a
        // twentieth more. Tiles of less than 64 rows leave the tensor cores more products than the time of their bytes. 22016 rows of gate
        // and up in 276 tiles of 80 instead of 172 of 128: 34.8 -> 32.7 us with 32 tokens, 37.5 -> 34.4 with 64. (Clusters of three: 12288
        // rows in 288 CTAs instead of 192 20.8 -> 31.) A chain over K is never cut over fewer CTAs than
        // above: its error goes with its length, 2.3e-7 of the result over 256, 4.7e-7 over 512, 2.1e-6 over 2048.
        static const int sizes[] = {1, 2, 4, 8}, fit[] = {296, 148, 71, 33};
        const int least = short_chains(a) ? 1 : cut.cs;
        long long best = 0;
        const long long bytes = 2LL * a.N * a.K / 128;
        for (int i = 0; i < 4; ++i) {
            if (sizes[i] < least) continue;
            if (sizes[i] > 1 && nch / sizes[i] < 4) break;
            for (int rows = TN; rows >= 64; rows -= 8) {
                const int units = two ? rows / 2 : rows;
                if (units % 8 || (a.act == kActRope && units != 64 && units != 32)) continue;
                const int tiles = (all + units - 1) / units;
                int smem;
                long long way = tiles <= fit[i] ? (long long)tiles * sizes[i] * stages(rows, ntok, smem) * rows : 0;
                if (way > bytes) way = bytes;
                if (way * 20 > best * 21) best = way, cut = {units, rows, sizes[i], 0};
            }
        }
    }
    return cut;
}

static cudaError_t by_eights(const Args& a, cudaStream_t st) {
    const int size = a.c_fp32 ? 4 : 2;
    for (int m = 0; m < a.M; m += 8) {
        Args b = a;
        b.M = a.M - m < 8 ? a.M - m : 8;
        b.first = a.first + m;
        b.A += m * a.lda;
        b.C = static_cast<char*>(a.C) + m * a.ldc * size;
        if (a.R) b.R = static_cast<const char*>(a.R) + m * a.ldr * size;
        const cudaError_t e = launch(b, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
cudaError_t launch(const Args& a, cudaStream_t st) {
    const bool grouped = a.tiles != nullptr, two = paired(a);
    const int nch = (a.K + BK - 1) / BK, all = units_of(a);
    // Up to eight tokens the mma.sync kernel: as fast as the other or faster (K = 2048, N = 2048: 4.5 against 5.8 us), and ten
    // times as exact. Routed experts have 0 to 64 tokens per tile, known only on the device.
    if (!grouped && a.M <= 8) {
        // Cut along K until the grid holds as many CTAs as are resident at once (four for each of the 148 SMs), as long as a CTA keeps four
        // slices of K.
        const int units = two ? BN / 2 : BN, tiles = (all + units - 1) / units;
        int cs = 1;
        while (cs < 8 && tiles * cs * 2 <= 592 && nch / (cs * 2) >= 4) cs *= 2;
        return a.c_fp32 ? go_mma<float>(a, cs, tiles, st) : go_mma<bf16_t>(a, cs, tiles, st);
    }
    // Rows closer to each other than K (one token's row for all tokens, windows of a sequence) are none that a tensor map is specified for
    if (!grouped && (a.ldw < a.K || (a.lda < a.K && a.M > 32))) return by_eights(a, st);
    const Cut cut = cut_of(a);
#define LLARK_SKINNY(N_, GR_, CH_) (a.c_fp32 ? go_tc<N_, float, GR_, CH_>(a, cut, st) : go_tc<N_, bf16_t, GR_, CH_>(a, cut, st))
    if (grouped) return LLARK_SKINNY(64, true, 1);
    if (short_chains(a)) {
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

extern "C" int llark_few_rows_plan(int M, int N, int K, int act, int max_tiles, long long* out) {
    using namespace llark::skinny;
    if (N <= 0 || K <= 0 || !out || (max_tiles <= 0 && (M <= 8 || M > kMaxRows))) return LLARK_EINVAL;
    static const int one = 0;
    Args a = {};
    a.M = M, a.N = N, a.K = K, a.act = act, a.max_tiles = max_tiles, a.tiles = max_tiles > 0 ? &one : nullptr;
    const Cut c = cut_of(a);
    const Boxes b = boxes_of(a, c);
    const long long v[] = {c.units, c.rows, c.cs, b.rows, b.inner, b.outer, b.experts};
    for (int i = 0; i < 7; ++i) out[i] = v[i];
    return LLARK_OK;
}
