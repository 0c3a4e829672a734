// Matrix recurrences of prompts, 16 tokens at a time as products on the tensor cores. Per head and request S is [D, E] and
//
//     S_t = diag(d_t) S_(t-1) + p_t u_t^T,     o_t = S_t^T q_t,
//
// with u_t = v_t (HGRN2: d = f, p = 1 - f; state-space layers) or, for the gated delta rules, u_t = v_t - S_(t-1)^T z_t, z = d . k
// and p = beta k. With b_t the product of d over the block's tokens up to t and w_s,t = p_s . d_(s+1) ... d_t (elementwise):
//
//     S_t^T x = S_0^T (b_t . x) + sum_(s <= t) (w_s,t x) u_s
//
// so a block of 16 tokens needs, beside S_0: Q' = b_t . q_t, Z' = b_(t-1) . z_t, the 16 x 16 matrices A[t, s] = w_s,t q_t (s <= t) and
// L[t, s] = w_s,(t-1) z_t (s < t), P = w_s,15 and b_15. Every product of decays is taken as such, front to back (never as a quotient of
// two of them), so nothing overflows however small a decay is. The correction u solves (1 + L) U = V - Z' S_0; with T = (1 + L)^-1,
// Z = T Z', Q = Q' - A Z and A' = A T both the outputs and U are direct functions of S_0 and V:
//
//     O = Q S_0 + A' V,    U = T V - Z S_0,    S = diag(b_15) S_0 + P^T U.
//
//   chunk_prep_kernel   all of that which does not depend on S, from the projections: a warp per block of tokens and head, every
//                       block at once, fp32
//   chunk_scan_kernel   the walk over the blocks: two warps keep 16 columns of S, transposed, half of the rows each, in registers
//                       that are directly the A operand of S^T Q^T; their partial results meet in shared memory. Every product as
//                       three TF32 products of split operands (x = hi + lo, without lo lo). The tensor cores cut their sums
//                       instead of rounding them, so chains are kept short (2 products) and a block's update of S starts from
//                       zero and is added with an FMA.
//
// The token-by-token kernels (seq_mixers.cu, seq_delta.cu) walk a chain of shared-memory reads and FMAs per token and stay for short
// steps, other sizes, the general rule and fp32 mode. What bounds this: one chain of blocks per head and 16 columns, in which a warp waits
// for its own results most of the time. With one warp for all rows the walk took 1.6 times as long. Measured on a B200, heads of 128, us,
// scan / here: HGRN2, 16 heads, 2048 + 1500 + 700 + 333 tokens 691 / 272; delta rule, 1777 + 1700 + 1500 tokens, a decay per head 1119 /
// 416; 1000 + 600 tokens, a decay per channel 533 / 199, state space 425 / 112.
#include "common.cuh"

#include <utility>

namespace llark {
extern thread_local int g_last_cuda_error;
namespace chunk {

constexpr int C = 16;  // tokens per block

enum { kChannel = 0, kGlr = 1, kScalar = 2, kState = 3 };  // gated delta with a decay per channel / HGRN2 / with one decay / state space

__host__ __device__ constexpr int block_floats(int D, bool correct) {  // Z | Q | P | b | T | A'
    return (correct ? 3 : 2) * C * D + D + (correct ? 2 : 1) * C * C;
}

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }

template <int N> struct Vec { float v[N]; };
template <int N> __device__ __forceinline__ Vec<N> ldv(const float* p) {
    Vec<N> r;
    if constexpr (N == 4) {
        const float4 f = *reinterpret_cast<const float4*>(p);
        r.v[0] = f.x, r.v[1] = f.y, r.v[2] = f.z, r.v[3] = f.w;
    } else {
        const float2 f = *reinterpret_cast<const float2*>(p);
        r.v[0] = f.x, r.v[1] = f.y;
    }
    return r;
}
template <int N> __device__ __forceinline__ void stv(float* p, const Vec<N>& r) {
    if constexpr (N == 4)
        *reinterpret_cast<float4*>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
    else
        *reinterpret_cast<float2*>(p) = make_float2(r.v[0], r.v[1]);
}
template <int N> __device__ __forceinline__ float dot(const Vec<N>& a, const Vec<N>& b) {
    float s = a.v[0] * b.v[0];
#pragma unroll
    for (int i = 1; i < N; ++i) s = fmaf(a.v[i], b.v[i], s);
    return s;
}

// 32 values per lane -> lane i holds the sum of value i over the lanes (31 shuffles)
__device__ __forceinline__ float reduce32(float (&v)[32], int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const bool up = lane & o;
            const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    return v[0];
}

template <int I> struct Const {
    static constexpr int value = I;
    __host__ __device__ constexpr operator int() const { return I; }
};
// f(0), f(1), .. f(N - 1) with constants: what indexes registers has to be known at compile time
template <typename F, int... I> __device__ __forceinline__ void each_(F&& f, std::integer_sequence<int, I...>) {
    (f(Const<I>{}), ...);
}
template <int N, typename F> __device__ __forceinline__ void each(F&& f) { each_(f, std::make_integer_sequence<int, N>{}); }

__device__ __forceinline__ float softplusf_(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }
struct PrepArgs {
    const float *q, *k, *dec, *mix;  // k, mix: not with kGlr (dec = f there); mix: not with kState
    long long q_ld, k_ld, dec_ld, mix_ld;
    const float *bias, *rate_log;    // of the decay; kGlr: bias = the lower bound (or NULL), no rate
    float unit_eps;
    float* ws;                       // [blocks of this pass, H]
    const int *blocks, *cu;          // (request, block of it) of every block of the pass
    int H, G, src;
};

// Four CTAs per SM: HGRN2's form for D = 128 spills some 300 bytes a thread for it, and takes 6 us more of 332 with three and no spill.
template <int D, int SRC>
__global__ void __launch_bounds__(128, 4)
chunk_prep_kernel(const PrepArgs p) {
    constexpr int N = D / 32;
    constexpr bool CORRECT = SRC == kChannel || SRC == kScalar;
    __shared__ float flat_[4][CORRECT ? 256 : 160], sT_[4][CORRECT ? C * C : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y * 4 + warp, b = p.blocks[2 * blockIdx.x], c = p.blocks[2 * blockIdx.x + 1];
    if (h >= p.H) return;  // no barrier of the block below
    const int row_b = p.cu[b], left = p.cu[b + 1] - row_b - c * C, cnt = left < C ? left : C;
    const long long row0 = row_b + c * C;
    float* flat = flat_[warp];
    float* out = p.ws + ((long long)blockIdx.x * p.H + h) * block_floats(D, CORRECT);
    float* oZ = out;
    float* oQ = out + (CORRECT ? C * D : 0);
    float* oP = oQ + C * D;
    float* oB = oP + C * D;
    float* oT = oB + D;
    float* oA = oT + (CORRECT ? C * C : 0);
    const int d0 = lane * N, g = SRC == kGlr ? h : h / (p.H / p.G);
    const float* qp = p.q + row0 * p.q_ld + (long long)g * D + d0;
    const float* kp = SRC == kGlr ? nullptr : p.k + row0 * p.k_ld + (long long)g * D + d0;
    const bool wide = SRC == kChannel || SRC == kGlr;  // a decay per channel
    const float* dp = p.dec + row0 * p.dec_ld + (wide ? (long long)h * D + d0 : h);
    const float rate = SRC == kGlr ? 0.f : expf(p.rate_log[h]);
    Vec<N> low, cum;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        cum.v[i] = 1.f;
        low.v[i] = wide && p.bias ? p.bias[h * D + d0 + i] : 0.f;
    }
    // numbers of a token: lane t keeps those of token t
    float beta = 0.f, decay = 1.f, step = 0.f, rq = 0.f, rk = 0.f;
    if (!wide || CORRECT) {
        const int t = lane & 15;
        if (t < cnt) {
            if (CORRECT) beta = sigmoidf_(p.mix[(row0 + t) * p.mix_ld + h]);
            if (!wide) {
                step = softplusf_(dp[t * p.dec_ld] + p.bias[h]);
                decay = expf(-rate * step);
            }
        }
    }
    float v[32];
    if (CORRECT) {  // squared norms of q (lanes 0 .. 15) and k (16 .. 31)
        each<C>([&](auto T) {
            constexpr int t = T;
            v[t] = v[t + 16] = 0.f;
            if (t < cnt) {
                const Vec<N> q = ldv<N>(qp + t * p.q_ld), k = ldv<N>(kp + t * p.k_ld);
                v[t] = dot(q, q);
                v[t + 16] = dot(k, k);
            }
        });
        const float n2 = 1.0f / sqrtf(reduce32(v, lane) + p.unit_eps);
        rq = n2 / sqrtf((float)D);
        rk = __shfl_down_sync(0xffffffffu, n2, 16);  // of lanes 0 .. 15
    }
    Vec<N> w[C];
    constexpr int G = 2;  // tokens whose rows are requested together
    each<C / G>([&](auto T0) {
        constexpr int t0 = T0 * G;
        Vec<N> q[G], d[G], pp[G], z[G];
        each<G>([&](auto I) {
            constexpr int i = I, t = t0 + i;
            if (t < cnt) {
                q[i] = ldv<N>(qp + t * p.q_ld);
                if (SRC != kGlr) pp[i] = ldv<N>(kp + t * p.k_ld);
                if (wide) d[i] = ldv<N>(dp + t * p.dec_ld);
            }
        });
        each<G>([&](auto I) {
            constexpr int i = I, t = t0 + i;
            float fb = 0.f, fd = 1.f, fs = 0.f, fq = 1.f, fk = 1.f;
            if (CORRECT) {
                fb = __shfl_sync(0xffffffffu, beta, t);
                fq = __shfl_sync(0xffffffffu, rq, t);
                fk = __shfl_sync(0xffffffffu, rk, t);
            }
            if (!wide) fd = __shfl_sync(0xffffffffu, decay, t);
            if (SRC == kState) fs = __shfl_sync(0xffffffffu, step, t);
#pragma unroll
            for (int e = 0; e < N; ++e) {
                if (t >= cnt) {  // nothing read, nothing written, nothing lost
                    q[i].v[e] = pp[i].v[e] = z[i].v[e] = 0.f;
                    d[i].v[e] = 1.f;
                } else if (SRC == kGlr) {
                    const float x = q[i].v[e];
                    q[i].v[e] = x * sigmoidf_(x);
                    d[i].v[e] = low.v[e] + (1.0f - low.v[e]) * sigmoidf_(d[i].v[e]);
                    pp[i].v[e] = 1.0f - d[i].v[e];
                } else if (SRC == kState) {
                    d[i].v[e] = fd;
                    pp[i].v[e] *= fs;
                } else {
                    if (wide) d[i].v[e] = expf(-rate * softplusf_(d[i].v[e] + low.v[e]));
                    else d[i].v[e] = fd;
                    const float kh = pp[i].v[e] * fk;
                    q[i].v[e] *= fq;
                    z[i].v[e] = kh * d[i].v[e];
                    pp[i].v[e] = fb * kh;
                }
            }
            auto put = [&](auto IDX, float x) {
                constexpr int idx = decltype(IDX)::value;
                v[idx & 31] = x;
                if constexpr ((idx & 31) == 31) flat[idx - 31 + lane] = reduce32(v, lane);
            };
            if constexpr (CORRECT) {
                Vec<N> zb;
#pragma unroll
                for (int e = 0; e < N; ++e) zb.v[e] = z[i].v[e] * cum.v[e];
                stv<N>(oZ + t * D + d0, zb);
                each<t>([&](auto S) { put(Const<t * t + S>{}, dot(z[i], w[S])); });  // L[t, s]
            }
            each<t>([&](auto S) {
#pragma unroll
                for (int e = 0; e < N; ++e) w[S].v[e] *= d[i].v[e];
            });
            w[t] = pp[i];
            each<t + 1>([&](auto S) {  // A[t, s]
                put(Const<(CORRECT ? t * t + t + S : t * (t + 1) / 2 + S)>{}, dot(q[i], w[S]));
            });
            Vec<N> qb;
#pragma unroll
            for (int e = 0; e < N; ++e) {
                cum.v[e] *= d[i].v[e];
                qb.v[e] = q[i].v[e] * cum.v[e];
            }
            stv<N>(oQ + t * D + d0, qb);
        });
    });
    each<C>([&](auto S) { stv<N>(oP + S * D + d0, w[S]); });
    stv<N>(oB + d0, cum);
    if constexpr (!CORRECT) {
        flat[128 + lane] = reduce32(v, lane);  // entries 128 .. 135, and left-overs behind them
        __syncwarp();
#pragma unroll
        for (int i = 0; i < C * C; i += 32) {
            const int t = (i + lane) >> 4, s = (i + lane) & 15;
            oA[i + lane] = s <= t ? flat[t * (t + 1) / 2 + s] : 0.f;
        }
    } else {
        __syncwarp();
        // ---- T = (1 + L)^-1 and A' = A T, a column per lane (both halves of the warp do the same)
        float* sT = sT_[warp];
        {
            const int j = lane & 15;
            float col[C];
            each<C>([&](auto I) {
                constexpr int i = I;
                float a = 0.f;
                each<i>([&](auto K) { a = fmaf(flat[i * i + K], col[K], a); });
                col[i] = i == j ? 1.f : (i > j ? -a : 0.f);
            });
            each<C>([&](auto I) {
                constexpr int i = I;
                float a = 0.f;
                each<i + 1>([&](auto K) { a = fmaf(flat[i * i + i + K], col[K], a); });
                if (lane < 16) {
                    sT[i * C + j] = col[i];
                    oT[i * C + j] = col[i];
                    oA[i * C + j] = a;
                }
            });
        }
        __syncwarp();
        // ---- Z = T Z' (from the last token back, so that the rows it reads are still Z'), Q = Q' - A Z; rows of this thread's own
        each<C>([&](auto T) { w[T] = ldv<N>(oZ + T * D + d0); });
        each<C>([&](auto R) {
            constexpr int t = C - 1 - R;
            each<t>([&](auto S) {
                const float f = sT[t * C + S];
#pragma unroll
                for (int e = 0; e < N; ++e) w[t].v[e] = fmaf(f, w[S].v[e], w[t].v[e]);
            });
        });
        each<C>([&](auto T) {
            constexpr int t = T;
            stv<N>(oZ + t * D + d0, w[t]);
            Vec<N> qb = ldv<N>(oQ + t * D + d0);
            each<t + 1>([&](auto S) {
                const float f = flat[t * t + t + S];
#pragma unroll
                for (int e = 0; e < N; ++e) qb.v[e] = fmaf(-f, w[S].v[e], qb.v[e]);
            });
            stv<N>(oQ + t * D + d0, qb);
        });
    }
}

// ------------------------------------------------------------------------------------------------ the walk
// x = hi + lo + (what neither holds, < 2^-21 |x|): hi rounded to TF32 on its bits, so that the rest has either sign; the tensor cores cut
// lo to TF32 themselves. With hi cut as well every part errs the same way and the products with it: outputs 4.5e-7 off against 1.1e-7,
// where FMAs token by token are 0.7 to 1.6e-7 off (2048 tokens, heads of 128).
__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// The sum of the leading products and that of the small ones. The adders cut, so that a chain of one or two products comes out 2^-25 too
// small on average, and every state with it (3.3e-8 for HGRN2, 6e-8 for the delta rule): that much is added.
__device__ __forceinline__ float whole(float lead, float small) { return lead + fmaf(lead, 0x1p-25f, small); }
struct FragA {
    uint32_t hi[4], lo[4];
    __device__ __forceinline__ void set(float x0, float x1, float x2, float x3) {
        split(x0, hi[0], lo[0]);
        split(x1, hi[1], lo[1]);
        split(x2, hi[2], lo[2]);
        split(x3, hi[3], lo[3]);
    }
};
struct FragB {
    uint32_t hi[2], lo[2];
    __device__ __forceinline__ void set(float x0, float x1) {
        split(x0, hi[0], lo[0]);
        split(x1, hi[1], lo[1]);
    }
};
__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}

struct ScanArgs {
    PrepArgs prep;     // for the blocks that the products cannot take
    const float* ws;
    const float* v;    // value of token row r, head h, channel e at v[r * v_ld + h * E + e]
    long long v_ld;
    float *state, *o;  // [slots, H, D, E], [n_tok, H * E]
    const int *requests, *cu, *slot;  // (request, its first block in ws, how many, the first one's place in the request) of the pass
    int H, E;
};

// shared memory of a stage, in floats: Z [16][D + 8] | Q [16][D + 8] | P [16][PP] | b [D] | T [16][20] | A' [16][20] | V [16][cols + 8]
template <int D, bool CORRECT> struct Layout {
    static constexpr int DS = D + 8, PP = CORRECT ? D + 4 : D + 8, TS = C + 4;  // pitches without bank conflicts for their reads
    static constexpr int Q = CORRECT ? C * DS : 0, P = Q + C * DS, B = P + C * PP, T = B + D, A = T + (CORRECT ? C * TS : 0), V = A + C * TS;
    __host__ __device__ static constexpr int stage(int cols) { return V + C * (cols + 8); }
};

// A block with an infinity or a NaN in it, or in the state: its tokens one after another, by FMAs, so that nothing reaches the tokens in
// front of it (0 times infinity above the diagonal would) and infinities stay what they are (their low part is NaN). Two warps, half of
// the rows of 16 columns each, as in the walk below: S are this thread's entries of the state, laid out as there, V the block's values from
// this column group on, xu the group's exchange buffer (128 floats a warp). Inlined:
// with a call in it the walk was given 128 registers and took 342 us instead of 301 (HGRN2, 4 requests of 333 to 2048 tokens).
struct Outputs { float mine[4], give[4]; };  // of the walk: four outputs of this warp's tokens, four of the other's
template <int D, bool CORRECT>
__device__ __forceinline__ Outputs block_by_tokens(const PrepArgs& p, int h, long long row0, int cnt, int half, const float* V, int VS,
                                                   float* xu, int barrier, float (&S)[D / 16][4]) {
    constexpr int NT = D / 16;
    Outputs out = {};
    const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3, hd = half * (D / 2);
    const bool wide = p.src == kChannel || p.src == kGlr;
    const int kh = p.src == kGlr ? h : h / (p.H / p.G);
    const float rate = p.src == kGlr ? 0.f : expf(p.rate_log[h]);
#pragma unroll 1
    for (int t = 0; t < cnt; ++t) {
        const float* q = p.q + (row0 + t) * p.q_ld + (long long)kh * D;
        const float* k = p.src == kGlr ? nullptr : p.k + (row0 + t) * p.k_ld + (long long)kh * D;
        const float* dec = p.dec + (row0 + t) * p.dec_ld + (wide ? (long long)h * D : h);
        float fq = 1.f, fk = 1.f, beta = 1.f, decay = 1.f, step = 0.f;
        if (CORRECT) {
            float sq = 0.f, sk = 0.f;
#pragma unroll 1
            for (int d = lane; d < D; d += 32) {
                sq = fmaf(q[d], q[d], sq);
                sk = fmaf(k[d], k[d], sk);
            }
            fq = 1.0f / sqrtf(warp_sum(sq) + p.unit_eps) / sqrtf((float)D);
            fk = 1.0f / sqrtf(warp_sum(sk) + p.unit_eps);
            beta = sigmoidf_(p.mix[(row0 + t) * p.mix_ld + h]);
        }
        if (!wide) {
            step = softplusf_(dec[0] + p.bias[h]);
            decay = expf(-rate * step);
        }
        float z[2 * NT], pp[2 * NT], dd[2 * NT], qq[2 * NT];  // of rows hd + 8 nt + 2 t4, + 1
#pragma unroll 1
        for (int i = 0; i < 2 * NT; ++i) {
            const int d = hd + 8 * (i >> 1) + 2 * t4 + (i & 1);
            dd[i] = decay;
            z[i] = 0.f;
            if (p.src == kGlr) {
                const float low = p.bias ? p.bias[h * D + d] : 0.f;
                qq[i] = q[d] * sigmoidf_(q[d]);
                dd[i] = low + (1.0f - low) * sigmoidf_(dec[d]);
                pp[i] = 1.0f - dd[i];
            } else if (p.src == kState) {
                qq[i] = q[d];
                pp[i] = k[d] * step;
            } else {
                if (wide) dd[i] = expf(-rate * softplusf_(dec[d] + p.bias[h * D + d]));
                qq[i] = q[d] * fq;
                z[i] = k[d] * fk * dd[i];
                pp[i] = beta * (k[d] * fk);
            }
        }
        float u[2] = {V[t * VS + g], V[t * VS + g + 8]}, o[2] = {0.f, 0.f};
        if (CORRECT) {
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                float a = 0.f;
#pragma unroll 1
                for (int i = 0; i < 2 * NT; ++i) a = fmaf(S[i >> 1][(i & 1) + 2 * c], z[i], a);
                a += __shfl_xor_sync(0xffffffffu, a, 1);
                a += __shfl_xor_sync(0xffffffffu, a, 2);
                if (t4 == 0) xu[half * 128 + g + 8 * c] = a;
            }
            asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
            for (int c = 0; c < 2; ++c) u[c] -= xu[g + 8 * c] + xu[128 + g + 8 * c];
            asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");  // both have read them
        }
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
#pragma unroll 1
            for (int i = 0; i < 2 * NT; ++i) {
                float& s = S[i >> 1][(i & 1) + 2 * c];
                s = fmaf(dd[i], s, pp[i] * u[c]);
                o[c] = fmaf(s, qq[i], o[c]);
            }
            o[c] += __shfl_xor_sync(0xffffffffu, o[c], 1);
            o[c] += __shfl_xor_sync(0xffffffffu, o[c], 2);
#pragma unroll
            for (int e = 0; e < 4; ++e)  // constant indexes: registers
                if (t4 == (t & 7) >> 1 && e == (t & 1) + 2 * c) (t >> 3 == half ? out.mine[e] : out.give[e]) = o[c];
        }
    }
    return out;
}

// Columns of S per CTA: 32 or 64, four threads each. PER_SM: CTAs that the registers have to leave room for. Without the correction two of
// 64 columns fit with 128 registers a thread (16 requests of 512 tokens, 32 heads: HGRN2 740 us, 859 with 174 registers and one CTA); with
// it they would spill. With it three of 32 columns fit with 168 registers, and are ahead once there are more than two for every SM (3
// requests of 2048 tokens, 32 heads 961 -> 786 us; 3 of 1500 to 1777, 16 heads 409 -> 425).
template <int D, bool CORRECT, int COLS, int PER_SM>
__global__ void __launch_bounds__(COLS * 4, PER_SM)
chunk_scan_kernel(const __grid_constant__ ScanArgs p) {
    constexpr int NT = D / 16;  // groups of eight rows of S that a warp keeps: half of them
    typedef Layout<D, CORRECT> Y;
    constexpr int M = CORRECT ? 2 : 1;  // Q alone, or Q and Z
    extern __shared__ __align__(16) float sm[];
    constexpr int cols = COLS, VS = cols + 8, stage_floats = Y::stage(cols);
    const int* rq = p.requests + 4 * blockIdx.z;
    const int h = blockIdx.y, b = rq[0], nblk = rq[2], c0 = rq[3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int half = warp & 1, e0 = blockIdx.x * cols, wc = (warp >> 1) * 16;
    const int row_b = p.cu[b], n = p.cu[b + 1] - row_b;
    const int hd = half * (D / 2);
    // partial results that the two warps of a column group hand each other: [2][warps][32] float4 of outputs, [warps][2][32] of U
    float4* xo = reinterpret_cast<float4*>(sm + 2 * stage_floats);
    float4* xu = xo + 2 * blockDim.x;
    float* st = p.state + ((long long)p.slot[b] * p.H + h) * (long long)D * p.E + (long long)hd * p.E + e0 + wc;
    const float* wsb = p.ws + ((long long)rq[1] * p.H + h) * block_floats(D, CORRECT);
    const long long ws_step = (long long)p.H * block_floats(D, CORRECT);
    float S[NT][4];  // rows g, g + 8 (columns of S) x entries d = hd + 8 nt + 2 t4, + 1
    auto each_entry = [&](auto&& f) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int c = 0; c < 4; ++c) f(S[nt][c], st + (long long)(8 * nt + 2 * t4 + (c & 1)) * p.E + g + (c >> 1) * 8);
    };
    auto fetch = [&](int k, float* dst) {
        const float* s = wsb + k * ws_step;
        auto rows = [&](float* to, int pitch) {  // 16 rows of D
            for (int i = threadIdx.x; i < C * (D / 4); i += blockDim.x)
                copy16(to + (i / (D / 4)) * pitch + (i % (D / 4)) * 4, s + i * 4, true);
            s += C * D;
        };
        auto square = [&](float* to) {
            for (int i = threadIdx.x; i < C * C / 4; i += blockDim.x) copy16(to + (i >> 2) * Y::TS + (i & 3) * 4, s + i * 4, true);
            s += C * C;
        };
        if (CORRECT) rows(dst, Y::DS);
        rows(dst + Y::Q, Y::DS);
        rows(dst + Y::P, Y::PP);
        for (int i = threadIdx.x; i < D / 4; i += blockDim.x) copy16(dst + Y::B + i * 4, s + i * 4, true);
        s += D;
        if (CORRECT) square(dst + Y::T);
        square(dst + Y::A);
        const int r0 = (c0 + k) * C, q = cols / 4;
        for (int i = threadIdx.x; i < C * q; i += blockDim.x) {
            const int t = i / q, e = (i % q) * 4;
            const bool live = r0 + t < n;
            copy16(dst + Y::V + t * VS + e, p.v + (live ? (long long)(row_b + r0 + t) * p.v_ld + h * p.E + e0 + e : 0), live);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // The outputs of eight tokens: this warp finishes tokens 8 half .. 8 half + 7 of a block, one block later (the other warp's part
    // is then there without a wait of its own). Rows g, g + 8 are channels, columns 2 t4, 2 t4 + 1 tokens.
    float mine[4];
    auto finish = [&](int k) {
        const int r0 = (c0 + k) * C + 8 * half;
        const float4 o4 = xo[(k & 1) * blockDim.x + (warp ^ 1) * 32 + lane];
        const float other[4] = {o4.x, o4.y, o4.z, o4.w};
        float* op = p.o + (long long)(row_b + r0) * p.H * p.E + (long long)h * p.E + e0 + wc + g;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int t = 2 * t4 + (c & 1);
            if (r0 + t < n) op[(long long)t * p.H * p.E + (c >> 1) * 8] = mine[c] + other[c];
        }
    };
    // Whether a block's results were finite is known at the barrier behind it, off the chain that the walk waits for. If they were not, the
    // walk begins again (the state in memory is still that in front of it) and goes token by token from that block on, until every entry of
    // the state is NaN: the products give what follows then (a request whose hidden states are NaN: one block, and not 10 us for every
    // token of it).
    int slow = nblk;
    bool odd = false, lost = false;
again:
    fetch(0, sm);
    each_entry([&](float& s, float* at) { s = *at; });
    for (int k = 0; k < nblk; ++k) {
        const float* x = sm + (k & 1) * stage_floats;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        const bool flag = __syncthreads_or(odd);  // this block is here, and everybody is done with the one before
        if (slow == nblk) {
            if (flag) {
                slow = k - 1;
                odd = false;
                goto again;
            }
        } else if (k > slow && !flag) {
            lost = true;
        }
        if (k + 1 < nblk) fetch(k + 1, sm + ((k + 1) & 1) * stage_floats);
        if (k) finish(k - 1);
        if (k >= slow && !lost) {
            const int r0 = (c0 + k) * C;
            float kept[NT][4];  // indexed at run time, so not S itself
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) kept[nt][c] = S[nt][c];
            const Outputs out = block_by_tokens<D, CORRECT>(p.prep, h, row_b + r0, n - r0 < C ? n - r0 : C, half, x + Y::V + wc, VS,
                                                            reinterpret_cast<float*>(xu + (warp & ~1) * 64), 1 + (warp >> 1), kept);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) S[nt][c] = kept[nt][c];
#pragma unroll
            for (int c = 0; c < 4; ++c) mine[c] = out.mine[c];
            xo[(k & 1) * blockDim.x + warp * 32 + lane] = make_float4(out.give[0], out.give[1], out.give[2], out.give[3]);
            odd = false;
            each_entry([&](float& s, float*) { odd |= s == s; });  // something that is not NaN
            continue;
        }
        // ---- this warp's rows of S^T Q^T (and S^T Z^T)
        constexpr int NC = NT / 2;  // leading products in chains of two, the small ones in a chain of their own
        float hh[M][2][NC][4] = {}, xx[M][2][4] = {};
        auto total = [&](int m, int j, int c) {
            float a = hh[m][j][0][c];
#pragma unroll
            for (int i = 1; i < NC; ++i) a += hh[m][j][i][c];
            return whole(a, xx[m][j][c]);
        };
#pragma unroll
        for (int kk = 0; kk < NT; ++kk) {
            FragA a;
            a.set(S[kk][0], S[kk][2], S[kk][1], S[kk][3]);  // slot t4 <-> entry 2 t4, slot t4 + 4 <-> entry 2 t4 + 1
            FragB f[M][2];
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 y = *reinterpret_cast<const float2*>(x + (m == 0 ? Y::Q : 0) + (8 * j + g) * Y::DS + hd + 8 * kk + 2 * t4);
                    f[m][j].set(y.x, y.y);
                }
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int j = 0; j < 2; ++j) mma_tf32(hh[m][j][kk % NC], a.hi, f[m][j].hi);
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int j = 0; j < 2; ++j) mma_tf32(xx[m][j], a.lo, f[m][j].hi);
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int j = 0; j < 2; ++j) mma_tf32(xx[m][j], a.hi, f[m][j].lo);
        }
        // ---- and, for tokens 8 half .. 8 half + 7, V^T A'^T (and V^T T^T); nothing above the diagonal
        FragA av[2];
        float vv[M][4] = {}, vx[M][4] = {};
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const float* vp = x + Y::V + (8 * ks + t4) * VS + wc + g;
            av[ks].set(vp[0], vp[8], vp[4 * VS], vp[4 * VS + 8]);
            if (ks <= half) {  // the same for the whole warp
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    const float* tp = x + (m == 0 ? Y::A : Y::T) + (8 * half + g) * Y::TS + 8 * ks + t4;
                    FragB f;
                    f.set(tp[0], tp[4]);
                    mma_tf32(vx[m], av[ks].lo, f.hi);
                    mma_tf32(vx[m], av[ks].hi, f.lo);
                    mma_tf32(vv[m], av[ks].hi, f.hi);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) vv[m][c] = whole(vv[m][c], vx[m][c]);
        float part[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) part[j][c] = total(0, j, c);
        float give[4], all[4] = {};  // all: finite only if everything that follows from this block's numbers is
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            mine[c] = (half ? part[1][c] : part[0][c]) + vv[0][c];
            give[c] = half ? part[0][c] : part[1][c];
            all[0] += mine[c];
            all[1] += give[c];
        }
        // ---- S <- b S + P^T U
        FragA au[2];
        float u[2][4];
        if (CORRECT) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    u[j][c] = -total(M - 1, j, c);
                    if (j == half) u[j][c] += vv[M - 1][c];
                    all[2 + j] += u[j][c];
                }
                xu[(warp * 2 + j) * 32 + lane] = make_float4(u[j][0], u[j][1], u[j][2], u[j][3]);
            }
        }
        xo[(k & 1) * blockDim.x + warp * 32 + lane] = make_float4(give[0], give[1], give[2], give[3]);
        odd = slow == nblk && !(fabsf((all[0] + all[1]) + (all[2] + all[3])) < INFINITY);
        if (CORRECT) {
            asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");  // the two warps of these columns
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 y = xu[((warp ^ 1) * 2 + j) * 32 + lane];
                // slot t4 <-> token 2 t4, slot t4 + 4 <-> token 2 t4 + 1; the same sum in both warps
                au[j].set(u[j][0] + y.x, u[j][2] + y.z, u[j][1] + y.y, u[j][3] + y.w);
            }
        }
#pragma unroll
        for (int n0 = 0; n0 < NT; n0 += 4) {
            float acc[2][4][4] = {}, ax[4][4] = {};
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const FragA& a = CORRECT ? au[ks] : av[ks];
                FragB f[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float* pp = x + Y::P + (8 * ks + (CORRECT ? 2 * t4 : t4)) * Y::PP + hd + 8 * (n0 + i) + g;
                    f[i].set(pp[0], pp[(CORRECT ? 1 : 4) * Y::PP]);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_tf32(ax[i], a.lo, f[i].hi);
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_tf32(ax[i], a.hi, f[i].lo);
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_tf32(acc[ks][i], a.hi, f[i].hi);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 bb = *reinterpret_cast<const float2*>(x + Y::B + hd + 8 * (n0 + i) + 2 * t4);
                S[n0 + i][0] = fmaf(S[n0 + i][0], bb.x, whole(acc[0][i][0] + acc[1][i][0], ax[i][0]));
                S[n0 + i][1] = fmaf(S[n0 + i][1], bb.y, whole(acc[0][i][1] + acc[1][i][1], ax[i][1]));
                S[n0 + i][2] = fmaf(S[n0 + i][2], bb.x, whole(acc[0][i][2] + acc[1][i][2], ax[i][2]));
                S[n0 + i][3] = fmaf(S[n0 + i][3], bb.y, whole(acc[0][i][3] + acc[1][i][3], ax[i][3]));
            }
        }
    }
    if (__syncthreads_or(odd) && slow == nblk) {
        slow = nblk - 1;
        odd = false;
        goto again;
    }
    finish(nblk - 1);
    each_entry([&](float& s, float* at) { *at = s; });
}

// ------------------------------------------------------------------------------------------------ the plan
// One CTA: which requests have more than `done` blocks, where their blocks of this pass begin (a running sum over the requests), and the
// list of blocks. A few us, once per step.
constexpr int kPlanThreads = 1024;
__global__ void __launch_bounds__(kPlanThreads)
chunk_plan_kernel(const int* __restrict__ cu, int n_seq, int done, int each, int* __restrict__ requests, int* __restrict__ blocks) {
    __shared__ int2 sums[32];  // requests, blocks of a warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int r0 = 0, b0 = 0;
    for (int at = 0; at < n_seq; at += kPlanThreads) {
        const int b = at + threadIdx.x;
        int n = b < n_seq ? (cu[b + 1] - cu[b] + C - 1) / C - done : 0;
        n = n < 0 ? 0 : n > each ? each : n;
        int r = n > 0, f = n;  // up to this request, it included
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, r, o), y = __shfl_up_sync(0xffffffffu, f, o);
            if (lane >= o) r += x, f += y;
        }
        if (lane == 31) sums[warp] = make_int2(r, f);
        __syncthreads();
        for (int w = 0; w < warp; ++w) r += sums[w].x, f += sums[w].y;
        if (n > 0) {
            int* q = requests + 4 * (r0 + r - 1);
            q[0] = b, q[1] = b0 + f - n, q[2] = n, q[3] = done;
            for (int i = 0; i < n; ++i) {
                int* e = blocks + 2 * (b0 + f - n + i);
                e[0] = b, e[1] = done + i;
            }
        }
        for (int w = 0; w < kPlanThreads / 32; ++w) r0 += sums[w].x, b0 += sums[w].y;
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------ host
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int D, int SRC>
static int run(PrepArgs a, ScanArgs s, int n_blocks, int n_requests, cudaStream_t st) {
    constexpr bool CORRECT = SRC == kChannel || SRC == kScalar;
    // columns of S per CTA: few heads and requests are spread over the SMs, many share the blocks' operands
    const long long heads = (long long)n_requests * a.H;
    int cols = 32;
    while (cols < 64 && s.E % (2 * cols) == 0 && heads * (s.E / cols) > 148 * 4) cols *= 2;
    auto bytes = [](int c) { return (2 * Layout<D, CORRECT>::stage(c) + 4 * (c * 4) * 4) * (int)sizeof(float); };
    auto scan = cols == 32 ? chunk_scan_kernel<D, CORRECT, 32, 1> : chunk_scan_kernel<D, CORRECT, 64, CORRECT ? 1 : 2>;
    if constexpr (CORRECT)
        if (cols == 32 && heads * (s.E / cols) > 148 * 2) scan = chunk_scan_kernel<D, CORRECT, 32, 3>;
    cudaError_t e = cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes(cols));  // of this kernel always the same
    if (e == cudaSuccess) {
        chunk_prep_kernel<D, SRC><<<dim3(n_blocks, (a.H + 3) / 4), 128, 0, st>>>(a);
        scan<<<dim3(s.E / cols, a.H, n_requests), cols * 4, bytes(cols), st>>>(s);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

}  // namespace chunk
}  // namespace llark

using namespace llark;

extern "C" long long llark_seq_chunk_block_bytes(int D, int correct) { return 4LL * chunk::block_floats(D, correct != 0); }

extern "C" int llark_seq_chunk_plan(const int* cu, int n_seq, int done, int each, int* requests, int* blocks, cudaStream_t st) {
    if (!cu || n_seq <= 0 || done < 0 || each <= 0 || !requests || !blocks) return LLARK_EINVAL;
    chunk::chunk_plan_kernel<<<1, chunk::kPlanThreads, 0, st>>>(cu, n_seq, done, each, requests, blocks);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return LLARK_ECUDA;
    }
    return LLARK_OK;
}

static bool bad_sizes(int n_blocks, int n_requests, int H, int D, int E) {
    return n_blocks <= 0 || n_requests <= 0 || n_requests > 65535 || H <= 0 || H > 65535 || (D != 64 && D != 128) || E <= 0 || E % 32;
}

extern "C" int llark_seq_glr_chunks(const float* src, long long ld, int q_off, int f_off, int v_off, const float* lower, float* state,
                                    float* o, float* ws, const int* blocks, int n_blocks, const int* requests, int n_requests,
                                    const int* cu, const int* slot, int H, int D, int E, cudaStream_t st) {
    if (bad_sizes(n_blocks, n_requests, H, D, E) || !src || !state || !o || !ws || !blocks || !requests || !cu || !slot || ld % 4 ||
        q_off % 4 || f_off % 4 || v_off % 4 || !chunk::aligned16(src) || !chunk::aligned16(ws))
        return LLARK_EINVAL;
    const chunk::PrepArgs a = {src + q_off, nullptr, src + f_off, nullptr, ld,  0,  ld, 0, lower,
                               nullptr,     0.f,     ws,          blocks,  cu, H, H,  chunk::kGlr};
    const chunk::ScanArgs s = {a, ws, src + v_off, ld, state, o, requests, cu, slot, H, E};
    return D == 64 ? chunk::run<64, chunk::kGlr>(a, s, n_blocks, n_requests, st)
                   : chunk::run<128, chunk::kGlr>(a, s, n_blocks, n_requests, st);
}

extern "C" int llark_seq_delta_chunks(int rule, const float* q, long long q_ld, const float* k, long long k_ld, const float* dec,
                                      long long dec_ld, const float* dec_bias, const float* rate_log, const float* mix,
                                      long long mix_ld, float unit_eps, const float* v, long long v_ld, float* state, float* o,
                                      float* ws, const int* blocks, int n_blocks, const int* requests, int n_requests, const int* cu,
                                      const int* slot, int H, int G, int D, int E, cudaStream_t st) {
    if (bad_sizes(n_blocks, n_requests, H, D, E) || (rule != 0 && rule != 2 && rule != 3) || G <= 0 || H % G || !q || !k || !dec ||
        !dec_bias || !rate_log || (!mix && rule != 3) || !v || !state || !o || !ws || !blocks || !requests || !cu || !slot || q_ld % 4 ||
        k_ld % 4 || v_ld % 4 || !chunk::aligned16(q) || !chunk::aligned16(k) || !chunk::aligned16(v) || !chunk::aligned16(ws) ||
        (rule == 0 && (dec_ld % 4 || !chunk::aligned16(dec))))
        return LLARK_EINVAL;
    const int kind = rule == 0 ? chunk::kChannel : rule == 2 ? chunk::kScalar : chunk::kState;
    const chunk::PrepArgs a = {q,        k,        dec, mix,    q_ld, k_ld, dec_ld, mix_ld, dec_bias,
                               rate_log, unit_eps, ws,  blocks, cu,   H,    G,      kind};
    const chunk::ScanArgs s = {a, ws, v, v_ld, state, o, requests, cu, slot, H, E};
#define LLARK_CHUNKS(SRC_) \
    (D == 64 ? chunk::run<64, SRC_>(a, s, n_blocks, n_requests, st) : chunk::run<128, SRC_>(a, s, n_blocks, n_requests, st))
    return rule == 0 ? LLARK_CHUNKS(chunk::kChannel) : rule == 2 ? LLARK_CHUNKS(chunk::kScalar) : LLARK_CHUNKS(chunk::kState);
#undef LLARK_CHUNKS
}
