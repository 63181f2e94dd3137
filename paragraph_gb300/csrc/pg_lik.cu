// pg_lik.cu -- log-likelihood of a growth trace under theta = (alpha, tau, gamma, beta), and its
// adjoint, batched over up to 64 parameter points per launch.  No counterpart in the reference:
// this is the density of the sampling law the growth step draws from
// (w_j beta^[j in N_a], successive sampling without replacement).
//
// Weights: w_j = 2^(x2_j), x2_j = log2(e) (gamma log f_j + alpha log(indeg_j+1) - (t-t_j)/tau), the
// exponent carried as an unevaluated fp32 pair h + l: the per-point constants are split into fp32
// high and low parts and log(indeg+1) is stored as a high/low pair.  A feature or constant rounded
// once to fp32 is a fixed error of every node that shares it -- it does not average out over the
// trace and moves the gradient by the Hessian times a 2^-24 shift of the data or of theta, which
// shows where the gradient nearly vanishes (the generating point of a trace).  Two arithmetic
// modes:
//   default     h by one FMA chain (its roundings are dropped), log f in fp32, 2^h from the
//               special-function unit (PTX ex2.approx.ftz.f32, relative error < 2^-22; results
//               below 2^-126 flush to zero) scaled by 1 + l ln 2, ball sums pairwise over four
//               weights: ~1e-5 of the gradient's norm at the generating point of a 200k-node trace,
//               1e-7 elsewhere;
//   exact_exp2  every product and sum of the exponent keeps its rounding error, log f is an FP64 log
//               carried as high part plus packed remainder, 2^(h + l) from exp2_exact (fp32
//               arithmetic, about 2 ulp), and every ball weight and product is summed on its own
//               (BallSum): ~3e-7 of the gradient's norm there, at about half of the throughput.
// The same weight function feeds every sum below, so the normalisers and the citations' prefix
// sums agree: an error that is a smooth function of the weight (such as the unit's) largely
// cancels between them.  The per-epoch sums over all nodes are shared by every agent of the epoch, so they are
// accumulated in FP64 (an fp32 partial's rounding would be common to all of the epoch's
// citations); the per-agent ball sums use compensated fp32.
//
// Per launch (forward or adjoint):
//   k_lik_global      per epoch: sum_{j<n_e} w_j (forward) or sum_j w_j g_j (adjoint), one CTA per
//                     1024-node chunk, to 64-bit accuracy (32 terms in fp32 with the roundings kept, then
//                     FP64, in a fixed order, so results are reproducible).  It also writes the epochs' weight
//                     table (LikBatch::wt) when the agent pass gathers from one.
//   k_lik_global_sum  chunks -> one FP64 value per (epoch, point).
//   k_lik_ball        (once per trace, or per chunk of agents and pass) the agent's 2-hop ball as
//                     a bitmap over [0, n_e) in shared memory, compacted to ascending ids.
//   k_lik_table1/2    one warp per agent: every point sums its ball weights S_a (adjoint: also
//                     sum w g), reading each ball element once for all points, its weights from the
//                     table.  A weight depends on the epoch, the node and the point, not on the agent,
//                     and a node is in many balls: 2.35M table rows for 405M ball elements of a
//                     200k-node trace.  Then the citations are walked in draw order with running
//                     sums: D_i = Z_a - sum_{l<i} W_{c_l}, log-likelihood sum x_i - log D_i, and in
//                     the adjoint g_i - (dZ_a - dP_i) / D_i.  The adjoint rebuilds the table and
//                     reads only the forward's per-agent Z_a.
//   k_lik_eval        the same with every weight evaluated where it is summed, for traces with few ball
//                     elements for their table rows (the line depends on the points: run_lik), and where
//                     a table has no room.
//   k_lik_sum         agents -> totals per point (fixed order).
#include "pg_lik.cuh"
#include "pg_sums.cuh"

#include <cuda_fp16.h>

namespace pg {

namespace {

constexpr double kLn2d = 0x1.62e42fefa39efp-1;
constexpr float kLn2f = 0x1.62e430p-1f;

struct Kahan {
    float s = 0.f, c = 0.f;
};

// Compensated summation (Kahan 1965); the build has no FMA contraction and no reassociation.
__device__ __forceinline__ void kadd(Kahan& k, float v) {
    const float y = v - k.c;
    const float t = k.s + y;
    k.c = (t - k.s) - y;
    k.s = t;
}
__device__ __forceinline__ double kval(const Kahan& k) { return (double)k.s - (double)k.c; }

// A ball's sums for one point: S = sum w (and, in the adjoint, sum w g for the three continuous
// features).  Default: four weights summed pairwise, products in FMA chains, then compensated fp32.
// EXACT: every weight and every rounded product enters the compensated sums on its own and the
// products' rounding errors (FMA residuals) are summed beside them, so a ball sum keeps no
// rounding of its own above the compensated sum's (these per-agent errors otherwise reach ~3e-6
// of the gradient where it nearly vanishes).
template <bool ADJ, bool EXACT>
struct BallSum {
    Kahan s, t0, t1, t2;
    float r0 = 0.f, r1 = 0.f, r2 = 0.f;
    __device__ __forceinline__ void add1(const float w, const float4 f) {
        kadd(s, w);
        if (ADJ) {
            const float p0 = w * f.y, p1 = w * f.z, p2 = w * f.x;
            kadd(t0, p0);
            kadd(t1, p1);
            kadd(t2, p2);
            if (EXACT) {
                r0 += __fmaf_rn(w, f.y, -p0);
                r1 += __fmaf_rn(w, f.z, -p1);
                r2 += __fmaf_rn(w, f.x, -p2);
            }
        }
    }
    __device__ __forceinline__ void add4(const float w0, const float w1, const float w2, const float w3,
                                         const float4 f0, const float4 f1, const float4 f2, const float4 f3) {
        if (EXACT) {
            add1(w0, f0);
            add1(w1, f1);
            add1(w2, f2);
            add1(w3, f3);
            return;
        }
        kadd(s, (w0 + w1) + (w2 + w3));
        if (ADJ) {
            kadd(t0, __fmaf_rn(w3, f3.y, __fmaf_rn(w2, f2.y, __fmaf_rn(w1, f1.y, w0 * f0.y))));
            kadd(t1, __fmaf_rn(w3, f3.z, __fmaf_rn(w2, f2.z, __fmaf_rn(w1, f1.z, w0 * f0.z))));
            kadd(t2, __fmaf_rn(w3, f3.x, __fmaf_rn(w2, f2.x, __fmaf_rn(w1, f1.x, w0 * f0.x))));
        }
    }
    __device__ __forceinline__ double S() const { return kval(s); }
    __device__ __forceinline__ double T0() const { return kval(t0) + (double)r0; }
    __device__ __forceinline__ double T1() const { return kval(t1) + (double)r1; }
    __device__ __forceinline__ double T2() const { return kval(t2) + (double)r2; }
};

// Two points per lane as a packed pair of fp32 (PTX .f32x2, sm_100 and later: two IEEE operations
// per instruction, each rounded as its scalar form, so the sums are the scalar ones bit for bit).
using F2 = unsigned long long;
__device__ __forceinline__ F2 f2_of(float x, float y) {
    return ((unsigned long long)__float_as_uint(y) << 32) | __float_as_uint(x);
}
__device__ __forceinline__ float f2_get(F2 a, int p) { return __uint_as_float((uint32_t)(p ? a >> 32 : a)); }
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) {  // a - b = a + (-1) b, exact before the one rounding
    return f2_fma(b, 0xBF800000BF800000ull, a);
}

// BallSum of two points at once.  A feature row comes as (y, y), (z, z) and (x, x) pairs.
struct Feat2 {
    F2 y, z, x;
};
template <bool ADJ, bool EXACT>
struct BallSum2 {
    F2 s = 0, sc = 0, t[3] = {0, 0, 0}, tc[3] = {0, 0, 0}, r[3] = {0, 0, 0};
    static __device__ __forceinline__ void kadd2(F2& s, F2& c, F2 v) {
        const F2 y = f2_sub(v, c);
        const F2 n = f2_add(s, y);
        c = f2_sub(f2_sub(n, s), y);
        s = n;
    }
    __device__ __forceinline__ void add1(const F2 w, const Feat2 f) {
        kadd2(s, sc, w);
        if (ADJ) {
            const F2 g[3] = {f.y, f.z, f.x};
            const F2 nw = EXACT ? f2_mul(w, 0xBF800000BF800000ull) : 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const F2 p = f2_mul(w, g[k]);
                kadd2(t[k], tc[k], p);
                if (EXACT) r[k] = f2_sub(r[k], f2_fma(nw, g[k], p));  // r + (w g - p)
            }
        }
    }
    __device__ __forceinline__ void add4(const F2* w, const Feat2* f) {
        if (EXACT) {
#pragma unroll
            for (int u = 0; u < 4; ++u) add1(w[u], f[u]);
            return;
        }
        kadd2(s, sc, f2_add(f2_add(w[0], w[1]), f2_add(w[2], w[3])));
        if (ADJ) {
            kadd2(t[0], tc[0], f2_fma(w[3], f[3].y, f2_fma(w[2], f[2].y, f2_fma(w[1], f[1].y, f2_mul(w[0], f[0].y)))));
            kadd2(t[1], tc[1], f2_fma(w[3], f[3].z, f2_fma(w[2], f[2].z, f2_fma(w[1], f[1].z, f2_mul(w[0], f[0].z)))));
            kadd2(t[2], tc[2], f2_fma(w[3], f[3].x, f2_fma(w[2], f[2].x, f2_fma(w[1], f[1].x, f2_mul(w[0], f[0].x)))));
        }
    }
    __device__ __forceinline__ BallSum<ADJ, EXACT> point(int p) const {
        BallSum<ADJ, EXACT> o;
        o.s.s = f2_get(s, p), o.s.c = f2_get(sc, p);
        o.t0.s = f2_get(t[0], p), o.t0.c = f2_get(tc[0], p), o.r0 = f2_get(r[0], p);
        o.t1.s = f2_get(t[1], p), o.t1.c = f2_get(tc[1], p), o.r1 = f2_get(r[1], p);
        o.t2.s = f2_get(t[2], p), o.t2.c = f2_get(tc[2], p), o.r2 = f2_get(r[2], p);
        return o;
    }
};

// First position of x's backward row whose source is >= ne (rows ascending).
__device__ __forceinline__ int64_t bwd_cut(const LikTrace& T, int64_t x, int64_t ne) {
    int64_t lo = T.bo[x], hi = T.bo[x + 1];
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if ((int64_t)T.bc[mid] < ne)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ LikC lik_c(const double* pp) {
    const float4 a = *reinterpret_cast<const float4*>(pp + 8), b = *reinterpret_cast<const float4*>(pp + 10);
    return LikC{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

// The exact layout's fourth word: the fp32 remainders of log(d+1) (low half) and of log f (high
// half), each times 2^24 as an IEEE half.  A remainder is at most 2^-25 of its high part, so 11 bits
// of it carry the pair to about 2^-35.
__device__ __forceinline__ float lik_pack_lows(float ly_rem24, float lx_rem24) {
    const uint32_t y = __half_as_ushort(__float2half_rn(ly_rem24));
    const uint32_t x = __half_as_ushort(__float2half_rn(lx_rem24));
    return __uint_as_float(y | (x << 16));
}
__device__ __forceinline__ void lik_unpack_lows(float w, float& ly_rem24, float& lx_rem24) {
    const uint32_t b = __float_as_uint(w);
    ly_rem24 = __half2float(__ushort_as_half((unsigned short)(b & 0xFFFFu)));
    lx_rem24 = __half2float(__ushort_as_half((unsigned short)(b >> 16)));
}
// 2^x on the special-function unit (PTX ex2.approx.ftz.f32).
__device__ __forceinline__ float ex2_sfu(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// log2 of the weight, ga2 log f + al2 log(d+1) - it2 (t - t_j), as h + l.  Features: f.y = log(d+1)
// (fp32 high part), f.z = t - t_j (an exact integer); default layout: f.x = log f in fp32 (logf_pg),
// f.w = the remainder of log(d+1); exact layout: f.x = the fp32 high part of the FP64 log f,
// f.w = both logs' remainders, packed (lik_pack_lows).
struct X2 {
    float h, l;
};
// the low-order terms of the exponent: the constants' remainders times the features' high parts,
// the constants times the features' remainders (the exact layout also carries log f's)
template <bool EXACT>
__device__ __forceinline__ float lik_tail(const float4 f, const LikC& c) {
    const float base = __fmaf_rn(c.al2l, f.y, __fmaf_rn(c.ga2l, f.x, -(c.it2l * f.z)));
    if (!EXACT) return __fmaf_rn(c.al2, f.w, base);
    float ly, lx;
    lik_unpack_lows(f.w, ly, lx);
    return __fmaf_rn(c.al2s, ly, __fmaf_rn(c.ga2s, lx, base));
}
template <bool EXACT>
__device__ __forceinline__ X2 lik_x2(const float4 f, const LikC& c) {
    X2 x;
    if (EXACT) {
        // every product and sum keeps its rounding error (FMA residuals, two-sums): h + l is the
        // exponent to about 2^-40, so no node's weight carries a fixed error of its own
        const float p3 = c.ga2 * f.x, e3 = __fmaf_rn(c.ga2, f.x, -p3);
        const float p1 = c.al2 * f.y, e1 = __fmaf_rn(c.al2, f.y, -p1);
        const float p2 = -c.it2 * f.z, e2 = __fmaf_rn(-c.it2, f.z, -p2);
        float r1, r2;
        const float s1 = two_sum(p3, p1, r1);
        x.h = two_sum(s1, p2, r2);
        x.l = ((e1 + e2) + (e3 + (r1 + r2))) + lik_tail<true>(f, c);
    } else {
        x.h = __fmaf_rn(c.al2, f.y, __fmaf_rn(-c.it2, f.z, c.ga2 * f.x));
        x.l = lik_tail<false>(f, c);
    }
    return x;
}
// 2^(h + l) for |l| < 2^-18 in fp32 arithmetic: n = rint(h), f = h - n (exact), t = (f + l) ln 2
// in [-0.35, 0.35], e^t by its Taylor series through t^7/7! (truncation below 5e-9 relative), times
// 2^n built in the exponent field: about 2 ulp, with rounding errors that vary from node to node.
__device__ __forceinline__ float exp2_exact(const X2 x) {
    const float n = rintf(x.h);
    const int ni = (int)n;
    if (ni < -126) return 0.0f;
    const float t = __fmaf_rn(x.h - n, kLn2f, x.l * kLn2f);
    float p = 1.0f / 5040.0f;
    p = __fmaf_rn(p, t, 1.0f / 720.0f);
    p = __fmaf_rn(p, t, 1.0f / 120.0f);
    p = __fmaf_rn(p, t, 1.0f / 24.0f);
    p = __fmaf_rn(p, t, 1.0f / 6.0f);
    p = __fmaf_rn(p, t, 0.5f);
    p = __fmaf_rn(p, t, 1.0f);
    p = __fmaf_rn(p, t, 1.0f);
    return p * __int_as_float((ni > 127 ? 255 : ni + 127) << 23);
}
// the weight 2^(h + l): EXACT selects exp2_exact, else the special-function unit's 2^h scaled by
// 1 + l ln 2 + O(l^2)
template <bool EXACT>
__device__ __forceinline__ float lik_w(const X2 x) {
    if (EXACT) return exp2_exact(x);
    const float e = ex2_sfu(x.h);
    return __fmaf_rn(e, x.l * kLn2f, e);
}

// Double-float numbers (a pair of fp32, h + l with |l| <= ulp(h) / 2; Dekker 1971, Knuth's two-sum):
// about 44 significant bits from fp32 arithmetic.  The citation loops run in them: GB300's FP64
// rate is a small fraction of its fp32 rate, and FP64 there cost as much as the ball sums.
struct DF {
    float h, l;
};
__device__ __forceinline__ DF df_of(double x) {
    DF r;
    r.h = (float)x;
    r.l = (float)(x - (double)r.h);
    return r;
}
__device__ __forceinline__ double df_val(const DF a) { return (double)a.h + (double)a.l; }
__device__ __forceinline__ DF df_norm(float s, float e) {  // s + e as a pair, any magnitudes
    float r;
    const float h = two_sum(s, e, r);
    return DF{h, r};
}
__device__ __forceinline__ DF df_add(const DF a, const DF b) {
    float e;
    const float s = two_sum(a.h, b.h, e);
    return df_norm(s, e + (a.l + b.l));
}
__device__ __forceinline__ DF df_neg(const DF a) { return DF{-a.h, -a.l}; }
__device__ __forceinline__ DF df_mul(const DF a, const DF b) {
    const float p = a.h * b.h;
    const float e = __fmaf_rn(a.h, b.h, -p);
    return df_norm(p, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, e)));
}
__device__ __forceinline__ DF df_mulf(const DF a, float b) {
    const float p = a.h * b;
    const float e = __fmaf_rn(a.h, b, -p);
    return df_norm(p, __fmaf_rn(a.l, b, e));
}
__device__ __forceinline__ bool df_gt(const DF a, const DF b) { return a.h > b.h || (a.h == b.h && a.l > b.l); }
// 1/a for a > 0: the fp32 reciprocal r, then one Newton step r + r (1 - a r) in double-float
__device__ __forceinline__ DF df_recip(const DF a) {
    const float r = 1.0f / a.h;
    const DF e = df_add(DF{1.0f, 0.0f}, df_neg(df_mulf(a, r)));
    return df_add(DF{r, 0.0f}, df_mulf(e, r));
}

// log(1 - u) for u in [0, 0.5): -2 atanh(t), t = u / (2 - u) in [0, 1/3), by the odd Taylor series
// of atanh, t + t^3/3 + ... + t^17/17 (truncation below 1e-9 relative at t = 1/3).
__device__ __forceinline__ float log1m_pg(float u) {
    const float t = u / (2.0f - u);
    const float s = t * t;
    float p = 1.0f / 17.0f;
    p = p * s + 1.0f / 15.0f;
    p = p * s + 1.0f / 13.0f;
    p = p * s + 1.0f / 11.0f;
    p = p * s + 1.0f / 9.0f;
    p = p * s + 1.0f / 7.0f;
    p = p * s + 1.0f / 5.0f;
    p = p * s + 1.0f / 3.0f;
    p = p * s + 1.0f;
    return -2.0f * t * p;
}

}  // namespace

// EXACT selects the exact layout (see lik_x2)
template <bool EXACT>
__global__ void __launch_bounds__(256) k_lik_features(LikTrace T) {
    const int e = blockIdx.y;
    const int64_t ne = T.epoch_nodes[e];
    const int32_t te = T.epoch_t[e];
    float4* F = T.feat + (int64_t)e * T.n;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < ne;
         j += (int64_t)gridDim.x * blockDim.x) {
        const int64_t d = bwd_cut(T, j, ne) - T.bo[j];
        const double ly = log_pg((double)(d + 1));
        float4 f;
        f.y = (float)ly;
        f.z = (float)(te - T.pub[j]);
        if (EXACT) {
            const double lx = log_pg((double)T.fit[j]);
            f.x = (float)lx;
            f.w = lik_pack_lows((float)((ly - (double)f.y) * 0x1p24), (float)((lx - (double)f.x) * 0x1p24));
        } else {
            f.x = logf_pg(T.fit[j]);
            f.w = (float)(ly - (double)f.y);
        }
        F[j] = f;
    }
}

template <bool ADJ, bool EXACT>
__global__ void __launch_bounds__(kLikThreads) k_lik_global(LikTrace T, LikBatch P) {
    __shared__ double red[kLikThreads * 4];
    const int e = P.e0 + blockIdx.y, tid = threadIdx.x;
    const int64_t ne = T.epoch_nodes[e];
    const int64_t lo = (int64_t)blockIdx.x * kLikChunk;
    const int BE = P.BE, B = P.B;
    const int b = tid & (BE - 1), sub = tid / BE, nsub = kLikThreads / BE;
    // Sums of at most 32 terms in fp32 with their rounding errors (ErrSum: the exact sum to 64 bits), then FP64:
    // GB300 does two FP64 operations per clock and SM, and the adjoint's four FP64 operations and four
    // conversions per weight were 2.87 ms of a 64-point pass of a 200k-node trace, now 0.65
    // (forward 0.34).  Terms out of ErrSum's range (weights of the batch together above 2^90 or below 2^-60)
    // are summed in FP64.
    double s = 0.0, t0 = 0.0, t1 = 0.0, t2 = 0.0;
    if (b < B && lo < ne) {
        const LikC c = lik_c(P.pp + b * kLikPP);
        const int64_t hi = ne < lo + kLikChunk ? ne : lo + kLikChunk;
        const float4* F = T.feat + (int64_t)e * T.n;
        float* tab = P.wt ? P.wt + blockIdx.y * P.wt_n * BE + b : nullptr;
        for (int64_t j = lo + sub; j < hi;) {
            const int64_t j0 = j;
            ErrSum ps, p0, p1, p2;
#pragma unroll 4
            for (int q = 0; q < 32; ++q, j += nsub) {
                if (j >= hi) break;
                const float4 f = F[j];
                const float w = lik_w<EXACT>(lik_x2<EXACT>(f, c));
                if (tab) tab[j * BE] = w;
                err_add(ps, w);
                if (ADJ) {
                    err_add_product(p0, w, f.y);
                    err_add_product(p1, w, f.z);
                    err_add_product(p2, w, f.x);
                }
            }
            if (err_ranges_hold(ps)) {
                s += err_value(ps);
                t0 += err_value(p0);
                t1 += err_value(p1);
                t2 += err_value(p2);
            } else {
#pragma unroll 1
                for (int64_t i = j0; i < j; i += nsub) {
                    const float4 f = F[i];
                    const double w = (double)lik_w<EXACT>(lik_x2<EXACT>(f, c));
                    s += w;
                    if (ADJ) {
                        t0 = __fma_rn(w, (double)f.y, t0);
                        t1 = __fma_rn(w, (double)f.z, t1);
                        t2 = __fma_rn(w, (double)f.x, t2);
                    }
                }
            }
        }
    }
    red[tid * 4 + 0] = s;
    red[tid * 4 + 1] = t0;
    red[tid * 4 + 2] = t1;
    red[tid * 4 + 3] = t2;
    __syncthreads();
    if (sub == 0 && b < B) {
        constexpr int K = ADJ ? 4 : 1;
        double acc[K] = {};
        for (int q = 0; q < nsub; ++q)
#pragma unroll
            for (int k = 0; k < K; ++k) acc[k] += red[(q * BE + b) * 4 + k];
        double* o = P.gpart + (((int64_t)e * T.chunks + blockIdx.x) * B + b) * K;
#pragma unroll
        for (int k = 0; k < K; ++k) o[k] = acc[k];
    }
}

// Sum over rows [lo, hi) of column threadIdx.x of the row-major matrix m with C columns, in threads
// 0..C-1 (Cp: C rounded up to a power of two, at most kLikSumThreads): the threads take rows in turn,
// then the rows' sums are added pairwise, in a fixed order.  Whole CTA; r: one double per thread.
__device__ __forceinline__ double column_sum(const double* m, int64_t lo, int64_t hi, int C, int Cp, double* r) {
    const int c = threadIdx.x & (Cp - 1), row = threadIdx.x / Cp, rows = kLikSumThreads / Cp;
    double acc = 0.0;
    if (c < C) {
#pragma unroll 8
        for (int64_t a = lo + row; a < hi; a += rows) acc += __ldcg(m + a * C + c);
    }
    r[threadIdx.x] = acc;
    __syncthreads();
    for (int h = kLikSumThreads / 2; h >= Cp; h >>= 1) {
        if ((int)threadIdx.x < h) r[threadIdx.x] += r[threadIdx.x + h];
        __syncthreads();
    }
    return r[c];
}

// One CTA per epoch: its chunks' partial sums.
template <bool ADJ>
__global__ void __launch_bounds__(kLikSumThreads) k_lik_global_sum(LikTrace T, LikBatch P) {
    __shared__ double r[kLikSumThreads];
    const int e = P.e0 + blockIdx.x, C = P.B * (ADJ ? 4 : 1);
    const double v = column_sum(P.gpart + (int64_t)e * T.chunks * C, 0, T.chunks, C, P.BE * (ADJ ? 4 : 1), r);
    if ((int)threadIdx.x >= C) return;
    if (!ADJ) {
        P.zglob[e * P.B + threadIdx.x] = v;
        return;
    }
    const int b = threadIdx.x >> 2, k = threadIdx.x & 3;  // (w, alpha, tau, gamma)
    const double tau = P.theta[b * 4 + 1];
    if (k) P.gglob[((int64_t)e * P.B + b) * 3 + k - 1] = k == 2 ? v * (1.0 / (tau * tau)) : v;
}

// The 2-hop ball of agents [a0, a1) in the epoch-start graph, one CTA per agent, as a bitmap over
// [0, n_e) in shared memory (passes of bitmap_words * 32 ids).  EMIT = false: ball sizes (and the
// adjacency entries read) into Bl.cnt; EMIT = true: the ids, ascending, at Bl.ids[boff[a] - base]
// and the ball membership of each citation into Bl.cflag.
template <bool EMIT>
__global__ void __launch_bounds__(kLikThreads) k_lik_ball(LikTrace T, LikBalls Bl, int64_t a0, int64_t a1) {
    extern __shared__ __align__(16) unsigned char lik_smem[];
    uint32_t* bits = reinterpret_cast<uint32_t*>(lik_smem);  // [bitmap_words]
    __shared__ int64_t seg[2 * PG_MAX_ANCHORS_DEV + 1];       // prefix of the anchors' row lengths
    __shared__ int64_t rowb[2 * PG_MAX_ANCHORS_DEV];          // first entry of each anchor row
    __shared__ int32_t anc[PG_MAX_ANCHORS_DEV];
    __shared__ int32_t nanc;
    __shared__ int32_t scan_ws[33];
    __shared__ unsigned long long adj_read;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t pass_ids = (int64_t)T.bitmap_words * 32;
    for (int64_t a = a0 + blockIdx.x; a < a1; a += gridDim.x) {
        const int e = T.agent_epoch[a];
        const int64_t ne = T.epoch_nodes[e];
        const int64_t c0 = T.coff[a];
        const int k = (int)(T.coff[a + 1] - c0);
        if (tid == 0) {
            int na = 0;
            for (int i = 0; i < T.num_anchors; ++i) {
                const int32_t x = T.anchors[a * 4 + i];
                if (x >= 0) anc[na++] = x;
            }
            nanc = na;
            int64_t acc = 0;
            for (int i = 0; i < na; ++i) {
                const int64_t x = anc[i];
                rowb[2 * i] = T.fo[x];
                seg[2 * i] = acc;
                acc += T.fo[x + 1] - T.fo[x];
                rowb[2 * i + 1] = T.bo[x];
                seg[2 * i + 1] = acc;
                acc += bwd_cut(T, x, ne) - T.bo[x];
            }
            seg[2 * na] = acc;
            adj_read = (unsigned long long)acc;
        }
        __syncthreads();
        const int na = nanc;
        const int64_t L1 = seg[2 * na];
        int64_t written = EMIT ? Bl.boff[a] - Bl.base : 0;
        unsigned long long ball = 0;
        for (int64_t lo = 0; lo < ne; lo += pass_ids) {
            const int64_t hi = ne < lo + pass_ids ? ne : lo + pass_ids;
            const int nw = (int)((hi - lo + 31) >> 5);
            uint32_t* cache = Bl.bmap ? Bl.bmap + a * Bl.bmap_stride + (lo / pass_ids) * T.bitmap_words : nullptr;
            if (EMIT && cache) {
                // the count pass left this agent's bitmap: no row walk
                for (int w = tid; w < nw; w += kLikThreads) bits[w] = cache[w];
                __syncthreads();
            } else {
                for (int w = tid; w < nw; w += kLikThreads) bits[w] = 0u;
                __syncthreads();
                auto mark = [&](int64_t v) {
                    if (v >= lo && v < hi) {
                        const int64_t o = v - lo;
                        atomicOr(&bits[o >> 5], 1u << (o & 31));
                    }
                };
                if (tid < na) mark(anc[tid]);
                // every 1-hop node y (one warp each) and the rows of y
                for (int64_t q = warp; q < L1; q += kLikThreads / 32) {
                    int sg = 0;
                    while (seg[sg + 1] <= q) ++sg;
                    const int32_t* col = (sg & 1) ? T.bc : T.fc;
                    const int64_t y = col[rowb[sg] + (q - seg[sg])];
                    if (lane == 0) mark(y);
                    const int64_t f1 = T.fo[y + 1];
                    for (int64_t p = T.fo[y] + lane; p < f1; p += 32) mark(T.fc[p]);
                    const int64_t b1 = bwd_cut(T, y, ne);
                    for (int64_t p = T.bo[y] + lane; p < b1; p += 32) mark(T.bc[p]);
                    if (!EMIT && lane == 0 && lo == 0)
                        atomicAdd(&adj_read, (unsigned long long)((f1 - T.fo[y]) + (b1 - T.bo[y])));
                }
                __syncthreads();
                if (!EMIT && cache)
                    for (int w = tid; w < nw; w += kLikThreads) cache[w] = bits[w];
            }
            if (EMIT) {
                for (int i = tid; i < k; i += kLikThreads) {
                    const int64_t c = T.cites[c0 + i];
                    if (c >= lo && c < hi) {
                        const int64_t o = c - lo;
                        Bl.cflag[c0 + i] = (uint8_t)((bits[o >> 5] >> (o & 31)) & 1u);
                    }
                }
            }
            // each thread owns a contiguous run of words; a block scan of their popcounts places
            // its ids so the ball comes out ascending
            const int wpt = (nw + kLikThreads - 1) / kLikThreads;
            const int w0 = tid * wpt < nw ? tid * wpt : nw;
            const int w1 = w0 + wpt < nw ? w0 + wpt : nw;
            int cnt = 0;
            for (int w = w0; w < w1; ++w) cnt += __popc(bits[w]);
            int total = 0;
            const int off = block_excl_scan<int>(cnt, scan_ws, &total);
            if (EMIT && cnt > 0) {
                int32_t* out = Bl.ids + written + off;
                int r = 0;
                for (int w = w0; w < w1; ++w) {
                    uint32_t m = bits[w];
                    while (m) {
                        const int bit = __ffs(m) - 1;
                        m &= m - 1u;
                        out[r++] = (int32_t)(lo + ((int64_t)w << 5) + bit);
                    }
                }
            }
            written += total;
            ball += (unsigned long long)total;
            __syncthreads();  // the bitmap is cleared by the next pass
        }
        if (!EMIT && tid == 0) {
            Bl.cnt[a] = (int64_t)ball;
            Bl.adj[a] = (int64_t)adj_read;
        }
        __syncthreads();
    }
}

// One agent at one point, by one lane: the normaliser Z_a from the ball's sums (S = sum w, T = sum w g)
// and the citations walked in draw order:  D_i = Z_a - P_i,  log D_i = log Z_a + log(1 - P_i / Z_a), and
// in the adjoint g_i - (dZ_a - dP_i) / D_i.
template <bool ADJ, bool EXACT>
__device__ __forceinline__ void lik_agent(const LikTrace& T, const LikBatch& P, const LikBalls& Bl, int64_t a, int e,
                                          const float4* F, int b, const LikC& c, double S, double T0, double T1,
                                          double T2) {
    const double* pp = P.pp + b * kLikPP;
    const double beta = pp[3], lbe = pp[4], ibe = pp[5], itau2 = pp[6];
    const int64_t c0 = T.coff[a];
    const int k = (int)(T.coff[a + 1] - c0);
    double Z;
    double dz[4] = {0.0, 0.0, 0.0, 0.0};
    if (!ADJ) {
        Z = P.zglob[e * P.B + b] + (beta - 1.0) * S;
        P.zagent[a * P.B + b] = Z;
    } else {
        Z = P.zagent[a * P.B + b];
        const double* gg = P.gglob + ((int64_t)e * P.B + b) * 3;
        dz[0] = gg[0] + (beta - 1.0) * T0;
        dz[1] = gg[1] + (beta - 1.0) * (T1 * itau2);
        dz[2] = gg[2] + (beta - 1.0) * T2;
        dz[3] = S;
    }
    if (!(Z > 0.0)) {
        atomicOr(P.error, 2u);
        return;
    }
    // the citations in draw order, in fp32 / double-float arithmetic (FP64 only per agent
    // and in the rare u >= 1/2 case): W_i = w_i beta^[in ball], P the weight drawn before
    if (!ADJ) {
        // l_a = ln2 sum x_i + n_in log beta - (k log Z_a + sum log(1 - u_i)), u_i = P_i / Z_a;
        // the sums of x_i (its two parts), of log(1 - u_i) and of P compensated in fp32
        const double logZ = log_pg(Z);
        const float invZ = 1.0f / (float)Z, betaf = (float)beta;
        Kahan sh, sl, slr, pc;
        // Where more than half of Z is drawn (1 - u is small) the term is log(Z - P) - log Z from the FP64
        // difference.  The differences are multiplied up and one logarithm taken of the product, whose exponent
        // is kept apart in an integer: a factor's rounding is 2^-53 of itself, less than that of its logarithm
        // would be.  A logarithm per citation: 5.83 ms for the forward pass of 64 points of a 200k-node trace, now
        // 4.84; 64 points one at a time, with their adjoints, 180.6 to 157.7 ms.
        double prod = 1.0, odd = 0.0;
        int pexp = 0, far = 0;
        int n_in = 0;
        for (int i = 0; i < k; ++i) {
            const bool in = Bl.cflag[c0 + i] != 0;
            const float4 f = F[T.cites[c0 + i]];
            const X2 x2 = lik_x2<EXACT>(f, c);
            const float w = lik_w<EXACT>(x2);
            const float W = in ? w * betaf : w;
            const float u = (pc.s - pc.c) * invZ;
            if (u < 0.5f)
                kadd(slr, log1m_pg(u));
            else {
                const double D = Z - kval(pc);
                const int dh = __double2hiint(D);
                if (dh >= (23 << 20) && dh < (2023 << 20)) {  // 2^-1000 <= D < 2^1000
                    prod = prod * D;
                    const int hi = __double2hiint(prod), ex = (hi >> 20) - 1023;
                    prod = __hiloint2double(hi - (ex << 20), __double2loint(prod));  // in [1, 2)
                    pexp += ex;
                    ++far;
                } else {
                    odd += log_pg(D) - logZ;
                }
            }
            kadd(sh, x2.h);
            kadd(sl, x2.l);
            n_in += in ? 1 : 0;
            kadd(pc, W);
        }
        if (far > 0) {
            const double pe = (double)pexp;
            odd += __fma_rn(pe, kLn2Hi, __fma_rn(pe, kLn2Lo, log_pg(prod)));
        }
        const double l = (kval(sh) + kval(sl)) * kLn2d + (double)n_in * lbe -
                         ((double)(k - far) * logZ + kval(slr) + odd);
        P.out[a * P.B + b] = l;
    } else {
        // g_k = sum_i [gk_i - (dZ_k - dP_k,i) / D_i],  D_i = Z_a - P_i,  dP_k,i = sum_{j<i} W_j gk_j
        const DF Zd = df_of(Z), betad = df_of(beta), itau2d = df_of(itau2), ibed = df_of(ibe);
        DF dzd[4], dP[4], g[4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            dzd[kk] = df_of(dz[kk]);
            dP[kk] = DF{0.0f, 0.0f};
            g[kk] = DF{0.0f, 0.0f};
        }
        DF Pc{0.0f, 0.0f};
        for (int i = 0; i < k; ++i) {
            const bool in = Bl.cflag[c0 + i] != 0;
            const float4 f = F[T.cites[c0 + i]];
            const X2 x2 = lik_x2<EXACT>(f, c);
            const float w = lik_w<EXACT>(x2);
            const DF W = in ? df_mulf(betad, w) : DF{w, 0.0f};
            const DF D = df_add(Zd, df_neg(Pc));
            const DF id = df_recip(df_gt(D, W) ? D : W);
            const DF gk[4] = {DF{f.y, 0.0f}, df_mulf(itau2d, f.z), DF{f.x, 0.0f}, in ? ibed : DF{0.0f, 0.0f}};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const DF t = df_mul(df_add(dzd[kk], df_neg(dP[kk])), id);
                g[kk] = df_add(g[kk], df_add(gk[kk], df_neg(t)));
                dP[kk] = df_add(dP[kk], df_mul(W, gk[kk]));
            }
            Pc = df_add(Pc, W);
        }
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) P.out[(a * P.B + b) * 4 + kk] = df_val(g[kk]);
    }
}

// Forward (ADJ = false) or adjoint pass over agents [a0, a1) whose balls are in Bl, every weight
// evaluated where it is summed.  One warp per (agent, group of points).  NP = 2 (33..64 points): lane l
// holds points l and l + 32, and every lane walks the whole ball, so each ball element is read once for
// all points.  NP = 1 (<= 32 points): lane = point p + BW * slice; the slices split the ball, so a
// single point spreads its ball over the whole warp.  Ball sums: fp32 weights, four elements summed
// pairwise, then compensated fp32 per lane, FP64 across slices.  The slice-0 lane of each point then
// walks the citations (lik_agent).
template <bool ADJ, int NP, bool EXACT>
__global__ void __launch_bounds__(kLikThreads, ADJ ? 2 : 3)
    k_lik_eval(LikTrace T, LikBatch P, LikBalls Bl, int64_t a0, int64_t a1) {
    __shared__ float4 lik_stage[kLikThreads / 32][32];
    const int lane = threadIdx.x & 31;
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int BW = NP == 2 ? 32 : P.BW, SL = 32 / BW;
    const int groups = NP == 2 ? 1 : (P.B + BW - 1) / BW;
    const int pl = lane & (BW - 1), sl = lane / BW;
    const int64_t items = (a1 - a0) * groups;
    for (int64_t it = wid; it < items; it += nwarps) {
        const int64_t a = a0 + it / groups;
        int bq[NP];
        bool act[NP];
        LikC cq[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            bq[p] = NP == 2 ? lane + 32 * p : (int)(it % groups) * BW + pl;
            act[p] = bq[p] < P.B;
            cq[p] = lik_c(P.pp + (act[p] ? bq[p] : 0) * kLikPP);
        }
        const int e = T.agent_epoch[a];
        const float4* F = T.feat + (int64_t)e * T.n;
        const int64_t j0 = Bl.boff[a] - Bl.base, j1 = Bl.boff[a + 1] - Bl.base;
        BallSum<ADJ, EXACT> acc[NP];
        if constexpr (NP == 2) {
            // the ball in batches of 32: lane l loads element l's id and feature row, the next
            // batch's loads are issued before this batch is summed, and the rows are read back
            // from the warp's shared buffer in the same groups of four (same sums) as below
            float4* buf = lik_stage[threadIdx.x >> 5];
            float4 cur = make_float4(0.f, 0.f, 0.f, 0.f);
            if (j0 + lane < j1) cur = F[Bl.ids[j0 + lane]];
            for (int64_t b0 = j0; b0 < j1; b0 += 32) {
                const int cnt = j1 - b0 < 32 ? (int)(j1 - b0) : 32;
                float4 nxt = make_float4(0.f, 0.f, 0.f, 0.f);
                if (b0 + 32 + lane < j1) nxt = F[Bl.ids[b0 + 32 + lane]];
                __syncwarp();
                buf[lane] = cur;
                __syncwarp();
                int i = 0;
                for (; i + 3 < cnt; i += 4) {
                    const float4 f0 = buf[i], f1 = buf[i + 1], f2 = buf[i + 2], f3 = buf[i + 3];
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        const float w0 = lik_w<EXACT>(lik_x2<EXACT>(f0, cq[p])), w1 = lik_w<EXACT>(lik_x2<EXACT>(f1, cq[p])),
                                    w2 = lik_w<EXACT>(lik_x2<EXACT>(f2, cq[p])), w3 = lik_w<EXACT>(lik_x2<EXACT>(f3, cq[p]));
                        acc[p].add4(w0, w1, w2, w3, f0, f1, f2, f3);
                    }
                }
                for (; i < cnt; ++i) {
                    const float4 f = buf[i];
#pragma unroll
                    for (int p = 0; p < NP; ++p) acc[p].add1(lik_w<EXACT>(lik_x2<EXACT>(f, cq[p])), f);
                }
                cur = nxt;
            }
        }
        int64_t q = NP == 2 ? j1 : j0 + sl;
        for (; q + 3 * SL < j1; q += 4 * SL) {
            const int32_t i0 = Bl.ids[q], i1 = Bl.ids[q + SL], i2 = Bl.ids[q + 2 * SL], i3 = Bl.ids[q + 3 * SL];
            const float4 f0 = F[i0], f1 = F[i1], f2 = F[i2], f3 = F[i3];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const float w0 = lik_w<EXACT>(lik_x2<EXACT>(f0, cq[p])), w1 = lik_w<EXACT>(lik_x2<EXACT>(f1, cq[p])),
                            w2 = lik_w<EXACT>(lik_x2<EXACT>(f2, cq[p])), w3 = lik_w<EXACT>(lik_x2<EXACT>(f3, cq[p]));
                acc[p].add4(w0, w1, w2, w3, f0, f1, f2, f3);
            }
        }
        for (; q < j1; q += SL) {
            const float4 f = F[Bl.ids[q]];
#pragma unroll
            for (int p = 0; p < NP; ++p) acc[p].add1(lik_w<EXACT>(lik_x2<EXACT>(f, cq[p])), f);
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            double S = acc[p].S(), T0 = 0.0, T1 = 0.0, T2 = 0.0;
            if (ADJ) {
                T0 = acc[p].T0();
                T1 = acc[p].T1();
                T2 = acc[p].T2();
            }
            for (int o = BW; o < 32; o <<= 1) {
                S += __shfl_xor_sync(0xffffffffu, S, o);
                if (ADJ) {
                    T0 += __shfl_xor_sync(0xffffffffu, T0, o);
                    T1 += __shfl_xor_sync(0xffffffffu, T1, o);
                    T2 += __shfl_xor_sync(0xffffffffu, T2, o);
                }
            }
            if (act[p] && sl == 0) lik_agent<ADJ, EXACT>(T, P, Bl, a, e, F, bq[p], cq[p], S, T0, T1, T2);
        }
    }
}

// The pass of k_lik_eval with the weights gathered from the global pass's table (LikBatch::wt: the same
// fp32 values, summed in the same order, so the same results): a ball element is one row of BE floats,
// read by the whole warp, instead of an exponent and a 2^x per point.  One warp (its own CTA) per agent.
// What bounds the forward pass is the rows' way from L2, 256 B per element at 64 points at 64 B per
// clock and SM: 405M elements (200k-node trace, 10 epochs) in 5.4 ms, 19 TB/s (direct: 18.7 ms).  The
// adjoint's four compensated sums take 7.75 packed fp32 operations per element: 9.9 ms (27.6).  Balls
// differ a hundredfold in size and a point's sum is one dependent chain, so long balls are taken first
// (LikBalls::order; as numbered: 9.1 and 14.4 ms).  Measured and slower: rows through a shared ring of
// asynchronous copies (10.2 and 15.7 ms: the ring's writes and reads share L1's bandwidth), fewer warps
// with 32 rows in flight each (6.1 ms).
template <bool ADJ, bool EXACT>
__global__ void __launch_bounds__(32, ADJ ? 20 : 32) k_lik_table2(LikTrace T, LikBatch P, LikBalls Bl, int64_t a0) {
    // 33..64 points: lane l holds points 2l and 2l + 1 (packed arithmetic); every lane walks the whole ball
    __shared__ __align__(16) int32_t s_id[32];
    __shared__ __align__(16) F2 s_feat[ADJ ? 32 : 1][4];  // a batch's feature pairs (y, y), (z, z), (x, x)
    const int lane = threadIdx.x;
    const int64_t a = Bl.order ? Bl.order[a0 + blockIdx.x] : a0 + blockIdx.x;
    const int e = T.agent_epoch[a];
    const float4* F = T.feat + (int64_t)e * T.n;
    const int32_t* ids = Bl.ids + (Bl.boff[a] - Bl.base);
    const int len = (int)(Bl.boff[a + 1] - Bl.boff[a]), nb = (len + 31) >> 5;
    const F2* W = reinterpret_cast<const F2*>(P.wt) + (e - P.e0) * P.wt_n * 32 + lane;
    // batches of 32 elements: lane l holds element l's id (adjoint: and its feature row), shared through
    // the warp's buffer; ids are loaded two batches ahead, feature rows one, and sixteen table rows are
    // in flight before they are summed.  Past the end id 0: a row that exists and is not summed.
    auto id_at = [&](int t) { return 32 * t + lane < len ? __ldg(ids + 32 * t + lane) : 0; };
    auto row = [&](int u) { return __ldg(W + (int64_t)s_id[u] * 32); };
    auto feat = [&](int u) {
        Feat2 f{0, 0, 0};
        if (ADJ) {
            const ulonglong2 yz = *reinterpret_cast<const ulonglong2*>(&s_feat[u][0]);
            f.y = yz.x, f.z = yz.y, f.x = s_feat[u][2];
        }
        return f;
    };
    BallSum2<ADJ, EXACT> sum;
    int i0 = id_at(0), i1 = id_at(1);
    float4 cur = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ADJ) cur = F[i0];
    for (int t = 0; t < nb; ++t) {
        const int i2 = id_at(t + 2);
        float4 nxt = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ADJ) nxt = F[i1];
        __syncwarp();
        s_id[lane] = i0;
        if (ADJ) {
            *reinterpret_cast<ulonglong2*>(&s_feat[lane][0]) = make_ulonglong2(f2_of(cur.y, cur.y), f2_of(cur.z, cur.z));
            s_feat[lane][2] = f2_of(cur.x, cur.x);
        }
        __syncwarp();
        const int cnt = len - 32 * t;
        if (cnt >= 32) {
#pragma unroll
            for (int h = 0; h < 32; h += 16) {
                F2 w[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) w[u] = row(h + u);
#pragma unroll
                for (int u = 0; u < 16; u += 4) {
                    const Feat2 f[4] = {feat(h + u), feat(h + u + 1), feat(h + u + 2), feat(h + u + 3)};
                    sum.add4(w + u, f);
                }
            }
        } else {
            int u = 0;
            for (; u + 3 < cnt; u += 4) {
                const F2 w[4] = {row(u), row(u + 1), row(u + 2), row(u + 3)};
                const Feat2 f[4] = {feat(u), feat(u + 1), feat(u + 2), feat(u + 3)};
                sum.add4(w, f);
            }
            for (; u < cnt; ++u) sum.add1(row(u), feat(u));
        }
        cur = nxt;
        i0 = i1;
        i1 = i2;
    }
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const BallSum<ADJ, EXACT> o = sum.point(p);
        const int b = 2 * lane + p;
        if (b < P.B)
            lik_agent<ADJ, EXACT>(T, P, Bl, a, e, F, b, lik_c(P.pp + b * kLikPP), o.S(), ADJ ? o.T0() : 0.0, ADJ ? o.T1() : 0.0,
                                  ADJ ? o.T2() : 0.0);
    }
}

// <= 32 points: lane = point p + BW * slice, the slices split the ball as in k_lik_eval.  Eight elements
// per slice and step (four in the adjoint), the next step's ids loaded before this step's sums.
template <bool ADJ, bool EXACT>
__global__ void __launch_bounds__(32, ADJ ? 20 : 32) k_lik_table1(LikTrace T, LikBatch P, LikBalls Bl, int64_t a0) {
    const int lane = threadIdx.x;
    const int64_t a = Bl.order ? Bl.order[a0 + blockIdx.x] : a0 + blockIdx.x;
    const int e = T.agent_epoch[a];
    const float4* F = T.feat + (int64_t)e * T.n;
    const int BW = P.BW, SL = 32 / BW, pl = lane & (BW - 1), sl = lane / BW;
    const int32_t* ids = Bl.ids + (Bl.boff[a] - Bl.base) + sl;
    const int all = (int)(Bl.boff[a + 1] - Bl.boff[a]);
    const int len = all > sl ? (all - sl + SL - 1) / SL : 0;  // this lane's elements
    const float* W = P.wt + (e - P.e0) * P.wt_n * BW + pl;
    BallSum<ADJ, EXACT> sum;
    auto ids_at = [&](int q, int* to) {
#pragma unroll
        for (int u = 0; u < 8; ++u) to[u] = q + u < len ? __ldg(ids + (int64_t)(q + u) * SL) : 0;
    };
    int id[8], nx[8];
    ids_at(0, id);
    ids_at(8, nx);
    int q = 0;
    auto eight = [&](auto next) {
        float w[8];
        float4 f[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            w[u] = __ldg(W + (int64_t)id[u] * BW);
            f[u] = ADJ ? F[id[u]] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) id[u] = nx[u];
        next();
        sum.add4(w[0], w[1], w[2], w[3], f[0], f[1], f[2], f[3]);
        sum.add4(w[4], w[5], w[6], w[7], f[4], f[5], f[6], f[7]);
    };
    const int32_t* ahead = ids + 16 * SL;
    for (; q + 23 < len; q += 8, ahead += 8 * SL)  // the ids two steps ahead exist: no bounds checks
        eight([&]() {
#pragma unroll
            for (int u = 0; u < 8; ++u) nx[u] = __ldg(ahead + u * SL);
        });
    for (; q + 7 < len; q += 8) eight([&]() { ids_at(q + 16, nx); });
    auto one = [&](int x) { sum.add1(__ldg(W + (int64_t)x * BW), ADJ ? F[x] : make_float4(0.f, 0.f, 0.f, 0.f)); };
    if (q + 3 < len) {
        float w[4];
        float4 f[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            w[u] = __ldg(W + (int64_t)id[u] * BW);
            f[u] = ADJ ? F[id[u]] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        sum.add4(w[0], w[1], w[2], w[3], f[0], f[1], f[2], f[3]);
        q += 4;
#pragma unroll
        for (int u = 0; u < 3; ++u)
            if (q + u < len) one(id[4 + u]);
    } else {
#pragma unroll
        for (int u = 0; u < 3; ++u)
            if (q + u < len) one(id[u]);
    }
    double v[4] = {sum.S(), 0.0, 0.0, 0.0};
    if (ADJ) v[1] = sum.T0(), v[2] = sum.T1(), v[3] = sum.T2();
    for (int o = BW; o < 32; o <<= 1)
#pragma unroll
        for (int k = 0; k < (ADJ ? 4 : 1); ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (pl < P.B && sl == 0)
        lik_agent<ADJ, EXACT>(T, P, Bl, a, e, F, pl, lik_c(P.pp + pl * kLikPP), v[0], v[1], v[2], v[3]);
}

// Totals over agents: every CTA sums a contiguous range of agents' rows (C = B K columns, read
// coalesced), the last one to finish adds the CTAs' sums; the order of every sum is fixed.  68,788
// agents x 64 points: 17 us (adjoint 70 us, bound by FP64 adds); one CTA per column, its threads a row
// apart, took 65 and 195 us.
__global__ void __launch_bounds__(kLikSumThreads) k_lik_sum(const double* out, int64_t agents, int C, int Cp, double* part,
                                                            unsigned int* ticket, double* res) {
    __shared__ double r[kLikSumThreads];
    __shared__ bool last;
    const int64_t per = (agents + gridDim.x - 1) / gridDim.x;
    const int64_t lo = per * blockIdx.x, hi = lo + per < agents ? lo + per : agents;
    const double mine = column_sum(out, lo, hi, C, Cp, r);
    if (threadIdx.x < C) __stcg(part + (int64_t)blockIdx.x * C + threadIdx.x, mine);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double total = column_sum(part, 0, gridDim.x, C, Cp, r);
    if (threadIdx.x < C) res[threadIdx.x] = total;
    if (threadIdx.x == 0) *ticket = 0u;  // for the next launch
}

size_t lik_ball_smem(int bitmap_words) { return sizeof(uint32_t) * (size_t)bitmap_words; }

cudaError_t init_lik_kernels(int bitmap_words, int* ball_per_sm, int* eval_per_sm) {
    // eval_per_sm[0]: forward, [1]: adjoint
    const int smem = (int)lik_ball_smem(bitmap_words);
    cudaError_t e = cudaFuncSetAttribute(k_lik_ball<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_lik_ball<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int b0 = 1, b1 = 1, v0 = 1, v1 = 1;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_lik_ball<false>, kLikThreads, smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_lik_ball<true>, kLikThreads, smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v0, k_lik_eval<false, 2, false>, kLikThreads, 0);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v1, k_lik_eval<true, 2, false>, kLikThreads, 0);
    *ball_per_sm = b0 < b1 ? (b0 < 1 ? 1 : b0) : (b1 < 1 ? 1 : b1);
    eval_per_sm[0] = v0 < 1 ? 1 : v0;
    eval_per_sm[1] = v1 < 1 ? 1 : v1;
    return e;
}

void launch_lik_ball(const LikTrace& T, const LikBalls& Bl, int emit, int64_t a0, int64_t a1, int grid,
                     cudaStream_t s) {
    if (a1 <= a0) return;
    int64_t g = a1 - a0 < grid ? a1 - a0 : grid;
    const size_t smem = lik_ball_smem(T.bitmap_words);
    if (emit)
        k_lik_ball<true><<<(unsigned)g, kLikThreads, smem, s>>>(T, Bl, a0, a1);
    else
        k_lik_ball<false><<<(unsigned)g, kLikThreads, smem, s>>>(T, Bl, a0, a1);
}

void launch_lik_global(const LikTrace& T, const LikBatch& P, int adjoint, cudaStream_t s) {
    const dim3 gg((unsigned)T.chunks, (unsigned)(P.e1 - P.e0));
    const unsigned gs = (unsigned)(P.e1 - P.e0);
    const bool x = P.exact_exp2 != 0;
    if (adjoint) {
        if (x)
            k_lik_global<true, true><<<gg, kLikThreads, 0, s>>>(T, P);
        else
            k_lik_global<true, false><<<gg, kLikThreads, 0, s>>>(T, P);
        k_lik_global_sum<true><<<gs, kLikSumThreads, 0, s>>>(T, P);
    } else {
        if (x)
            k_lik_global<false, true><<<gg, kLikThreads, 0, s>>>(T, P);
        else
            k_lik_global<false, false><<<gg, kLikThreads, 0, s>>>(T, P);
        k_lik_global_sum<false><<<gs, kLikSumThreads, 0, s>>>(T, P);
    }
}

void launch_lik_eval(const LikTrace& T, const LikBatch& P, const LikBalls& Bl, int adjoint, int64_t a0,
                     int64_t a1, int grid, cudaStream_t s) {
    if (a1 <= a0) return;
    const bool two = P.B > 32;
    const int groups = two ? 1 : (P.B + P.BW - 1) / P.BW;
    const int64_t warps = (a1 - a0) * groups;
    const bool x = P.exact_exp2 != 0;
    int64_t g = (warps + kLikThreads / 32 - 1) / (kLikThreads / 32);
    if (g > grid) g = grid;
    const unsigned gt = (unsigned)(a1 - a0);
#define PG_LIK_EVAL(ADJ, NP, EX)                                                                    \
    (!P.wt ? k_lik_eval<ADJ, NP, EX><<<(unsigned)g, kLikThreads, 0, s>>>(T, P, Bl, a0, a1)           \
           : (NP == 2 ? k_lik_table2<ADJ, EX><<<gt, 32, 0, s>>>(T, P, Bl, a0)                       \
                      : k_lik_table1<ADJ, EX><<<gt, 32, 0, s>>>(T, P, Bl, a0)))
    if (adjoint) {
        if (two)
            x ? PG_LIK_EVAL(true, 2, true) : PG_LIK_EVAL(true, 2, false);
        else
            x ? PG_LIK_EVAL(true, 1, true) : PG_LIK_EVAL(true, 1, false);
    } else {
        if (two)
            x ? PG_LIK_EVAL(false, 2, true) : PG_LIK_EVAL(false, 2, false);
        else
            x ? PG_LIK_EVAL(false, 1, true) : PG_LIK_EVAL(false, 1, false);
    }
#undef PG_LIK_EVAL
}

void launch_lik_sum(const LikTrace& T, const LikBatch& P, int adjoint, cudaStream_t s) {
    const int C = P.B * (adjoint ? 4 : 1);
    int Cp = 1;
    while (Cp < C) Cp <<= 1;
    const int64_t g = (T.agents * C + 8 * kLikSumThreads - 1) / (8 * kLikSumThreads);
    k_lik_sum<<<(unsigned)(g < 1 ? 1 : (g > kLikSumCtas ? kLikSumCtas : g)), kLikSumThreads, 0, s>>>(
        P.out, T.agents, C, Cp, P.spart, P.error + 1, P.res);
}

// one warp per agent
__global__ void __launch_bounds__(256) k_trace_edges(const int64_t* coff, const int32_t* cites, int64_t agents,
                                                     int64_t n0, int64_t ns, int32_t* src, int32_t* dst) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t a = warp; a < agents; a += nwarps) {
        const int64_t p1 = coff[a + 1];
        for (int64_t p = coff[a] + lane; p < p1; p += 32) {
            src[ns + p] = (int32_t)(n0 + a);
            dst[ns + p] = cites[p];
        }
    }
}

void launch_trace_edges(const int64_t* coff, const int32_t* cites, int64_t agents, int64_t n0, int64_t ns,
                        int32_t* src, int32_t* dst, int num_sms, cudaStream_t s) {
    if (agents <= 0) return;
    int64_t g = (agents + 7) / 8;
    if (g > (int64_t)num_sms * 16) g = (int64_t)num_sms * 16;
    k_trace_edges<<<(unsigned)g, 256, 0, s>>>(coff, cites, agents, n0, ns, src, dst);
}

void launch_lik_features(const LikTrace& T, int exact, int num_sms, cudaStream_t s) {
    int64_t gx = (T.n + 255) / 256;
    if (gx > (int64_t)num_sms * 8) gx = (int64_t)num_sms * 8;
    if (gx < 1) gx = 1;
    const dim3 grid((unsigned)gx, (unsigned)T.epochs);
    if (exact)
        k_lik_features<true><<<grid, 256, 0, s>>>(T);
    else
        k_lik_features<false><<<grid, 256, 0, s>>>(T);
}

}  // namespace pg
