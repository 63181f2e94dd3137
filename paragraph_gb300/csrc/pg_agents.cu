// pg_agents.cu -- per-agent citation sampling of the preferential-attachment epoch.
//
// Replaces kernelCallStage1/_warped/2/3/4 and the fused ABMKernel (src/kernel.cu:17-402,436-573;
// device bodies src/abm.cu:376-565,577-994).  One warp (thinning) or one CTA (enumeration,
// refcompat streams) owns one agent (new paper).  The enumeration sampler does:
//   1. global race: k draws without replacement from the replica's quantised CDF.  Draw i picks the
//      smallest j with cdf[j] - C(j) > y, where C(j) sums the weights already chosen at ids <= j;
//      the warp searches 32-ary (32 probes per round, ballot), which gives the same j as any other
//      search because the function is monotone and integer.  Arrival times are exponential
//      increments E / R with R the remaining weight.
//   2. neighbourhood race: the 2-hop undirected ball of the anchors (forward and backward rows,
//      the reference's GetOneAndTwoHopNeighborhood semantics) is streamed with load-balanced
//      expansion (32 neighbours' rows at a time, owner found by a shuffle search).  Each element j
//      gets the key E_j / w_j with E_j drawn from Philox keyed by (agent, j), so duplicates in the
//      stream share a key and the k smallest distinct keys are found without deduplicating the
//      ball and without depending on traversal order -- the Efraimidis-Spirakis top-k of the
//      reference (src/abm.cu:529-564) in exponential-clock form.
//   3. merge: the first k distinct nodes of the two races by (time, id) are the agent's citations
//      (weights w_j beta^[j in ball]); they are sorted and appended to the forward CSR, and each
//      cited node's in-degree counter returns the edge's rank for the backward append.
// No per-agent O(n) state exists (the reference clears O(n) bitmaps per agent,
// includes/abm.cuh:178-184, src/abm.cu:722-726).
#include "pg_engine.cuh"
#include "pg_rc.cuh"
#include "pg_scan.cuh"
#include "pg_weights.cuh"
#include "pg_csr.cuh"

namespace pg {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ bool key_less(float ka, int ia, float kb, int ib) {
    return ka < kb || (ka == kb && ia < ib);
}

// Offer one candidate per lane to the warp's sorted top-k list (bk, bi)[0..nb) of S.
template <typename SM>
__device__ __forceinline__ void topk_offer(bool valid, float key, int id, int k, int& nb, SM& S) {
    const int lane = lane_id();
    bool pass = valid && (nb < k || key_less(key, id, S.bk[k - 1], S.bi[k - 1]));
    unsigned mask = __ballot_sync(kFull, pass);
    while (mask) {
        const int leader = __ffs(mask) - 1;
        const float ck = __shfl_sync(kFull, key, leader);
        const int cid = __shfl_sync(kFull, id, leader);
        int less_cnt = 0;
        bool dup = false;
        for (int i = lane; i < nb; i += 32) {
            const int ii = S.bi[i];
            if (ii == cid) dup = true;
            if (key_less(S.bk[i], ii, ck, cid)) ++less_cnt;
        }
        if (!__any_sync(kFull, dup)) {
            const int pos = __reduce_add_sync(kFull, less_cnt);
            const int last = nb < k ? nb : k - 1;
            for (int hi = last; hi > pos; hi -= 32) {
                const int i = hi - 1 - lane;
                const bool act = i >= pos;
                float tk = 0.0f;
                int ti = 0;
                if (act) {
                    tk = S.bk[i];
                    ti = S.bi[i];
                }
                __syncwarp();
                if (act) {
                    S.bk[i + 1] = tk;
                    S.bi[i + 1] = ti;
                }
                __syncwarp();
            }
            if (lane == 0) {
                S.bk[pos] = ck;
                S.bi[pos] = cid;
            }
            __syncwarp();
            nb = nb < k ? nb + 1 : k;
        }
        pass = pass && lane != leader && (nb < k || key_less(key, id, S.bk[k - 1], S.bi[k - 1]));
        mask = __ballot_sync(kFull, pass);
    }
}

// The agent's targets sorted (bitonic network in registers, R entries per lane), written to its
// forward row and the edge list, and counted into the in-degree increments.
template <int R>
__device__ __forceinline__ void emit_sorted(const Arena& A, const Replica& rp, int64_t e0, int64_t row0,
                                            const int32_t* arr, int taken, int lane) {
    int v[R];
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = i * 32 + lane < taken ? arr[i * 32 + lane] : 0x7fffffff;
    warp_bitonic<R>(v, lane);
    int32_t* fcol = A.fwd_col + rp.ebase;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int q = i * 32 + lane;
        if (q < taken) {
            const int d = v[i];
            fcol[row0 + q] = d;
            A.e_dst[e0 + q] = d;
            A.e_rank[e0 + q] = atomicAdd(&A.inc[rp.nbase + d], 1);
        }
    }
}

// Append one agent's citations: arrival order to the trace, the sorted row to the forward CSR and
// the epoch edge list, one in-degree increment (whose old value is the edge's rank in the cited
// node's new backward entries) per citation, and the byte-model counters.
template <int KCAP>
__device__ void emit_row(const Arena& A, const Replica& rp, int64_t a, int64_t al, int64_t n,
                         const int32_t* arr, int taken, long long rows, long long elems, long long draws) {
    const int lane = lane_id();
    const int64_t e0 = A.eoff[a];
    if (A.arrivals)
        for (int q = lane; q < taken; q += 32) A.arrivals[e0 + q] = arr[q];
    const int64_t row0 = rp.m + (e0 - A.eoff[rp.abase]);
    if (taken <= 32)
        emit_sorted<1>(A, rp, e0, row0, arr, taken, lane);
    else if (KCAP <= 64 || taken <= 64)
        emit_sorted<2>(A, rp, e0, row0, arr, taken, lane);
    else if (KCAP <= 128 || taken <= 128)
        emit_sorted<4>(A, rp, e0, row0, arr, taken, lane);
    else
        emit_sorted<8>(A, rp, e0, row0, arr, taken, lane);
    if (lane == 0) {
        A.fwd_off[rp.obase + n + al + 1] = row0 + taken;
        atomicAdd(&A.st->rows_expanded, (unsigned long long)rows);
        atomicAdd(&A.st->elems_streamed, (unsigned long long)elems);
        atomicAdd(&A.st->draws, (unsigned long long)draws);
    }
    __syncwarp();
}

#include "pg_thin.cuh"
#include "pg_rc_agent.cuh"

// ---------------------------------------------------------------- the enumeration sampler
// What the enumeration sampler's stream needs.
struct EnCtx {
    const float* w;
    const int64_t* fo;
    const int32_t* fc;
    const BRow* br;
    const int32_t* bc;
    uint64_t seed;
    uint32_t rep, ep, unit;
};

// E_z / w_z, E_z exponential from the Philox stream of (agent, z); valid for a positive weight
__device__ __forceinline__ float en_key(const EnCtx& C, int32_t z, float wz) {
    const u32x4 x = draw(C.seed, kStreamBoost, C.rep, C.ep, C.unit, (uint32_t)z);
    return -logf_pg(u01f(x.x[0])) / wz;
}

// As rc_queue, with the keys left to the flush: an element joins the queue (with its weight) unless an
// estimate of its key is clear of the threshold.  The estimate's E is -ln 2 lg2.approx(u), within
// 2^-22 absolute of the logarithm for u in (1/2, 1] and 2^-22 relative below (PTX), logf_pg is within two ulp:
// 4e-7 + 1e-5 E covers both and the threshold's product.  The logarithm and the division of
// en_key are 50 of a chunk's 165 instructions, and few elements of a ball pass.
__device__ __forceinline__ void en_flush(const EnCtx& C, RcTop& T, RcSmem& S) {
    const int lane = lane_id(), at = (T.nq < 32 ? 0 : T.nq - 32) + lane;
    __syncwarp();
    if (at < T.nq) S.qk[at] = en_key(C, S.qi[at], S.qk[at]);
    rc_flush(T, S);
}
__device__ __forceinline__ void en_queue(const EnCtx& C, RcTop& T, bool valid, int32_t z, float wz, RcSmem& S) {
    const u32x4 x = draw(C.seed, kStreamBoost, C.rep, C.ep, C.unit, (uint32_t)z);
    float l;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(u01f(x.x[0])));
    const float E = -0x1.62e430p-1f * l;
    const bool can = valid && E * (1.0f - 1e-5f) - 4e-7f <= T.thr * wz;
    const unsigned m = __ballot_sync(kFull, can);
    if (!m) return;
    if (can) {
        const int at = T.nq + __popc(m & ((1u << lane_id()) - 1u));
        S.qk[at] = wz;
        S.qi[at] = z;
    }
    T.nq += __popc(m);
    if (T.nq >= 32) en_flush(C, T, S);
}

// The rows of up to 32 papers (this lane's: base, its entries from ys on in their concatenation of tot
// entries), of which this warp takes every nw-th 32-entry chunk from number `warp`.  As in rc_group, four
// chunks' entries and then weights are in flight at once, and one copy of the key code takes them in
// turn.
template <typename I>
__device__ __forceinline__ void en_group(const EnCtx& C, int warp, int nw, const int32_t* base, I ys, I tot, RcTop& T,
                                         RcSmem& S) {
    constexpr int U = 4;
    const int lane = lane_id();
    const int32_t* rel = base - ys;
    for (I t0 = (I)32 * warp; t0 < tot; t0 += (I)32 * nw * U) {
        int32_t z[U];
        bool in[U];
        float w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const I t = t0 + (I)32 * nw * u + lane;
            in[u] = t < tot;
            const I tt = in[u] ? t : tot - 1;
            int o = 0;  // owner: the last lane whose row starts at or before tt
#pragma unroll
            for (int b = 16; b >= 1; b >>= 1)
                if (__shfl_sync(kFull, ys, o + b) <= tt) o += b;
            const int32_t* p = (const int32_t*)__shfl_sync(kFull, (unsigned long long)rel, o);
            z[u] = p[tt];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = C.w[z[u]];
        T.thr = fminf(T.thr, __int_as_float(*(volatile int*)T.shared_thr));
#pragma unroll 1
        for (int u = 0; u < U; ++u) {
            en_queue(C, T, in[0] && w[0] > 0.0f, z[0], w[0], S);
#pragma unroll
            for (int v = 0; v + 1 < U; ++v) {
                z[v] = z[v + 1];
                in[v] = in[v + 1];
                w[v] = w[v + 1];
            }
        }
    }
}
// the same with 64-bit positions, out of line: 2^30 entries or more
__device__ __noinline__ void en_group_long(const EnCtx& C, int warp, int nw, const int32_t* base, int64_t ys, int64_t tot,
                                           RcTop* Tp, RcSmem* S) {
    RcTop T = *Tp;
    en_group<int64_t>(C, warp, nw, base, ys, tot, T, *S);
    *Tp = T;
}

// Shared memory of one agent: the warps' lists, and the global race.
struct EnSmem {
    RcSmem top[kAgentWarps];
    double g_t[kKMax];
    uint64_t c_cq[kKMax];   // chosen so far, by id: their cumulative weight
    uint64_t c_cdf[kKMax];  // and their CDF entries
    int32_t g_id[kKMax];
    int32_t out[kKMax];
    int nb[kAgentWarps];
    int thr;
    long long item;
};

// The global race, one warp: k draws without replacement from the quantised CDF (g_id, g_t); their number.
// The draws depend on one another only through the integer weights left (R): the exponentials are
// taken 32 at a time, one per lane, before the searches and divided by their R after them, so no FP64
// operation but the k additions of t is in the chain (GB300 does two FP64 operations per clock and SM;
// a log and a division per draw, in turn, were two thirds of an agent).
__device__ __forceinline__ int en_race(const Arena& A, const Replica& rp, const EnCtx& C, int k, EnSmem& S) {
    const int lane = lane_id();
    const int64_t n = rp.n;
    const uint64_t* cdf = A.cdf + rp.nbase;
    const int s = cdf_shift(bitsf(rp.wmax_bits), n);
    const double scale = bitsd((uint64_t)(1023 - s) << 52);
    uint64_t R = rp.wq_total;
    double t = 0.0;
    int nc = 0;
    uint64_t own_r = 0;  // R before this lane's draw
    double own_e = 0.0;
    uint64_t own_u = 0;
    // the first round of every search probes the same 32 places
    int64_t p0 = n > 32 ? (int64_t)(lane + 1) * ((n + 31) / 32) - 1 : lane;
    if (p0 > n - 1) p0 = n - 1;
    const uint64_t cdf0 = cdf[p0];
    // the times of draws i0 .. i0 + cnt - 1
    auto times = [&](int i0, int cnt) {
        const double dt = own_e / ((double)own_r * scale);
        for (int q = 0; q < cnt; ++q) {
            t = t + __shfl_sync(kFull, dt, q);
            if (lane == q) S.g_t[i0 + q] = t;
        }
    };
    for (int i = 0; i < k; ++i) {
        if (R == 0) break;
        if ((i & 31) == 0) {
            if (i) times(i - 32, 32);
            const u32x4 x = draw(C.seed, kStreamGlobal, C.rep, C.ep, C.unit, (uint32_t)(i + lane));
            own_e = -log_pg(u01d(x.x[0], x.x[1]));
            own_u = u64of(x.x[2], x.x[3]);
        }
        if (lane == (i & 31)) own_r = R;
        const uint64_t y = mulhi64(__shfl_sync(kFull, own_u, i & 31), R);
        // The answer is the smallest j with cdf[j] - C(j) > y, C(j) the weight chosen at ids <= j.  A chosen
        // c leaves an empty interval at cdf[c] - C(c); those at or below y are the chosen ids below j, and
        // y plus their weight is a place of the plain CDF.
        int m = 0;
        for (int q0 = 0; q0 < nc; q0 += 32) {
            const int q = q0 + lane;
            m += __popc(__ballot_sync(kFull, q < nc && S.c_cdf[q] - S.c_cq[q] <= y));
        }
        const uint64_t chosen = m ? S.c_cq[m - 1] : 0, at = y + chosen;
        // 32-ary search of the CDF
        int64_t lo = 0, hi = n;
        while (true) {
            const int64_t span = hi - lo;
            const int64_t step = span > 32 ? (span + 31) / 32 : 1;
            int64_t p = lo + (int64_t)(lane + 1) * step - 1;
            if (p > hi - 1) p = hi - 1;
            const unsigned b = __ballot_sync(kFull, (lo == 0 && hi == n ? cdf0 : cdf[p]) > at);
            if (b == 0) {  // cdf[hi-1] > at is an invariant; report instead of probing out of range
                if (lane == 0) atomicOr(&A.st->error, kErrArg);
                lo = 0;
                break;
            }
            const int L = __ffs(b) - 1;  // the first lane at or past the answer
            const int64_t pL = lo + (int64_t)(L + 1) * step - 1 < hi ? lo + (int64_t)(L + 1) * step - 1 : hi - 1;
            if (span <= 32) {
                lo = pL;
                break;
            }
            hi = pL + 1;
            if (L > 0) lo += (int64_t)L * step;
        }
        const int j = (int)lo;
        const uint64_t cj = cdf[j], qj = cj - (j > 0 ? cdf[j - 1] : 0);
        // j into the sorted chosen list, at m
        for (int top = nc; top > m; top -= 32) {
            const int q = top - 1 - lane;
            const bool act = q >= m;
            uint64_t tc = 0, tq = 0;
            if (act) {
                tc = S.c_cdf[q];
                tq = S.c_cq[q];
            }
            __syncwarp();
            if (act) {
                S.c_cdf[q + 1] = tc;
                S.c_cq[q + 1] = tq + qj;
            }
            __syncwarp();
        }
        if (lane == 0) {
            S.c_cdf[m] = cj;
            S.c_cq[m] = chosen + qj;
            S.g_id[i] = j;
        }
        __syncwarp();
        ++nc;
        R -= qj;
    }
    if (nc) times((nc - 1) & ~31, ((nc - 1) & 31) + 1);
    __syncwarp();
    return nc;
}

// One CTA per agent: warp 0 draws the global race, the other warps stream the 2-hop ball, each keeping
// the k smallest keys of its chunks; the lists are merged and warp 0 merges the two races and emits.
// What bounds it is latency: the race is k dependent searches, and a ball's elements are two dependent
// loads, a Philox block and a logarithm each.  One warp per agent took both in turn and balls differ a
// hundredfold: 30k nodes, 1,500 agents an epoch, 383 us an epoch; now 150 (4, 5, 8 CTAs per SM: 200,
// 161, 164).
__global__ void __launch_bounds__(kAgentWarps * 32, 6) k_agents_enum(Arena A, int64_t agents) {
    __shared__ EnSmem S;
    if (cta_error(A)) return;
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    while (true) {
        if (threadIdx.x == 0) {
            S.item = (long long)atomicAdd(&A.st->queue_small, 1ull);
            S.thr = 0x7f800000;
        }
        __syncthreads();
        const int64_t a = S.item;
        if (a >= agents) break;
        const int k = A.kk[a];
        const int r = replica_of_agent(A.rep, A.R, a);
        const Replica& rp = A.rep[r];
        const int64_t n = rp.n, al = a - rp.abase;
        EnCtx C;
        C.w = A.w + rp.nbase;
        C.fo = A.fwd_off + rp.obase;
        C.fc = A.fwd_col + rp.ebase;
        C.br = A.brow + rp.nbase;
        C.bc = A.bcol + rp.bbase;
        C.seed = A.seed;
        C.rep = (uint32_t)(r + A.rep_base);
        C.ep = (uint32_t)A.st->epoch;
        C.unit = (uint32_t)al;
        RcTop T = rc_top(k, &S.thr);
        RcSmem& L = S.top[warp];
        long long rows = 0, elems = 0;
        int ng = 0;
        if (warp == 0) {
            ng = en_race(A, rp, C, k, S);
        }
        if (rp.beta_m1 > 0.0) {
            const int na = rp.anchors;
            const u32x4 xa = draw(C.seed, kStreamAnchor, C.rep, C.ep, C.unit, 0);
            const uint32_t xr = lane == 0 ? xa.x[0] : (lane == 1 ? xa.x[1] : (lane == 2 ? xa.x[2] : xa.x[3]));
            const int anchor = (int)bounded32(xr, (uint32_t)n);
            rows += na;
            elems += na;
            // the chunks of all groups are dealt to the streaming warps in turn (warp 0 only counts)
            constexpr int kS = kAgentWarps - 1;
            const int me = warp - 1;
            int turn = 0;
            auto my_turn = [&]() { return me >= 0 && turn == me; };
            if (my_turn()) {
                const float wz = lane < na ? C.w[anchor] : 0.0f;
                en_queue(C, T, wz > 0.0f, anchor, wz, L);
            }
            turn = (turn + 1) % kS;
            for (int ai = 0; ai < na; ++ai) {
                const int x = __shfl_sync(kFull, anchor, ai);
                const int64_t fb = C.fo[x], lf = C.fo[x + 1] - fb;
                int64_t bb, be;
                bspan(C.br, x, bb, be);
                const int64_t deg1 = lf + (be - bb);
                rows += deg1;
                elems += deg1;
                for (int64_t g0 = 0; g0 < deg1; g0 += 32) {
                    const int64_t idx = g0 + lane;
                    const bool valid = idx < deg1;
                    const int y = valid ? (idx < lf ? C.fc[fb + idx] : C.bc[bb + idx - lf]) : 0;
                    if (my_turn()) {
                        const float wy = valid ? C.w[y] : 0.0f;
                        en_queue(C, T, wy > 0.0f, y, wy, L);
                    }
                    turn = (turn + 1) % kS;
                    // a cited paper's forward row has a copy right before its backward entries: one run
                    int64_t yd = 0;
                    const int32_t* base = C.fc;
                    if (valid) {
                        const int64_t yf = C.fo[y], ylf = C.fo[y + 1] - yf;
                        int64_t yb, ye;
                        bspan(C.br, y, yb, ye);
                        yd = ylf + (ye - yb);
                        base = ye > yb ? C.bc + (yb - ylf) : C.fc + yf;
                    }
                    const int64_t incl = warp_incl_scan<int64_t>(yd);
                    const int64_t tot = __shfl_sync(kFull, incl, 31);
                    elems += tot;
                    if (me >= 0) {
                        const int mine = me >= turn ? me - turn : me - turn + kS;
                        if (tot < (1ll << 30)) {
                            en_group<int>(C, mine, kS, base, (int)(incl - yd), (int)tot, T, L);
                        } else {
                            RcTop t = T;
                            en_group_long(C, mine, kS, base, incl - yd, tot, &t, &L);
                            T = t;
                        }
                    }
                    turn = (int)((turn + (tot + 31) / 32) % kS);
                }
            }
            if (T.nq) en_flush(C, T, L);
        }
        if (lane == 0) S.nb[warp] = T.nb;
        __syncthreads();
        // warp 0's list is empty: it takes warp 1's part of the merges
        for (int h = 1; h < kAgentWarps; h <<= 1) {
            if ((warp & (2 * h - 1)) == 0) {
                const int w = warp + h, nw = S.nb[w];
                for (int q0 = 0; q0 < nw; q0 += 32) {
                    const int q = q0 + lane;
                    const bool v = q < nw;
                    T.nb = rc_offer(v, v ? S.top[w].bk[q] : 0.0f, v ? S.top[w].bi[q] : 0, k, T.nb, &L);
                }
                if (lane == 0) S.nb[warp] = T.nb;
            }
            __syncthreads();
        }
        if (warp == 0) {
            // the first k distinct nodes of the two races by (time, id)
            int taken = 0, gi = 0, bj = 0;
            const int nb = T.nb;
            double* b_t = reinterpret_cast<double*>(S.c_cq);  // the race is done with its list
            for (int q = lane; q < nb; q += 32) b_t[q] = (double)L.bk[q] / rp.beta_m1;
            __syncwarp();
            while (taken < k && (gi < ng || bj < nb)) {
                const double tb = bj < nb ? b_t[bj] : 0.0;
                const bool take_g =
                    bj >= nb || (gi < ng && (S.g_t[gi] < tb || (S.g_t[gi] == tb && S.g_id[gi] <= L.bi[bj])));
                const int id = take_g ? S.g_id[gi] : L.bi[bj];
                if (take_g)
                    ++gi;
                else
                    ++bj;
                bool dup = false;
                for (int q = lane; q < taken; q += 32) dup |= (S.out[q] == id);
                if (!__any_sync(kFull, dup)) {
                    if (lane == 0) S.out[taken] = id;
                    __syncwarp();
                    ++taken;
                }
            }
            if (taken != k && lane == 0) atomicOr(&A.st->error, kErrArg);
            emit_row<kKMax>(A, rp, a, al, n, S.out, taken, rows, elems, ng);
        }
        __syncthreads();  // the shared memory is the next agent's
    }
}


// ---------------------------------------------------------------- setup: out-degree + new nodes
__device__ __forceinline__ void d_agent_setup(const Arena& A, int64_t agents, int vb) {
    if (A.st->error) return;
    const int64_t a = (int64_t)vb * blockDim.x + threadIdx.x;
    if (a >= agents) return;
    const int r = replica_of_agent(A.rep, A.R, a);
    const Replica& rp = A.rep[r];
    const int64_t al = a - rp.abase;
    const uint32_t ep = (uint32_t)A.st->epoch;
    const bool rc = A.weight_model == 1;
    // out-degree: Poisson (baseline) or the out-degree bag (refcompat), both as a 257-entry CDF
    const u32x4 x = draw(A.seed, kStreamOutDegree, (uint32_t)(r + A.rep_base), ep, (uint32_t)al, 0);
    const int kraw = poisson_draw(A.tables + (int64_t)r * kTableEntries, kTableEntries,
                                  u64of(x.x[0], x.x[1]));
    int64_t k = kraw < 1 ? 1 : kraw;
    if (rc) {
        const int64_t kmax = rp.n - 1 < kRcMaxOutDegree ? rp.n - 1 : kRcMaxOutDegree;
        if (k > kmax) k = kmax;
    } else {
        if (k > rp.n) k = rp.n;
        if (k > rp.npos) k = rp.npos;
    }
    A.kk[a] = (int32_t)k;
    if (!rc && k > kKSmall) {
        const unsigned long long i = atomicAdd(&A.st->big_count, 1ull);
        A.big_list[i] = (int32_t)a;
    }
    const int64_t slot = rp.nbase + rp.n + al;
    A.pub[slot] = (int32_t)A.st->epoch;
    if (rc) {
        // peak fitness from the power-law table, static window (ABM::AssignPeakFitnessValues,
        // AssignFitnessLagDuration, AssignFitnessPeakDuration; includes/abm.cuh:447-484)
        const u32x4 xf = draw(A.seed, kStreamRcFitness, (uint32_t)(r + A.rep_base), ep, (uint32_t)al, 0);
        A.fit[slot] = (float)rc_peak_draw(A.rc_ftab, u64of(xf.x[0], xf.x[1]));
        A.rc_lag[slot] = 0;
        A.rc_dur[slot] = 1000;
    } else {
        A.fit[slot] = lognormal_fitness(A.seed, (uint32_t)(r + A.rep_base), ep, (uint32_t)al);
    }
    A.indeg[slot] = 0;
    int heavy = 0;
    if (rc) {
        double w3[3], alpha;
        int32_t gen;
        rc_agent_params(A.seed, (uint32_t)(r + A.rep_base), ep, (uint32_t)al, rp.n, rp.rc_w, rp.rc_alpha, w3,
                        &alpha, &gen);
        double* o = A.rc_agent + a * 6;  // the agent kernels read them back (and pg_rc_copy_agents)
        o[0] = w3[0];
        o[1] = w3[1];
        o[2] = w3[2];
        o[3] = alpha;
        o[4] = (double)gen;
        o[5] = (double)k;
    }
    if (!rc && A.sampler == kSamplerThinning && rp.p_global < 1.0) {
        // the anchors (the same draw the agent kernel makes): flag the hubs among them, whose
        // hub-pair rows are the only ones read, and mark the agent heavy when an anchor is a hub or
        // the anchors' rows would not all fit the smaller shared frontier (the agent then tests
        // memberships against global rows); heavy agents are taken first, so none starts late
        const u32x4 xa = draw(A.seed, kStreamAnchor, (uint32_t)(r + A.rep_base), ep, (uint32_t)al, 0);
        const int64_t* fo = A.fwd_off + rp.obase;
        const BRow* br = A.brow + rp.nbase;
        int64_t zsize = rp.anchors;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (i >= rp.anchors) break;
            const int64_t x = bounded32(xa.x[i], (uint32_t)rp.n);
            const int hs = A.hslot[rp.nbase + x];
            if (hs >= 0) {
                atomicOr(&A.hub_need[(int64_t)r * (kHeavyMax / 32) + (hs >> 5)], 1u << (hs & 31));
                heavy = 1;
            } else {
                zsize += (fo[x + 1] - fo[x]) + blen(br, x);
            }
        }
        if (zsize > kZCap / 2) heavy = 1;
        if (heavy && k <= kKSmall) A.heavy_list[atomicAdd(&A.st->heavy_count, 1ull)] = (int32_t)a;
    }
    A.heavy_mark[a] = heavy;
    if (A.anchors_out) {
        // the same draw the agent kernels make for the neighbourhood (recorded for traces)
        const u32x4 xa = draw(A.seed, kStreamAnchor, (uint32_t)(r + A.rep_base), ep, (uint32_t)al, 0);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            A.anchors_out[a * 4 + i] = i < rp.anchors ? (int32_t)bounded32(xa.x[i], (uint32_t)rp.n) : -1;
    }
}

__global__ void __launch_bounds__(256) k_agent_setup(Arena A, int64_t agents) {
    pdl_begin();
    d_agent_setup(A, agents, blockIdx.x);
}

// Refcompat, after the setup: a generator with many row entries, or a few long ones, makes a long
// 2-hop stream; such agents are listed for the CTA-wide pass (k_rc_big), mark = list slot + 1.  One
// warp per agent, a lane per generator row entry: the row lengths of a generator are loads that
// depend on its row, and one thread taking them in turn was latency all through.  Setup and route of an
// epoch of 7,000 agents: 75 us in one thread per agent, now 8 + 10 us.
__global__ void __launch_bounds__(256) k_rc_route(Arena A, int64_t agents) {
    if (A.st->error) return;
    const int lane = lane_id();
    const int64_t a = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (a >= agents || A.kk[a] < 2) return;
    const int r = replica_of_agent(A.rep, A.R, a);
    const Replica& rp = A.rep[r];
    const int32_t gen = (int32_t)A.rc_agent[a * 6 + 4];
    const int64_t* fo = A.fwd_off + rp.obase;
    const BRow* br = A.brow + rp.nbase;
    int64_t gb0, gb1;
    bspan(br, gen, gb0, gb1);
    const int64_t f0 = fo[gen], lf = fo[gen + 1] - f0, gd = lf + (gb1 - gb0);
    int64_t len = 0;
    for (int64_t q = lane; q < gd; q += 32) {
        const int32_t y = q < lf ? A.fwd_col[rp.ebase + f0 + q] : A.bcol[rp.bbase + gb0 + (q - lf)];
        len += (fo[y + 1] - fo[y]) + blen(br, y);
    }
    len = warp_sum(len);
    if (lane == 0 && (gd >= kRcBigGd || len >= kRcBigStream)) {
        const unsigned long long q = atomicAdd(&A.st->rc_big_count, 1ull);
        if (q < (unsigned long long)kRcBigCap) {
            A.heavy_list[q] = (int32_t)a;
            A.heavy_mark[a] = (int)q + 1;
            // a stream of several parts takes an item more for each; without room it stays one
            int parts = len >= 64ll * kRcPart ? 64 : (int)((len + kRcPart - 1) / kRcPart);
            int first = 0;
            if (parts > 1) {
                const unsigned long long i = atomicAdd(&A.st->rc_part_count, (unsigned long long)(parts - 1));
                if (i + (unsigned long long)(parts - 1) <= (unsigned long long)kRcParts) {
                    first = (int)i;
                    for (int p = 1; p < parts; ++p) A.rc_item[i + p - 1] = make_int2((int)q, p);
                } else {
                    for (unsigned long long j = i; j < (unsigned long long)kRcParts && j < i + parts - 1; ++j)
                        A.rc_item[j] = make_int2(-1, 0);  // reserved, not used
                    parts = 1;
                }
            }
            A.rc_part[q] = make_int2(parts < 1 ? 1 : parts, first);
        }
    }
}

// After the edge-offset scan: totals and capacity checks.
__device__ __forceinline__ void d_edges_check(const Arena& A, int64_t agents) {
    if (A.st->error) return;
    const int64_t E = A.eoff[agents];
    if (threadIdx.x == 0) {
        A.st->edges = E;
        if (E > A.edge_cap) atomicOr(&A.st->error, kErrCapacity);
    }
    for (int r = threadIdx.x; r < A.R; r += blockDim.x) {
        const Replica& rp = A.rep[r];
        const int64_t er = A.eoff[rp.abase + rp.delta] - A.eoff[rp.abase];
        if (rp.m + er > rp.m_cap) atomicOr(&A.st->error, kErrCapacity);
    }
}

__global__ void k_edges_check(Arena A, int64_t agents) {
    pdl_begin();
    d_edges_check(A, agents);
}

// Shapes of the k <= 64 thinning kernel (pg_tuning.small_hash = HS): 0 -- a 2048-slot frontier hash
// and 512-entry stage buffers (the lean instance: 1024 slots, a filter of 512 words and 768-entry stages); 1 -- 1024
// slots, a filter of 256 words and 1024-entry stages; both 4 CTAs per SM.  The k <= 256 kernel always
// has 1024 slots, 256 filter words and 512-entry stages.  Shapes with more resident warps were
// measured on the PA workload and were slower: 1024 slots and 512-entry stages at 5 CTAs per SM (96
// registers) by 9 %, and 2048 slots and 256-entry stages at 5 CTAs per SM with the heavy agents'
// instance out of line (the lean one then fits 96 registers) by 8 %.
template <int KCAP, int HS>
struct ThinStage {
    static constexpr int value = (KCAP <= kKSmall && HS == 1) ? 1024 : 512;
};
template <int KCAP, int HS>
struct ThinHash {
    static constexpr int value = (KCAP <= kKSmall && HS == 0) ? 2 * kZCap : kZCap;
};
template <int KCAP, int HS>
__host__ __device__ constexpr size_t thin_smem_bytes() {
    return sizeof(ThinSmem<KCAP, ThinHash<KCAP, HS>::value, ThinStage<KCAP, HS>::value>) * kAgentWarps;
}

// The agent loop of one warp of the thinning sampler.  The warp's shared memory is dsm + warp * stride
// (the calling kernel's dynamic shared memory; stride >= sizeof of this variant's ThinSmem).
template <int KCAP, bool BIG, int HS = 0>
__device__ __forceinline__ void d_agents(const Arena& A, int64_t agents, unsigned char* dsm, size_t stride) {
    constexpr int HCAP = ThinHash<KCAP, HS>::value;
    constexpr int STAGE = ThinStage<KCAP, HS>::value;
    using Smem = ThinSmem<KCAP, HCAP, STAGE>;
    Smem& S = *reinterpret_cast<Smem*>(dsm + (threadIdx.x >> 5) * stride);
    if (A.st->error) return;
    const int lane = lane_id();
    // the small thinning kernel walks the heavy list, then every agent not on it
    constexpr bool kHeavyFirst = !BIG;
    const int64_t hc = kHeavyFirst ? (int64_t)A.st->heavy_count : 0;
    const int64_t limit = BIG ? (int64_t)A.st->big_count : agents + hc;
    uint32_t phase = 0;
    if (lane == 0) {
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
    }
    fence_proxy_async();
    __syncwarp();
    while (true) {
        long long q = 0;
        if (lane == 0)
            q = (long long)atomicAdd(BIG ? &A.st->queue_big : &A.st->queue_small, 1ull);
        q = __shfl_sync(kFull, q, 0);
        if (q >= limit) break;
        int64_t a;
        bool general = true;  // heavy agents take the general instance
        if (BIG) {
            a = (int64_t)A.big_list[q];
            general = A.heavy_mark[a] != 0;  // the rest lean: 6.00 to 5.70 ms, 12 epochs of Poisson(55)
        } else if (q < hc) {
            a = (int64_t)A.heavy_list[q];
        } else {
            a = q - hc;
            if (kHeavyFirst && A.heavy_mark[a]) continue;
            general = !kHeavyFirst;
        }
        const int k = A.kk[a];
        if (!BIG && k > KCAP) continue;
        const bool ok = general ? process_agent_thin<KCAP, HCAP, STAGE, true>(A, a, k, S, phase)
                                : process_agent_thin<KCAP, HCAP, STAGE, false>(A, a, k, S, phase);
        if (!ok) break;
    }
    // every copy this warp issued has been waited for: the barriers' memory can be reused
    __syncwarp();
    if (lane == 0) {
        mbar_inval(&S.bar[0]);
        mbar_inval(&S.bar[1]);
    }
    __syncwarp();
}

template <int KCAP, bool BIG, int HS = 0>
__global__ void __launch_bounds__(kAgentWarps * 32, 4) k_agents(Arena A, int64_t agents) {
    pdl_begin();
    // two stage buffers per warp go past 48 KiB: dynamic
    extern __shared__ __align__(16) unsigned char agent_dsm[];
    constexpr size_t stride = thin_smem_bytes<KCAP, HS>() / kAgentWarps;
    d_agents<KCAP, BIG, HS>(A, agents, agent_dsm, stride);
}

// LISTED: the agents whose 2-hop lists k_rc_big has made; else all others, which do not wait for it.
template <bool LISTED>
__global__ void __launch_bounds__(kAgentWarps * 32, 6) k_agents_rc(Arena A, int64_t agents) {
    __shared__ RcSmem smem[kAgentWarps];
    __shared__ int32_t arr[kAgentWarps][kKMax];  // citations in arrival order
    __shared__ __align__(16) int32_t set[kAgentWarps][1 << kRcSetBits];
    if (A.st->error) return;
    RcSmem& S = smem[threadIdx.x >> 5];
    const int lane = lane_id();
    const unsigned long long listed = A.st->rc_big_count;
    const int64_t limit = LISTED ? (int64_t)(listed < (unsigned long long)kRcBigCap ? listed : kRcBigCap) : agents;
    while (true) {
        long long q = 0;
        if (lane == 0) q = (long long)atomicAdd(LISTED ? &A.st->queue_big : &A.st->queue_small, 1ull);
        q = __shfl_sync(kFull, q, 0);
        if (q >= limit) break;
        const int64_t a = LISTED ? A.heavy_list[q] : q;
        if (!LISTED && A.heavy_mark[a] > 0) continue;
        process_agent_rc(A, a, A.kk[a], S, arr[threadIdx.x >> 5], set[threadIdx.x >> 5]);
    }
}

// The 2-hop streams of the refcompat agents that k_rc_route listed (long streams), a CTA per work item: a
// stream, or a part of one that is longer than kRcPart entries (the longest, alone on a CTA, was the
// launch's tail).  Each warp keeps the top of its share; the lists are merged pairwise (dropping entries
// that two warps both reached; the smallest distinct (key, id) pairs do not depend on the merge
// order), an agent's last item merges its items' lists, and the sorted ids and the stream's counters
// are stored for k_agents_rc<true>.  Bound by issue (about 165 instructions per 32 elements, half of them
// Philox) and by instruction fetch.  200k papers, 10 epochs of 3 %: 0.60 ms an epoch in the last with
// FP64 keys, 0.09 now.
constexpr int kRcBigWarps = 8;
constexpr int kRcBigSetBits = 12;  // the generator's 1-hop set: 4,096 slots

__global__ void __launch_bounds__(kRcBigWarps * 32, 3) k_rc_big(Arena A) {
    __shared__ RcSmem sm[kRcBigWarps];
    __shared__ __align__(16) int32_t set[1 << kRcBigSetBits];
    __shared__ int s_nb[kRcBigWarps];
    __shared__ long long s_cnt[2];
    __shared__ long long s_item;
    // the warps' smallest full-list threshold (float bits); an odd score was met; the agent's last item
    __shared__ int s_thr, s_odd, s_last;
    if (cta_error(A)) return;
    const int warp = threadIdx.x >> 5, lane = lane_id();
    RcSmem& S = sm[warp];
    const long long listed = (long long)A.st->rc_big_count;
    const long long agents = listed < kRcBigCap ? listed : kRcBigCap;
    const long long asked = (long long)A.st->rc_part_count;
    const long long more = asked < kRcParts ? asked : kRcParts;
    // one pairwise merge of the warps' lists, log2(warps) rounds: warp w takes warp w + h's list when
    // w % 2h == 0; the result is warp 0's
    auto merge = [&](int cap, int nb) {
        if (lane == 0) s_nb[warp] = nb;
        __syncthreads();
        for (int h = 1; h < kRcBigWarps; h <<= 1) {
            if ((warp & (2 * h - 1)) == 0) {
                const int w = warp + h;
                const int nw = s_nb[w];
                for (int q0 = 0; q0 < nw; q0 += 32) {
                    const int q = q0 + lane;
                    const bool v = q < nw;
                    nb = rc_offer(v, v ? sm[w].bk[q] : 0.0f, v ? sm[w].bi[q] : 0, cap, nb, &S);
                }
                if (lane == 0) s_nb[warp] = nb;
            }
            __syncthreads();
        }
        return nb;
    };
    // the whole stream's part `part` of `parts` into the warps' merged list
    auto walk = [&](const RcCtx& X, const int32_t* H, int part, int parts, bool exact, int cap) {
        if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
        if (threadIdx.x == 0) {
            s_thr = 0x7f800000;
            s_odd = 0;
        }
        __syncthreads();
        RcTop T = rc_top(cap, &s_thr);
        long long rows = 0, elems = 0;
        const bool odd = rc_2hop_slice(X, warp, kRcBigWarps, part, parts, exact, T, rows, elems, S, H, kRcBigSetBits);
        if (lane == 0) {
            atomicAdd((unsigned long long*)&s_cnt[0], (unsigned long long)rows);
            atomicAdd((unsigned long long*)&s_cnt[1], (unsigned long long)elems);
            if (odd) s_odd = 1;
        }
        return merge(cap, T.nb);
    };
    while (true) {
        // the items of many-part streams first (they are the long ones), then every agent's first part
        if (threadIdx.x == 0) s_item = (long long)atomicAdd(&A.st->rc_big_queue, 1ull);
        __syncthreads();
        const long long q = s_item;
        __syncthreads();
        if (q >= agents + more) break;
        const int2 own = q < more ? A.rc_item[q] : make_int2((int)(q - more), 0);
        const int slot = own.x, part = own.y;
        if (slot < 0) continue;
        const int2 pf = A.rc_part[slot];
        const int64_t a = A.heavy_list[slot];
        RcCtx X;
        rc_ctx(A, a, X);
        const int k = A.kk[a];
        const int kcap = k < kKMax ? k : kKMax;
        const int32_t* H = rc_set(X, set, kRcBigSetBits, (int)threadIdx.x, kRcBigWarps * 32, true) ? set : nullptr;
        int nb = walk(X, H, part, pf.x, false, kcap + kRcSlack);
        long long rows = s_cnt[0], elems = s_cnt[1];
        bool odd = s_odd != 0;
        if (pf.x > 1) {
            // the item's list and counters to memory; the agent's last item merges them all
            const int64_t it = part == 0 ? slot : kRcBigCap + pf.y + part - 1;
            if (warp == 0) {
                int2* l = A.rc_item_list + it * kRcItemList;
                for (int i = lane; i < nb; i += 32) __stcg(l + i, make_int2(__float_as_int(S.bk[i]), S.bi[i]));
                if (lane == 0) {
                    long long* m = A.rc_item_meta + it * 4;
                    __stcg(m + 0, (long long)nb);
                    __stcg(m + 1, rows);
                    __stcg(m + 2, elems);
                    __stcg(m + 3, (long long)odd);
                }
                __threadfence();
                __syncwarp();
                if (lane == 0) s_last = atomicAdd(&A.rc_ticket[slot], 1u) == (unsigned)pf.x - 1u;
            }
            __syncthreads();
            const bool last = s_last != 0;
            __syncthreads();
            if (!last) continue;
            __threadfence();
            if (threadIdx.x == 0) A.rc_ticket[slot] = 0u;
            nb = 0;
            rows = elems = 0;
            odd = false;
            for (int p = 0; p < pf.x; ++p) {
                const int64_t ip = p == 0 ? slot : kRcBigCap + pf.y + p - 1;
                const long long* m = A.rc_item_meta + ip * 4;
                rows += __ldcg(m + 1);
                elems += __ldcg(m + 2);
                odd |= __ldcg(m + 3) != 0;
                if (p % kRcBigWarps != warp) continue;
                const int np = (int)__ldcg(m);
                const int2* l = A.rc_item_list + ip * kRcItemList;
                for (int i0 = 0; i0 < np; i0 += 32) {
                    const bool v = i0 + lane < np;
                    const int2 e = v ? __ldcg(l + i0 + lane) : make_int2(0, 0);
                    nb = rc_offer(v, __int_as_float(e.x), e.y, kcap + kRcSlack, nb, &S);
                }
            }
            nb = merge(kcap + kRcSlack, nb);
        }
        // the approximate keys first; the exact ones for the whole stream when those cannot decide
        if (warp == 0) {
            const bool done = !odd && rc_refine(X, kcap, nb, S);
            if (lane == 0) s_last = done ? 1 : 0;
        }
        __syncthreads();
        const bool done = s_last != 0;
        __syncthreads();
        if (!done) {
            nb = walk(X, H, 0, 1, true, kcap);
            rows = s_cnt[0];
            elems = s_cnt[1];
        }
        if (warp == 0) {
            int32_t* ids = A.rc_big_id + (int64_t)slot * kKMax;
            for (int i = lane; i < nb; i += 32) ids[i] = S.bi[i];
            if (lane == 0) {
                long long* meta = A.rc_big_meta + (int64_t)slot * 3;
                meta[0] = nb;
                meta[1] = rows;
                meta[2] = elems;
            }
        }
        __syncthreads();  // the lists and counters are reused by the next item
    }
}

static int g_blocks_rc = 0;

cudaError_t init_rc_kernels() {
    if (g_blocks_rc) return cudaSuccess;
    const cudaError_t e =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_blocks_rc, k_agents_rc<false>, kAgentWarps * 32, 0);
    if (g_blocks_rc < 1) g_blocks_rc = 1;
    return e;
}

void launch_rc_agents(const Arena& A, int64_t agents, int num_sms, cudaStream_t s, cudaStream_t side, cudaEvent_t fork,
                      cudaEvent_t join) {
    if (agents <= 0) return;
    int64_t grid = (int64_t)num_sms * (g_blocks_rc ? g_blocks_rc : 1);
    const int64_t need = (agents + kAgentWarps - 1) / kAgentWarps;
    if (grid > need) grid = need;
    // the long streams beside the other agents; then the agents that read their lists
    cudaEventRecord(fork, s);
    cudaStreamWaitEvent(side, fork, 0);
    k_rc_big<<<(unsigned)num_sms * 2, kRcBigWarps * 32, 0, side>>>(A);
    cudaEventRecord(join, side);
    k_agents_rc<false><<<(unsigned)grid, kAgentWarps * 32, 0, s>>>(A, agents);
    cudaStreamWaitEvent(s, join, 0);
    k_agents_rc<true><<<(unsigned)grid, kAgentWarps * 32, 0, s>>>(A, agents);
}

static int g_blocks_enum = 0, g_blocks_big = 0;  // enumeration; thinning, k > 64
static int g_blocks_hs[2] = {0, 0};             // thinning, k <= 64, by shape (small_hash)

// The hub pairs (for the hubs the setup found among the anchors) need the setup alone, and the agents need
// them and the offsets: beside the scan and its check they cost the epoch little of their own (three epochs of
// 5,000 agents: 654 to 644 us).
void launch_agent_setup(const Arena& A, int64_t agents, int num_sms, cudaStream_t s, cudaStream_t side,
                        cudaEvent_t fork, cudaEvent_t join) {
    if (agents <= 0) return;
    launch_dependent(k_agent_setup, (agents + 255) / 256, 256, 0, s, A, agents);
    if (A.weight_model == 1) {
        k_rc_route<<<(unsigned)((agents + 7) / 8), 256, 0, s>>>(A, agents);
    }
    if (side) {
        cudaEventRecord(fork, s);
        cudaStreamWaitEvent(side, fork, 0);
        launch_hub_pairs(A, num_sms, side);
        cudaEventRecord(join, side);
    }
    scan_impl<int32_t>(A.kk, A.eoff, agents, A.blocksum, s, false);
    launch_dependent(k_edges_check, 1, 256, 0, s, A, agents);
    if (side) cudaStreamWaitEvent(s, join, 0);
}

// Occupancy of the persistent agent kernels; called once per process before any capture.
cudaError_t init_agent_kernels() {
    if (g_blocks_enum) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    const int th = kAgentWarps * 32;
    int en = 0;
    constexpr size_t d0 = thin_smem_bytes<kKSmall, 0>(), d1 = thin_smem_bytes<kKSmall, 1>(),
                     db = thin_smem_bytes<kKMax, 0>();
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_agents<kKSmall, false, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d0);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_agents<kKSmall, false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_agents<kKMax, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)db);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_blocks_hs[0], k_agents<kKSmall, false, 0>, th, d0);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_blocks_hs[1], k_agents<kKSmall, false, 1>, th, d1);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_blocks_big, k_agents<kKMax, true>, th, db);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&en, k_agents_enum, th, 0);
    if (g_blocks_big < 1) g_blocks_big = 1;
    for (int& b : g_blocks_hs)
        if (b < 1) b = 1;
    g_blocks_enum = en < 1 ? 1 : en;
    return e;
}

// Warps of the thinning kernels that can be resident at once (the rows of the global anchor table).
int64_t agent_warp_slots(int num_sms) {
    int mb = g_blocks_big;
    for (int b : g_blocks_hs) mb = b > mb ? b : mb;
    const int64_t sep = (int64_t)num_sms * mb * kAgentWarps;
    const int64_t per = (int64_t)(2 * num_sms) * 8;  // the epoch kernel: 2 CTAs of 8 warps per SM at most
    return sep > per ? sep : per;
}

int agent_occupancy(int thin, int small_hash) {
    if (!thin) return g_blocks_enum;
    return g_blocks_hs[small_hash == 1 ? 1 : 0];
}

void launch_agents(const Arena& A, int64_t agents, int num_sms, cudaStream_t s) {
    if (agents <= 0) return;
    const int t = A.sampler == kSamplerThinning ? 1 : 0;
    const int hs = t && A.tune_small_hash == 1 ? 1 : 0;
    int per_sm = agent_occupancy(t, hs);
    if (A.tune_agent_ctas > 0 && A.tune_agent_ctas < per_sm) per_sm = A.tune_agent_ctas;
    const int64_t need = t ? (agents + kAgentWarps - 1) / kAgentWarps : agents;
    int64_t grid = (int64_t)num_sms * per_sm;
    if (grid > need) grid = need;
    const int th = kAgentWarps * 32;
    if (!t) {
        k_agents_enum<<<(unsigned)grid, th, 0, s>>>(A, agents);
        return;
    }
    if (hs == 1)
        launch_dependent(k_agents<kKSmall, false, 1>, grid, th, thin_smem_bytes<kKSmall, 1>(), s, A, agents);
    else
        launch_dependent(k_agents<kKSmall, false, 0>, grid, th, thin_smem_bytes<kKSmall, 0>(), s, A, agents);
    launch_dependent(k_agents<kKMax, true>, num_sms * g_blocks_big, th, thin_smem_bytes<kKMax, 0>(), s, A, agents);
}


// ---------------------------------------------------------------- one persistent kernel per epoch
// The thinning epoch of every replica as ONE cooperative launch (one CTA pair per SM, all CTAs
// resident), instead of the two dozen launches above.  The phases are the same device bodies the
// separate kernels run -- tiles and blocks walked by the CTAs in turn, single-CTA steps on one CTA,
// grid-stride loops as they are -- so every result is bit-identical to the launch sequence.  A grid
// barrier separates dependent phases; independent stages share a phase (the hub index beside the
// weights and the CDF, the old-entry copy beside the placement of the new ones).  Each barrier
// wait is bounded: on expiry the CTA sets the timeout bit of the error word and goes on, and every
// later phase sees the bit and skips its work, so the launch always ends.
constexpr int kEpochThreads = 256;
constexpr int kEpochWarps = kEpochThreads / 32;
constexpr uint32_t kGridWaitPolls = 1u << 24;  // with a 64 ns back-off: about a second at least

__device__ __forceinline__ void grid_sync(const Arena& A) {
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned int* gen = &A.st->gbar_gen;
        const unsigned int g = *gen;
        __threadfence();
        if (atomicAdd(&A.st->gbar_count, 1u) == gridDim.x - 1) {
            atomicExch(&A.st->gbar_count, 0u);
            __threadfence();
            atomicAdd(&A.st->gbar_gen, 1u);
        } else {
            for (uint32_t i = 0; *gen == g; ++i) {
                if (i >= kGridWaitPolls) {
                    atomicOr(&A.st->error, kErrTimeout);
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    __syncthreads();
}

// per-warp shared memory of the agent phase: the larger of the two thinning variants it runs (the
// k <= 64 one with the 1024-slot frontier and 1024-entry stages)
constexpr size_t kEpochWarpSmem =
    thin_smem_bytes<kKSmall, 1>() > thin_smem_bytes<kKMax, 0>() ? thin_smem_bytes<kKSmall, 1>() / kAgentWarps
                                                                  : thin_smem_bytes<kKMax, 0>() / kAgentWarps;
constexpr size_t kEpochSmem = kEpochWarps * kEpochWarpSmem;

__global__ void __launch_bounds__(kEpochThreads, 2) k_epoch(Arena A, int64_t epoch, int64_t agents, int G) {
    extern __shared__ __align__(16) unsigned char ep_dsm[];
    const int T = A.ntiles;
    const int hub_items = A.R * G;
    // epoch start: new-node counts and agent offsets
    if (blockIdx.x == 0) d_epoch_begin(A, epoch, -1);
    grid_sync(A);
    // hub histogram and weights
    for (int t = blockIdx.x; t < T; t += gridDim.x) {
        d_hub_hist(A, t);
        d_weights(A, t);
        __syncthreads();
    }
    grid_sync(A);
    // hub threshold; tile-local CDF scans
    for (int r = blockIdx.x; r < A.R; r += gridDim.x) d_hub_pick(A, r);
    for (int t = blockIdx.x; t < T; t += gridDim.x) {
        d_cdf_tiles(A, t);
        __syncthreads();
    }
    grid_sync(A);
    // hubs leaving and joining; tile offsets of the CDF (on the last CTA, so CTA 0 is not the only
    // one with extra work)
    for (int t = blockIdx.x; t < T; t += gridDim.x) d_hub_collect(A, t);
    if (blockIdx.x == gridDim.x - 1) d_tile_scan(A);
    grid_sync(A);
    // hub bits; CDF offsets and guide marks
    d_hub_assign(A);
    for (int t = blockIdx.x; t < T; t += gridDim.x) {
        d_cdf_add(A, t);
        __syncthreads();
    }
    grid_sync(A);
    // bits cleared by the hubs that left; guide table; per-agent out-degrees, new nodes, heavy lists
    for (int i = blockIdx.x; i < hub_items; i += gridDim.x) d_hub_mask<false>(A, G, i);
    for (int t = blockIdx.x; t < T; t += gridDim.x) {
        d_guide_fill(A, t);
        __syncthreads();
    }
    const int setup_blocks = (int)((agents + 255) / 256);
    for (int b = blockIdx.x; b < setup_blocks; b += gridDim.x) d_agent_setup(A, agents, b);
    grid_sync(A);
    // bits set by the hubs that joined; edge offsets: exclusive scan of the out-degrees (reduce,
    // block sums, apply)
    for (int i = blockIdx.x; i < hub_items; i += gridDim.x) d_hub_mask<true>(A, G, i);
    const int nb = (int)((agents + kScanBlock - 1) / kScanBlock);
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        d_scan_reduce<int32_t>(A.kk, agents, A.blocksum, b);
        __syncthreads();
    }
    grid_sync(A);
    if (blockIdx.x == 0) d_scan_blocksums(A.blocksum, nb);
    grid_sync(A);
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        d_scan_apply<int32_t>(A.kk, agents, A.blocksum, nb, A.eoff, b);
        __syncthreads();
    }
    grid_sync(A);
    // capacity check; hub-pair rows for the hub anchors
    if (blockIdx.x == 0) d_edges_check(A, agents);
    for (int i = blockIdx.x; i < hub_items; i += gridDim.x) {
        d_hub_pairs(A, G, i);
        __syncthreads();
    }
    grid_sync(A);
    // the agents: k <= 256 queue, then the k <= 64 queue (heavy list first)
    d_agents<kKMax, true>(A, agents, ep_dsm, kEpochWarpSmem);
    d_agents<kKSmall, false, 1>(A, agents, ep_dsm, kEpochWarpSmem);
    grid_sync(A);
    // backward append: the cited rows' new lengths, new spans for the rows that outgrew theirs
    d_bwd_grow(A, agents);
    grid_sync(A);
    // the moved rows' old entries copied, new entries placed (disjoint positions)
    d_bwd_reloc(A);
    d_bwd_place(A, agents);
    d_copy_out(A, agents, reinterpret_cast<int32_t*>(ep_dsm));  // this phase uses no other shared memory
    grid_sync(A);
    // appended segments sorted
    d_sort_small(A);
    __syncthreads();
    d_sort_large(A, reinterpret_cast<uint32_t*>(ep_dsm), (int64_t)(kEpochSmem / 4));
    grid_sync(A);
    if (blockIdx.x == 0) d_epoch_end(A, agents);
}

static int g_epoch_ctas = 0;

cudaError_t init_epoch_kernel(int num_sms) {
    if (g_epoch_ctas) return cudaSuccess;
    int dev = 0, coop = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEpochSmem);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_epoch, kEpochThreads, kEpochSmem);
    if (e != cudaSuccess || !coop || per_sm < 1) {
        cudaGetLastError();
        g_epoch_ctas = -1;  // not available on this device: the launch sequence is used
        return cudaSuccess;
    }
    g_epoch_ctas = num_sms * (per_sm < 2 ? per_sm : 2);
    return cudaSuccess;
}

int epoch_kernel_ctas() { return g_epoch_ctas > 0 ? g_epoch_ctas : 0; }

cudaError_t launch_epoch_kernel(const Arena& A, int64_t epoch, int64_t agents, cudaStream_t s) {
    if (g_epoch_ctas <= 0) return cudaErrorNotSupported;
    Arena a = A;
    int G = hub_ctas(A.R, g_epoch_ctas / 2);
    void* args[] = {&a, &epoch, &agents, &G};
    return cudaLaunchCooperativeKernel((const void*)k_epoch, dim3((unsigned)g_epoch_ctas), dim3(kEpochThreads), args,
                                       kEpochSmem, s);
}

}  // namespace pg
