// pg_rc_agent.cuh -- the refcompat agent: ParAGraph's own per-paper citation rule (included by
// pg_agents.cu after the top-k and emit helpers).
//
// One warp owns one agent (new paper) of out-degree d and, in arrival order, cites
//   its generator g (uniform over the existing papers; getGeneratorNode, src/abm.cu:567-574),
//   a paper of its own epoch when it is a same-year citer (MakeSameYearCitations, src/abm.cu:376-384),
//   the `in` best of the generator's 1-hop set N1 and the `out` best of its 2-hop set N2 (N2 without
//   N1 and g) by Efraimidis-Spirakis keys on the linear score (ABMKernelStage2/3 with
//   MakePopulateCitations, src/abm.cu:461-565; budget split src/kernel.cu:230-273,320-343),
//   and uniformly drawn papers from [0, n-1) that are neither g nor already cited
//   (MakeUniformRandomCitations, src/abm.cu:386-432).
// The 2-hop stream is load-balanced over the warp: 32 entries of N1 at a time, their rows
// concatenated and split evenly over the lanes.  Keys are functions of (agent, node), so the stream
// is never deduplicated and its order does not matter.

constexpr int kRcSlack = 8;          // list entries beyond k while keys are approximate
constexpr int kRcList = kKMax + 32;  // list capacity: kKMax + kRcSlack in whole warps
constexpr int kRcSetBits = 8;        // a warp's set of its generator's 1-hop ids: 256 slots

struct RcSmem {
    float bk[kRcList];    // top-k keys, ascending
    int32_t bi[kRcList];  // their ids
    int32_t out[kRcList]; // scratch
    float qk[64];         // elements below the list's threshold, not yet offered (rc_queue)
    int32_t qi[64];
};

__device__ __forceinline__ bool rc_in_rows(const int64_t* fo, const int32_t* fc, const BRow* br,
                                           const int32_t* bc, int32_t g, int32_t v) {
    if (contains(fc, fo[g], fo[g + 1], v)) return true;
    int64_t b0, b1;
    bspan(br, g, b0, b1);
    return contains(bc, b0, b1, v);
}

// Offer one candidate per lane to the top-k list.  When more than two pass the list's threshold
// they are merged as a batch: sorted across the lanes by (key, id), duplicates dropped (equal
// neighbours, or already listed), and list entries and candidates written at their merged ranks,
// the first k kept.  The result is the one candidate-by-candidate insertion gives: the k smallest
// distinct (key, id) pairs offered.  S.out is scratch.
__device__ __forceinline__ void rc_topk_offer(bool valid, float key, int id, int k, int& nb, RcSmem& S) {
    const int lane = lane_id();
    const bool pass = valid && (nb < k || key_less(key, id, S.bk[k - 1], S.bi[k - 1]));
    const unsigned pm = __ballot_sync(kFull, pass);
    if (!pm) return;
    if (__popc(pm) <= 2) {
        topk_offer(valid, key, id, k, nb, S);
        return;
    }
    float ck = pass ? key : __int_as_float(0x7f800000);  // not passing: +inf, sorted last
    int cid = pass ? id : 0x7fffffff;
#pragma unroll
    for (int w = 2; w <= 32; w <<= 1) {
#pragma unroll
        for (int j = w >> 1; j > 0; j >>= 1) {
            const float ok = __shfl_xor_sync(kFull, ck, j);
            const int oi = __shfl_xor_sync(kFull, cid, j);
            const bool up = (lane & w) == 0, lower = (lane & j) == 0;
            if ((lower == up) ? key_less(ok, oi, ck, cid) : key_less(ck, cid, ok, oi)) {
                ck = ok;
                cid = oi;
            }
        }
    }
    const int np = __popc(pm);
    const float pk = __shfl_up_sync(kFull, ck, 1);
    const int pi = __shfl_up_sync(kFull, cid, 1);
    bool keep = lane < np && !(lane > 0 && pk == ck && pi == cid);
    int below = 0;  // list entries ahead of the candidate
    if (lane < np) {
        int lo = 0, hi = nb;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (key_less(S.bk[mid], S.bi[mid], ck, cid))
                lo = mid + 1;
            else
                hi = mid;
        }
        below = lo;
        if (lo < nb && S.bk[lo] == ck && S.bi[lo] == cid) keep = false;
    }
    const unsigned km = __ballot_sync(kFull, keep);
    const int nk = __popc(km);
    if (!nk) return;
    const int rank = __popc(km & ((1u << lane) - 1u));
    if (keep) S.out[rank] = below;
    float tk[kRcList / 32];
    int ti[kRcList / 32];
#pragma unroll
    for (int j = 0; j < kRcList / 32; ++j) {
        const int i = lane + 32 * j;
        tk[j] = 0.0f;
        ti[j] = 0;
        if (i < nb) {
            tk[j] = S.bk[i];
            ti[j] = S.bi[i];
        }
    }
    __syncwarp();  // every read of the old list (and the scratch writes) done
#pragma unroll
    for (int j = 0; j < kRcList / 32; ++j) {
        const int i = lane + 32 * j;
        if (i < nb) {
            int lo = 0, hi = nk;  // kept candidates ahead of entry i: those with below <= i
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (S.out[mid] <= i)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            const int p = i + lo;
            if (p < k) {
                S.bk[p] = tk[j];
                S.bi[p] = ti[j];
            }
        }
    }
    if (keep && below + rank < k) {
        S.bk[below + rank] = ck;
        S.bi[below + rank] = cid;
    }
    __syncwarp();
    nb = nb + nk < k ? nb + nk : k;
}

// The same out of line, returning the new list length: the streams call it only for chunks with an
// element below their threshold, and one copy of it keeps their loops short.
__device__ __noinline__ int rc_offer(bool valid, float key, int id, int k, int nb, RcSmem* S) {
    rc_topk_offer(valid, key, id, k, nb, *S);
    return nb;
}

// A warp's list in the making: candidates below the threshold wait in a queue and are offered 32 at a
// time, since an offer costs some 300 instructions however few of its lanes carry one.
struct RcTop {
    int cap, nb, nq;   // list capacity, its length, queued
    float thr;         // nothing above it can matter
    int* shared_thr;   // the smallest full-list threshold of the CTA's warps (float bits), or null
};
__device__ __forceinline__ RcTop rc_top(int cap, int* shared_thr) {
    return RcTop{cap, 0, 0, __int_as_float(0x7f800000), shared_thr};
}
// offers the last min(nq, 32) queued
__device__ __forceinline__ void rc_flush(RcTop& T, RcSmem& S) {
    const int lane = lane_id(), n = T.nq < 32 ? T.nq : 32;
    __syncwarp();
    T.nq -= n;
    const bool v = lane < n;
    T.nb = rc_offer(v, v ? S.qk[T.nq + lane] : 0.0f, v ? S.qi[T.nq + lane] : 0, T.cap, T.nb, &S);
    if (T.nb == T.cap) {
        T.thr = fminf(T.thr, S.bk[T.cap - 1]);
        if (T.shared_thr) {
            if (lane == 0) atomicMin(T.shared_thr, __float_as_int(T.thr));
            T.thr = fminf(T.thr, __int_as_float(*(volatile int*)T.shared_thr));
        }
    }
    __syncwarp();
}
__device__ __forceinline__ void rc_queue(RcTop& T, bool valid, float key, int id, RcSmem& S) {
    const bool can = valid && key <= T.thr;
    const unsigned m = __ballot_sync(kFull, can);
    if (!m) return;
    if (can) {
        const int at = T.nq + __popc(m & ((1u << lane_id()) - 1u));
        S.qk[at] = key;
        S.qi[at] = id;
    }
    T.nq += __popc(m);
    if (T.nq >= 32) rc_flush(T, S);
}

// What the streams of one refcompat agent need.
struct RcCtx {
    const int64_t* fo;
    const int32_t* fc;
    const BRow* br;
    const int32_t* bc;
    const double* pa;
    const double* rec;
    const double* fit;
    const float4* s32;
    double w3[3];
    float w32[3];
    uint64_t seed;
    uint32_t rep, ep, unit;
    int32_t gen;
    int64_t gf0, glf, gb0, gd;  // the generator's forward row start and length, backward start, degree
};

__device__ __forceinline__ void rc_ctx(const Arena& A, int64_t a, RcCtx& X) {
    const int r = replica_of_agent(A.rep, A.R, a);
    const Replica& rp = A.rep[r];
    X.fo = A.fwd_off + rp.obase;
    X.fc = A.fwd_col + rp.ebase;
    X.br = A.brow + rp.nbase;
    X.bc = A.bcol + rp.bbase;
    X.pa = A.rc_pa + rp.nbase;
    X.rec = A.rc_rec + rp.nbase;
    X.fit = A.rc_fit + rp.nbase;
    X.s32 = A.rc_s32 + rp.nbase;
    X.seed = A.seed;
    X.rep = (uint32_t)(r + A.rep_base);
    X.ep = (uint32_t)A.st->epoch;
    X.unit = (uint32_t)(a - rp.abase);
    const double* o = A.rc_agent + a * 6;  // drawn by the setup
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        X.w3[i] = o[i];
        X.w32[i] = (float)o[i];
    }
    X.gen = (int32_t)o[4];
    X.gf0 = X.fo[X.gen];
    X.glf = X.fo[X.gen + 1] - X.gf0;
    int64_t gb1;
    bspan(X.br, X.gen, X.gb0, gb1);
    X.gd = X.glf + (gb1 - X.gb0);
}

__device__ __forceinline__ double rc_score(const RcCtx& X, int32_t j) {
    return X.w3[0] * X.pa[j] + X.w3[1] * X.rec[j] + X.w3[2] * X.fit[j];
}

// the exact key, out of line: rare, and its FP64 log is long
__device__ __noinline__ float rc_key_exact(const RcCtx& X, int32_t j) {
    return rc_key(X.seed, X.rep, X.ep, X.unit, j, rc_score(X, j));
}

__device__ __forceinline__ float rc_score32(const RcCtx& X, const float4 s) {
    return __fmaf_rn(X.w32[2], s.z, __fmaf_rn(X.w32[1], s.y, X.w32[0] * s.x));
}

// ---- approximate keys.  An exact key takes an FP64 log, division and score, some hundred FP64
// operations, and GB300 does two per clock and SM: the FP64 pipe was what the streams waited for.  Only
// the order of the k smallest keys of a stream matters, so the stream is ranked by an fp32
// approximation of the key whose relative error is below kRcEps, and exact keys are taken only where
// approximations come within twice the error of one another (rc_refine).
//
// The error: u = ((x >> 11) + 1) 2^-53 and d = 1 - u come from the integer exactly up to their one
// fp32 rounding (2^-23 relative with the two-part conversion).  E = -log u is d (1 + d/2 + ... + d^5/6)
// for d < 1/16 (truncation d^6/7 < 1e-8) and -ln2 lg2.approx(u) else, where E >= 0.064: the unit's
// absolute error 2^-22 in lg2 (relative 2^-22 below u = 1/2) is at most 4e-6 of E.  The score is a sum of three nonnegative
// products of values rounded once (4e-7), the division adds 2 ulp.  Together below 5e-6; kRcEps is
// 2^-16 = 1.5e-5.  Scores below 2^-100 in fp32 (a score of zero among them) are reported as odd.
constexpr float kRcEps = 0x1p-16f;

__device__ __forceinline__ float rc_key_approx(const RcCtx& X, int32_t j, float score) {
    const u32x4 r = draw(X.seed, kStreamRcKey, X.rep, X.ep, X.unit, (uint32_t)j);
    const uint32_t lo = r.x[0] & ~0x7FFu, nlo = ~r.x[0] & ~0x7FFu;
    const float u = __fmaf_rn((float)r.x[1], 0x1p-32f, (float)lo * 0x1p-64f + 0x1p-53f);
    const float d = __fmaf_rn((float)~r.x[1], 0x1p-32f, (float)nlo * 0x1p-64f);
    float l;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(u));
    float p = 1.0f / 6.0f;
    p = __fmaf_rn(p, d, 1.0f / 5.0f);
    p = __fmaf_rn(p, d, 1.0f / 4.0f);
    p = __fmaf_rn(p, d, 1.0f / 3.0f);
    p = __fmaf_rn(p, d, 1.0f / 2.0f);
    p = __fmaf_rn(p, d, 1.0f);
    const float E = d < 0.0625f ? d * p : -0x1.62e430p-1f * l;
    return __fdividef(E, score);
}

// The generator's 1-hop set in shared memory (2^bits slots, hash_insert's table), built by `threads`
// threads of which this is number t (a warp, or with cta = true a CTA).  False, and no set, when the
// rows would fill more than three quarters of it: membership is then a search of the rows.  (Searching the
// rows for the elements that a bit signature let through was what most chunks waited for: the
// bisection's dependent loads, four chunks in turn.)
__device__ __forceinline__ bool rc_set(const RcCtx& X, int32_t* H, int bits, int t, int threads, bool cta) {
    if (X.gd > (3ll << bits) / 4) return false;
    for (int q = t; q < 1 << bits; q += threads) H[q] = -1;
    if (cta)
        __syncthreads();
    else
        __syncwarp();
    for (int64_t q = t; q < X.gd; q += threads) hash_insert(H, bits, q < X.glf ? X.fc[X.gf0 + q] : X.bc[X.gb0 + (q - X.glf)]);
    if (cta)
        __syncthreads();
    else
        __syncwarp();
    return true;
}

// One group's share of the stream (rc_2hop_slice), positions in I (int when the group's rows hold
// fewer than 2^30 entries).  base: this lane's row, both directions as one run;
// ys: its start in the concatenation; this warp takes every nw-th 32-entry chunk from number `warp`.
// Four chunks are taken together, so that their row entries, then their scores, are in flight at
// once.  Elements of the 1-hop set H (null: search the rows) are not valid.
template <typename I>
__device__ __forceinline__ bool rc_group(const RcCtx& X, int warp, int nw, const int32_t* base, I ys, I tot, bool exact,
                                         RcTop& T, long long& elems, RcSmem& S, const int32_t* H, int bits) {
    constexpr int U = 4;
    const int lane = lane_id();
    bool odd = false;
    const int32_t* rel = base - ys;
    for (I t0 = (I)32 * warp; t0 < tot; t0 += (I)32 * nw * U) {
        int32_t z[U];
        bool in[U];
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
        float4 sc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) sc[u] = __ldg(X.s32 + z[u]);
        if (T.shared_thr) T.thr = fminf(T.thr, __int_as_float(*(volatile int*)T.shared_thr));
        // one copy of the key and list code, the chunks' values moving through the first: four copies
        // made the instruction fetch the wait that led
#pragma unroll 1
        for (int u = 0; u < U; ++u) {
            bool valid = in[0] && z[0] != X.gen;
            if (H) {
                if (hash_contains(H, bits, z[0])) valid = false;
            } else if (valid) {
                valid = !rc_in_rows(X.fo, X.fc, X.br, X.bc, X.gen, z[0]);
            }
            float key = 0.0f;
            if (!exact) {
                const float s = rc_score32(X, sc[0]);
                key = rc_key_approx(X, z[0], s);
                odd |= in[0] && !(s > 0x1p-100f);
            } else if (valid) {
                key = rc_key_exact(X, z[0]);
            }
            elems += __popc(__ballot_sync(kFull, valid));
            rc_queue(T, valid, key, z[0], S);
#pragma unroll
            for (int v = 0; v + 1 < U; ++v) {
                z[v] = z[v + 1];
                in[v] = in[v + 1];
                sc[v] = sc[v + 1];
            }
        }
    }
    return odd;
}

// the same out of line with 64-bit positions: a group of 2^30 row entries or more
__device__ __noinline__ bool rc_group_long(const RcCtx& X, int warp, int nw, const int32_t* base, int64_t ys, int64_t tot,
                                           bool exact, RcTop* Tp, long long* elems_p, RcSmem* S, const int32_t* H,
                                           int bits) {
    RcTop T = *Tp;
    long long elems = *elems_p;
    const bool odd = rc_group<int64_t>(X, warp, nw, base, ys, tot, exact, T, elems, *S, H, bits);
    *Tp = T;
    *elems_p = elems;
    return odd;
}

// The 2-hop stream (N2 without N1 and g) of the generator's 1-hop groups (32 entries of N1 each):
// every group's rows are concatenated and split into 32-entry chunks, each valid entry keyed (approximately, or exactly) and offered to the warp's list of
// capacity T.cap.  The stream is shared by `parts` CTAs of nw warps (or is one warp's): part and warp
// number this one.  A stream of at least as many groups as parts is dealt out by groups, whose chunks
// the part's warps take in turn; else all the parts' warps take the chunks in turn.  rows and elems
// count the byte model (every row and element once over all parts and warps).  Returns whether some
// score was too small for the approximation.
__device__ __forceinline__ bool rc_2hop_slice(const RcCtx& X, int warp, int nw, int part, int parts, bool exact, RcTop& T,
                                              long long& rows, long long& elems, RcSmem& S, const int32_t* H,
                                              int bits) {
    const bool by_group = X.gd > 32ll * (parts - 1);
    const int w = by_group ? warp : part * nw + warp, n = by_group ? nw : parts * nw;
    int turn = 0;  // chunks of the groups so far, modulo n
    const int lane = lane_id();
    bool odd = false;
    for (int64_t q0 = by_group ? 32ll * part : 0; q0 < X.gd; q0 += by_group ? 32ll * parts : 32) {
        const int64_t q = q0 + lane;
        int32_t y = -1;
        if (q < X.gd) {
            y = q < X.glf ? X.fc[X.gf0 + q] : X.bc[X.gb0 + (q - X.glf)];
            if (y == X.gen) y = -1;
        }
        const int nrow = __popc(__ballot_sync(kFull, y >= 0));
        if (w == 0) rows += nrow;
        // a cited paper's forward row has a copy right before its backward entries: one run; a paper
        // never cited is its forward row
        int64_t yd = 0;
        const int32_t* base = X.fc;
        if (y >= 0) {
            const int64_t f0 = X.fo[y], lf = X.fo[y + 1] - f0;
            int64_t b0, b1;
            bspan(X.br, y, b0, b1);
            yd = lf + (b1 - b0);
            base = b1 > b0 ? X.bc + (b0 - lf) : X.fc + f0;
        }
        const int64_t incl = warp_incl_scan(yd);
        const int64_t tot = __shfl_sync(kFull, incl, 31), ys = incl - yd;
        const int mine = w >= turn ? w - turn : w - turn + n;
        turn = (int)((turn + (tot + 31) / 32) % n);
        if (tot < (1ll << 30)) {
            odd |= rc_group<int>(X, mine, n, base, (int)ys, (int)tot, exact, T, elems, S, H, bits);
        } else {
            RcTop t = T;
            long long el = elems;
            odd |= rc_group_long(X, mine, n, base, ys, tot, exact, &t, &el, &S, H, bits);
            T = t;
            elems = el;
        }
    }
    if (T.nq) rc_flush(T, S);
    return __any_sync(kFull, odd);
}

// The exact keys of the list's n leading elements by approximate key, and the k smallest of them as the
// new list (ascending, ties by id); returns its length.
__device__ __noinline__ int rc_exact_list(const RcCtx& X, int k, int n, RcSmem* Sp) {
    RcSmem& S = *Sp;
    const int lane = lane_id();
    for (int q = lane; q < n; q += 32) S.bk[q] = rc_key_exact(X, S.bi[q]);
    __syncwarp();
    // the list's arrays are reused by the offers: its entries wait in registers
    float key[kRcList / 32];
    int32_t id[kRcList / 32];
#pragma unroll
    for (int j = 0; j < kRcList / 32; ++j) {
        const int q = lane + 32 * j;
        key[j] = q < n ? S.bk[q] : 0.0f;
        id[j] = q < n ? S.bi[q] : 0;
    }
    __syncwarp();
    int nb = 0;
#pragma unroll
    for (int j = 0; j < kRcList / 32; ++j)
        if (32 * j < n) nb = rc_offer(lane + 32 * j < n, key[j], id[j], k, nb, Sp);
    __syncwarp();
    return nb;
}

// The list of a stream's nb <= k + kRcSlack leading elements by approximate key becomes the list of its
// k smallest exact keys, ascending (ties by id).  Only the order is used, so no exact key is needed while
// neighbours up to the k-th and the one after are more than twice the error apart (all but a few in
// a thousand lists of 15); else the whole list's are taken.  False: elements outside the list could
// belong to it.
__device__ __forceinline__ bool rc_refine(const RcCtx& X, int k, int& nb, RcSmem& S) {
    const int lane = lane_id();
    auto apart = [&](int i, int j) { return S.bk[j] * (1.0f - 2.0f * kRcEps) > S.bk[i] * (1.0f + kRcEps); };
    bool close = false;
    for (int i = lane; i < k && i + 1 < nb; i += 32) close |= !apart(i, i + 1);
    if (!__any_sync(kFull, close)) {
        nb = nb < k ? nb : k;
        return true;
    }
    // with room left the list holds the whole stream; else what it lacks is at or above its last entry
    if (nb == k + kRcSlack && !apart(k - 1, nb - 1)) return false;
    nb = rc_exact_list(X, k, nb, &S);
    return true;
}

__device__ void process_agent_rc(const Arena& A, int64_t a, int k, RcSmem& S, int32_t* arr, int32_t* set) {
    const int lane = lane_id();
    const unsigned below = (1u << lane) - 1u;
    const int r = replica_of_agent(A.rep, A.R, a);
    const Replica& rp = A.rep[r];
    const int64_t n = rp.n, al = a - rp.abase;
    const uint32_t ep = (uint32_t)A.st->epoch, unit = (uint32_t)al, rep = (uint32_t)(r + A.rep_base);
    RcCtx X;
    rc_ctx(A, a, X);
    const double alpha = A.rc_agent[a * 6 + 3];
    const int32_t gen = X.gen;

    int c = 1;
    if (lane == 0) arr[0] = gen;
    int32_t tgt = 0;
    const int sy = k >= 2 ? rc_same_year(A.seed, rep, ep, al, rp.delta, rp.rc_sy, n, &tgt) : 0;
    if (sy) {
        if (lane == 0) arr[c] = tgt;
        ++c;
    }
    const int rsv = (int)floor(rp.rc_frc * (double)k);
    const int rem1 = k - 1 - sy - rsv;
    int in_t = rem1 > 0 ? (int)ceil((double)rem1 * alpha) : 0;
    if (in_t > rem1) in_t = rem1 > 0 ? rem1 : 0;
    long long rows = 1, elems = 0, draws = 0;
    // ---- the 1-hop set
    int in = 0;
    if (in_t > 0) {
        int nb = 0;
        long long e1 = 0;
        for (int exact = 0; exact < 2; ++exact) {  // as the 2-hop streams: approximate keys, exact ones if they cannot decide
            nb = 0;
            e1 = 0;
            bool odd = false;
            for (int64_t q0 = 0; q0 < X.gd; q0 += 32) {
                const int64_t q = q0 + lane;
                bool valid = false;
                int32_t y = 0;
                float key = 0.0f;
                if (q < X.gd) {
                    y = q < X.glf ? X.fc[X.gf0 + q] : X.bc[X.gb0 + (q - X.glf)];
                    valid = y != gen;
                    if (exact) {
                        if (valid) key = rc_key_exact(X, y);
                    } else {
                        const float sc = rc_score32(X, __ldg(X.s32 + y));
                        key = rc_key_approx(X, y, sc);
                        odd |= !(sc > 0x1p-100f);
                    }
                }
                e1 += __popc(__ballot_sync(kFull, valid));
                nb = rc_offer(valid, key, y, exact ? in_t : in_t + kRcSlack, nb, &S);
            }
            if (exact || (!__any_sync(kFull, odd) && rc_refine(X, in_t, nb, S))) break;
        }
        elems += e1;
        in = nb;
        __syncwarp();
        for (int q = lane; q < in; q += 32) arr[c + q] = S.bi[q];
        __syncwarp();
        c += in;
    }

    // ---- the 2-hop set (without N1 and g)
    const int rem2 = k - 1 - sy - rsv - in;
    int out = 0;
    if (rem2 > 0) {
        int nb = 0;
        const int big = A.heavy_mark[a];
        if (big > 0) {
            // listed by the setup: k_rc_big has walked the stream with a whole CTA; its sorted
            // top min(k, kKMax) starts with this agent's top rem2
            const long long* meta = A.rc_big_meta + (int64_t)(big - 1) * 3;
            const int have = (int)meta[0];
            nb = have < rem2 ? have : rem2;
            for (int q = lane; q < nb; q += 32) S.bi[q] = A.rc_big_id[(int64_t)(big - 1) * kKMax + q];
            rows += meta[1];
            elems += meta[2];
            __syncwarp();
        } else {
            const int32_t* H = rc_set(X, set, kRcSetBits, lane, 32, false) ? set : nullptr;
            long long r2 = 0, e2 = 0;
            for (int exact = 0; exact < 2; ++exact) {  // exact keys when the approximate ones cannot decide
                RcTop T = rc_top(exact ? rem2 : rem2 + kRcSlack, nullptr);
                r2 = e2 = 0;
                const bool odd = rc_2hop_slice(X, 0, 1, 0, 1, exact != 0, T, r2, e2, S, H, kRcSetBits);
                nb = T.nb;
                if (exact || (!odd && rc_refine(X, rem2, nb, S))) break;
            }
            rows += r2;
            elems += e2;
        }
        out = nb;
        __syncwarp();
        for (int q = lane; q < out; q += 32) arr[c + q] = S.bi[q];
        __syncwarp();
        c += out;
    }

    // ---- uniform fill over [0, n-1) without g and earlier choices; the 32 lanes draw the next 32
    // candidates (4 per Philox block) and take them in order, exactly as one at a time
    int rnd = k - 1 - sy - in - out;
    uint32_t cidx = 0;
    while (rnd > 0) {
        if (cidx >= 4u * kRcFillBlocks) {
            if (lane == 0) atomicOr(&A.st->error, kErrArg);
            break;
        }
        const uint32_t my = cidx + (uint32_t)lane;
        const u32x4 x = draw(A.seed, kStreamUniformFill, rep, ep, unit, my >> 2);
        const uint32_t xr = (my & 3u) == 0 ? x.x[0] : ((my & 3u) == 1 ? x.x[1] : ((my & 3u) == 2 ? x.x[2] : x.x[3]));
        const int32_t v = (int32_t)bounded32(xr, (uint32_t)(n - 1));
        bool pre = false;
        for (int q = 0; q < c; ++q) pre |= arr[q] == v;
        const unsigned grp = __match_any_sync(kFull, v);
        const unsigned gc = grp & __ballot_sync(kFull, !pre);
        const int first = gc ? __ffs(gc) - 1 : 32;
        const unsigned am = __ballot_sync(kFull, !pre && lane == first);
        unsigned consumed = kFull;
        if (__popc(am) >= rnd) {
            unsigned m = am;
            for (int q = 1; q < rnd; ++q) m &= m - 1u;
            const int L = __ffs(m) - 1;
            consumed = L == 31 ? kFull : ((1u << (L + 1)) - 1u);
        }
        draws += __popc(consumed);
        const unsigned took = am & consumed;
        __syncwarp();
        if ((took >> lane) & 1u) arr[c + __popc(took & below)] = v;
        __syncwarp();
        c += __popc(took);
        rnd -= __popc(took);
        cidx += 32;
    }
    if (c != k && lane == 0) atomicOr(&A.st->error, kErrArg);
    emit_row<kKMax>(A, rp, a, al, n, arr, c < k ? c : k, rows, elems, draws);
}
