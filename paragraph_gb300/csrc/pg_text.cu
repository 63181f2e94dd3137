// pg_text.cu -- the edge list as text, formatted on the device (the output writer of the growth
// step).
//
// Restates Graph::WriteGraph (src/graph.cu:909-1003): one "source,target\n" line per edge, sources
// in ascending sequence id, targets ascending within a source, both printed as the caller's
// original ids.  The reference formats on the host threads with std::to_chars; here one pass
// measures tiles of kTextTile lines, the engine's scan turns their sizes into offsets, and a second
// pass formats every tile in shared memory and stores it whole, so a 60M-edge graph becomes text in a
// few milliseconds and leaves the device in one copy.
#include "pg_engine.cuh"
#include "pg_fmt.cuh"

namespace pg {

__device__ __forceinline__ uint64_t magnitude(int64_t v) { return v < 0 ? (uint64_t)(-(v + 1)) + 1u : (uint64_t)v; }

__device__ __forceinline__ int dec_len(int64_t v) {
    uint64_t u = magnitude(v);
    int n = v < 0 ? 2 : 1;
    for (; u >= 1000000000u; u /= 1000000000u) n += 9;  // 32 bits from here
    const uint32_t w = (uint32_t)u;
    return n + (w >= 10u) + (w >= 100u) + (w >= 1000u) + (w >= 10000u) + (w >= 100000u) + (w >= 1000000u) +
           (w >= 10000000u) + (w >= 100000000u);
}

// writes the decimal text of v into p[0, len)
__device__ __forceinline__ void dec_write(char* p, int64_t v, int len) {
    uint64_t u = magnitude(v);
    int i = len - 1;
    for (; u >= 1000000000u; u /= 1000000000u) {
        uint32_t w = (uint32_t)(u % 1000000000u);
        for (int k = 0; k < 9; ++k) {
            p[i--] = (char)('0' + (int)(w % 10u));
            w /= 10u;
        }
    }
    uint32_t w = (uint32_t)u;
    do {
        p[i--] = (char)('0' + (int)(w % 10u));
        w /= 10u;
    } while (w);
    if (v < 0) p[0] = '-';
}

// The CTA's staged text, stage[(dst & 15) ..) so that both sides are aligned alike, to dst: whole
// 16-byte vectors, and bytes at the two ends (neighbouring tiles share those vectors).
__device__ __forceinline__ void store_text(char* __restrict__ dst, const char* __restrict__ stage, int bytes) {
    const int skew = (int)((uintptr_t)dst & 15u);
    char* const base = dst - skew;
    const int end = skew + bytes;
    for (int v = threadIdx.x * 16; v < end; v += blockDim.x * 16) {
        if (v >= skew && v + 16 <= end) {
            *reinterpret_cast<int4*>(base + v) = *reinterpret_cast<const int4*>(stage + v);
        } else {
            for (int i = v < skew ? skew : v; i < v + 16 && i < end; ++i) base[i] = stage[i];
        }
    }
}

constexpr int kTextThreads = 256;

// Rows of the tile's edges [e0, e1), EDGES consecutive ones per thread, all kTextThreads threads.  They
// come from the tile's own row starts: each row marks its first edge (the last of several rows that
// start at one edge, the others being empty, is the source), and a running maximum carries the marks on.
// Where nearly all rows are empty a tile spans a great many of them, and its edges are searched between the
// tile's first and last row instead.  500 edges of 2M rows: sources copied out in 43 us and text in 280, where
// walking the rows took 2,030 and 6,260; one gap of 2M rows among 1.4M edges 110 and 1,890 (2,060 and 7,750).
// The line: from 1,024 rows to 16,384 nothing differs by 3 % at 1 to 4,000 rows per edge; with 65,536, 31,000
// edges of 2M rows take 72 us instead of 43.
constexpr int kMarkRows = 4096;
template <int EDGES>
__device__ __forceinline__ void tile_sources(const int64_t* __restrict__ fo, int64_t n, int64_t e0, int64_t e1,
                                             int64_t (&row)[EDGES]) {
    __shared__ int s_row[kTextThreads * EDGES];
    __shared__ int s_max[kTextThreads / 32];
    __shared__ int64_t s_span[2];  // the first and last edge's rows
    const int lane = lane_id(), wid = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kTextThreads * EDGES; i += kTextThreads) s_row[i] = 0;
    if (wid < 2) {
        const int64_t e = wid == 0 ? e0 : e1 - 1;
        const int64_t r = warp_last_below(n, [&](int64_t i) { return fo[i] <= e; });
        if (lane == 0) s_span[wid] = r;
    }
    __syncthreads();
    const int64_t first = s_span[0], rows = s_span[1] - first;
    if (rows > kMarkRows) {
#pragma unroll
        for (int k = 0; k < EDGES; ++k) row[k] = first;
        for (int64_t step = 1ll << (63 - __clzll(rows)); step; step >>= 1) {
#pragma unroll
            for (int k = 0; k < EDGES; ++k) {
                const int64_t r = row[k] + step;
                if (r - first <= rows && fo[r] <= e0 + threadIdx.x * EDGES + k) row[k] = r;
            }
        }
        __syncthreads();  // the shared arrays are the next tile's
        return;
    }
    for (int r = 1 + (int)threadIdx.x; r <= (int)rows; r += kTextThreads) atomicMax(&s_row[fo[first + r] - e0], r);
    __syncthreads();
    int mark[EDGES], run = 0;
#pragma unroll
    for (int k = 0; k < EDGES; ++k) {
        run = max(run, s_row[threadIdx.x * EDGES + k]);
        mark[k] = run;
    }
    int incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl = max(incl, y);
    }
    if (lane == 31) s_max[wid] = incl;
    int before = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) before = 0;
    __syncthreads();
    for (int w = 0; w < wid; ++w) before = max(before, s_max[w]);
#pragma unroll
    for (int k = 0; k < EDGES; ++k) row[k] = first + max(before, mark[k]);
    __syncthreads();  // the shared arrays are the next tile's
}

// A tile of kTextTile edges.  The pass without an output leaves the tile's bytes in `sums`, the writing
// pass places the tile at off[tile].  1.2M edges: 12 us to measure and 25 to write, where a thread per
// edge, each with its bisection, took 31 and 62.
constexpr int kTextEdges = 2;
constexpr int kTextTile = kTextThreads * kTextEdges;
constexpr int kLineMax = 42;  // two 64-bit ids of 20 characters, a comma and a newline

template <bool WRITE>
__global__ void __launch_bounds__(kTextThreads) k_text(const int64_t* __restrict__ fo, const int32_t* __restrict__ fc,
                                                       int64_t n, int64_t m, const int64_t* __restrict__ ids,
                                                       int32_t* __restrict__ sums, const int64_t* __restrict__ off,
                                                       char* __restrict__ out) {
    __shared__ int s_scan[33];
    __shared__ __align__(16) char stage[WRITE ? kTextTile * kLineMax + 16 : 16];
    const int64_t tiles = (m + kTextTile - 1) / kTextTile;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int64_t e0 = t * kTextTile;
        const int64_t e1 = e0 + kTextTile < m ? e0 + kTextTile : m;
        int64_t row[kTextEdges];
        tile_sources<kTextEdges>(fo, n, e0, e1, row);
        int64_t a[kTextEdges], b[kTextEdges];
        int la[kTextEdges], lb[kTextEdges], mine = 0;
#pragma unroll
        for (int k = 0; k < kTextEdges; ++k) {
            const int64_t e = e0 + threadIdx.x * kTextEdges + k;
            la[k] = lb[k] = 0;
            if (e < e1) {
                a[k] = ids[row[k]];
                b[k] = ids[fc[e]];
                la[k] = dec_len(a[k]);
                lb[k] = dec_len(b[k]);
                mine += la[k] + lb[k] + 2;
            }
        }
        int total;
        int at = block_excl_scan<int>(mine, s_scan, &total);
        if constexpr (WRITE) {
            char* const dst = out + off[t];
            at += (int)((uintptr_t)dst & 15u);
#pragma unroll
            for (int k = 0; k < kTextEdges; ++k) {
                if (la[k]) {
                    dec_write(stage + at, a[k], la[k]);
                    stage[at + la[k]] = ',';
                    dec_write(stage + at + la[k] + 1, b[k], lb[k]);
                    stage[at + la[k] + 1 + lb[k]] = '\n';
                    at += la[k] + lb[k] + 2;
                }
            }
            __syncthreads();
            store_text(dst, stage, total);
        } else if (threadIdx.x == 0) {
            sums[t] = total;
        }
        __syncthreads();  // the next tile's
    }
}

// Sources of the edges [first, first + count), a tile of kSrcTile edges per CTA and step, stored whole (a
// thread per row wrote its row entry by entry: 125 us for 10M edges of 100-entry rows, now 33).
constexpr int kSrcEdges = 4;
constexpr int kSrcTile = kTextThreads * kSrcEdges;
__global__ void __launch_bounds__(kTextThreads) k_edge_sources(const int64_t* __restrict__ fo, int64_t n, int64_t first,
                                                               int64_t count, int32_t* __restrict__ out) {
    for (int64_t t0 = (int64_t)blockIdx.x * kSrcTile; t0 < count; t0 += (int64_t)gridDim.x * kSrcTile) {
        const int64_t t1 = t0 + kSrcTile < count ? t0 + kSrcTile : count;
        int64_t row[kSrcEdges];
        tile_sources<kSrcEdges>(fo, n, first + t0, first + t1, row);
        const int64_t at = t0 + threadIdx.x * kSrcEdges;
        if (at + kSrcEdges <= t1) {  // `out` is an allocation's start: 16-byte aligned
            *reinterpret_cast<int4*>(out + at) = make_int4((int)row[0], (int)row[1], (int)row[2], (int)row[3]);
        } else {
#pragma unroll
            for (int k = 0; k < kSrcEdges; ++k)
                if (at + k < t1) out[at + k] = (int32_t)row[k];
        }
    }
}

void launch_edge_sources(const int64_t* fo, int64_t n, int64_t first, int64_t count, int32_t* out,
                         int num_sms, cudaStream_t s) {
    if (count <= 0 || n <= 0) return;
    int64_t g = (count + kSrcTile - 1) / kSrcTile;
    if (g > (int64_t)num_sms * 8) g = (int64_t)num_sms * 8;
    k_edge_sources<<<(unsigned)g, kTextThreads, 0, s>>>(fo, n, first, count, out);
}

int64_t text_tiles(int64_t m) { return (m + kTextTile - 1) / kTextTile; }

// out == nullptr: the tiles' bytes into sums
void launch_text(const int64_t* fo, const int32_t* fc, int64_t n, int64_t m, const int64_t* ids, int32_t* sums,
                 const int64_t* off, char* out, int num_sms, cudaStream_t s) {
    if (m <= 0) return;
    int64_t g = text_tiles(m);
    if (g > (int64_t)num_sms * 8) g = (int64_t)num_sms * 8;
    if (out)
        k_text<true><<<(unsigned)g, kTextThreads, 0, s>>>(fo, fc, n, m, ids, sums, off, out);
    else
        k_text<false><<<(unsigned)g, kTextThreads, 0, s>>>(fo, fc, n, m, ids, sums, off, out);
}

// ---------------------------------------------------------------- the attribute file
// Restates Graph::WriteAttributes (src/graph.cu:1057-1218): one line per node,
//   id,type,year,pa_weight,rec_weight,fit_weight,fit_lag_duration,fit_peak_value,
//   fit_peak_duration,alpha,in_degree,out_degree,assigned_out_degree,planted_line,generators
// with the weights and alpha as "%.10g", the peak as "%d" (refcompat's integer peak) or "%.9g" of
// the fp32 fitness, seeds typed "seed" with "no_generators", agents typed "agent" with their
// generator ids joined by ';' ("-1" when there is none).  Year, fitness and degrees come from the
// arena; the per-paper draws, printed ids and generators from the caller.  Pass 1 measures tiles of
// kAttrNodes lines (no output buffer), the scan places them, pass 2 formats and stores them.


// Eight lanes per line, a field or a run of integer fields each, so that a line waits for one "%g" and
// not for five in a row: fewer nodes than threads fit the GPU, and the conversions' chains are what the
// pass waits for.  Each lane's text goes to its own shared-memory slot, a scan over the CTA places the
// slots, and the tile is stored whole.  109,000 lines: 32 us to measure and 54 to write, where a thread per
// line took 93 and 159.
constexpr int kAttrThreads = 256;
constexpr int kAttrLanes = 8;
constexpr int kAttrNodes = kAttrThreads / kAttrLanes;
constexpr int kFieldMax = 92;  // a lane's text: at most four 64-bit generator ids (84); an odd number of words
constexpr int kAttrLineMax = 320;  // 38 + 4 x 18 + 42 + 56 + 85, and slack

struct FieldOut {
    char* p;
    int n;
    __device__ __forceinline__ void put(char c) { p[n++] = c; }
    __device__ __forceinline__ void str(const char* s) {
        while (*s) put(*s++);
    }
    __device__ __forceinline__ void dec(int64_t v) {
        const int l = dec_len(v);
        dec_write(p + n, v, l);
        n += l;
    }
};

// part j of node v's line into p; returns its length
__device__ __forceinline__ int attr_part(const AttrCols& C, int64_t v, int j, char* p) {
    FieldOut o{p, 0};
    const bool seed = v < C.n_seed;
    const int32_t* q = C.ints + v * 4;
    // integers before the lane's "%g"
    if (j == 0) {
        o.dec(C.ids[v]);
        o.str(seed ? ",seed," : ",agent,");
        o.dec(C.pub[v]);
    } else if (j == 4) {
        o.put(',');
        o.dec(q[0]);
    }
    // 1..3: the three weights, 4: the peak, 5: alpha
    if (j >= 1 && j <= 5) {
        o.put(',');
        if (j == 4 && C.peak_int) {
            o.dec((int64_t)(int32_t)C.fit[v]);
        } else {
            const double x = j == 4 ? (double)C.fit[v] : C.draws[v * 4 + (j == 5 ? 3 : j - 1)];
            o.n += fmt_g(x, j == 4 ? 9 : 10, o.p + o.n);
        }
    }
    if (j == 4) {
        o.put(',');
        o.dec(q[1]);
    } else if (j == 6) {
        o.put(',');
        o.dec(C.indeg[v]);
        o.put(',');
        o.dec(C.fo[v + 1] - C.fo[v]);
        o.put(',');
        o.dec(q[2]);
        o.put(',');
        o.dec(q[3]);
    } else if (j == 7) {
        o.put(',');
        if (seed) {
            o.str("no_generators");
        } else {
            int k = 0;
            for (int i = 0; i < 4; ++i) {
                const int64_t gid = C.gens[v * 4 + i];
                if (gid < 0) continue;
                if (k++) o.put(';');
                o.dec(gid);
            }
            if (!k) o.str("-1");
        }
        o.put('\n');
    }
    return o.n;
}

template <bool WRITE>
__global__ void __launch_bounds__(kAttrThreads) k_attr(AttrCols C, int32_t* __restrict__ sums,
                                                       const int64_t* __restrict__ off, char* __restrict__ out) {
    __shared__ char s_part[kAttrThreads * kFieldMax];
    __shared__ int s_scan[33];
    __shared__ __align__(16) char stage[WRITE ? kAttrNodes * kAttrLineMax + 16 : 16];
    const int64_t tiles = (C.n + kAttrNodes - 1) / kAttrNodes;
    char* const part = s_part + threadIdx.x * kFieldMax;
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int64_t v = t * kAttrNodes + threadIdx.x / kAttrLanes;
        const int l = v < C.n ? attr_part(C, v, threadIdx.x % kAttrLanes, part) : 0;
        int total;
        int at = block_excl_scan<int>(l, s_scan, &total);
        if constexpr (WRITE) {
            char* const dst = out + off[t];
            at += (int)((uintptr_t)dst & 15u);
            for (int i = 0; i < l; ++i) stage[at + i] = part[i];
            __syncthreads();
            store_text(dst, stage, total);
        } else if (threadIdx.x == 0) {
            sums[t] = total;
        }
        __syncthreads();  // the next tile's
    }
}

int64_t attr_tiles(int64_t n) { return (n + kAttrNodes - 1) / kAttrNodes; }

void launch_attr_text(const AttrCols& C, int32_t* sums, const int64_t* off, char* out, int num_sms,
                      cudaStream_t s) {
    if (C.n <= 0) return;
    int64_t g = attr_tiles(C.n);
    if (g > (int64_t)num_sms * 16) g = (int64_t)num_sms * 16;
    if (out)
        k_attr<true><<<(unsigned)g, kAttrThreads, 0, s>>>(C, sums, off, out);
    else
        k_attr<false><<<(unsigned)g, kAttrThreads, 0, s>>>(C, sums, off, out);
}

}  // namespace pg

// C's "%.<precision>g" of x (the device attribute writer's conversion, compiled for the host).
extern "C" int32_t pg_format_g_host(double x, int32_t precision, char* out) {
    if (precision < 1) precision = 1;
    if (precision > 13) precision = 13;
    return pg::fmt_g(x, precision, out);
}
