// bm_kernels.cuh -- sm_100a device code of the swap-delta engine.
//
// Notation (0-based inside the engine; the C ABI is 1-based like the
// reference):  G1 vertices a,b,u,v in [0,n);  G2 vertices f,g in [0,n);
// p: G1 -> G2 (value n = unmatched, "NONE");  pinv: G2 -> G1 (n = NONE).
// W2 is G2's dense (n+1)x(n+1) weight matrix whose row and column n are 0,
// which plays the role of the reference's unused row/column 0.
//
// Profit matrix.  For every ordered pair (a,b) of G1 vertices
//     S[a][b] = sum_{(a,v,w) in out1(a)} min(w, W2[p b][p v])
//             + sum_{(u,a,w) in in1(a)}  min(w, W2[p u][p b])
//             + unary self-loop terms + per-edge corner corrections
// i.e. the score a would earn by taking p(b) while everyone else stays.
// S[a][a] is a's current contribution, and the exact swap delta is
//     delta(a,b) = S[a][b] + S[b][a] - S[a][a] - S[b][b]
// once the corner corrections below are folded into S.  This is the same
// arithmetic as calculate_swap_delta (src/graph-alignment-optimized.c:321-408)
// regrouped by row: the reference skips the partner in each edge list and adds
// the two a<->b edges separately; here those terms are removed or replaced by
// the correction  min(x,W2[pa][pb]) + min(x,W2[pb][pa]) - min(x,W2[pa][pa])
// - min(x,W2[pb][pb])  added to S[a][b] for every G1 edge a->b of weight x.
//
// S is accumulated sparse x sparse: for each out-edge (a,v,w1) of a, every
// G2 in-edge (g -> p(v), w2) contributes min(w1,w2) to S[a][pinv(g)]; for each
// in-edge (u,a,w1), every G2 out-edge (p(u) -> g, w2) contributes to
// S[a][pinv(g)].  Only nonzero min terms are ever touched.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace bm {

// ---- list entries: (id, weight) packed per storage mode ----
template <bool W16> struct Ent;
template <> struct Ent<true> {
    typedef uint32_t T;  // id in bits 0..15, weight in bits 16..31
    static __host__ __device__ __forceinline__ int id(T e) { return (int)(e & 0xFFFFu); }
    static __host__ __device__ __forceinline__ int w(T e) { return (int)(e >> 16); }
    static __host__ __device__ __forceinline__ T make(int i, int w) { return (uint32_t)i | ((uint32_t)w << 16); }
};
template <> struct Ent<false> {
    typedef int2 T;  // x = id, y = weight
    static __host__ __device__ __forceinline__ int id(T e) { return e.x; }
    static __host__ __device__ __forceinline__ int w(T e) { return e.y; }
    static __host__ __device__ __forceinline__ T make(int i, int w) { return make_int2(i, w); }
};
template <bool W16> struct Dense;
template <> struct Dense<true> { typedef uint16_t T; };
template <> struct Dense<false> { typedef int32_t T; };

// Row pitch of the profit matrix S: rows start on 16-byte boundaries at every n,
// so that S is read and written in 16-byte pieces and by TMA.  Columns n .. pitch
// - 1 hold no meaning.
__host__ __device__ __forceinline__ int s_pitch(int n) { return (n + 3) & ~3; }
// Shared memory of a profit row's accumulator: n + 1 ints in whole 16-byte words.
__host__ __device__ __forceinline__ size_t row_smem(int n) { return (size_t)((n + 4) & ~3) * sizeof(int); }

// Device view of a context.
template <bool W16> struct DevView {
    typedef typename Ent<W16>::T E;
    typedef typename Dense<W16>::T D;
    int n;
    const int* off1o; const E* ent1o;   // G1 out-lists (id = dst)
    const int* off1i; const E* ent1i;   // G1 in-lists  (id = src)
    const int* off2o; const E* ent2o;   // G2 out-lists (id = dst)
    const int* off2i; const E* ent2i;   // G2 in-lists  (id = src)
    const int* offs;  const int* selfw; // G1 self-loops per vertex
    E* ent1oP; E* ent1iP;               // G1 lists with ids mapped through p
    E* ent2oP; E* ent2iP;               // G2 lists with ids mapped through pinv
    const int* off2oH; E* ent2oHP;      // G2 out-entries above the hub threshold, mapped through pinv
    const D* W2;                        // dense (n+1)^2, row/col n zero
    const D* W2T;                       // its transpose (columns of W2 read as rows)
    const int* W2D;                     // its diagonal W2[f][f], f = 0..n
    int* p; int* pinv;                  // n+1 entries, [n] = n
    int* S;                             // profit matrix, n rows of s_pitch(n)
    __device__ __forceinline__ int w2(int f, int g) const {
        return (int)W2[(size_t)f * (size_t)(n + 1) + (size_t)g];
    }
    // same value as w2(f, g), read from row g of the transpose
    __device__ __forceinline__ int w2t(int f, int g) const {
        return (int)W2T[(size_t)g * (size_t)(n + 1) + (size_t)f];
    }
    // S[a][b]
    __device__ __forceinline__ size_t at(int a, int b) const { return (size_t)a * s_pitch(n) + b; }
    // same value as w2(f, f)
    __device__ __forceinline__ int w2d(int f) const { return W2D[f]; }
};

// Polls of a wait that the stall test hook (bm_test_stall) makes run out.
constexpr int kStallPolls = 1 << 12;

__device__ __forceinline__ int imin(int a, int b) { return a < b ? a : b; }

// ---------------------------------------------------------------------------
// Relabel list ids through a map (p for G1 lists, pinv for G2 lists), all lists
// in one launch: 16 bytes per thread, the lists end to end.  Five launches of
// 4-byte entries took 48 us at E = 5e6, this one 33 (160 MB).  Thread 0 also
// clears the rebuild's counters.
constexpr int kRelabelLists = 5;
template <bool W16> struct RelabelLists {
    const typename Ent<W16>::T* in[kRelabelLists];
    typename Ent<W16>::T* out[kRelabelLists];
    const int* map[kRelabelLists];
    long long len[kRelabelLists];
    int* row_counter;
    unsigned long long* work_total;
};
template <bool W16>
__global__ void __launch_bounds__(256) k_relabel(const __grid_constant__ RelabelLists<W16> a) {
    typedef Ent<W16> EN;
    typedef typename EN::T E;
    constexpr int V = 16 / sizeof(E);   // entries per 16 bytes
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    if (tid == 0) { *a.row_counter = 0; *a.work_total = 0; }
#pragma unroll
    for (int l = 0; l < kRelabelLists; l++) {
        const E* in = a.in[l];
        E* out = a.out[l];
        const int* map = a.map[l];
        const long long m = a.len[l], mv = m / V;
        for (long long i = tid; i < mv; i += step) {
            union { uint4 q; E e[V]; } x;
            x.q = reinterpret_cast<const uint4*>(in)[i];
#pragma unroll
            for (int u = 0; u < V; u++) x.e[u] = EN::make(__ldg(&map[EN::id(x.e[u])]), EN::w(x.e[u]));
            reinterpret_cast<uint4*>(out)[i] = x.q;
        }
        for (long long i = mv * V + tid; i < m; i += step) out[i] = EN::make(__ldg(&map[EN::id(in[i])]), EN::w(in[i]));
    }
}

// ---------------------------------------------------------------------------
// Profit rows.  Persistent CTAs take rows from `order` (heaviest first) via an
// atomic counter, accumulate the row in shared memory (n+1 ints: slot n
// absorbs terms for unmatched G2 vertices) and write it to S[a][0..n).
// Inside a row, warps take the row's G1 edges round robin and scatter the
// matching G2 list; lists longer than kLongList are queued and then scattered
// by the whole CTA, so a few hub lists cannot hold the row's barrier.
// The queue is small enough (1 KB) that three CTAs of 512 threads with an
// N = 18,524 row each (74 KB) share one SM; a row that queues more scatters
// the rest warp by warp.
constexpr int kLongList = 4096;
constexpr int kLongQueue = 128;

// Scatters min(w1, w2) over list[i0, i1) into acc, lanes striding by `step`.
template <bool W16>
__device__ __forceinline__ void scatter_list(int* acc, const typename Ent<W16>::T* __restrict__ list,
                                             int i0, int i1, int w1, int first, int step) {
    typedef Ent<W16> EN;
    typedef typename EN::T E;
    int i = i0 + first;
    for (; i + 7 * step < i1; i += 8 * step) {  // eight loads in flight per thread
        E x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) x[u] = list[i + u * step];
#pragma unroll
        for (int u = 0; u < 8; u++) atomicAdd(&acc[EN::id(x[u])], imin(w1, EN::w(x[u])));
    }
    for (; i + 3 * step < i1; i += 4 * step) {
        const E x0 = list[i], x1 = list[i + step], x2 = list[i + 2 * step], x3 = list[i + 3 * step];
        atomicAdd(&acc[EN::id(x0)], imin(w1, EN::w(x0)));
        atomicAdd(&acc[EN::id(x1)], imin(w1, EN::w(x1)));
        atomicAdd(&acc[EN::id(x2)], imin(w1, EN::w(x2)));
        atomicAdd(&acc[EN::id(x3)], imin(w1, EN::w(x3)));
    }
    for (; i < i1; i += step) { const E x = list[i]; atomicAdd(&acc[EN::id(x)], imin(w1, EN::w(x))); }
}

// Hub residual: terms of a hub in-edge (u,a,w1) above the threshold T that
// the tensor-core GEMM does not cover, min(w1,w2) - T for w1 > T, over the
// G2 out-entries of p(u) whose weight w2 is above T.
template <bool W16>
__device__ __forceinline__ void scatter_residual(int* acc, const typename Ent<W16>::T* __restrict__ list,
                                                 int i0, int i1, int w1, int thr, int first, int step) {
    typedef Ent<W16> EN;
    for (int i = i0 + first; i < i1; i += step) {
        const typename EN::T x = list[i];
        atomicAdd(&acc[EN::id(x)], imin(w1, EN::w(x)) - thr);
    }
}

// One profit row of S by a group of threads that all call it together: the
// whole block (NT = 0), or the NT threads (a power of two) of the block's
// NT-aligned group; `sync` is a barrier over exactly those threads.  It ends
// with a barrier.  acc holds row_smem(n) bytes of
// shared memory on a 16-byte boundary.
// With `work_total`, the row adds its scattered min terms to it.
template <bool W16, int NT, typename Sync>
__device__ __forceinline__ void profit_row_on(const DevView<W16>& g, int a, int* acc, int2* s_long, int* s_nlong,
                                              const unsigned char* __restrict__ is_hub, int hub_thr, int* s_terms,
                                              unsigned long long* work_total, Sync sync) {
    static_assert(NT == 0 || (NT & (NT - 1)) == 0, "group size is a power of two");
    typedef Ent<W16> EN;
    typedef typename EN::T E;
    const int n = g.n;
    const int tid = NT ? (int)(threadIdx.x & (NT - 1)) : (int)threadIdx.x;
    const int nthr = NT ? NT : (int)blockDim.x;
    const int lane = tid & 31, wid = tid >> 5, nw = nthr >> 5;
    if (tid == 0) {
        *s_nlong = 0;
        if (work_total) *s_terms = 0;
    }
    // the row's scattered terms start from zero; with hubs, the tensor-core
    // hub terms already in S are added when the row is written back
    {
        int4* a4 = reinterpret_cast<int4*>(acc);
        for (int i = tid; i < ((n + 4) >> 2); i += nthr) a4[i] = make_int4(0, 0, 0, 0);
    }
    sync();
    // out-edges of a against G2 in-lists of p(v), then in-edges against out-lists of p(u)
    const int so = g.off1o[a], lo = g.off1o[a + 1] - so;
    const int si = g.off1i[a], li = g.off1i[a + 1] - si;
    // the warp's edges are j = wid + nw * t; lane t loads the set-up of its t-th
    // edge (entry, list extent, kind) so one round of loads serves 32 edges
    const int tot = lo + li;
    for (int base = wid; base < tot; base += nw * 32) {
        const int j = base + nw * lane;
        int f = 0, w1 = 0, b0 = 0, b1 = 0, kind = 0;  // kind: 0 none, 1 out-edge, 2 in-edge, 3 hub residual
        if (j < tot) {
            const bool out = j < lo;
            const E ea = out ? g.ent1oP[so + j] : g.ent1iP[si + (j - lo)];
            f = EN::id(ea);
            w1 = EN::w(ea);
            if (!out && is_hub && is_hub[EN::id(g.ent1i[si + (j - lo)])]) {
                // hub in-edge: the GEMM has its terms up to the threshold
                if (w1 > hub_thr) { kind = 3; b0 = g.off2oH[f]; b1 = g.off2oH[f + 1]; }
            } else {
                kind = out ? 1 : 2;
                const int* off = out ? g.off2i : g.off2o;
                b0 = off[f];
                b1 = off[f + 1];
            }
        }
        if (work_total) {   // the chunk's scattered terms
            int c = kind ? b1 - b0 : 0;
            for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
            if (lane == 0 && c) atomicAdd(s_terms, c);
        }
        const int cnt = min(32, (tot - base + nw - 1) / nw);
        for (int t = 0; t < cnt; t++) {
            const int kt = __shfl_sync(0xffffffffu, kind, t);
            const int w1t = __shfl_sync(0xffffffffu, w1, t);
            const int b0t = __shfl_sync(0xffffffffu, b0, t);
            const int b1t = __shfl_sync(0xffffffffu, b1, t);
            const int ft = __shfl_sync(0xffffffffu, f, t);
            if (kt == 0) continue;
            if (kt == 3) {
                scatter_residual<W16>(acc, g.ent2oHP, b0t, b1t, w1t, hub_thr, lane, 32);
                continue;
            }
            const bool out = kt == 1;
            if (b1t - b0t > kLongList) {
                int q = 0;
                if (lane == 0) q = atomicAdd(s_nlong, 1);
                q = __shfl_sync(0xffffffffu, q, 0);
                if (q < kLongQueue) {
                    if (lane == 0) s_long[q] = make_int2(ft, w1t | (out ? 0 : (int)0x80000000));
                    continue;
                }
            }
            scatter_list<W16>(acc, out ? g.ent2iP : g.ent2oP, b0t, b1t, w1t, lane, 32);
        }
    }
    sync();
    // long lists, one at a time, by the whole block
    const int nl = min(*s_nlong, kLongQueue);
    for (int q = 0; q < nl; q++) {
        const int2 e = s_long[q];
        const bool out = e.y >= 0;
        const int w1 = e.y & 0x7fffffff;
        const int* off = out ? g.off2i : g.off2o;
        const E* list = out ? g.ent2iP : g.ent2oP;
        scatter_list<W16>(acc, list, off[e.x], off[e.x + 1], w1, tid, nthr);
    }
    // corner corrections for every G1 edge a->b
    {
        const int pa = g.p[a];
        const int dpa = g.w2d(pa);
        for (int j = tid; j < lo; j += nthr) {
            const int b = EN::id(g.ent1o[so + j]);
            const E ep = g.ent1oP[so + j];
            const int pb = EN::id(ep), x = EN::w(ep);
            const int c = imin(x, g.w2(pa, pb)) + imin(x, g.w2t(pb, pa))
                        - imin(x, dpa) - imin(x, g.w2d(pb));
            if (c) atomicAdd(&acc[b], c);
        }
    }
    // unary terms of G1 self-loops: a taking p(b) earns min(s, W2[p b][p b])
    {
        const int q0 = g.offs[a], q1 = g.offs[a + 1];
        if (q1 > q0) {
            sync();
            for (int b = tid; b < n; b += nthr) {
                const int pb = g.p[b];
                const int d = g.w2d(pb);
                int t = 0;
                for (int q = q0; q < q1; q++) t += imin(g.selfw[q], d);
                acc[b] += t;
            }
        }
    }
    sync();
    if (work_total && tid == 0) atomicAdd(work_total, (unsigned long long)*s_terms);
    {
        const int n4 = s_pitch(n) >> 2;
        int4* r4 = reinterpret_cast<int4*>(g.S + g.at(a, 0));
        const int4* a4 = reinterpret_cast<const int4*>(acc);
        if (is_hub) {
            int i = tid;
            for (; i + 3 * (int)nthr < n4; i += 4 * nthr) {
                int4 h[4];
#pragma unroll
                for (int u = 0; u < 4; u++) h[u] = r4[i + u * nthr];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int4 v = a4[i + u * nthr];
                    r4[i + u * nthr] = make_int4(h[u].x + v.x, h[u].y + v.y, h[u].z + v.z, h[u].w + v.w);
                }
            }
            for (; i < n4; i += nthr) {
                const int4 h = r4[i], v = a4[i];
                r4[i] = make_int4(h.x + v.x, h.y + v.y, h.z + v.z, h.w + v.w);
            }
        } else {
            for (int i = tid; i < n4; i += nthr) r4[i] = a4[i];
        }
    }
    sync();
}

// One profit row of S by the whole block (all threads call it together; it
// ends with a barrier).
template <bool W16>
__device__ __forceinline__ void profit_row(const DevView<W16>& g, int a, int* acc, int2* s_long, int* s_nlong,
                                           const unsigned char* __restrict__ is_hub, int hub_thr,
                                           int* s_terms = nullptr, unsigned long long* work_total = nullptr) {
    profit_row_on<W16, 0>(g, a, acc, s_long, s_nlong, is_hub, hub_thr, s_terms, work_total,
                          [] { __syncthreads(); });
}

template <bool W16>
__global__ void __launch_bounds__(512, 3)
k_profit(DevView<W16> g, const int* __restrict__ order, int* __restrict__ counter,
         const unsigned char* __restrict__ is_hub, int hub_thr, unsigned long long* __restrict__ work_total) {
    extern __shared__ __align__(16) int acc[];
    __shared__ int s_row, s_nlong, s_terms;
    __shared__ int2 s_long[kLongQueue];  // (G2 vertex, w1 | kind << 31)
    for (;;) {
        if (threadIdx.x == 0) s_row = atomicAdd(counter, 1);
        __syncthreads();
        const int r = s_row;
        if (r >= g.n) break;
        profit_row<W16>(g, order[r], acc, s_long, &s_nlong, is_hub, hub_thr, &s_terms, work_total);
    }
}

// ---------------------------------------------------------------------------
// Per-row best partner as a packed key  (delta + 2^31) << 32 | ~b  (larger
// delta, then smaller b, wins).
__device__ __forceinline__ unsigned long long pack_best(int d, int b) {
    return ((unsigned long long)(unsigned)(d + 0x80000000u) << 32) | (unsigned)(~b);
}
__device__ __forceinline__ unsigned long long kmax(unsigned long long x, unsigned long long y) {
    return x > y ? x : y;
}

// Appends the warp's keys (lanes with `has`) to keys[*count ...], in any order.
// All lanes call it.
__device__ __forceinline__ void append_key(bool has, unsigned long long key, unsigned long long* __restrict__ keys,
                                           int* __restrict__ count) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (!m) return;
    int at = 0;
    if (lane == 0) at = atomicAdd(count, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (has) keys[at + __popc(m & ((1u << lane) - 1u))] = key;
}

// Counters reported by the commit kernels.
struct CommitStats {
    long long total_delta;
    int scanned, verified, committed, steps;
    long long entries;
    int carried, pad;
};

// Control words of a set commit, zeroed before it.
struct SetCtl {
    unsigned arrived;    // arrivals of the CTAs, all steps
    unsigned released;   // steps decided so far, or kSetAbort
    int err;             // bit 1: a wait ran out
    int pad;
};
// What the host reads after it, in one copy.
struct alignas(16) SetResult {
    SetCtl ctl;
    CommitStats st;
};

// Candidate keys: one per row whose best partner improves, deduplicated when
// two rows pick each other.  Sort key: (0x7fffffff - delta) << 32 | lo << 16 | hi
// -> ascending order = delta desc, lo asc, hi asc.  ctl: of the set commit that
// follows, cleared here.
static __global__ void k_candidates(const unsigned long long* __restrict__ rowbest, int n,
                             unsigned long long* __restrict__ keys, int* __restrict__ ncand,
                             int* __restrict__ best_delta, SetCtl* __restrict__ ctl) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a == 0) *ctl = SetCtl{};
    const unsigned long long k = a < n ? rowbest[a] : 0ull;
    unsigned long long out = ~0ull;
    int d = 0;
    if (k) {
        d = max((int)((unsigned)(k >> 32) - 0x80000000u), 0);
        const int b = (int)(~(unsigned)(k & 0xffffffffu));
        if (d > 0) {
            const unsigned long long kb = rowbest[b];
            const int bb = (int)(~(unsigned)(kb & 0xffffffffu));
            const bool mutual = (kb != 0) && (bb == a);
            if (!mutual || a < b) {
                const int lo = a < b ? a : b, hi = a < b ? b : a;
                out = ((unsigned long long)(0x7fffffffu - (unsigned)d) << 32) |
                      ((unsigned long long)lo << 16) | (unsigned long long)hi;
            }
        }
    }
    d = __reduce_max_sync(0xffffffffu, d);
    if ((threadIdx.x & 31) == 0 && d > 0) atomicMax(best_delta, d);
    append_key(out != ~0ull, out, keys, ncand);
}

// Sort key of every profit row, heaviest first: (2^32 - 1 - terms) << 32 | row, a
// warp per row.  The terms of a row are half those on a random matching (`mean`
// G2 entries per G1 edge) and half those on one that matches degrees; in-edges
// from hubs are the tensor cores'.  *count = n.
template <bool W16>
__global__ void __launch_bounds__(256) k_row_keys(DevView<W16> g, const unsigned char* __restrict__ is_hub, float mean,
                                                  unsigned long long* __restrict__ keys, int* __restrict__ count) {
    typedef Ent<W16> EN;
    const int lane = threadIdx.x & 31, a = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0) *count = g.n;
    if (a >= g.n) return;
    unsigned long long t = 0;   // entries of the lists the row's edges meet, and the edges
    unsigned edges = 0;
#pragma unroll 4
    for (int i = g.off1o[a] + lane; i < g.off1o[a + 1]; i += 32) {
        const int v = EN::id(g.ent1o[i]);
        t += g.off1i[v + 1] - g.off1i[v];
        edges++;
    }
#pragma unroll 4
    for (int i = g.off1i[a] + lane; i < g.off1i[a + 1]; i += 32) {
        const int u = EN::id(g.ent1i[i]);
        if (is_hub && is_hub[u]) continue;
        t += g.off1o[u + 1] - g.off1o[u];
        edges++;
    }
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    edges = __reduce_add_sync(0xffffffffu, edges);
    t = min(t + (unsigned long long)(mean * edges), 0xffffffffull);
    if (lane == 0) keys[a] = (0xffffffffull - t) << 32 | (unsigned)a;
}
static __global__ void k_row_order(const unsigned long long* __restrict__ keys, int n, int* __restrict__ order) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) order[i] = (int)(unsigned)keys[i];
}

// Sorts keys[0, *count) (distinct, or with DUP any) into sorted[0, *count) and
// fills sorted[*count, n) with ~0: each key's place is the number of smaller
// keys (equal ones by index), a warp counting for kRankKeys keys at once.  Quadratic, but one launch that
// reads the keys from L1 (980, 5,200 and 17,000 keys: 6, 17 and 57 us) where a
// radix sort of 64-bit keys takes ten launches over all n (12 us for a single
// tile, 65 to 80 us from a few thousand keys); beyond kRankMax keys the radix
// sort wins.
constexpr int kRankKeys = 4, kRankMax = 20480;
template <bool DUP>
__global__ void __launch_bounds__(256) k_rank_sort(const unsigned long long* __restrict__ keys,
                                                          const int* __restrict__ count, int n,
                                                          unsigned long long* __restrict__ sorted) {
    constexpr int per = 8 * kRankKeys;   // keys of a block
    const int m = *count;
    const int lane = threadIdx.x & 31;
    {
        const int i = blockIdx.x * per + threadIdx.x;
        if (threadIdx.x < per && i >= m && i < n) sorted[i] = ~0ull;
    }
    const int i0 = blockIdx.x * per + (threadIdx.x >> 5) * kRankKeys;
    if (i0 >= m) return;
    unsigned long long k[kRankKeys];
    int at[kRankKeys];
#pragma unroll
    for (int u = 0; u < kRankKeys; u++) { k[u] = keys[min(i0 + u, m - 1)]; at[u] = 0; }
#pragma unroll 8
    for (int j = lane; j < m; j += 32) {
        const unsigned long long x = __ldg(&keys[j]);
#pragma unroll
        for (int u = 0; u < kRankKeys; u++) at[u] += x < k[u] || (DUP && x == k[u] && j < i0 + u);
    }
#pragma unroll
    for (int u = 0; u < kRankKeys; u++) {
        at[u] = __reduce_add_sync(0xffffffffu, at[u]);
        if (lane == u && i0 + u < m) sorted[at[u]] = k[u];
    }
}

// ---------------------------------------------------------------------------
// Exact swap delta of (a,b) by `parts` warps, img(v) the matching: the sum of
// part 0 .. parts - 1, each returned to every lane of its warp.  The four edge
// lists of a and b as calculate_swap_delta walks them
// (src/graph-alignment-optimized.c:321-408), plus the exact self-loop terms.
// Lanes load the list extents in one round, then take four entries each per
// round: their entries, images and W2 terms are in flight together, so a pair
// of 128 list entries costs three dependent loads instead of twelve.
template <bool W16, typename Img>
__device__ __forceinline__ int swap_delta_warp(const DevView<W16>& g, Img img, int a, int b, int lane, int part = 0,
                                               int parts = 1) {
    typedef Ent<W16> EN;
    constexpr int U = 4;
    const int pa = img(a), pb = img(b);
    int ext = 0;   // lanes 0..7: out- and in-list of a, of b; lanes 8..11: their self-loops
    {
        const int v = (lane >> 1 & 1) ? b : a;
        const int* off = lane < 4 ? g.off1o : lane < 8 ? g.off1i : g.offs;
        if (lane < 12) ext = off[v + (lane & 1)];
    }
    const int oa = __shfl_sync(0xffffffffu, ext, 0), ob = __shfl_sync(0xffffffffu, ext, 2);
    const int ia = __shfl_sync(0xffffffffu, ext, 4), ib = __shfl_sync(0xffffffffu, ext, 6);
    const int e0 = __shfl_sync(0xffffffffu, ext, 1) - oa;          // ends of: out a,
    const int e1 = e0 + __shfl_sync(0xffffffffu, ext, 3) - ob;     // out b,
    const int e2 = e1 + __shfl_sync(0xffffffffu, ext, 5) - ia;     // in a,
    const int e3 = e2 + __shfl_sync(0xffffffffu, ext, 7) - ib;     // in b
    int d = 0;
    for (int k0 = 32 * U * part; k0 < e3; k0 += 32 * U * parts) {
        typename EN::T e[U];
        int lo[U], ln[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = k0 + 32 * u + lane;
            if (k < e3) e[u] = k < e1 ? g.ent1o[k < e0 ? oa + k : ob + (k - e0)] : g.ent1i[k < e2 ? ia + (k - e1) : ib + (k - e2)];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = k0 + 32 * u + lane;
            lo[u] = ln[u] = 0;
            if (k >= e3) continue;
            const bool out = k < e1, isa = out ? k < e0 : k < e2;
            const int v = EN::id(e[u]);
            const int po = isa ? pa : pb, pn = isa ? pb : pa;       // this end's image, and the one it takes
            const bool other = v == (isa ? b : a);
            if (other && !out) continue;                            // counted from its source's out-list
            const int q = img(v), qn = other ? po : q;
            lo[u] = out ? g.w2(po, q) : g.w2t(q, po);
            ln[u] = out ? g.w2(pn, qn) : g.w2t(q, pn);
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (k0 + 32 * u + lane < e3) d += imin(EN::w(e[u]), ln[u]) - imin(EN::w(e[u]), lo[u]);
    }
    const int sa = __shfl_sync(0xffffffffu, ext, 8), ta = __shfl_sync(0xffffffffu, ext, 9);
    const int sb = __shfl_sync(0xffffffffu, ext, 10), tb = __shfl_sync(0xffffffffu, ext, 11);
    if (part == 0 && (ta > sa || tb > sb)) {   // G1 self-loops
        const int da = g.w2d(pa), db = g.w2d(pb);
        for (int q = sa + lane; q < ta; q += 32) d += imin(g.selfw[q], db) - imin(g.selfw[q], da);
        for (int q = sb + lane; q < tb; q += 32) d += imin(g.selfw[q], da) - imin(g.selfw[q], db);
    }
    return __reduce_add_sync(0xffffffffu, d);
}

// One warp per requested pair.
template <bool W16>
__global__ void k_pair_deltas(DevView<W16> g, const int* __restrict__ pa, const int* __restrict__ pb,
                              long long k, int* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (; w < k; w += nw) {
        const int d = swap_delta_warp<W16>(g, [&](int v) { return g.p[v]; }, pa[w], pb[w], lane);
        if (lane == 0) out[w] = d;
    }
}

// Row of CSR entry i: the last row r with off[r] <= i, r in [0, n).
__device__ __forceinline__ int row_of(const int* __restrict__ off, int n, int i) {
    int lo = 0, hi = n;   // off[lo] <= i < off[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (off[mid] <= i) lo = mid; else hi = mid;
    }
    return lo;
}

// The same, one i for a warp: its lanes try 32 rows at once, so n = 1,000 takes two
// dependent loads instead of ten.
__device__ __forceinline__ int row_of_warp(const int* __restrict__ off, int n, int i, int lane) {
    int lo = 0, hi = n;   // off[lo] <= i < off[hi]
    while (hi - lo > 1) {
        const int step = (hi - lo + 32) / 33, x = lo + (lane + 1) * step;
        lo += step * __popc(__ballot_sync(0xffffffffu, x < hi && off[x] <= i));
        hi = min(hi, lo + step);
    }
    return lo;
}

// Alignment score (src/graph-alignment-optimized.c:292-307).  A warp takes a run of
// consecutive G1 entries, whatever their rows: with a warp per row the
// power-law rows' longest held the launch (54 us at n = 8,192 / E = 1e6).  Runs
// of 128 entries, or of 32 where that leaves warps without one (each entry's row
// is walked to from the run's first: n = 500 / E = 7,500, 23.3 us a call with a binary
// search and runs of 128, 20.2 with a warp per row, now 19.4).
constexpr int kScoreRun = 128;
__host__ __device__ __forceinline__ int score_blocks(long long m, int most) {   // of 256 threads
    return m / 256 + 1 < most ? (int)(m / 256 + 1) : most;
}
__device__ __forceinline__ int score_run(int m, int nwarps) {
    return min(kScoreRun, (m / nwarps + 32) & ~31);
}
template <bool W16>
__device__ __forceinline__ void add_score(const DevView<W16>& g, int m, unsigned long long* __restrict__ out, int block,
                                          int blocks) {
    typedef Ent<W16> EN;
    const int lane = threadIdx.x & 31;
    const int warp = (block * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (blocks * blockDim.x) >> 5;
    long long s = 0;
    const int run = score_run(m, nwarps);
    for (long long r0 = (long long)warp * run; r0 < m; r0 += (long long)nwarps * run) {
        int a = row_of_warp(g.off1o, g.n, (int)r0, lane), end = g.off1o[a + 1];
        const int len = (int)min((long long)run, m - r0);   // lists of up to 2^31 - 1 entries
#pragma unroll
        for (int u = 0; u < kScoreRun / 32; u++) {
            if (32 * u + lane >= len) continue;
            const int i = (int)r0 + 32 * u + lane;
            while (i >= end) end = g.off1o[++a + 1];
            const typename EN::T e = g.ent1o[i];
            s += imin(EN::w(e), g.w2(g.p[a], g.p[EN::id(e)]));
        }
    }
    const int loops = g.offs[g.n];   // G1 self-loops
    for (int i = block * blockDim.x + threadIdx.x; i < loops; i += blocks * blockDim.x)
        s += imin(g.selfw[i], g.w2d(g.p[row_of(g.offs, g.n, i)]));
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0 && s) atomicAdd(out, (unsigned long long)s);
}
template <bool W16>
__global__ void k_score(DevView<W16> g, int m, unsigned long long* __restrict__ out) {
    add_score<W16>(g, m, out, blockIdx.x, gridDim.x);
}

// C[a] += what vertex a's G1 edges and self-loops earn now; one pass over the
// G1 entries, dealt as in k_score (C zero before).  Most terms of an early
// matching are zero and add nothing.
template <bool W16>
__global__ void k_contrib(DevView<W16> g, int m, int* __restrict__ C) {
    typedef Ent<W16> EN;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int run = score_run(m, nwarps);
    for (long long r0 = (long long)warp * run; r0 < m; r0 += (long long)nwarps * run) {
        int a = row_of_warp(g.off1o, g.n, (int)r0, lane), end = g.off1o[a + 1];
        const int len = (int)min((long long)run, m - r0);   // lists of up to 2^31 - 1 entries
#pragma unroll
        for (int u = 0; u < kScoreRun / 32; u++) {
            if (32 * u + lane >= len) continue;
            const int i = (int)r0 + 32 * u + lane;
            while (i >= end) end = g.off1o[++a + 1];
            const typename EN::T e = g.ent1o[i];
            const int v = EN::id(e), t = imin(EN::w(e), g.w2(g.p[a], g.p[v]));
            if (t) { atomicAdd(&C[a], t); atomicAdd(&C[v], t); }
        }
    }
    const int loops = g.offs[g.n];   // G1 self-loops
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < loops; i += gridDim.x * blockDim.x) {
        const int a = row_of(g.offs, g.n, i), t = imin(g.selfw[i], g.w2d(g.p[a]));
        if (t) atomicAdd(&C[a], t);
    }
}

}  // namespace bm
