// bm_batch.cu -- many independent alignment instances of uneven size swept
// together.
//
// Each instance is an ordinary context (bm_create: same preprocessing, same
// storage, same exact arithmetic); the batch adds device tables of the
// instances' buffers and runs the shared per-row, per-tile and per-instance
// bodies of the single-instance path in one of two schedules:
//   * the launch sequence: relabel (all lists of all instances) -> row work +
//     one LPT sort over all (instance, row) items -> one persistent
//     profit-row launch over every item -> one combine launch over every
//     (instance, tile) item -> reduce -> candidates -> one segmented sort ->
//     one commit launch (a CTA per instance);
//   * one persistent launch (k_b_sweep): the same phases in one cooperative
//     grid, the candidate sort in shared memory, and sparse instances' row
//     bests without their profit matrix (direct_row).
// One sweep of the whole batch is captured once as a CUDA graph and replayed.
// The schedule and its launch shapes (profit-row block size, combine tile)
// are picked by bm_batch_autotune, which times the candidates on the batch
// itself; results do not depend on the choice.  Hub tensor-core terms are
// not used here: the instances are built with BM_FLAG_NO_HUB_GEMM.
#include <climits>
#include <cstdio>
#include <cstring>
#include <vector>
#include <algorithm>
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_segmented_radix_sort.cuh>
#include <cub/block/block_radix_sort.cuh>
#include "bm.h"
#include "bm_internal.cuh"
#include "bm_select.cuh"

namespace {

// Per-instance device record of the batch.
struct BatchInst {
    int n;
    int tiles;            // combine tiles per side for the current tile size
    long long tile_base;  // first global (instance, tile) item
    int row_base;         // first global (instance, row) item / candidate slot
    int* S;
    unsigned long long* rowbest;
    unsigned long long* part;
    unsigned long long* keys;
    unsigned long long* keys_sorted;
    int* diag;            // direct instances: S[x][x]
};

__device__ __forceinline__ int find_inst(const int* __restrict__ base, int nb, long long it) {
    int lo = 0, hi = nb;  // base[lo] <= it < base[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (base[mid] <= it) lo = mid; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ int find_inst_ll(const long long* __restrict__ base, int nb, long long it) {
    int lo = 0, hi = nb;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (base[mid] <= it) lo = mid; else hi = mid;
    }
    return lo;
}

template <bool W16>
__global__ void k_b_relabel(const DevView<W16>* __restrict__ views, const long long* __restrict__ e1,
                            const long long* __restrict__ e2, const typename Ent<W16>::T* const* __restrict__ src,
                            int nb) {
    typedef Ent<W16> EN;
    const int b = blockIdx.y;
    const DevView<W16> g = views[b];
    // lists: 0 G1 out, 1 G1 in (through p); 2 G2 out, 3 G2 in (through pinv)
    const int lst = blockIdx.z;
    const long long m = lst < 2 ? e1[b] : e2[b];
    const typename EN::T* in = src[4 * b + lst];
    typename EN::T* out = lst == 0 ? g.ent1oP : lst == 1 ? g.ent1iP : lst == 2 ? g.ent2oP : g.ent2iP;
    const int* map = lst < 2 ? g.p : g.pinv;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (long long)gridDim.x * blockDim.x) {
        const typename EN::T e = in[i];
        out[i] = EN::make(map[EN::id(e)], EN::w(e));
    }
}

// Matchings of the instances in and out of one staging buffer: p, then pinv, of
// instance b from 2 (row_base[b] + b).  Instances along x: the other dimensions
// end at 65,535.  64 instances took 4 ms per set and get as copies, scores and
// waits of their own (8 sweeps of the smallest).
template <bool W16>
__global__ void k_b_maps_in(const DevView<W16>* __restrict__ views, const int* __restrict__ row_base,
                            const int* __restrict__ stage) {
    const int b = blockIdx.x;
    const DevView<W16>& g = views[b];
    const int* s = stage + 2 * ((size_t)row_base[b] + b);
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i <= g.n; i += gridDim.y * blockDim.x) {
        g.p[i] = s[i];
        g.pinv[i] = s[g.n + 1 + i];
    }
}
template <bool W16>
__global__ void k_b_maps_out(const DevView<W16>* __restrict__ views, const int* __restrict__ row_base,
                             int* __restrict__ stage) {
    const int b = blockIdx.x;
    const DevView<W16>& g = views[b];
    int* s = stage + 2 * ((size_t)row_base[b] + b);
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i <= g.n; i += gridDim.y * blockDim.x) s[i] = g.p[i];
}
template <bool W16>
__global__ void k_b_score(const DevView<W16>* __restrict__ views, const long long* __restrict__ e1,
                          unsigned long long* __restrict__ out) {
    add_score<W16>(views[blockIdx.x], (int)e1[blockIdx.x], out + blockIdx.x, blockIdx.y, gridDim.y);
}

template <bool W16>
__global__ void k_b_row_work(const DevView<W16>* __restrict__ views, const int* __restrict__ row_base, int nb,
                             int total, unsigned long long* __restrict__ key, int* __restrict__ val) {
    typedef Ent<W16> EN;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < total; it += nwarps) {
        const int b = find_inst(row_base, nb, it);
        const DevView<W16>& g = views[b];
        const int a = it - row_base[b];
        long long w = 0;
        for (int i = g.off1o[a] + lane; i < g.off1o[a + 1]; i += 32) {
            const int f = EN::id(g.ent1oP[i]);
            w += g.off2i[f + 1] - g.off2i[f];
        }
        for (int i = g.off1i[a] + lane; i < g.off1i[a + 1]; i += 32) {
            const int f = EN::id(g.ent1iP[i]);
            w += g.off2o[f + 1] - g.off2o[f];
        }
        for (int o = 16; o; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (lane == 0) {
            w += (g.off1o[a + 1] - g.off1o[a]) + (g.off1i[a + 1] - g.off1i[a]) + 64;
            if (g.offs[a + 1] > g.offs[a]) w += g.n;
            key[it] = (unsigned long long)w;
            val[it] = it;
        }
    }
}

template <bool W16>
__global__ void __launch_bounds__(512)
k_b_profit(const DevView<W16>* __restrict__ views, const int* __restrict__ row_base, int nb, int total,
           const int* __restrict__ order, int* __restrict__ counter) {
    extern __shared__ __align__(16) int acc[];
    __shared__ int s_item, s_nlong;
    __shared__ int2 s_long[kLongQueue];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int r = s_item;
        if (r >= total) break;
        const int it = order[r];
        const int b = find_inst(row_base, nb, it);
        const DevView<W16> g = views[b];
        profit_row<W16>(g, it - row_base[b], acc, s_long, &s_nlong, nullptr, 0);
    }
}

// (instance, tile) items: the upper triangle of each instance, row-major.
template <int T>
__global__ void __launch_bounds__(256)
k_b_combine(const BatchInst* __restrict__ inst, const long long* __restrict__ tile_base, int nb, long long total) {
    for (long long it = blockIdx.x; it < total; it += gridDim.x) {
        const int b = find_inst_ll(tile_base, nb, it);
        const BatchInst I = inst[b];
        long long t = it - tile_base[b];
        int ti = 0;
        while (t >= I.tiles - ti) { t -= I.tiles - ti; ti++; }
        const int tj = ti + (int)t;
        combine_tile<T>(I.S, I.n, ti, tj, I.part, nullptr);
        __syncthreads();
    }
}

__global__ void k_b_reduce(const BatchInst* __restrict__ inst, int nb) {
    const int b = blockIdx.y;
    const BatchInst I = inst[b];
    for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < I.n; x += gridDim.x * blockDim.x) {
        unsigned long long k = 0;
        for (int t = 0; t < I.tiles; t++) k = kmax(k, I.part[(size_t)t * I.n + x]);
        I.rowbest[x] = k;
    }
}

// Candidate keys of every instance (the single-instance rule, k_candidates).
__global__ void k_b_candidates(const BatchInst* __restrict__ inst, int nb) {
    const int b = blockIdx.y;
    const BatchInst I = inst[b];
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < I.n; a += gridDim.x * blockDim.x) {
        const unsigned long long k = I.rowbest[a];
        unsigned long long out = ~0ull;
        if (k) {
            const int d = (int)((unsigned)(k >> 32) - 0x80000000u);
            const int p = (int)(~(unsigned)(k & 0xffffffffu));
            if (d > 0) {
                const unsigned long long kb = I.rowbest[p];
                const int pp = (int)(~(unsigned)(kb & 0xffffffffu));
                const bool mutual = (kb != 0) && (pp == a);
                if (!mutual || a < p) {
                    const int lo = a < p ? a : p, hi = a < p ? p : a;
                    out = ((unsigned long long)(0x7fffffffu - (unsigned)d) << 32) |
                          ((unsigned long long)lo << 16) | (unsigned long long)hi;
                }
            }
        }
        I.keys[a] = out;
    }
}

template <bool W16>
__global__ void __launch_bounds__(1024)
k_b_commit(const DevView<W16>* __restrict__ views, const BatchInst* __restrict__ inst, int max_scan,
           int max_verify, CommitStats* __restrict__ st, long long* __restrict__ acc_delta,
           long long* __restrict__ acc_commits) {
    extern __shared__ unsigned char smem[];
    const int b = blockIdx.x;
    const DevView<W16> g = views[b];
    const BatchInst I = inst[b];
    const int lim = (max_scan > 0 && max_scan < I.n) ? max_scan : I.n;
    commit_group<W16, kCGBatch>(g, I.keys_sorted, lim, max_verify, &st[b], smem);
    __syncthreads();
    if (threadIdx.x == 0) {
        acc_delta[b] += st[b].total_delta;
        acc_commits[b] += st[b].committed;
    }
}

// ---------------------------------------------------------------------------
// Direct rows (persistent schedule): a sparse instance's row bests without the
// profit matrix.  delta(a,b) + S[a][a] = S[a][b] + S[b][a] - S[b][b], and both
// S[a][.] and S[.][a] are sums over short lists: S[a][.] as in profit_row_on,
// and S[b][a] over G2's lists of p(a) -- a G2 edge p(a) -> g of weight x meets
// every G1 in-edge (b, w) of pinv(g) with min(w, x), and likewise with both
// directions turned.  So a group of threads adds all four kinds into one
// shared-memory row that starts at -S[b][b], takes its maximum, and neither
// writes n^2 profits nor reads them back in tiles.  Every min term is computed
// twice (for a and for b), which is why only sparse instances take this path
// (direct_instance).  A call of three sweeps of 64 instances of 500 to 8,000
// vertices, 20 edges each: 23.9 -> 15.9 ms, the set commit's wider steps included.
constexpr double kDirectTerms = 1.5;   // most terms per pair of vertices (direct_instance)
constexpr int kDirectRows = 4;    // rows of a task per accumulator
constexpr int kDirectLong = 64;   // longer lists take a whole warp instead of 8 lanes,
constexpr int kDirectAll = 1024;  // and longer ones than this all of the row's threads

// S[a][a], by L lanes of a warp that call it together (mask); all get the sum.
template <bool W16, int L>
__device__ __forceinline__ int direct_diag(const DevView<W16>& g, int a, unsigned mask) {
    const int sub = threadIdx.x & (L - 1);
    typedef Ent<W16> EN;
    typedef typename EN::T E;
    const int pa = g.p[a];
    const int so = g.off1o[a], lo = g.off1o[a + 1] - so;
    const int si = g.off1i[a], tot = lo + g.off1i[a + 1] - si;
    int d = 0;
    for (int j0 = sub; j0 < tot; j0 += 4 * L) {
        int w[4], f[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int j = j0 + L * u;
            w[u] = 0; f[u] = g.n;
            if (j < tot) {
                const E e = j < lo ? g.ent1o[so + j] : g.ent1i[si + (j - lo)];
                w[u] = EN::w(e);
                f[u] = g.p[EN::id(e)];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++)   // both from row p(a): of W2 for out-edges, of its transpose for in-edges
            d += imin(w[u], j0 + L * u < lo ? g.w2(pa, f[u]) : g.w2t(f[u], pa));
    }
    for (int q = g.offs[a] + sub; q < g.offs[a + 1]; q += L) d += imin(g.selfw[q], g.w2d(pa));
    for (int o = L / 2; o; o >>= 1) d += __shfl_xor_sync(mask, d, o);
    return d;
}

// A list to add: its entries, their number, and the weight they are capped by.
struct __align__(16) DirectHead {
    const void* list;
    int len, w;
};
constexpr int kDirectHeads = 128;   // per 128 threads, one each
static_assert(sizeof(DirectHead) * kDirectHeads >= sizeof(int2) * kLongQueue, "profit_row_on's queue fits the heads");

// Best partner of vertex a (packed key, 0 if it has none) by NT threads of the
// block's NT-aligned group; `sync` is a barrier over exactly those threads.
// acc: row_smem(n) bytes of shared memory; head, longs: NT of each; nlong: 2;
// red: NT / 32 keys.  Thread 0 of the group gets the key; the group may start
// another row at once.
//
// What bounds it: latency and issue, not bytes -- a row of a 20-edge-per-vertex
// instance is about 80 lists of 20 entries.  So every thread first sets up one
// list (entry, extent and corner: three dependent loads, taken while the
// accumulator is started), and the lists are then added from shared memory by 8
// lanes each, two lists of up to 32 entries in flight.
template <bool W16, int NT, typename Sync>
__device__ __forceinline__ unsigned long long direct_row(const DevView<W16>& g, const int* __restrict__ diag, int a,
                                                         int* acc, DirectHead* head, uint16_t* longs, int* nlong,
                                                         unsigned long long* red, Sync sync) {
    typedef Ent<W16> EN;
    typedef typename EN::T E;
    constexpr int nw = NT / 32, ng = NT / 8;
    const int n = g.n;
    const int tid = (int)(threadIdx.x & (NT - 1)), lane = tid & 31, wid = tid >> 5, sub = lane & 7;
    const int pa = g.p[a];
    // list heads: 0 G1 out-edges of a, 1 its in-edges, 2 G2 out-edges of p(a), 3 its in-edges
    const int h0 = g.off1o[a], h1 = g.off1i[a], h2 = g.off2o[pa], h3 = g.off2i[pa];
    const int c0 = g.off1o[a + 1] - h0, c1 = c0 + g.off1i[a + 1] - h1;
    const int c2 = c1 + g.off2o[pa + 1] - h2, tot = c2 + g.off2i[pa + 1] - h3;
    if (tid == 0) nlong[0] = nlong[1] = 0;
    int base = 0, par = 0;
    do {
        const int j = base + tid;
        DirectHead h = {nullptr, 0, 0};
        int cb = 0, cv = 0;   // corner of a G1 edge between a and b: in S[a][b] for a -> b, in S[b][a] for b -> a
        if (j < tot) {
            const int kind = j < c0 ? 0 : j < c1 ? 1 : j < c2 ? 2 : 3;
            const int at = kind == 0 ? h0 + j : kind == 1 ? h1 + (j - c0) : kind == 2 ? h2 + (j - c1) : h3 + (j - c2);
            const E e = (kind == 0 ? g.ent1oP : kind == 1 ? g.ent1iP : kind == 2 ? g.ent2oP : g.ent2iP)[at];
            const int f = EN::id(e);
            h.w = EN::w(e);
            const int* off = kind == 0 ? g.off2i : kind == 1 ? g.off2o : kind == 2 ? g.off1i : g.off1o;
            const int b0 = off[f];
            h.len = off[f + 1] - b0;
            h.list = (kind == 0 ? g.ent2iP : kind == 1 ? g.ent2oP : kind == 2 ? g.ent1i : g.ent1o) + b0;
            if (kind < 2) {
                cb = EN::id((kind == 0 ? g.ent1o : g.ent1i)[at]);
                cv = imin(h.w, g.w2(pa, f)) + imin(h.w, g.w2t(f, pa)) - imin(h.w, g.w2d(pa)) - imin(h.w, g.w2d(f));
            }
        }
        if (base == 0)
            for (int i = tid; i < (n + 4) >> 2; i += NT) {   // diag is padded to whole 16-byte words
                const int4 v = __ldcg(reinterpret_cast<const int4*>(diag) + i);
                reinterpret_cast<int4*>(acc)[i] = make_int4(-v.x, -v.y, -v.z, -v.w);
            }
        sync();   // the accumulator is started, the heads before these are done
        head[tid] = h;
        if (cv) atomicAdd(&acc[cb], cv);
        if (h.len > kDirectLong) longs[atomicAdd(&nlong[par], 1)] = (uint16_t)tid;
        if (tid == 0) nlong[par ^ 1] = 0;
        sync();
        const int cnt = min(NT, tot - base);
        for (int t = tid >> 3; t < cnt; t += 2 * ng) {
            DirectHead q[2];
            E x[2][4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                q[k].len = 0;
                if (t + k * ng < cnt) q[k] = head[t + k * ng];
                if (q[k].len > kDirectLong) q[k].len = 0;
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (sub + 8 * u < q[k].len) x[k][u] = static_cast<const E*>(q[k].list)[sub + 8 * u];
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (sub + 8 * u < q[k].len) atomicAdd(&acc[EN::id(x[k][u])], imin(q[k].w, EN::w(x[k][u])));
                for (int i = sub + 32; i < q[k].len; i += 8) {
                    const E e = static_cast<const E*>(q[k].list)[i];
                    atomicAdd(&acc[EN::id(e)], imin(q[k].w, EN::w(e)));
                }
            }
        }
        __syncwarp();
        const int nl = nlong[par];
        for (int q = 0; q < nl; q++) {   // a warp each, the longest by all
            const DirectHead x = head[longs[q]];
            if (x.len > kDirectAll) scatter_list<W16>(acc, static_cast<const E*>(x.list), 0, x.len, x.w, tid, NT);
            else if (q % nw == wid) scatter_list<W16>(acc, static_cast<const E*>(x.list), 0, x.len, x.w, lane, 32);
        }
        base += NT;
        par ^= 1;
    } while (base < tot);
    if (g.offs[n] > 0) {   // self-loops: of a in S[a][b], of b in S[b][a]
        const int dpa = g.w2d(pa);
        for (int b = tid; b < n; b += NT) {
            int t = 0;
            const int d = g.w2d(g.p[b]);
            for (int q = g.offs[a]; q < g.offs[a + 1]; q++) t += imin(g.selfw[q], d);
            for (int q = g.offs[b]; q < g.offs[b + 1]; q++) t += imin(g.selfw[q], dpa);
            if (t) atomicAdd(&acc[b], t);
        }
    }
    sync();
    // the best partner: largest delta, then smallest id
    int bd = INT_MIN, bi = -1;
    for (int i = tid; i < (n + 3) >> 2; i += NT) {
        const int4 v = reinterpret_cast<const int4*>(acc)[i];
        const int x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int b = 4 * i + e;
            if (b < n && b != a && (bi < 0 || x[e] > bd)) { bd = x[e]; bi = b; }
        }
    }
    unsigned long long k = bi < 0 ? 0ull : pack_best(bd - __ldcg(&diag[a]), bi);
    for (int o = 16; o; o >>= 1) k = kmax(k, __shfl_xor_sync(0xffffffffu, k, o));
    if (lane == 0) red[wid] = k;
    sync();
    if (tid == 0)
        for (int q = 1; q < nw; q++) k = kmax(k, red[q]);
    return k;
}

// ---------------------------------------------------------------------------
// One batch sweep as one persistent launch: a cooperative grid of one
// 1024-thread CTA per SM.  The relabel of every list of every instance comes
// first, behind one bounded grid barrier; then a dataflow over the instances
// (no further grid barrier, see the kernel): four 256-thread groups per CTA
// take profit rows and combine tile pairs from one task counter, and each
// instance's row bests, candidates, in-kernel candidate sort and set commit
// run on the CTA that owns it as soon as its own tile pairs are done.  Row
// order does not matter for the result (integer sums).
constexpr int kBThreads = 1024;
constexpr int kBSortItems = 8;                           // candidate keys per thread
constexpr int kBSortMax = kBThreads * kBSortItems;       // instances up to 8,192 vertices
constexpr unsigned kBSpinLimit = 1u << 24;               // polls of one grid-barrier wait (~1 s)
typedef cub::BlockRadixSort<unsigned long long, kBThreads, kBSortItems> BSort;

template <bool W16>
struct BSweepArgs {
    const DevView<W16>* views;
    const BatchInst* inst;
    const long long* ebase;   // 4 count + 1: list segments laid end to end
    const typename Ent<W16>::T* const* lists;
    int nb;
    const int* iorder;     // instances, largest first: the order of their tasks
    const int* rpt;        // rows per row task
    const int* ways;       // accumulators the task uses: 2 when two of the instance's rows fit a group's
                           // shared memory; negative for direct rows
    const long long* tbase;   // 2 (count + 1): first row task, then first tile-pair task (from the
                              // first tile-pair task) of each instance in that order
    const int* row_base;   // first vertex of each instance, laid end to end; rows_total vertices
    int rows_total;
    int total_tasks;       // every instance's rows and tile pairs
    size_t group_bytes;    // shared memory of one 256-thread group (a row accumulator or a tile stage)
    int* counter;          // tasks taken
    int* done;             // 2 count: rows and tile pairs finished, per instance
    unsigned* bar;         // grid barrier: arrivals, generation, error
    int max_scan, max_verify;
    int stall;             // test hook: the first grid barrier never completes
    CommitStats* st;
    long long* acc_delta;
    long long* acc_commits;
};

__device__ __forceinline__ unsigned b_ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid-wide barrier of the co-resident CTAs.  A wait that runs out sets the
// error word (bar[2]); every CTA leaves at its next barrier.  Returns false
// once the error word is set.  With `stall` (the bm_test_stall hook) CTA 0
// does not arrive and every CTA polls only a few thousand times, so the
// barrier never completes and every CTA leaves at it.
__device__ bool b_grid_barrier(unsigned* bar, bool stall = false) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        __threadfence();
        const unsigned gen = b_ld_acquire(&bar[1]);
        const unsigned limit = stall ? (1u << 12) : kBSpinLimit;
        if (!(stall && blockIdx.x == 0) && atomicAdd(&bar[0], 1u) == gridDim.x - 1) {
            atomicExch(&bar[0], 0u);
            __threadfence();
            atomicAdd(&bar[1], 1u);
        } else {
            unsigned it = 0;
            while (b_ld_acquire(&bar[1]) == gen) {
                if (b_ld_acquire(&bar[2]) || ++it > limit) {
                    atomicExch(&bar[2], 1u);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
        s_ok = ok && !b_ld_acquire(&bar[2]);
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ void b_group_sync(int grp) {
    asm volatile("bar.sync %0, 256;" :: "r"(grp + 1) : "memory");
}

template <bool W16, int T>
__global__ void __launch_bounds__(kBThreads, 1) k_b_sweep(BSweepArgs<W16> a) {
    typedef Ent<W16> EN;
    extern __shared__ __align__(16) unsigned char bsm[];
    const int tid = threadIdx.x;
    // relabel every instance's lists (G1 through p, G2 through pinv): the
    // lists laid end to end (segment 4b + lst starts at ebase[4b + lst]), each
    // CTA one contiguous range of that
    {
        const long long tot = a.ebase[4 * a.nb];
        const long long per = (tot + gridDim.x - 1) / gridDim.x;
        const long long lo = (long long)blockIdx.x * per, hi = min(tot, lo + per);
        for (int sg = lo < hi ? find_inst_ll(a.ebase, 4 * a.nb, lo) : 4 * a.nb; sg < 4 * a.nb; sg++) {
            const long long s0 = max(lo, a.ebase[sg]), s1 = min(hi, a.ebase[sg + 1]);
            if (s0 >= hi) break;
            if (s0 >= s1) continue;
            const int b = sg >> 2, lst = sg & 3;
            const DevView<W16>& g = a.views[b];
            const typename EN::T* in = a.lists[sg];
            typename EN::T* out = lst == 0 ? g.ent1oP : lst == 1 ? g.ent1iP : lst == 2 ? g.ent2oP : g.ent2iP;
            const int* map = lst < 2 ? g.p : g.pinv;
            const long long end = s1 - a.ebase[sg];
            for (long long i = s0 - a.ebase[sg] + tid; i < end; i += 4 * kBThreads) {   // four entries in flight
                typename EN::T e[4];
                int f[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i + u * kBThreads < end) e[u] = in[i + u * kBThreads];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i + u * kBThreads < end) f[u] = map[EN::id(e[u])];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i + u * kBThreads < end) out[i + u * kBThreads] = EN::make(f[u], EN::w(e[u]));
            }
        }
    }
    // S[x][x] of the direct instances, 8 lanes per vertex; a warp takes its
    // vertices of many edges with all lanes (8 lanes took 0.2 ms for the largest hub)
    {
        const int gw = (blockIdx.x * kBThreads + tid) >> 5, nw = gridDim.x * (kBThreads / 32), q = (tid & 31) >> 3;
        for (int it0 = 4 * gw; it0 < a.rows_total; it0 += 4 * nw) {
            const int it = it0 + q;
            int b = -1, v = 0, deg = 0;
            if (it < a.rows_total) {
                b = find_inst(a.row_base, a.nb, it);
                v = it - a.row_base[b];
                if (a.ways[b] >= 0) b = -1;
            }
            if (b >= 0) {
                const DevView<W16>& g = a.views[b];
                deg = g.off1o[v + 1] - g.off1o[v] + g.off1i[v + 1] - g.off1i[v];
                if (deg <= 256) {
                    const int d = direct_diag<W16, 8>(g, v, 0xffu << (8 * q));
                    if ((tid & 7) == 0) a.inst[b].diag[v] = d;
                }
            }
            for (unsigned m = __ballot_sync(0xffffffffu, deg > 256 && (tid & 7) == 0); m; m &= m - 1) {
                const int src = __ffs(m) - 1;
                const int bb = __shfl_sync(0xffffffffu, b, src), vv = __shfl_sync(0xffffffffu, v, src);
                const int d = direct_diag<W16, 32>(a.views[bb], vv, 0xffffffffu);
                if ((tid & 31) == 0) a.inst[bb].diag[vv] = d;
            }
        }
    }
    // the dataflow's counters start from zero (read only after the barrier)
    if (blockIdx.x == 0) {
        if (tid == 0) *a.counter = 0;
        for (int i = tid; i < 2 * a.nb; i += blockDim.x) a.done[i] = 0;
    }
    if (!b_grid_barrier(a.bar, a.stall != 0)) return;
    // Dataflow over the instances, with no further grid barrier: the tasks are
    // every instance's rows, then every instance's tile pairs, each part with
    // the largest instance first (iorder), and the four 256-thread groups of
    // every CTA take them one at a time from a global counter.  A tile pair of
    // instance i waits until all of i's rows are written (they were taken
    // long before); the CTA that owns i (CTA i mod grid) stops taking tasks
    // once all of i's tile pairs are done and runs i's row bests, candidates,
    // candidate sort and set commit with all its threads -- so the largest
    // instances' commits overlap the other instances' tile pairs.
    // Dependencies point only to earlier tasks, which the groups that took
    // them finish without waiting on later ones.
    int* rows_done = a.done;
    int* tiles_done = a.done + a.nb;
    const int grp = tid >> 8, gtid = tid & 255;
    unsigned char* gsm = bsm + (size_t)grp * a.group_bytes;     // the group's row accumulator or tile stage
    int* acc = reinterpret_cast<int*>(gsm);
    CombineSmem<T>& cs = *reinterpret_cast<CombineSmem<T>*>(gsm);
    __shared__ int s_task[4], s_go[4];
    __shared__ int s_nlong[16];
    __shared__ DirectHead s_head[8][kDirectHeads];   // per half-group (a group uses two)
    __shared__ uint16_t s_longs[8][kDirectHeads];
    int2* s_long = reinterpret_cast<int2*>(s_head[2 * grp + (gtid >> 7)]);   // profit rows: their long lists
    __shared__ unsigned long long s_red[kBThreads / 32];
    __shared__ int s_stop;
    for (int own = blockIdx.x;; own += gridDim.x) {
        // what the commit of `own` waits for: its tile pairs, or its direct rows
        const bool odir = own < a.nb && a.ways[own] < 0;
        const int target = own >= a.nb ? 0 : odir ? a.inst[own].n : a.inst[own].tiles * (a.inst[own].tiles + 1) / 2;
        const unsigned* fin = (const unsigned*)(odir ? rows_done : tiles_done) + own;
        for (;;) {
            if (gtid == 0) {
                int go = !b_ld_acquire(&a.bar[2]);
                if (go && own < a.nb && (int)b_ld_acquire(fin) >= target) go = 0;
                int t = -1;
                if (go && (t = atomicAdd(a.counter, 1)) >= a.total_tasks) go = 0;
                s_task[grp] = t;
                s_go[grp] = go;
            }
            b_group_sync(grp);
            if (!s_go[grp]) break;
            const int t = s_task[grp];
            const bool row = t < a.tbase[a.nb];
            const long long* base = row ? a.tbase : a.tbase + a.nb + 1;
            const int k = find_inst_ll(base, a.nb, row ? t : t - a.tbase[a.nb]);
            const int i = a.iorder[k];
            const BatchInst I = a.inst[i];
            const int local = (row ? t : t - (int)a.tbase[a.nb]) - (int)base[k] + (row ? 0 : I.n);
            if (row) {
                const DevView<W16>& g = a.views[i];
                const int ways = a.ways[i], rpt = a.rpt[i];
                if (ways < 0) {        // direct rows, by the whole group or by each 128-thread half
                    const int per = rpt / -ways, end = min(I.n, (local + 1) * rpt);
                    if (ways == -1) {
                        for (int r = local * rpt; r < end; r++) {
                            const unsigned long long k = direct_row<W16, 256>(
                                a.views[i], I.diag, r, acc, s_head[2 * grp], s_longs[2 * grp], &s_nlong[4 * grp],
                                s_red + 8 * grp,
                                [grp] { b_group_sync(grp); });
                            if (gtid == 0) I.rowbest[r] = k;
                        }
                    } else {
                        const int half = gtid >> 7, hb = 2 * grp + half;
                        const int r0 = local * rpt + half * per, r1 = min(end, r0 + per);
                        int* hacc = acc + half * (row_smem(I.n) / sizeof(int));
                        for (int r = r0; r < r1; r++) {
                            const unsigned long long k = direct_row<W16, 128>(
                                a.views[i], I.diag, r, hacc, s_head[hb], s_longs[hb], &s_nlong[2 * hb], s_red + 4 * hb,
                                [hb] { asm volatile("bar.sync %0, 128;" :: "r"(5 + hb) : "memory"); });
                            if ((gtid & 127) == 0) I.rowbest[r] = k;
                        }
                    }
                    __threadfence();
                    b_group_sync(grp);
                    if (gtid == 0) atomicAdd(&rows_done[i], end - local * rpt);
                } else if (ways == 1) {   // profit row `local` of instance i by the whole group
                    profit_row_on<W16, 256>(g, local, acc, reinterpret_cast<int2*>(s_head[2 * grp]), &s_nlong[4 * grp],
                                            nullptr, 0, nullptr, nullptr, [grp] { b_group_sync(grp); });
                    __threadfence();     // every thread's part of the row is visible before it counts
                    b_group_sync(grp);
                    if (gtid == 0) atomicAdd(&rows_done[i], 1);
                } else {               // rows 2 local and 2 local + 1, a 128-thread half and accumulator each
                    const int half = gtid >> 7, r = 2 * local + half;
                    const int hb = 2 * grp + half;   // the half's barrier: 5 + hb, 128 threads
                    if (r < I.n)
                        profit_row_on<W16, 128>(g, r, acc + half * (row_smem(I.n) / sizeof(int)), s_long, &s_nlong[2 * hb],
                                                nullptr, 0, nullptr, nullptr, [hb] {
                                                    asm volatile("bar.sync %0, 128;" :: "r"(5 + hb) : "memory");
                                                });
                    __threadfence();
                    b_group_sync(grp);
                    if (gtid == 0) atomicAdd(&rows_done[i], min(2, I.n - 2 * local));
                }
            } else {             // tile pair of instance i, once its rows are written
                if (gtid == 0) {
                    unsigned it = 0;
                    while ((int)b_ld_acquire((const unsigned*)&rows_done[i]) < I.n) {
                        if (b_ld_acquire(&a.bar[2]) || ++it > kBSpinLimit) { atomicExch(&a.bar[2], 1u); break; }
                        __nanosleep(64);
                    }
                    __threadfence();
                }
                b_group_sync(grp);
                long long q = local - I.n;
                int ti = 0;
                while (q >= I.tiles - ti) { q -= I.tiles - ti; ti++; }
                const int tj = ti + (int)q;
                combine_tile_on<T>(I.S, I.n, ti, tj, I.part, nullptr, cs, gtid, [grp] { b_group_sync(grp); });
                __threadfence();     // the tile's partial bests are visible before it counts
                b_group_sync(grp);   // (and cs is rewritten by the group's next task)
                if (gtid == 0) atomicAdd(&tiles_done[i], 1);
            }
        }
        __syncthreads();   // all four groups have stopped
        if (own >= a.nb) break;
        // ---- instance `own`: wait for its tile pairs, then its bests, candidates, sort and commit
        if (tid == 0) {
            unsigned it = 0;
            while ((int)b_ld_acquire(fin) < target) {
                if (b_ld_acquire(&a.bar[2]) || ++it > kBSpinLimit) { atomicExch(&a.bar[2], 1u); break; }
                __nanosleep(64);
            }
            __threadfence();
            s_stop = b_ld_acquire(&a.bar[2]) != 0;
        }
        __syncthreads();
        if (s_stop) break;
        const BatchInst I = a.inst[own];
        for (int x = tid; x < I.n && !odir; x += blockDim.x) {
            unsigned long long k = 0;
            for (int tt = 0; tt < I.tiles; tt++) k = kmax(k, __ldcg(&I.part[(size_t)tt * I.n + x]));
            I.rowbest[x] = k;
        }
        __syncthreads();
        // candidate keys (the single-instance rule, k_candidates)
        for (int xa = tid; xa < I.n; xa += blockDim.x) {
            const unsigned long long k = __ldcg(&I.rowbest[xa]);   // direct rows: written by other CTAs
            unsigned long long out = ~0ull;
            if (k) {
                const int d = (int)((unsigned)(k >> 32) - 0x80000000u);
                const int q = (int)(~(unsigned)(k & 0xffffffffu));
                if (d > 0) {
                    const unsigned long long kb = __ldcg(&I.rowbest[q]);
                    const int qq = (int)(~(unsigned)(kb & 0xffffffffu));
                    const bool mutual = (kb != 0) && (qq == xa);
                    if (!mutual || xa < q) {
                        const int lo = xa < q ? xa : q, hi = xa < q ? q : xa;
                        out = ((unsigned long long)(0x7fffffffu - (unsigned)d) << 32) |
                              ((unsigned long long)lo << 16) | (unsigned long long)hi;
                    }
                }
            }
            I.keys[xa] = out;
        }
        __syncthreads();
        {   // sort the candidate keys in shared memory
            typename BSort::TempStorage& ts = *reinterpret_cast<typename BSort::TempStorage*>(bsm);
            unsigned long long kk[kBSortItems];
#pragma unroll
            for (int q = 0; q < kBSortItems; q++) {
                const int x = tid * kBSortItems + q;
                kk[q] = x < I.n ? I.keys[x] : ~0ull;
            }
            BSort(ts).Sort(kk);
#pragma unroll
            for (int q = 0; q < kBSortItems; q++) {
                const int x = tid * kBSortItems + q;
                if (x < I.n) I.keys_sorted[x] = kk[q];
            }
        }
        __syncthreads();
        const DevView<W16> g = a.views[own];
        const int lim = (a.max_scan > 0 && a.max_scan < I.n) ? a.max_scan : I.n;
        commit_group<W16, kCGBatch>(g, I.keys_sorted, lim, a.max_verify, &a.st[own], bsm);
        __syncthreads();
        if (tid == 0) {
            a.acc_delta[own] += a.st[own].total_delta;
            a.acc_commits[own] += a.st[own].committed;
        }
        __syncthreads();
    }
}

}  // namespace

struct bm_batch {
    int count = 0, max_n = 0, total = 0;
    bool w16 = true;
    std::vector<bm_ctx*> ctx;
    cudaStream_t st = nullptr;
    char err[512] = {0};
    // tuning
    int profit_threads = 512, tile = 64;
    bool tuned = false;
    // device tables
    void* views = nullptr;                // DevView<W16>[count]
    BatchInst* inst = nullptr;
    int* row_base = nullptr;              // count+1
    long long* tile_base = nullptr;       // count+1
    long long *e1 = nullptr, *e2 = nullptr;
    long long* ebase = nullptr;           // 4 count + 1: the lists laid end to end (persistent relabel)
    // the persistent schedule's dataflow: instances largest first, the first
    // row task and tile-pair task of each in that order, per-instance
    // finished rows and tile pairs
    int* iorder = nullptr;
    int* rpt = nullptr;                   // rows per row task of each instance
    int* ways = nullptr;                  // accumulators of its row tasks, negative for direct rows
    int* diag = nullptr;
    int *stage = nullptr, *hstage = nullptr;                       // matchings, device and pinned host
    unsigned long long *scores = nullptr, *hscores = nullptr;
    long long* tbase = nullptr;
    long long total_tasks = 0;
    int* done = nullptr;
    void** lists = nullptr;               // 4 per instance: ent1o, ent1i, ent2o, ent2i
    unsigned long long *wkeys = nullptr, *wkeys_sorted = nullptr, *ckeys = nullptr, *ckeys_sorted = nullptr;
    int *wvals = nullptr, *order = nullptr;
    unsigned long long *rowbest = nullptr, *part = nullptr;
    void* cub_tmp = nullptr;
    size_t cub_bytes = 0;
    int* counter = nullptr;
    CommitStats* cstats = nullptr;
    long long *acc_delta = nullptr, *acc_commits = nullptr;
    long long total_tiles = 0;
    std::vector<BatchInst> hinst;
    // schedules: one persistent launch per sweep (k_b_sweep, possible when
    // every instance's candidates fit its in-kernel sort) or the launch
    // sequence above; the autotuner times both and keeps the faster
    bool can_persist = false, use_persist = false;
    size_t group_cap = 0;                 // most shared memory a 256-thread group of it can have
    unsigned* gbar = nullptr;             // its grid barrier
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_max_scan = 0, graph_max_verify = -1;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

static thread_local char g_batch_create_err[512];

template <bool W16>
static bm_status persistent_setup(bm_batch* B);
static size_t persistent_group_bytes(const bm_batch* B);

// Whether the persistent schedule finds an instance's row bests without its
// profit matrix (direct_row).  That computes each of the about 2 e1 e2 / n min
// terms of the matrix twice, and saves writing n^2 profits and reading them in
// tiles: the line is a number of terms per pair, 4 e1 e2 / n^3.  Measured, ms per
// sweep of 64 instances (24 at n = 4,000) through the matrix / direct: n = 1,600,
// 24 edges per vertex (1.4 terms) 2.5 / 2.3, 32 edges (2.6) 2.78 / 2.79, 40 edges
// (4.0) 3.21 / 3.45; n = 4,000, 40 edges (1.6) 4.39 / 4.45, 50 edges (2.5) 5.05 /
// 5.95, 63 edges (4.0) 5.8 / 9.4; n = 800, 24 edges (2.9) 1.10 / 1.03.
static bool direct_instance(const bm_ctx* c) {
    return 4.0 * (double)c->e1 * (double)c->e2 <= kDirectTerms * (double)c->n * c->n * c->n;
}

#define BK(call)                                                                         \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess) {                                                         \
            snprintf(B->err, sizeof B->err, "%s:%d: %s: %s", __FILE__, __LINE__, #call,  \
                     cudaGetErrorString(e_));                                            \
            return BM_E_CUDA;                                                            \
        }                                                                                \
    } while (0)

static void batch_free(bm_batch* B) {
    if (!B) return;
    if (B->exec) cudaGraphExecDestroy(B->exec);
    if (B->graph) cudaGraphDestroy(B->graph);
    void* bufs[] = {B->views, B->inst, B->row_base, B->tile_base, B->e1, B->e2, B->lists, B->wkeys,
                    B->wkeys_sorted, B->ckeys, B->ckeys_sorted, B->wvals, B->order, B->rowbest, B->part,
                    B->cub_tmp, B->counter, B->cstats, B->acc_delta, B->acc_commits, B->gbar, B->ebase,
                    B->iorder, B->tbase, B->done, B->rpt, B->ways, B->diag, B->stage, B->scores};
    for (void* p : bufs) if (p) cudaFree(p);
    if (B->hstage) cudaFreeHost(B->hstage);
    if (B->hscores) cudaFreeHost(B->hscores);
    if (B->ev0) cudaEventDestroy(B->ev0);
    if (B->ev1) cudaEventDestroy(B->ev1);
    if (B->st) cudaStreamDestroy(B->st);
    for (bm_ctx* c : B->ctx) bm_destroy(c);
    delete B;
}

extern "C" void bm_batch_destroy(bm_batch* B) { batch_free(B); }
extern "C" const char* bm_batch_last_error(const bm_batch* B) { return B ? B->err : g_batch_create_err; }

// (Re)builds the per-instance tile tables for the current tile size.  Every table
// is copied on the batch's stream: its launches do not wait for the legacy
// stream, where a copy from pageable memory may still be under way on return.
static bm_status batch_tiles(bm_batch* B) {
    std::vector<long long> tb(B->count + 1, 0);
    for (int i = 0; i < B->count; i++) {
        const int T = (B->hinst[i].n + B->tile - 1) / B->tile;
        B->hinst[i].tiles = T;
        B->hinst[i].tile_base = tb[i];
        tb[i + 1] = tb[i] + (long long)T * (T + 1) / 2;
    }
    B->total_tiles = tb[B->count];
    BK(cudaMemcpyAsync(B->tile_base, tb.data(), tb.size() * sizeof(long long), cudaMemcpyHostToDevice, B->st));
    if (B->iorder) {   // the persistent schedule's task layout: per instance, largest first, rows then tile pairs
        std::vector<int> ord(B->count);
        for (int i = 0; i < B->count; i++) ord[i] = i;
        std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return B->hinst[x].n > B->hinst[y].n; });
        // two rows at a time where both accumulators fit a group's shared memory; a
        // task of direct rows has several rows per accumulator (they are short)
        const size_t gb = persistent_group_bytes(B);
        std::vector<int> rpt(B->count), ways(B->count);
        for (int i = 0; i < B->count; i++) {
            const int w = 2 * row_smem(B->hinst[i].n) <= gb ? 2 : 1;
            const bool dir = direct_instance(B->ctx[i]);
            ways[i] = dir ? -w : w;
            rpt[i] = dir ? w * kDirectRows : w;
        }
        // [rows prefix (count + 1)][tile-pair prefix (count + 1)]
        std::vector<long long> tbase(2 * (size_t)B->count + 2, 0);
        for (int k = 0; k < B->count; k++) {
            const BatchInst& I = B->hinst[ord[k]];
            tbase[k + 1] = tbase[k] + (I.n + rpt[ord[k]] - 1) / rpt[ord[k]];
            tbase[B->count + 1 + k + 1] = tbase[B->count + 1 + k] +
                (ways[ord[k]] < 0 ? 0 : (long long)I.tiles * (I.tiles + 1) / 2);
        }
        B->total_tasks = tbase[B->count] + tbase[2 * (size_t)B->count + 1];
        if (B->total_tasks > 0x7fffffffLL) B->can_persist = B->use_persist = false;   // 32-bit task indices
        BK(cudaMemcpyAsync(B->iorder, ord.data(), ord.size() * sizeof(int), cudaMemcpyHostToDevice, B->st));
        BK(cudaMemcpyAsync(B->rpt, rpt.data(), rpt.size() * sizeof(int), cudaMemcpyHostToDevice, B->st));
        BK(cudaMemcpyAsync(B->ways, ways.data(), ways.size() * sizeof(int), cudaMemcpyHostToDevice, B->st));
        BK(cudaMemcpyAsync(B->tbase, tbase.data(), tbase.size() * sizeof(long long), cudaMemcpyHostToDevice, B->st));
    }
    BK(cudaMemcpyAsync(B->inst, B->hinst.data(), B->hinst.size() * sizeof(BatchInst), cudaMemcpyHostToDevice, B->st));
    return BM_OK;
}

template <bool W16>
static bm_status batch_tables(bm_batch* B) {
    std::vector<DevView<W16>> v(B->count);
    std::vector<void*> lists(4 * B->count);
    std::vector<long long> e1(B->count), e2(B->count);
    for (int i = 0; i < B->count; i++) {
        v[i] = view<W16>(B->ctx[i]);
        lists[4 * i + 0] = B->ctx[i]->ent1o;
        lists[4 * i + 1] = B->ctx[i]->ent1i;
        lists[4 * i + 2] = B->ctx[i]->ent2o;
        lists[4 * i + 3] = B->ctx[i]->ent2i;
        e1[i] = B->ctx[i]->e1;
        e2[i] = B->ctx[i]->e2;
    }
    BK(cudaMalloc(&B->views, v.size() * sizeof(DevView<W16>)));
    BK(cudaMemcpyAsync(B->views, v.data(), v.size() * sizeof(DevView<W16>), cudaMemcpyHostToDevice, B->st));
    BK(cudaMalloc(&B->lists, lists.size() * sizeof(void*)));
    BK(cudaMemcpyAsync(B->lists, lists.data(), lists.size() * sizeof(void*), cudaMemcpyHostToDevice, B->st));
    BK(cudaMalloc(&B->e1, B->count * sizeof(long long)));
    BK(cudaMalloc(&B->e2, B->count * sizeof(long long)));
    BK(cudaMemcpyAsync(B->e1, e1.data(), B->count * sizeof(long long), cudaMemcpyHostToDevice, B->st));
    BK(cudaMemcpyAsync(B->e2, e2.data(), B->count * sizeof(long long), cudaMemcpyHostToDevice, B->st));
    std::vector<long long> eb(4 * (size_t)B->count + 1, 0);
    for (int i = 0; i < B->count; i++)
        for (int l = 0; l < 4; l++) eb[4 * i + l + 1] = eb[4 * i + l] + (l < 2 ? e1[i] : e2[i]);
    BK(cudaMalloc(&B->ebase, eb.size() * sizeof(long long)));
    BK(cudaMemcpyAsync(B->ebase, eb.data(), eb.size() * sizeof(long long), cudaMemcpyHostToDevice, B->st));
    return BM_OK;
}

extern "C" bm_status bm_batch_create(bm_batch** out, int32_t count, const int32_t* n, const int64_t* e1,
                                     const int32_t* const* src1, const int32_t* const* dst1,
                                     const int32_t* const* w1, const int64_t* e2, const int32_t* const* src2,
                                     const int32_t* const* dst2, const int32_t* const* w2, uint32_t flags) {
    if (!out || count < 1 || !n || !e1 || !src1 || !dst1 || !w1 || !e2 || !src2 || !dst2 || !w2)
        return BM_E_INPUT;
    *out = nullptr;
    bm_batch* B = new (std::nothrow) bm_batch();
    if (!B) return BM_E_NOMEM;
    B->count = count;
    // every instance in one storage mode
    const uint32_t f = (flags | BM_FLAG_NO_HUB_GEMM);
    bool any32 = (flags & BM_FLAG_FORCE_I32) != 0;
    for (int pass = 0; pass < 2; pass++) {
        for (bm_ctx* c : B->ctx) bm_destroy(c);
        B->ctx.clear();
        for (int i = 0; i < count; i++) {
            bm_ctx* c = nullptr;
            bm_status s = bm_create(&c, n[i], e1[i], src1[i], dst1[i], w1[i], e2[i], src2[i], dst2[i], w2[i],
                                    f | (any32 ? BM_FLAG_FORCE_I32 : 0u));
            if (s != BM_OK) {
                snprintf(g_batch_create_err, sizeof g_batch_create_err, "instance %d: %s", i, bm_last_error(nullptr));
                batch_free(B);
                return s;
            }
            B->ctx.push_back(c);
        }
        bool mixed = false;
        for (bm_ctx* c : B->ctx) mixed |= !c->w16;
        if (!mixed || any32) break;
        any32 = true;  // some instance needs 32-bit entries: rebuild all that way
    }
    B->w16 = B->ctx[0]->w16;
    bm_status s;
    for (bm_ctx* c : B->ctx) {
        if ((s = ensure_S(c)) != BM_OK) {
            snprintf(g_batch_create_err, sizeof g_batch_create_err, "%s", c->err);
            batch_free(B);
            return s;
        }
        B->max_n = std::max(B->max_n, c->n);
        B->total += c->n;
    }
    auto body = [&]() -> bm_status {
        BK(cudaStreamCreateWithFlags(&B->st, cudaStreamNonBlocking));
        BK(cudaEventCreate(&B->ev0));
        BK(cudaEventCreate(&B->ev1));
        // concatenated per-instance buffers, sized for the smallest tile (32)
        std::vector<int> rb(count + 1, 0);
        long long part_total = 0;
        for (int i = 0; i < count; i++) {
            rb[i + 1] = rb[i] + B->ctx[i]->n;
            part_total += (long long)((B->ctx[i]->n + 31) / 32) * B->ctx[i]->n;
        }
        BK(cudaMalloc(&B->row_base, rb.size() * sizeof(int)));
        BK(cudaMemcpyAsync(B->row_base, rb.data(), rb.size() * sizeof(int), cudaMemcpyHostToDevice, B->st));
        BK(cudaMalloc(&B->tile_base, (count + 1) * sizeof(long long)));
        BK(cudaMalloc(&B->inst, count * sizeof(BatchInst)));
        const size_t tot = (size_t)B->total;
        BK(cudaMalloc(&B->wkeys, tot * sizeof(unsigned long long)));
        BK(cudaMalloc(&B->wkeys_sorted, tot * sizeof(unsigned long long)));
        BK(cudaMalloc(&B->ckeys, tot * sizeof(unsigned long long)));
        BK(cudaMalloc(&B->ckeys_sorted, tot * sizeof(unsigned long long)));
        BK(cudaMalloc(&B->wvals, tot * sizeof(int)));
        BK(cudaMalloc(&B->order, tot * sizeof(int)));
        BK(cudaMalloc(&B->rowbest, tot * sizeof(unsigned long long)));
        BK(cudaMalloc(&B->part, (size_t)part_total * sizeof(unsigned long long)));
        BK(cudaMalloc(&B->counter, sizeof(int)));
        BK(cudaMalloc(&B->cstats, count * sizeof(CommitStats)));
        BK(cudaMalloc(&B->stage, 2 * (tot + count) * sizeof(int)));
        BK(cudaMallocHost(&B->hstage, 2 * (tot + count) * sizeof(int)));
        BK(cudaMalloc(&B->scores, count * sizeof(unsigned long long)));
        BK(cudaMallocHost(&B->hscores, count * sizeof(unsigned long long)));
        BK(cudaMalloc(&B->acc_delta, count * sizeof(long long)));
        BK(cudaMalloc(&B->acc_commits, count * sizeof(long long)));
        size_t b1 = 0, b2 = 0;
        BK(cub::DeviceRadixSort::SortPairsDescending(nullptr, b1, B->wkeys, B->wkeys_sorted, B->wvals, B->order,
                                                     B->total));
        BK(cub::DeviceSegmentedRadixSort::SortKeys(nullptr, b2, B->ckeys, B->ckeys_sorted, B->total, count,
                                                   B->row_base, B->row_base + 1));
        B->cub_bytes = std::max(b1, b2);
        BK(cudaMalloc(&B->cub_tmp, B->cub_bytes));
        B->hinst.resize(count);
        long long poff = 0, doff = 0;
        for (int i = 0; i < count; i++) doff += row_smem(B->ctx[i]->n) / sizeof(int);
        BK(cudaMalloc(&B->diag, (size_t)doff * sizeof(int)));
        BK(cudaMemsetAsync(B->diag, 0, (size_t)doff * sizeof(int), B->st));   // the padding is read
        doff = 0;
        for (int i = 0; i < count; i++) {
            BatchInst& I = B->hinst[i];
            I.n = B->ctx[i]->n;
            I.row_base = rb[i];
            I.S = B->ctx[i]->S;
            I.rowbest = B->rowbest + rb[i];
            I.part = B->part + poff;
            poff += (long long)((I.n + 31) / 32) * I.n;
            I.diag = B->diag + doff;
            doff += row_smem(I.n) / sizeof(int);
            I.keys = B->ckeys + rb[i];
            I.keys_sorted = B->ckeys_sorted + rb[i];
        }
        bm_status s2 = B->w16 ? batch_tables<true>(B) : batch_tables<false>(B);
        if (s2) return s2;
        BK(cudaMalloc(&B->gbar, 4 * sizeof(unsigned)));
        BK(cudaMemsetAsync(B->gbar, 0, 4 * sizeof(unsigned), B->st));
        BK(cudaMalloc(&B->iorder, count * sizeof(int)));
        BK(cudaMalloc(&B->rpt, count * sizeof(int)));
        BK(cudaMalloc(&B->ways, count * sizeof(int)));
        BK(cudaMalloc(&B->tbase, 2 * (count + 1) * sizeof(long long)));
        BK(cudaMalloc(&B->done, 2 * count * sizeof(int)));
        s2 = B->w16 ? persistent_setup<true>(B) : persistent_setup<false>(B);
        if (s2) return s2;
        return batch_tiles(B);
    };
    s = body();
    if (s != BM_OK) {
        snprintf(g_batch_create_err, sizeof g_batch_create_err, "%s", B->err);
        batch_free(B);
        return s;
    }
    *out = B;
    return BM_OK;
}

template <bool W16>
static bm_status batch_maps_in(bm_batch* B, int k, size_t ints) {
    const DevView<W16>* views = (const DevView<W16>*)B->views;
    const dim3 grid(k, (B->max_n + 1024) / 1024);
    BK(cudaMemcpyAsync(B->stage, B->hstage, ints * sizeof(int), cudaMemcpyHostToDevice, B->st));
    BK(cudaMemsetAsync(B->scores, 0, k * sizeof(unsigned long long), B->st));
    k_b_maps_in<W16><<<grid, 256, 0, B->st>>>(views, B->row_base, B->stage);
    BK(cudaGetLastError());
    k_b_score<W16><<<dim3(k, 16), 256, 0, B->st>>>(views, B->e1, B->scores);
    BK(cudaGetLastError());
    BK(cudaMemcpyAsync(B->hscores, B->scores, k * sizeof(unsigned long long), cudaMemcpyDeviceToHost, B->st));
    BK(cudaStreamSynchronize(B->st));
    return BM_OK;
}

// A single instance is set and read by its own calls: the pass over all of them
// has a staging copy that pays from two instances on (n = 3,000, us to set: one 49
// through it and 40 without, two 54 and 89).
extern "C" bm_status bm_batch_set_mappings(bm_batch* B, const int32_t* const* maps) {
    if (!B || !maps) return BM_E_INPUT;
    bm_status bad = BM_OK;
    if (B->count == 1) {
        if ((bad = bm_set_mapping(B->ctx[0], maps[0]))) snprintf(B->err, sizeof B->err, "instance 0: %.480s", B->ctx[0]->err);
        return bad;
    }
    size_t at = 0;
    int k = 0;   // the instances before the first bad matching are set
    for (; k < B->count; k++) {
        const size_t n1 = (size_t)B->ctx[k]->n + 1;
        if ((bad = decode_mapping(B->ctx[k], maps[k], B->hstage + at, B->hstage + at + n1))) break;
        at += 2 * n1;
    }
    if (k) {
        bm_status s = B->w16 ? batch_maps_in<true>(B, k, at) : batch_maps_in<false>(B, k, at);
        if (s) return s;
        for (int i = 0; i < k; i++) {
            B->ctx[i]->mapped = true;
            B->ctx[i]->score = (long long)B->hscores[i];
        }
    }
    if (bad) snprintf(B->err, sizeof B->err, "instance %d: %.480s", k, B->ctx[k]->err);
    return bad;
}

extern "C" bm_status bm_batch_get_mappings(bm_batch* B, int32_t* const* maps) {
    if (!B || !maps) return BM_E_INPUT;
    size_t at = 0;
    int k = 0;
    if (B->count > 1)
        for (; k < B->count && B->ctx[k]->mapped && maps[k]; k++) at += 2 * ((size_t)B->ctx[k]->n + 1);
    if (k) {
        const dim3 grid(k, (B->max_n + 1024) / 1024);
        if (B->w16) k_b_maps_out<true><<<grid, 256, 0, B->st>>>((const DevView<true>*)B->views, B->row_base, B->stage);
        else k_b_maps_out<false><<<grid, 256, 0, B->st>>>((const DevView<false>*)B->views, B->row_base, B->stage);
        BK(cudaGetLastError());
        BK(cudaMemcpyAsync(B->hstage, B->stage, at * sizeof(int), cudaMemcpyDeviceToHost, B->st));
        BK(cudaStreamSynchronize(B->st));
    }
    const int* p = B->hstage;
    for (int i = 0; i < k; i++) {
        const int n = B->ctx[i]->n;
        maps[i][0] = 0;
        for (int a = 0; a < n; a++) maps[i][a + 1] = p[a] == n ? 0 : p[a] + 1;
        p += 2 * ((size_t)n + 1);
    }
    if (k == B->count) return BM_OK;
    bm_status s = bm_get_mapping(B->ctx[k], maps[k]);   // the only one, or the error of the first it cannot get
    if (s) snprintf(B->err, sizeof B->err, "instance %d: %.480s", k, B->ctx[k]->err);
    return s;
}

extern "C" bm_status bm_batch_scores(bm_batch* B, int64_t* scores) {
    if (!B || !scores) return BM_E_INPUT;
    for (int i = 0; i < B->count; i++) {
        bm_status s = bm_score(B->ctx[i], &scores[i]);
        if (s) { snprintf(B->err, sizeof B->err, "instance %d: %.480s", i, B->ctx[i]->err); return s; }
    }
    return BM_OK;
}

// Shared memory of one 256-thread group of k_b_sweep: a row accumulator or a
// tile stage, whichever is larger, and room for two accumulators of the
// direct instances as far as the SM has it.
static size_t persistent_group_bytes(const bm_batch* B) {
    size_t m = std::max(row_smem(B->max_n), B->tile == 32 ? sizeof(CombineSmem<32>) : sizeof(CombineSmem<64>));
    m = (m + 15) & ~(size_t)15;
    for (const bm_ctx* c : B->ctx)
        if (direct_instance(c) && 2 * row_smem(c->n) <= B->group_cap) m = std::max(m, 2 * row_smem(c->n));
    return m;
}

// Shared memory of k_b_sweep: the largest of its phases' needs.
static size_t persistent_smem(const bm_batch* B) {
    size_t m = 4 * persistent_group_bytes(B);                              // four groups
    m = std::max(m, sizeof(typename BSort::TempStorage));                  // the candidate sort
    m = std::max(m, commit_group_smem(B->max_n));                          // the set commit
    return (m + 15) & ~(size_t)15;
}

template <bool W16, int T>
static bool persistent_fits(bm_batch* B) {
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k_b_sweep<W16, T>) != cudaSuccess) { cudaGetLastError(); return false; }
    B->tile = T;
    const size_t room = B->ctx[0]->smem_optin - std::min(B->ctx[0]->smem_optin, fa.sharedSizeBytes);
    B->group_cap = (room / 4) & ~(size_t)15;
    const size_t sm = persistent_smem(B);
    // the limit is the same for every batch: one with smaller instances must not lower another's
    if (sm > room ||
        cudaFuncSetAttribute(k_b_sweep<W16, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_b_sweep<W16, T>, kBThreads, sm) != cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        return false;
    }
    return true;
}

// Whether every batch sweep can be one persistent launch: the instances'
// candidates fit the in-kernel sort and the kernel fits one CTA per SM with
// either combine tile.
template <bool W16>
static bm_status persistent_setup(bm_batch* B) {
    const int tile = B->tile;
    B->can_persist = B->max_n <= kBSortMax && persistent_fits<W16, 32>(B) && persistent_fits<W16, 64>(B);
    B->tile = tile;
    return BM_OK;
}

template <bool W16>
static bm_status enqueue_persistent(bm_batch* B, int max_scan, int max_verify, int stall = 0) {
    BSweepArgs<W16> a;
    a.views = (const DevView<W16>*)B->views;
    a.inst = B->inst;
    a.ebase = B->ebase;
    a.lists = (const typename Ent<W16>::T* const*)B->lists;
    a.nb = B->count;
    a.iorder = B->iorder;
    a.rpt = B->rpt;
    a.ways = B->ways;
    a.row_base = B->row_base;
    a.rows_total = B->total;
    a.tbase = B->tbase;
    a.total_tasks = (int)B->total_tasks;
    a.group_bytes = persistent_group_bytes(B);
    a.counter = B->counter;
    a.done = B->done;
    a.bar = B->gbar;
    a.max_scan = max_scan;
    a.max_verify = max_verify;
    a.stall = stall;
    a.st = B->cstats;
    a.acc_delta = B->acc_delta;
    a.acc_commits = B->acc_commits;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(B->ctx[0]->num_sms);
    cfg.blockDim = dim3(kBThreads);
    cfg.dynamicSmemBytes = persistent_smem(B);
    cfg.stream = B->st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (B->tile == 32) BK(cudaLaunchKernelEx(&cfg, k_b_sweep<W16, 32>, a));
    else BK(cudaLaunchKernelEx(&cfg, k_b_sweep<W16, 64>, a));
    return BM_OK;
}

// Enqueues the profit and combine stages of one batch sweep on B->st.
template <bool W16>
static bm_status enqueue_eval(bm_batch* B) {
    typedef typename Ent<W16>::T E;
    const DevView<W16>* views = (const DevView<W16>*)B->views;
    long long maxe = 0;
    for (bm_ctx* c : B->ctx) maxe = std::max(maxe, std::max(c->e1, c->e2));
    dim3 rg((unsigned)std::min<long long>((maxe + 255) / 256, 256), B->count, 4);
    k_b_relabel<W16><<<rg, 256, 0, B->st>>>(views, B->e1, B->e2, (const E* const*)B->lists, B->count);
    BK(cudaGetLastError());
    k_b_row_work<W16><<<(B->total + 7) / 8, 256, 0, B->st>>>(views, B->row_base, B->count, B->total, B->wkeys,
                                                            B->wvals);
    BK(cudaGetLastError());
    size_t tb = B->cub_bytes;
    BK(cub::DeviceRadixSort::SortPairsDescending(B->cub_tmp, tb, B->wkeys, B->wkeys_sorted, B->wvals, B->order,
                                                 B->total, 0, 64, B->st));
    BK(cudaMemsetAsync(B->counter, 0, sizeof(int), B->st));
    const size_t smem = row_smem(B->max_n);
    BK(allow_smem<k_b_profit<W16>>(smem));
    int per_sm = 0, sms = B->ctx[0]->num_sms;
    BK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_b_profit<W16>, B->profit_threads, smem));
    if (per_sm < 1) { snprintf(B->err, sizeof B->err, "profit kernel does not fit (max n %d)", B->max_n); return BM_E_INPUT; }
    k_b_profit<W16><<<sms * per_sm, B->profit_threads, smem, B->st>>>(views, B->row_base, B->count, B->total,
                                                                     B->order, B->counter);
    BK(cudaGetLastError());
    const unsigned cg = (unsigned)std::min<long long>(B->total_tiles, (long long)sms * 16);
    if (B->tile == 32) k_b_combine<32><<<cg, 256, 0, B->st>>>(B->inst, B->tile_base, B->count, B->total_tiles);
    else k_b_combine<64><<<cg, 256, 0, B->st>>>(B->inst, B->tile_base, B->count, B->total_tiles);
    BK(cudaGetLastError());
    dim3 cg2((B->max_n + 255) / 256, B->count);
    k_b_reduce<<<cg2, 256, 0, B->st>>>(B->inst, B->count);
    BK(cudaGetLastError());
    return BM_OK;
}

template <bool W16>
static bm_status enqueue_select_commit(bm_batch* B, int max_scan, int max_verify) {
    dim3 cg2((B->max_n + 255) / 256, B->count);
    k_b_candidates<<<cg2, 256, 0, B->st>>>(B->inst, B->count);
    BK(cudaGetLastError());
    size_t tb = B->cub_bytes;
    BK(cub::DeviceSegmentedRadixSort::SortKeys(B->cub_tmp, tb, B->ckeys, B->ckeys_sorted, B->total, B->count,
                                               B->row_base, B->row_base + 1, 0, 64, B->st));
    const size_t smem = commit_group_smem(B->max_n);
    BK(allow_smem<k_b_commit<W16>>(smem));
    k_b_commit<W16><<<B->count, 1024, smem, B->st>>>((const DevView<W16>*)B->views, B->inst, max_scan, max_verify,
                                                     B->cstats, B->acc_delta, B->acc_commits);
    BK(cudaGetLastError());
    return BM_OK;
}

static bm_status enqueue_sweep(bm_batch* B, int max_scan, int max_verify) {
    if (B->use_persist)
        return B->w16 ? enqueue_persistent<true>(B, max_scan, max_verify)
                      : enqueue_persistent<false>(B, max_scan, max_verify);
    bm_status s = B->w16 ? enqueue_eval<true>(B) : enqueue_eval<false>(B);
    if (s) return s;
    return B->w16 ? enqueue_select_commit<true>(B, max_scan, max_verify)
                  : enqueue_select_commit<false>(B, max_scan, max_verify);
}

extern "C" bm_status bm_batch_autotune(bm_batch* B, int32_t* profit_threads, int32_t* combine_tile) {
    if (!B) return BM_E_INPUT;
    for (bm_ctx* c : B->ctx)
        if (!c->mapped) { snprintf(B->err, sizeof B->err, "bm_batch_autotune: mappings not set"); return BM_E_STATE; }
    // candidate schedules: the persistent launch with either combine tile,
    // and the launch sequence with profit blocks of 256 or 512 threads and
    // either tile; each is timed on whole sweeps of the batch itself from the
    // same matchings, restored afterwards (results never depend on the choice)
    struct Sched { bool persist; int threads, tile; };
    std::vector<Sched> cand;
    if (B->can_persist) { cand.push_back({true, kBThreads, 32}); cand.push_back({true, kBThreads, 64}); }
    for (int pt : {256, 512})
        for (int tl : {32, 64}) cand.push_back({false, pt, tl});
    std::vector<std::vector<int32_t>> saved(B->count);
    std::vector<int32_t*> maps(B->count);
    for (int i = 0; i < B->count; i++) {
        saved[i].resize((size_t)B->ctx[i]->n + 1);
        maps[i] = saved[i].data();
    }
    bm_status got = bm_batch_get_mappings(B, maps.data());
    if (got) return got;
    auto restore = [&]() { return bm_batch_set_mappings(B, maps.data()); };
    float best = 1e30f;
    Sched pick = cand[0];
    for (const Sched& c : cand) {
        B->use_persist = c.persist;
        B->profit_threads = c.threads;
        B->tile = c.tile;
        bm_status s = batch_tiles(B);
        if (s) return s;
        // the second and third sweep from the saved matchings (the first
        // warms up and has a descent's first, commit-heavy candidate set)
        if ((s = restore())) return s;
        if ((s = enqueue_sweep(B, 0, -1))) return s;
        BK(cudaEventRecord(B->ev0, B->st));
        for (int rep = 0; rep < 2; rep++)
            if ((s = enqueue_sweep(B, 0, -1))) return s;
        BK(cudaEventRecord(B->ev1, B->st));
        BK(cudaEventSynchronize(B->ev1));
        float tot = 0;
        BK(cudaEventElapsedTime(&tot, B->ev0, B->ev1));
        if (tot < best) { best = tot; pick = c; }
    }
    bm_status s = restore();
    if (s) return s;
    B->use_persist = pick.persist;
    B->profit_threads = pick.threads;
    B->tile = pick.tile;
    if ((s = batch_tiles(B))) return s;
    B->tuned = true;
    if (B->exec) { cudaGraphExecDestroy(B->exec); B->exec = nullptr; }
    if (B->graph) { cudaGraphDestroy(B->graph); B->graph = nullptr; }
    if (profit_threads) *profit_threads = pick.threads;
    if (combine_tile) *combine_tile = pick.tile;
    return BM_OK;
}

extern "C" bm_status bm_batch_set_schedule(bm_batch* B, int32_t persistent, int32_t profit_threads,
                                           int32_t combine_tile) {
    if (!B) return BM_E_INPUT;
    if (combine_tile != 32 && combine_tile != 64) {
        snprintf(B->err, sizeof B->err, "bm_batch_set_schedule: combine_tile %d is not 32 or 64", combine_tile);
        return BM_E_INPUT;
    }
    if (persistent && !B->can_persist) {
        snprintf(B->err, sizeof B->err, "bm_batch_set_schedule: no persistent schedule (largest instance %d > %d or "
                 "the kernel does not fit)", B->max_n, kBSortMax);
        return BM_E_INPUT;
    }
    if (!persistent && profit_threads != 256 && profit_threads != 512) {
        snprintf(B->err, sizeof B->err, "bm_batch_set_schedule: profit_threads %d is not 256 or 512", profit_threads);
        return BM_E_INPUT;
    }
    B->use_persist = persistent != 0;
    B->profit_threads = persistent ? kBThreads : profit_threads;
    B->tile = combine_tile;
    bm_status s = batch_tiles(B);
    if (s) return s;
    if (B->exec) { cudaGraphExecDestroy(B->exec); B->exec = nullptr; }
    if (B->graph) { cudaGraphDestroy(B->graph); B->graph = nullptr; }
    return BM_OK;
}

extern "C" bm_status bm_batch_sweeps(bm_batch* B, int32_t sweeps, const bm_sweep_opts* opts,
                                     int64_t* committed, float* ms) {
    if (!B || sweeps < 0) return BM_E_INPUT;
    for (bm_ctx* c : B->ctx)
        if (!c->mapped) { snprintf(B->err, sizeof B->err, "bm_batch_sweeps: mappings not set"); return BM_E_STATE; }
    const int max_scan = opts ? opts->max_candidates : 0;
    const int max_verify = opts ? opts->max_verify : -1;
    // one sweep of the whole batch as a CUDA graph, captured once per option set
    if (B->exec && (max_scan != B->graph_max_scan || max_verify != B->graph_max_verify)) {
        cudaGraphExecDestroy(B->exec); B->exec = nullptr;
        cudaGraphDestroy(B->graph); B->graph = nullptr;
    }
    if (!B->exec) {
        BK(cudaStreamBeginCapture(B->st, cudaStreamCaptureModeThreadLocal));
        bm_status s = enqueue_sweep(B, max_scan, max_verify);
        cudaGraph_t g = nullptr;
        cudaError_t ce = cudaStreamEndCapture(B->st, &g);
        if (s) { if (g) cudaGraphDestroy(g); return s; }
        BK(ce);
        B->graph = g;
        BK(cudaGraphInstantiate(&B->exec, B->graph, 0));
        B->graph_max_scan = max_scan;
        B->graph_max_verify = max_verify;
    }
    BK(cudaMemsetAsync(B->acc_delta, 0, B->count * sizeof(long long), B->st));
    BK(cudaMemsetAsync(B->acc_commits, 0, B->count * sizeof(long long), B->st));
    // test hook (bm_test_stall): one sweep launched outside the graph whose
    // first grid barrier never completes
    const int stall = (B->use_persist && sweeps > 0) ? take_stall(BM_STALL_BATCH) : 0;
    BK(cudaEventRecord(B->ev0, B->st));
    if (stall) {
        bm_status s = B->w16 ? enqueue_persistent<true>(B, max_scan, max_verify, 1)
                             : enqueue_persistent<false>(B, max_scan, max_verify, 1);
        if (s) return s;
        sweeps = 0;
    }
    for (int i = 0; i < sweeps; i++) BK(cudaGraphLaunch(B->exec, B->st));
    BK(cudaEventRecord(B->ev1, B->st));
    std::vector<long long> dsum(B->count), csum(B->count);
    BK(cudaMemcpyAsync(dsum.data(), B->acc_delta, B->count * sizeof(long long), cudaMemcpyDeviceToHost, B->st));
    BK(cudaMemcpyAsync(csum.data(), B->acc_commits, B->count * sizeof(long long), cudaMemcpyDeviceToHost, B->st));
    unsigned gerr = 0;
    if (B->use_persist) BK(cudaMemcpyAsync(&gerr, B->gbar + 2, sizeof gerr, cudaMemcpyDeviceToHost, B->st));
    BK(cudaStreamSynchronize(B->st));
    if (gerr) {
        // a grid-barrier wait of the persistent sweep ran out: the matchings
        // may be partly committed; the caller sets them again
        BK(cudaMemsetAsync(B->gbar, 0, 4 * sizeof(unsigned), B->st));
        for (bm_ctx* c : B->ctx) { c->mapped = false; c->S_exact = false; }
        snprintf(B->err, sizeof B->err, "bm_batch_sweeps: persistent sweep grid barrier wait timed out");
        return BM_E_TIMEOUT;
    }
    for (int i = 0; i < B->count; i++) {
        B->ctx[i]->score += dsum[i];
        if (committed) committed[i] = csum[i];
    }
    if (ms) BK(cudaEventElapsedTime(ms, B->ev0, B->ev1));
    return BM_OK;
}

extern "C" bm_status bm_batch_info(const bm_batch* B, int32_t* count, int32_t* max_n, int64_t* total_pairs,
                                   int32_t* profit_threads, int32_t* combine_tile) {
    if (!B) return BM_E_INPUT;
    long long pairs = 0;
    for (bm_ctx* c : B->ctx) pairs += (long long)c->n * (c->n - 1) / 2;
    if (count) *count = B->count;
    if (max_n) *max_n = B->max_n;
    if (total_pairs) *total_pairs = pairs;
    if (profit_threads) *profit_threads = B->profit_threads;
    if (combine_tile) *combine_tile = B->tile;
    return BM_OK;
}
