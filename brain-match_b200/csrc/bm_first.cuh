// bm_first.cuh -- the reference's sequential first-improvement order
// (src/graph-alignment-optimized.c:515-577) in persistent kernels.
//
// The order visits the pairs (m1, m2), m2 != m1, row by row and commits every
// swap whose delta on the current matching is > 0.  A step evaluates the next
// pairs of that order at once on the current matching; the first improving one
// is the next commit, since no pair before it changes anything, and the order
// goes on right behind it.  Every CTA keeps the whole matching in shared memory
// and makes the same commits, so the only thing the CTAs exchange per step is 8
// bytes each: their first improving pair, tagged with the step.
//
// k_first_rows (n up to about 18,800, short lists): one cluster of 16 CTAs, a row of n
// deltas per CTA and step.  With C[v] the current contribution of v,
//     delta(a, b) = acc[b] - C[a] - C[b],
// acc[b] = what a would earn on b's image plus what b would earn on a's, is
// summed sparse x sparse in shared memory: a's G1 edges against the G2 lists
// of their ends' images, and the G2 edges of p(a) against the G1 lists of the
// vertices they are matched to; an edge between a and b is corrected.  A commit
// updates C at the neighbours of the two vertices.  Bound by the latency of a
// step, about 6 us: extents, lists and shared atomics 3, the search 1, the
// exchange through distributed shared memory and the slowest row 1, C 1.5.  One
// warp polls the words: with every warp polling, or a cluster barrier instead, a
// step took 1 us more (n = 600 / E = 12,000: 20.4 ms, now 17.8).
//
// k_first (otherwise): the whole grid, a warp per pair (several when the window
// has fewer pairs than there are warps), the words exchanged through slots in
// global memory that every CTA polls.  The window is four times the last
// distance between commits, so that few pairs behind the next commit are
// evaluated and waited for, and grows while nothing improves.  Bound by the W2
// gathers, one L1 line each, and the exchange (6 us).
//
// Three launches, a copy and a host wait per row scan took 189 ms at n = 600 /
// E = 12,000 (2,171 commits in 6 passes; now 18 ms) and 1,240 ms for one pass at
// n = 3,000 / E = 6e5 (now 423 ms).
#pragma once
#include "bm_kernels.cuh"

namespace bm {

constexpr int kFirstThreads = 512;
constexpr int kFirstMin = 256;               // k_first: pairs of the smallest window
constexpr int kFirstMult = 8;                // k_first: pairs per warp of the largest window
constexpr double kFirstLongLists = 1024;     // k_first: average entries of a pair's lists for more than one CTA per SM
constexpr int kRowsCluster = 16;             // k_first_rows: CTAs, rows per step
constexpr int kRowsThreads = 1024;
// k_first_rows: average terms of a row.  First pass, rows against grid: n = 600,
// degree 20 (1,600 terms) 18 / 25 ms for all passes, n = 1,500, degree 30
// (3,600) 79 / 85 ms, degree 60 (14,400) 118 / 93 ms, degree 130 203 / 102 ms.
constexpr double kRowsTerms = 4096;
constexpr int kFirstSteps = 1024;            // steps per launch (the host relaunches)
// Polls of one slot (seconds).  The kernels' STALL forms (bm_test_stall) poll a
// few thousand times, and their last CTA keeps its words to itself; they are
// kernels of their own because a run-time switch took 0.3 to 1.3%.
constexpr unsigned kFirstPolls = 1u << 22;
constexpr unsigned long long kFirstNone = (1ull << 51) - 1;   // (place << 31 | delta) of no pair

// The scan between launches; zero at the start.
struct FirstState {
    int m1, m2;              // next pair
    int in_pass, passes;     // commits of this pass, finished passes
    int done, err;
    long long delta, commits;
};

template <bool W16, bool STALL>
__global__ void __launch_bounds__(kFirstThreads) k_first(DevView<W16> g, FirstState* __restrict__ st,
                                                         unsigned long long* slots, int max_passes) {
    constexpr int NWARP = kFirstThreads / 32;
    extern __shared__ unsigned short p16[];   // the matching; unmatched = n
    __shared__ unsigned long long s_red[NWARP];
    __shared__ int s_part[NWARP];
    __shared__ int s_ok;
    const int n = g.n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int G = gridDim.x, nw = G * NWARP;
    for (int v = tid; v < n; v += kFirstThreads) p16[v] = (unsigned short)g.p[v];
    if (tid == 0) s_ok = 1;
    constexpr unsigned polls = STALL ? kStallPolls : kFirstPolls;
    const int most = nw * kFirstMult;
    int want = kFirstMin;
    int m1 = st->m1, m2 = st->m2, in_pass = st->in_pass, passes = st->passes, done = 0;
    long long delta = st->delta, commits = st->commits;
    __syncthreads();
    for (int step = 0; step < kFirstSteps && !done; step++) {
        const long long rest = (long long)(n - m1) * n - m2;   // pairs left in the pass
        const int win = (int)min((long long)want, rest);
        // ---- the first improving pair of the window among this CTA's ----
        unsigned long long best = kFirstNone;
        int parts = 1;                       // warps per pair, of one CTA
        while (2 * parts <= NWARP && 2 * parts * win <= nw) parts *= 2;
        auto img = [&](int v) { return (int)p16[v]; };
        if (parts > 1) {
            const int off = (wid / parts) * G + blockIdx.x;
            const int t = m2 + off, a = m1 + t / n, b = t % n;
            int d = 0;
            if (off < win && a != b) d = swap_delta_warp<W16>(g, img, a, b, lane, wid % parts, parts);
            if (lane == 0) s_part[wid] = d;
            __syncthreads();
            if (wid % parts == 0) {
                d = lane < parts ? s_part[wid + lane] : 0;
                d = __reduce_add_sync(0xffffffffu, d);
                if (d > 0) best = (unsigned long long)off << 31 | (unsigned)d;
            }
        } else {
            for (int off = wid * G + blockIdx.x; off < win; off += nw) {   // neighbouring pairs on different SMs
                const int t = m2 + off, a = m1 + t / n, b = t % n;
                if (a == b) continue;
                const int d = swap_delta_warp<W16>(g, img, a, b, lane);
                if (d > 0) { best = (unsigned long long)off << 31 | (unsigned)d; break; }
            }
        }
        if (lane == 0) s_red[wid] = best;
        __syncthreads();
        // ---- exchange: this CTA's slot of the step's copy, tagged ----
        unsigned long long* sl = slots + (step & 1) * G;
        const unsigned long long tag = (unsigned long long)(step + 1) << 51;
        if (wid == 0) {
            best = lane < NWARP ? s_red[lane] : kFirstNone;
            for (int o = 16; o; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane == 0 && !(STALL && (int)blockIdx.x == G - 1))
                asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(sl + blockIdx.x), "l"(tag | best) : "memory");
        }
        best = kFirstNone;
        for (int s = tid; s < G; s += kFirstThreads) {
            unsigned long long v;
            for (unsigned it = 0;;) {
                asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(sl + s) : "memory");
                if ((v & ~kFirstNone) == tag) break;
                if (++it > polls) { s_ok = 0; v = kFirstNone; break; }
            }
            best = min(best, v & kFirstNone);
        }
        for (int o = 16; o; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
        __syncthreads();     // s_red is read
        if (lane == 0) s_red[wid] = best;
        __syncthreads();
        if (!s_ok) {
            if (tid == 0) st->err = 1;
            return;
        }
        best = lane < NWARP ? s_red[lane] : kFirstNone;
        for (int o = 16; o; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
        // ---- commit, or go on behind the window ----
        int next;
        if (best != kFirstNone) {
            const int off = (int)(best >> 31), t = m2 + off, a = m1 + t / n, b = t % n;
            if (tid == 0) {
                const unsigned short f = p16[a];
                p16[a] = p16[b];
                p16[b] = f;
            }
            delta += (long long)(best & 0x7fffffffull);
            commits++;
            in_pass++;
            want = min(max(4 * (off + 1), kFirstMin), most);
            next = off + 1;
        } else {
            want = min(4 * want, most);
            next = win;
        }
        const int t = m2 + next;
        m1 += t / n;
        m2 = t % n;
        if (m1 >= n) {       // the pass is over
            passes++;
            done = in_pass == 0 || passes >= max_passes;
            m1 = m2 = in_pass = 0;
        }
        __syncthreads();     // the matching is swapped, s_red may be written
    }
    if (blockIdx.x) return;
    for (int v = tid; v < n; v += kFirstThreads) {
        const int f = p16[v];
        g.p[v] = f;
        if (f < n) g.pinv[f] = v;
    }
    if (tid == 0) {
        st->m1 = m1; st->m2 = m2; st->in_pass = in_pass; st->passes = passes;
        st->done = done; st->delta = delta; st->commits = commits;
    }
}

// Shared memory of k_first_rows: acc (n + 1), C (n), matching and its inverse.
__host__ __device__ inline size_t first_rows_smem(int n) {
    return (2 * (size_t)n + 1) * sizeof(int) + 2 * ((size_t)n + 1) * sizeof(unsigned short);
}

template <bool W16, bool STALL>
__global__ void __launch_bounds__(kRowsThreads, 1) k_first_rows(DevView<W16> g, FirstState* __restrict__ st,
                                                                int* __restrict__ Cg, int max_passes) {
    typedef Ent<W16> EN;
    typedef typename EN::T E;
    constexpr int T = kRowsThreads, NWARP = T / 32;
    extern __shared__ int acc[];                       // n + 1: slot n absorbs terms of unmatched G2 vertices
    __shared__ unsigned long long s_red[NWARP], s_slot[2][kRowsCluster], s_word;
    __shared__ int s_ok;
    const int n = g.n;
    int* C = acc + n + 1;
    unsigned short* p16 = reinterpret_cast<unsigned short*>(C + n);   // n + 1: G1 -> G2, unmatched n
    unsigned short* q16 = p16 + n + 1;                                // n + 1: G2 -> G1
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int v = tid; v <= n; v += T) {
        p16[v] = (unsigned short)(v < n ? g.p[v] : n);
        q16[v] = (unsigned short)(v < n ? g.pinv[v] : n);
        acc[v] = 0;
        if (v < n) C[v] = Cg[v];
    }
    if (tid == 0) s_ok = 1;
    if (tid < 2 * kRowsCluster) (&s_slot[0][0])[tid] = 0;
    const bool loops = g.offs[n] > 0;
    constexpr unsigned polls = STALL ? kStallPolls : kFirstPolls;
    int m1 = st->m1, m2 = st->m2, in_pass = st->in_pass, passes = st->passes, done = 0;
    long long delta = st->delta, commits = st->commits;
    int rows = 1, seen = 0;   // rows of this step; rows since the last commit
    __syncthreads();
    // every CTA's slots are cleared before anyone writes into them
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int step = 0; step < kFirstSteps && !done; step++) {
        const int a = m1 + (int)blockIdx.x;
        unsigned long long best = kFirstNone;
        if ((int)blockIdx.x < rows && a < n) {
            const int pa = p16[a];
            // ---- acc: list j of the row, for j in out(a), in(a), out2(p a), in2(p a) ----
            const int o1 = g.off1o[a], i1 = g.off1i[a], o2 = g.off2o[pa], i2 = g.off2i[pa];
            const int e0 = g.off1o[a + 1] - o1, e1 = e0 + g.off1i[a + 1] - i1;
            const int e2 = e1 + g.off2o[pa + 1] - o2, e3 = e2 + g.off2i[pa + 1] - i2;
            const int da = g.w2d(pa);
            for (int base = wid; base < e3; base += NWARP * 32) {
                // lane t sets up the warp's t-th list of this round
                const int j = base + NWARP * lane;
                int w = 0, b0 = 0, len = 0, kind = 0, x0 = -1, ca = 0, cb = 0, db = 0;
                if (j < e3) {
                    kind = j < e0 ? 0 : j < e1 ? 1 : j < e2 ? 2 : 3;
                    const E e = kind == 0 ? g.ent1o[o1 + j] : kind == 1 ? g.ent1i[i1 + (j - e0)]
                              : kind == 2 ? g.ent2o[o2 + (j - e1)] : g.ent2i[i2 + (j - e2)];
                    w = EN::w(e);
                    const int x = EN::id(e);
                    const int f = kind < 2 ? p16[x] : q16[x];
                    // out-edges meet in-lists, in-edges out-lists
                    const int* off = kind == 0 ? g.off2i : kind == 1 ? g.off2o : kind == 2 ? g.off1i : g.off1o;
                    b0 = off[f];
                    len = off[f + 1] - b0;
                    if (kind < 2) { x0 = x; ca = g.w2(pa, f); cb = g.w2t(f, pa); db = g.w2d(f); }
                }
                const int cnt = min(32, (e3 - base + NWARP - 1) / NWARP);
                constexpr int U = 4;
                for (int t = 0; t < cnt; t += U) {
                    E x[U];
                    int bt[U], lt[U], wt[U], kt[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int src = (t + u) & 31;
                        bt[u] = __shfl_sync(0xffffffffu, b0, src);
                        lt[u] = t + u < cnt ? __shfl_sync(0xffffffffu, len, src) : 0;
                        wt[u] = __shfl_sync(0xffffffffu, w, src);
                        kt[u] = __shfl_sync(0xffffffffu, kind, src);
                        const E* list = kt[u] == 0 ? g.ent2i : kt[u] == 1 ? g.ent2o : kt[u] == 2 ? g.ent1i : g.ent1o;
                        if (lane < lt[u]) x[u] = list[bt[u] + lane];
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const E* list = kt[u] == 0 ? g.ent2i : kt[u] == 1 ? g.ent2o : kt[u] == 2 ? g.ent1i : g.ent1o;
                        for (int k = lane; k < lt[u]; k += 32) {
                            const E y = k < 32 ? x[u] : list[bt[u] + k];
                            const int v = EN::id(y);
                            atomicAdd(&acc[kt[u] < 2 ? (int)q16[v] : v], imin(wt[u], EN::w(y)));
                        }
                    }
                }
                if (x0 >= 0) {   // an edge between a and x0: both ends move
                    const int c = imin(w, ca) + imin(w, cb) - imin(w, da) - imin(w, db);
                    if (c) atomicAdd(&acc[x0], c);
                }
            }
            if (loops) {   // G1 self-loops: a's on every image, every vertex's on a's image
                const int q0 = g.offs[a], q1 = g.offs[a + 1];
                for (int b = tid; b < n; b += T) {
                    int s = 0;
                    if (q1 > q0) {
                        const int d = g.w2d(p16[b]);
                        for (int q = q0; q < q1; q++) s += imin(g.selfw[q], d);
                    }
                    for (int q = g.offs[b]; q < g.offs[b + 1]; q++) s += imin(g.selfw[q], da);
                    if (s) atomicAdd(&acc[b], s);
                }
            }
            __syncthreads();
            const int start = blockIdx.x ? 0 : m2, cur = C[a];
            for (int b = tid; b <= n; b += T) {
                const int d = acc[b] - cur - (b < n ? C[b] : 0);
                acc[b] = 0;
                if (b >= start && b < n && b != a && d > 0 && best == kFirstNone)
                    best = (unsigned long long)(blockIdx.x << 16 | (unsigned)b) << 31 | (unsigned)d;
            }
        }
        for (int o = 16; o; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
        if (lane == 0) s_red[wid] = best;
        __syncthreads();
        // ---- exchange: this CTA's word into its slot of every CTA ----
        const int par = step & 1;
        const unsigned long long tag = (unsigned long long)(step + 1) << 51;
        if (wid == 0) {
            best = lane < NWARP ? s_red[lane] : kFirstNone;
            for (int o = 16; o; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane < kRowsCluster && !(STALL && (int)blockIdx.x == kRowsCluster - 1)) {
                const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&s_slot[par][blockIdx.x]);
                uint32_t peer;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(mine), "r"(lane));
                asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" :: "r"(peer), "l"(tag | best) : "memory");
            }
        }
        best = kFirstNone;
        if (wid == 0 && lane < kRowsCluster) {
            const uint32_t here = (uint32_t)__cvta_generic_to_shared(&s_slot[par][lane]);
            unsigned long long v;
            for (unsigned it = 0;;) {
                asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(here) : "memory");
                if ((v & ~kFirstNone) == tag) break;
                if (++it > polls) { s_ok = 0; v = kFirstNone; break; }
            }
            best = v & kFirstNone;
        }
        if (wid == 0) {
            for (int o = 16; o; o >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (lane == 0) s_word = best;
        }
        __syncthreads();     // the words are read
        if (!s_ok) break;
        best = s_word;
        if (best != kFirstNone) {
            // ---- commit: x takes y's image and y x's; C at their neighbours ----
            const int at = (int)(best >> 31), x = m1 + (at >> 16), y = at & 0xffff;
            const int px = p16[x], py = p16[y];
            __syncthreads();
            if (tid == 0) {
                p16[x] = (unsigned short)py;
                p16[y] = (unsigned short)px;
                if (py < n) q16[py] = (unsigned short)x;
                if (px < n) q16[px] = (unsigned short)y;
                C[x] = C[y] = 0;
            }
            __syncthreads();
            const int ox = g.off1o[x], oy = g.off1o[y], ix = g.off1i[x], iy = g.off1i[y];
            const int e0 = g.off1o[x + 1] - ox, e1 = e0 + g.off1o[y + 1] - oy;
            const int e2 = e1 + g.off1i[x + 1] - ix, e3 = e2 + g.off1i[y + 1] - iy;
            for (int k = tid; k < e3; k += T) {
                const bool out = k < e1, isx = out ? k < e0 : k < e2;
                const E e = out ? g.ent1o[isx ? ox + k : oy + (k - e0)] : g.ent1i[isx ? ix + (k - e1) : iy + (k - e2)];
                const int v = EN::id(e), w = EN::w(e);
                const int po = isx ? px : py, pn = isx ? py : px;
                const int q = p16[v];
                const int now = imin(w, out ? g.w2(pn, q) : g.w2t(q, pn));
                atomicAdd(&C[isx ? x : y], now);
                if (v != (isx ? y : x)) {
                    const int c = now - imin(w, out ? g.w2(po, q) : g.w2t(q, po));
                    if (c) atomicAdd(&C[v], c);
                }
            }
            if (loops) {
                for (int q = g.offs[x] + tid; q < g.offs[x + 1]; q += T) atomicAdd(&C[x], imin(g.selfw[q], g.w2d(py)));
                for (int q = g.offs[y] + tid; q < g.offs[y + 1]; q += T) atomicAdd(&C[y], imin(g.selfw[q], g.w2d(px)));
            }
            delta += (long long)(best & 0x7fffffffull);
            commits++;
            in_pass++;
            // as many rows as the last commit took, so that few rows behind the
            // next one are evaluated and waited for
            rows = min(seen + (at >> 16) + 1, kRowsCluster);
            seen = 0;
            m1 = x;
            m2 = y + 1;
            if (m2 == n) { m1++; m2 = 0; }
        } else {
            m1 += rows;
            m2 = 0;
            seen += rows;
            rows = min(2 * rows, kRowsCluster);
        }
        if (m1 >= n) {       // the pass is over
            passes++;
            done = in_pass == 0 || passes >= max_passes;
            m1 = m2 = in_pass = 0;
        }
        __syncthreads();     // C is updated, s_red may be written
    }
    // no CTA leaves while another may still write into its slots; every CTA gets here
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (!s_ok) {
        if (tid == 0) st->err = 1;
        return;
    }
    if (blockIdx.x) return;
    for (int v = tid; v < n; v += T) {
        g.p[v] = p16[v];
        g.pinv[v] = q16[v];
        Cg[v] = C[v];
    }
    if (tid == 0) {
        st->m1 = m1; st->m2 = m2; st->in_pass = in_pass; st->passes = passes;
        st->done = done; st->delta = delta; st->commits = commits;
    }
}

}  // namespace bm
