// bm_commit.cuh -- the set commit of a sweep, a 3-cycle round or a 4-set round.
//
// The rule is sequential over the sorted candidates (sets of K vertices, K = 2
// for swaps, that permute their images among themselves):
//   * skip the set if one of its vertices already moved;
//   * otherwise its current delta is its candidate delta plus, for every G1
//     edge from one of its vertices x to an already-moved vertex y outside it,
//     the change of what the set would make of that edge, between y's
//     pre-move image and its image now; a set with at least one moved
//     neighbour is the "re-verified" case (counted, limited by max_verify);
//   * commit iff the current delta is > 0.
// A vertex moves at most once per call, so the changes that committed sets
// make to another set's delta add up, and whole windows of the list can be
// decided together: a step takes the next W live candidates, the grid scans
// their G1 lists, and per list entry (x in set j, y)
//   * y moved in an earlier step: the change above goes into corr[j];
//   * y is in earlier sets i of the window: pair (j, i) is marked adjacent and
//     the change that set i's move would make goes into cc[j][i].
// CTA 0 then replays the sequential rule on corr and cc alone (set_decide) and
// publishes the committed sets.  The decisions, the re-verification budget
// included, are those of the one-at-a-time rule.
//
// What bounds it: the serial chain per step, at n = 18,524 / E = 5e6 about
// 20 us -- select and tables 2.3, list scan 6.3 (three dependent gathers),
// collecting the grid 2.9, loading and deciding 6, publishing 1.8 -- so few
// large steps win over many small ones as long as the window's dead sets
// (those that share a vertex with an earlier commit of the window) stay cheap
// to scan.  Measured against a cluster of 8 CTAs deciding 32 pairs per step
// (candidate sort included): n = 18,524 / E = 5e6 1.97 -> 0.63 ms (100 -> 29
// steps), n = 6,007 / E = 3e5 0.92 -> 0.34 ms, n = 1,000 / E = 2e4 0.18 ->
// 0.11 ms.
#pragma once
#include <climits>
#include "bm_kernels.cuh"

namespace bm {

constexpr int kSetThreads = 1024;
// Candidates per step: the fewest steps whose decision still fits shared
// memory at every n.  256 took 16 steps of 45 us at n = 18,524 / E = 5e6 where
// 128 take 29 of 20 us (more dead sets scanned, a longer decision).
constexpr int kSetW = 128, kSetWords = kSetW / 32;
constexpr unsigned kSetPolls = 1u << 22;    // polls of one wait (seconds)
constexpr unsigned kSetAbort = 0xffffffffu;

// Step results in global memory, two copies by step parity; zero between uses.
struct SetBuf {
    static constexpr int W = kSetW, kWords = kSetWords;
    static constexpr int oCorr = 0, oFlag = W, oAdj = oFlag + ((kWords + 3) & ~3), oCC = oAdj + W * kWords;
    static constexpr int kInts = oCC + ((W * (W - 1) / 2 + 3) & ~3);
};
constexpr size_t kSetBufInts = 2 * (size_t)SetBuf::kInts + 2 * kSetWords;

struct SetArgs {
    const unsigned long long* keys;   // sorted; ~0 ends the list
    const int4* sets;                 // K > 2: (v0 | v1 << 16, v2 | v3 << 16, source of each image by bytes, -)
    int lim, max_verify;
    CommitStats* st;
    SetCtl* ctl;
    int* buf;                         // kSetBufInts ints
    int* newp;                        // n ints: images of moved vertices
    int stall;                        // test hook (bm_test_stall): the last CTA skips its first arrival
};

template <int K> struct SetSmem {
    static constexpr int W = kSetW, kWords = kSetWords;
    static constexpr int oCC = 0;                                        // W (W - 1) / 2: cc[j][i], i < j
    static constexpr int oPre = oCC + ((W * (W - 1) / 2 + 3) & ~3);      // 2 K W + 1: prefix of the list lengths
    static constexpr int oOff = oPre + 2 * K * W + 4;                    // 2 K W: list starts
    static constexpr int oV = oOff + 2 * K * W;                          // K W: vertices
    static constexpr int oPo = oV + K * W, oPn = oPo + K * W;            // their images, and those they would take
    static constexpr int oD0 = oPn + K * W, oCorr = oD0 + W;
    static constexpr int oMemb = oCorr + W;                              // K W x kWords: sets that hold a window vertex
    static constexpr int kInts = oMemb + K * W * kWords;
    // per-vertex state: bit 15 moved, else window vertex + 1 (0: not in the window)
    __host__ __device__ static size_t bytes(int n) { return (size_t)kInts * 4 + 2 * (size_t)((n + 7) & ~7); }
};

__device__ __forceinline__ unsigned set_ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void set_st_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

// What one G1 edge of weight w adds to a set's delta when its outside end's
// image goes from q to r; its inside end has image po and would take pn.
template <bool W16>
__device__ __forceinline__ int set_change(const DevView<W16>& g, bool in, int w, int po, int pn, int q, int r) {
    if (in)   // W2 columns of the set's images: rows of the transpose
        return (imin(w, g.w2t(r, pn)) - imin(w, g.w2t(r, po))) - (imin(w, g.w2t(q, pn)) - imin(w, g.w2t(q, po)));
    return (imin(w, g.w2(pn, r)) - imin(w, g.w2(po, r))) - (imin(w, g.w2(pn, q)) - imin(w, g.w2(po, q)));
}

// The sets before set j among those of word h of a membership mask.
__device__ __forceinline__ unsigned set_earlier(unsigned bits, int h, int j) {
    return h < (j >> 5) ? bits : bits & ((1u << (j & 31)) - 1u);
}

// Shared memory of set_decide.
struct SetDecide {
    float lo[8][kSetW], hi[8][kSetW];   // partial bounds and sums of part p of set j
    int sum[8][kSetW];
    unsigned done[kSetWords], take[kSetWords];
    int verified;
};

// The sequential rule over one window, by all threads.  Thread (j, p), p = tid
// / 128, looks at the 16 earlier sets 16 p .. 16 p + 15 of set j, and warps 0-3
// (p = 0) decide.  d is set j's delta without the window's commits, moved
// whether an earlier step's move makes it re-verified, adj and share the
// earlier sets that are adjacent to it or share a vertex with it, cc[i] what
// set i's commit adds to d (all for p = 0; near16, cc for every part).  The
// sets are decided in rounds: a set is skipped once an earlier set that shares
// a vertex commits, and decided once no such set is undecided and its delta
// has one sign whatever its undecided neighbours do: in a window of hub pairs
// nearly every two sets are adjacent, and waiting for the neighbours would
// decide one set per round (32 rounds per 32 sets; with the bounds 3 to 5 per
// window).  A window that would exceed the re-verification budget is decided
// again, one set per round in order.  At the end D.done/take hold the decided
// and the committed sets; returns the delta of set j if it commits (p = 0).
__device__ __forceinline__ int set_decide(SetDecide& D, const int* cc, int cnt, int d0, bool moved, unsigned near16,
                                          const unsigned (&adj)[kSetWords], const unsigned (&share)[kSetWords],
                                          int max_verify) {
    const int tid = threadIdx.x, j = tid & (kSetW - 1), p = tid / kSetW;
    const int wj = j >> 5, hp = p >> 1;
    const unsigned bit = 1u << (j & 31);
    const bool lead = p == 0, in = lead && j < cnt;
    // bounds on what the undecided neighbours can still do, rounded outwards
    float neg0 = 0.f, pos0 = 0.f;
    for (unsigned x = near16; x; x &= x - 1) {
        const int v = cc[32 * hp + __ffs(x) - 1];
        neg0 = __fadd_rd(neg0, __int2float_rd(min(v, 0)));
        pos0 = __fadd_ru(pos0, __int2float_ru(max(v, 0)));
    }
    int gain = 0;
    for (int ordered = 0;; ordered = 1) {
        __syncthreads();
        const int verified0 = D.verified;
        if (tid < kSetWords) {
            D.take[tid] = 0;
            D.done[tid] = 32 * tid >= cnt ? ~0u : cnt - 32 * tid >= 32 ? 0u : ~((1u << (cnt - 32 * tid)) - 1u);
        }
        bool und = in, gone = false, near = moved, mine = false;
        unsigned left = near16;
        float neg = neg0, pos = pos0;
        int got = 0;   // what the decided neighbours did
        D.lo[p][j] = neg;
        D.hi[p][j] = pos;
        D.sum[p][j] = 0;
        for (;;) {
            __syncthreads();
            unsigned open = 0;
#pragma unroll
            for (int h = 0; h < kSetWords; h++) open |= ~D.done[h];
            unsigned x = left & D.done[hp];
            if (x) {
                const unsigned c = D.take[hp];
                left &= ~x;
                for (; x; x &= x - 1) {
                    const int i = __ffs(x) - 1, v = cc[32 * hp + i];
                    neg = __fsub_rd(neg, __int2float_ru(min(v, 0)));
                    pos = __fsub_ru(pos, __int2float_rd(max(v, 0)));
                    if ((c >> i) & 1u) got += v;
                }
                D.lo[p][j] = left ? neg : 0.f;
                D.hi[p][j] = left ? pos : 0.f;
                D.sum[p][j] = got;
            }
            __syncthreads();
            if (lead) {
                int d = d0;
                float lo = 0.f, hi = 0.f;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    d += D.sum[q][j];
                    lo = __fadd_rd(lo, D.lo[q][j]);
                    hi = __fadd_ru(hi, D.hi[q][j]);
                }
                unsigned before = 0;
                bool wait = false;
#pragma unroll
                for (int h = 0; h < kSetWords; h++) {
                    const unsigned u = ~D.done[h], c = D.take[h];
                    before |= h < wj ? u : h == wj ? u & (bit - 1u) : 0u;
                    wait = wait || (share[h] & u);
                    gone = gone || (share[h] & c);
                    near = near || (adj[h] & c);
                }
                __syncwarp();
                asm volatile("bar.sync 1, %0;" :: "n"(kSetW) : "memory");   // every set has read the words
                if (!open) {
                    gain = mine ? d : 0;
                } else if (und) {
                    bool now = false, count = false;
                    if (gone) {
                        now = true;
                    } else if (ordered) {
                        now = !before;
                        count = now && near && D.verified < max_verify;
                        mine = now && d > 0 && (!near || count);
                    } else if (!wait) {
                        mine = __fadd_rd(__int2float_rd(d), lo) > 0.f;
                        now = mine || __fadd_ru(__int2float_ru(d), hi) <= 0.f;
                    }
                    if (now) {
                        und = false;
                        if (count) ++D.verified;
                        atomicOr(&D.done[wj], bit);
                        if (mine) atomicOr(&D.take[wj], bit);
                    }
                }
            }
            if (!open) break;
        }
        if (ordered) break;
        // one re-verification per set that was not skipped and has a moved neighbour
        if (in && !gone && near) atomicAdd(&D.verified, 1);
        __syncthreads();
        if (max_verify < 0 || D.verified <= max_verify) break;
        __syncthreads();
        if (tid == 0) D.verified = verified0;
    }
    return gain;
}

template <bool W16, int K>
__global__ void __launch_bounds__(kSetThreads, 1) k_commit_sets(DevView<W16> g, SetArgs A) {
    typedef Ent<W16> EN;
    typedef typename EN::T E;
    typedef SetSmem<K> L;
    typedef SetBuf B;
    constexpr int W = kSetW, WW = kSetWords;
    static_assert(K * W <= kSetThreads, "a thread per window vertex");
    extern __shared__ __align__(16) int sm[];
    int* s_pre = sm + L::oPre;
    int* s_off = sm + L::oOff;
    int* s_v = sm + L::oV;
    int* s_po = sm + L::oPo;
    int* s_pn = sm + L::oPn;
    int* s_d0 = sm + L::oD0;
    int* s_corr = sm + L::oCorr;
    unsigned* s_memb = reinterpret_cast<unsigned*>(sm + L::oMemb);
    unsigned short* s_st = reinterpret_cast<unsigned short*>(sm + L::kInts);
    __shared__ unsigned s_flag[WW], s_cm[WW], s_sig[W];
    __shared__ int s_wsum[32], s_next, s_ok;
    __shared__ SetDecide s_dec;
    __shared__ unsigned long long s_total;
    const int n = g.n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int ct = blockIdx.x, nct = gridDim.x;
    for (int i = tid; i < (n + 1) / 2; i += kSetThreads) reinterpret_cast<unsigned*>(s_st)[i] = 0;
    for (int i = tid; i < K * W * WW; i += kSetThreads) s_memb[i] = 0;
    if (tid < W) s_corr[tid] = 0;
    if (tid < WW) s_flag[tid] = 0;
    if (tid == 0) { s_dec.verified = 0; s_total = 0; s_ok = 1; }
    unsigned* pub = reinterpret_cast<unsigned*>(A.buf + 2 * B::kInts);
    int k = 0, nval = 0;                 // next candidate; valid candidates seen
    unsigned step = 0;
    long long entries = 0;
    int committed = 0;
    unsigned long long pkey = tid < A.lim ? A.keys[tid] : ~0ull;   // candidate k + tid, loaded ahead
    __syncthreads();
    for (;;) {
        // ---- the next W live candidates; every CTA selects the same ones ----
        int cnt = 0;
        const int k0 = k;
        for (int base = k0; cnt < W && base < A.lim; ) {
            const int idx = base + tid;
            const unsigned long long key = base == k0 ? pkey : idx < A.lim ? A.keys[idx] : ~0ull;
            const bool valid = key != ~0ull;
            int v[4] = {0, 0, 0, 0};
            unsigned sig = 1u;           // K = 2: each takes the other's image
            if (valid) {
                if (K == 2) {
                    v[0] = (int)((key >> 16) & 0xffffu);
                    v[1] = (int)(key & 0xffffu);
                } else {
                    const int4 q = A.sets[idx];
                    v[0] = q.x & 0xffff; v[1] = (int)((unsigned)q.x >> 16);
                    v[2] = q.y & 0xffff; v[3] = (int)((unsigned)q.y >> 16);
                    sig = (unsigned)q.z;
                }
            }
            bool live = valid;
#pragma unroll
            for (int m = 0; m < K; m++) live = live && !(s_st[v[m]] & 0x8000u);
            const unsigned lm = __ballot_sync(0xffffffffu, live);
            if (lane == 0) s_wsum[wid] = __popc(lm);
            const int nvalid = __syncthreads_count(valid);
            int w = s_wsum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            const int all = __shfl_sync(0xffffffffu, w, 31);
            const int before = __shfl_sync(0xffffffffu, w, (wid + 31) & 31);
            const int pos = cnt + (wid ? before : 0) + __popc(lm & ((1u << lane) - 1u));
            if (live && pos < W) {
#pragma unroll
                for (int m = 0; m < K; m++) s_v[pos * K + m] = v[m];
                s_sig[pos] = sig;
                s_d0[pos] = (int)(0x7fffffffu - (unsigned)(key >> 32));
            }
            if (live && pos == W) s_next = idx;      // the first candidate left for the next step
            __syncthreads();
            nval = max(nval, base + nvalid);
            if (cnt + all > W) { cnt = W; k = s_next; break; }
            cnt += all;
            base += kSetThreads;
            k = nvalid < kSetThreads ? A.lim : min(base, A.lim);
            if (nvalid < kSetThreads) break;
        }
        if (cnt == 0) break;
        pkey = k + tid < A.lim ? A.keys[k + tid] : ~0ull;
        // ---- the window's tables: thread j K + m for vertex m of set j ----
        int len_o = 0, len_i = 0, off_o = 0, off_i = 0;
        const int slots = cnt * K;
        if (tid < slots) {
            const int x = s_v[tid], j = tid / K;
            off_o = g.off1o[x]; len_o = g.off1o[x + 1] - off_o;
            off_i = g.off1i[x]; len_i = g.off1i[x + 1] - off_i;
            s_po[tid] = g.p[x];          // a live vertex has not moved; g.p changes only at the end
            const unsigned old = atomicCAS(&s_st[x], (unsigned short)0, (unsigned short)(tid + 1));
            const int slot = old ? (int)old - 1 : tid;
            atomicOr(&s_memb[slot * WW + (j >> 5)], 1u << (j & 31));
        }
        int incl = len_o + len_i;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_wsum[wid] = incl;
        __syncthreads();
        int tot;
        {
            int w = s_wsum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            tot = __shfl_sync(0xffffffffu, w, 31);
            const int before = __shfl_sync(0xffffffffu, w, (wid + 31) & 31);
            incl += wid ? before : 0;
        }
        if (tid < slots) {
            const int j = tid / K, m = tid - j * K;
            s_pre[2 * tid] = incl - len_o - len_i;
            s_pre[2 * tid + 1] = incl - len_i;
            s_off[2 * tid] = off_o;
            s_off[2 * tid + 1] = off_i;
            s_pn[tid] = s_po[j * K + (K == 2 ? 1 - m : (int)((s_sig[j] >> (8 * m)) & 0xffu))];
        }
        if (tid == 0) s_pre[2 * slots] = tot;
        __syncthreads();
        // ---- scan the window's list entries ----
        const int par = (int)(step & 1u);
        int* buf = A.buf + par * B::kInts;
        {   // the other copy was read before the previous step was published
            int* other = A.buf + (par ^ 1) * B::kInts;
            const int z1 = (int)((long long)B::kInts * (ct + 1) / nct);
            for (int i = (int)((long long)B::kInts * ct / nct) + tid; i < z1; i += kSetThreads) other[i] = 0;
        }
        entries += tot;
        // units of 32 U entries dealt over the grid's warps, a CTA's warps far
        // apart: later sets have more earlier ones to compare with
        constexpr int U = 2;
        for (int e0 = (wid * nct + ct) * 32 * U; e0 < tot; e0 += nct * kSetThreads * U) {
            const int w1 = min(tot, e0 + 32 * U);
            int seg = 0;
            {
                int lo = 0, hi = 2 * slots;      // s_pre[lo] <= e0 < s_pre[hi]
                while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_pre[mid] <= e0) lo = mid; else hi = mid; }
                seg = lo;
            }
            {
                int slot[U], x[U], w[U], hits[U];
                unsigned s[U];
                bool in[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int e = e0 + 32 * u + lane;
                    slot[u] = -1;
                    if (e < w1) {
                        while (e >= s_pre[seg + 1]) seg++;
                        const E en = ((seg & 1) ? g.ent1i : g.ent1o)[s_off[seg] + (e - s_pre[seg])];
                        x[u] = EN::id(en); w[u] = EN::w(en);
                        slot[u] = seg >> 1; in[u] = seg & 1;
                    } else {
                        x[u] = 0; w[u] = 0; in[u] = false;
                    }
                }
                // the changes to evaluate: one if y moved, one per earlier set that
                // holds y if y is in the window outside set j
                int mine = 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int j = slot[u] / K;
                    s[u] = slot[u] >= 0 ? s_st[x[u]] : 0u;
                    hits[u] = (int)(s[u] >> 15);
                    if (s[u] != 0 && !(s[u] & 0x8000u)) {
                        bool inner = false;
#pragma unroll
                        for (int m = 0; m < K; m++) inner = inner || s_v[j * K + m] == x[u];
                        if (!inner) {
                            const unsigned* mb = s_memb + (s[u] - 1) * WW;
                            for (int h = 0; h <= (j >> 5); h++) {
                                const unsigned bits = set_earlier(mb[h], h, j);
                                if (bits) atomicOr(reinterpret_cast<unsigned*>(buf + B::oAdj + j * WW + h), bits);
                                hits[u] += __popc(bits);
                            }
                        }
                    }
                    mine += hits[u];
                }
                // spread evenly over the warp's lanes (a vertex that is the best partner
                // of many is in many sets), V of a lane's in flight together
                int upto = mine;
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += y;
                }
                const int total = __shfl_sync(0xffffffffu, upto, 31);
                constexpr int V = 2;
                for (int t0 = 0; t0 < total; t0 += 32 * V) {
                    int ej[V], ei[V], ew[V], q[V], r[V], po[V], pn[V], c[V];
                    bool ein[V];
#pragma unroll
                    for (int v = 0; v < V; v++) {
                        const int t = t0 + 32 * v + lane;
                        ej[v] = -1;
                        if (t0 + 32 * v >= total) continue;   // the whole warp
                        int src = 0;                          // first lane with upto > t
#pragma unroll
                        for (int o = 16; o; o >>= 1) {
                            const int y = __shfl_sync(0xffffffffu, upto, src + o - 1);
                            if (y <= t) src += o;
                        }
                        int rank = t - __shfl_sync(0xffffffffu, upto - mine, src);
                        int ex = 0, eslot = 0;
                        unsigned es = 0;
                        bool found = false;
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int hu = __shfl_sync(0xffffffffu, hits[u], src), xu = __shfl_sync(0xffffffffu, x[u], src);
                            const int wu = __shfl_sync(0xffffffffu, w[u], src);
                            const unsigned su = __shfl_sync(0xffffffffu, s[u] | (unsigned)(2 * slot[u] + (int)in[u]) << 16, src);
                            if (!found) {
                                if (rank < hu) { found = true; ex = xu; ew[v] = wu; es = su; }
                                else rank -= hu;
                            }
                        }
                        if (t >= total) continue;
                        ein[v] = (es >> 16) & 1u;
                        eslot = (int)(es >> 17);
                        es &= 0xffffu;
                        ej[v] = eslot / K;
                        po[v] = s_po[eslot]; pn[v] = s_pn[eslot];
                        if (es & 0x8000u) {      // moved: from its image before the call to its image now
                            ei[v] = -1;
                            q[v] = g.p[ex]; r[v] = __ldcg(&A.newp[ex]);
                        } else {                 // the rank-th earlier set that holds it
                            const unsigned* mb = s_memb + (es - 1) * WW;
                            int h = 0;
                            unsigned bits = set_earlier(mb[0], 0, ej[v]);
                            while (rank >= __popc(bits)) { rank -= __popc(bits); h++; bits = set_earlier(mb[h], h, ej[v]); }
                            for (; rank; rank--) bits &= bits - 1;
                            ei[v] = 32 * h + __ffs(bits) - 1;
                            int m = ei[v] * K;
                            while (s_v[m] != ex) m++;
                            q[v] = s_po[m]; r[v] = s_pn[m];
                        }
                    }
#pragma unroll
                    for (int v = 0; v < V; v++)
                        c[v] = ej[v] >= 0 ? set_change<W16>(g, ein[v], ew[v], po[v], pn[v], q[v], r[v]) : 0;
#pragma unroll
                    for (int v = 0; v < V; v++) {
                        if (ej[v] < 0) continue;
                        if (ei[v] < 0) {
                            if (c[v]) atomicAdd(&s_corr[ej[v]], c[v]);
                            atomicOr(&s_flag[ej[v] >> 5], 1u << (ej[v] & 31));
                        } else if (c[v]) {
                            atomicAdd(buf + B::oCC + ej[v] * (ej[v] - 1) / 2 + ei[v], c[v]);
                        }
                    }
                }
            }
        }
        __syncthreads();
        if (tid < cnt) {
            const int c = s_corr[tid];
            if (c) { atomicAdd(buf + B::oCorr + tid, c); s_corr[tid] = 0; }
        }
        if (tid < WW) {
            const unsigned f = s_flag[tid];
            if (f) { atomicOr(reinterpret_cast<unsigned*>(buf + B::oFlag + tid), f); s_flag[tid] = 0; }
        }
        // ---- collect, decide, publish ----
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            if (!(A.stall && step == 0 && nct > 1 && ct == nct - 1)) atomicAdd(&A.ctl->arrived, 1u);
            if (ct == 0) {
                const unsigned want = (unsigned)nct * (step + 1), limit = A.stall ? kStallPolls : kSetPolls;
                unsigned it = 0;
                while (set_ld_acquire(&A.ctl->arrived) != want)
                    if (++it > limit) { s_ok = 0; break; }
                if (!s_ok) {
                    atomicOr(&A.ctl->err, 2);
                    set_st_release(&A.ctl->released, kSetAbort);
                }
            }
        }
        if (ct == 0) {
            __syncthreads();
            if (!s_ok) return;
            int* s_cc = sm + L::oCC;
            {
                const int q4 = (cnt * (cnt - 1) / 2 + 3) / 4;
                const int4* src = reinterpret_cast<const int4*>(buf + B::oCC);
                for (int i = tid; i < q4; i += kSetThreads) reinterpret_cast<int4*>(s_cc)[i] = __ldcg(src + i);
            }
            unsigned adj[WW], share[WW], near16 = 0;   // earlier sets of the window: adjacent, sharing a vertex
            int d = 0;
            bool moved = false;
            const int j = tid & (W - 1), part = tid / W;
#pragma unroll
            for (int h = 0; h < WW; h++) { adj[h] = 0; share[h] = 0; }
            if (j < cnt) {
                const unsigned* gadj = reinterpret_cast<unsigned*>(buf + B::oAdj) + j * WW;
                near16 = __ldcg(gadj + (part >> 1)) & (0xffffu << (16 * (part & 1)));
                if (part == 0) {
                    d = s_d0[j] + __ldcg(buf + B::oCorr + j);
                    moved = (__ldcg(reinterpret_cast<unsigned*>(buf + B::oFlag) + (j >> 5)) >> (j & 31)) & 1u;
#pragma unroll
                    for (int h = 0; h < WW; h++) {
                        if (32 * h >= j) break;
                        adj[h] = __ldcg(gadj + h);
#pragma unroll
                        for (int m = 0; m < K; m++) share[h] |= s_memb[(s_st[s_v[j * K + m]] - 1) * WW + h];
                        share[h] = set_earlier(share[h], h, j);
                    }
                }
            }
            __syncthreads();   // cc has arrived
            const int gain = set_decide(s_dec, s_cc + j * (j - 1) / 2, cnt, d, moved, near16, adj, share, A.max_verify);
            if (tid < WW) s_cm[tid] = s_dec.take[tid];
            if (tid < W) {
                long long won = gain;
                for (int o = 16; o; o >>= 1) won += __shfl_xor_sync(0xffffffffu, won, o);
                if (lane == 0 && won) atomicAdd(&s_total, (unsigned long long)won);
            }
            __syncthreads();
            if (tid < WW) __stcg(&pub[par * WW + tid], s_cm[tid]);
            if (tid < slots) {
                const int j = tid / K;
                if ((s_cm[j >> 5] >> (j & 31)) & 1u) __stcg(&A.newp[s_v[tid]], s_pn[tid]);
            }
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                set_st_release(&A.ctl->released, step + 1);
                for (int q = 0; q < WW; q++) committed += __popc(s_cm[q]);
            }
        } else {
            if (tid == 0) {
                const unsigned limit = kSetPolls;
                unsigned it = 0, r;
                while ((r = set_ld_acquire(&A.ctl->released)) != step + 1) {
                    if (r == kSetAbort) { s_ok = 0; break; }
                    if (++it > limit) { s_ok = 0; atomicOr(&A.ctl->err, 2); break; }
                }
            }
            __syncthreads();
            if (!s_ok) return;
            if (tid < WW) s_cm[tid] = __ldcg(&pub[par * WW + tid]);
            __syncthreads();
        }
        // ---- every CTA: committed vertices are moved, the window is left ----
        for (int i = tid; i < slots * WW; i += kSetThreads) s_memb[i] = 0;
        if (tid < slots) s_st[s_v[tid]] = 0;
        __syncthreads();
        if (tid < slots) {
            const int j = tid / K;
            if ((s_cm[j >> 5] >> (j & 31)) & 1u) s_st[s_v[tid]] = 0x8000u;
        }
        step++;
        __syncthreads();
    }
    // the copy of the last step is cleared for the next launch, and the moved
    // vertices' images are written back (no CTA reads g.p or the copies again)
    if (step) {
        int* last = A.buf + ((step - 1) & 1u) * B::kInts;
        const int z1 = (int)((long long)B::kInts * (ct + 1) / nct);
        for (int i = (int)((long long)B::kInts * ct / nct) + tid; i < z1; i += kSetThreads) last[i] = 0;
    }
    const int v1 = (int)((long long)n * (ct + 1) / nct);
    for (int v = (int)((long long)n * ct / nct) + tid; v < v1; v += kSetThreads)
        if (s_st[v] & 0x8000u) {
            const int f = __ldcg(&A.newp[v]);
            g.p[v] = f;
            if (f < n) g.pinv[f] = v;
        }
    if (ct == 0 && tid == 0) {
        A.st->total_delta = (long long)s_total;
        A.st->scanned = min(nval, A.lim);
        A.st->verified = s_dec.verified;
        A.st->committed = committed;
        A.st->steps = (int)step;
        A.st->entries = entries;
        A.st->carried = 0;   // every set is decided in the step that scans it
    }
}

}  // namespace bm
