// bm_select.cuh -- pair combine and move selection of the sweep.
//
// k_combine64: 64x64 tiles of the upper triangle of S.  Each tile (I,J), I<=J,
//   reads S[I][J] and S[J][I] once (coalesced rows), forms
//   delta(a,b) = S[a][b] + S[b][a] - S[a][a] - S[b][b] and writes, for every
//   vertex of the tile, its best partner inside the tile to a partial array
//   P[tile column][vertex]; k_best_reduce folds the partials into rowbest.
//   No atomics; every (tile, vertex) slot is written exactly once.
// commit_group: the sequential set commit of a batched instance by one CTA
//   (candidates sorted by delta desc, skip a pair whose vertex already moved,
//   re-evaluate it on the current matching, commit iff > 0), several pairs per
//   step.  bm_commit.cuh has the set commit of a single instance.
#pragma once
#include <climits>
#include "bm_kernels.cuh"

namespace bm {

constexpr int kTile = 64;

// Shared memory of one combine tile pass.
template <int T> struct CombineSmem {
    static constexpr int kSegs = 128 / T;   // threads per owner: the partners in kSegs shares
    int sA[T][T + 1];               // sA[r][c] = S[a0+r][b0+c]
    int sB[T][T + 1];               // sB[r][c] = S[b0+r][a0+c]
    int dA[T], dB[T];
    int2 best[2][kSegs][T];         // (delta + own diagonal, partner) of each owner's share
};

// One TxT tile (ti <= tj) of the upper triangle by 256 threads (tid 0..255 among
// them; T = 32 or 64; `sync` is a barrier over exactly those threads), staged in
// `sm`.  A thread owns one vertex of the tile -- a row vertex (threads 0-127) or
// a column vertex -- and walks a share of its partners in ascending order, so a
// best is a compare and two moves in registers; reading the other tile
// transposed costs no more than the tile itself (rows padded by one word).
// Lanes holding rows, with a shuffle reduction per row and packed 64-bit keys,
// took 2.3 times the instructions.
template <int T, typename Sync>
__device__ __forceinline__ void combine_tile_on(const int* __restrict__ S, int n, int ti, int tj,
                                                unsigned long long* __restrict__ part, int* __restrict__ all_out,
                                                CombineSmem<T>& sm, int tid, Sync sync) {
    constexpr int SEGS = CombineSmem<T>::kSegs, L = T / SEGS;   // partners per share
    const int a0 = ti * T, b0 = tj * T;
    const size_t ld = s_pitch(n);
    // 16-byte streaming loads: a 4-column group that starts inside the matrix
    // lies inside its row's pitch
    for (int i = tid; i < T * T / 4; i += 256) {
        const int r = i / (T / 4), c = (i % (T / 4)) * 4;
        const int a = a0 + r, b = b0 + c;
        const int bb = b0 + r, aa = a0 + c;
        int4 va = make_int4(0, 0, 0, 0), vb = make_int4(0, 0, 0, 0);
        if (a < n && b < n) va = __ldcs(reinterpret_cast<const int4*>(S + a * ld + b));
        if (bb < n && aa < n) vb = __ldcs(reinterpret_cast<const int4*>(S + bb * ld + aa));
        sm.sA[r][c] = va.x; sm.sA[r][c + 1] = va.y; sm.sA[r][c + 2] = va.z; sm.sA[r][c + 3] = va.w;
        sm.sB[r][c] = vb.x; sm.sB[r][c + 1] = vb.y; sm.sB[r][c + 2] = vb.z; sm.sB[r][c + 3] = vb.w;
    }
    if (tid < T) {
        const int a = a0 + tid, b = b0 + tid;
        sm.dA[tid] = a < n ? S[a * ld + a] : 0;
        sm.dB[tid] = b < n ? S[b * ld + b] : 0;
    }
    sync();
    const bool diag = ti == tj;   // its row owners already cover both orders of every pair
    const int dir = tid >> 7, seg = (tid & 127) / T, o = tid & (T - 1);
    if (!(dir && diag)) {
        const int (*X)[T + 1] = dir ? sm.sB : sm.sA;   // X[o][c]: own row
        const int (*Y)[T + 1] = dir ? sm.sA : sm.sB;   // Y[c][o]: the partner's row
        const int* dP = dir ? sm.dA : sm.dB;
        const int p0 = dir ? a0 : b0;                  // partner c is vertex p0 + c
        const int skip = diag ? o : -1, last = min(L * (seg + 1), n - p0);
        int bd = INT_MIN, bi = -1;
        if (!diag && last == L * (seg + 1)) {
#pragma unroll 8
            for (int c = L * seg; c < L * (seg + 1); c++) {
                const int d = X[o][c] + Y[c][o] - dP[c];
                if (d > bd || bi < 0) { bd = d; bi = c; }
            }
        } else {
            for (int c = L * seg; c < last; c++) {
                const int d = X[o][c] + Y[c][o] - dP[c];
                if (c != skip && (d > bd || bi < 0)) { bd = d; bi = c; }
            }
        }
        sm.best[dir][seg][o] = make_int2(bd, bi);
    }
    if (all_out) {
        for (int i = tid; i < T * T; i += 256) {
            const int r = i / T, c = i % T, a = a0 + r, b = b0 + c;
            if (a < b && b < n)
                all_out[(long long)a * (2LL * n - a - 1) / 2 + (b - a - 1)] =
                    sm.sA[r][c] + sm.sB[c][r] - sm.dA[r] - sm.dB[c];
        }
    }
    sync();
    if (tid < 2 * T) {
        const int d = tid / T, q = tid & (T - 1), x = (d ? b0 : a0) + q;
        if (x < n && !(d && diag)) {
            int2 k = sm.best[d][0][q];
#pragma unroll
            for (int g = 1; g < SEGS; g++) {   // the lower share keeps ties: its partners are smaller
                const int2 y = sm.best[d][g][q];
                if (y.y >= 0 && (k.y < 0 || y.x > k.x)) k = y;
            }
            part[(size_t)(d ? ti : tj) * n + x] =
                k.y < 0 ? 0ull : pack_best(k.x - (d ? sm.dB[q] : sm.dA[q]), (d ? a0 : b0) + k.y);
        }
    }
}

// One tile pair by a 256-thread block.
template <int T>
__device__ __forceinline__ void combine_tile(const int* __restrict__ S, int n, int ti, int tj,
                                             unsigned long long* __restrict__ part, int* __restrict__ all_out) {
    __shared__ CombineSmem<T> sm;
    combine_tile_on<T>(S, n, ti, tj, part, all_out, sm, threadIdx.x, [] { __syncthreads(); });
}

static __global__ void __launch_bounds__(256)
k_combine64(const int* __restrict__ S, int n, unsigned long long* __restrict__ part,
            int* __restrict__ all_out) {
    const int ti = blockIdx.y, tj = blockIdx.x;
    if (ti > tj) return;
    combine_tile<kTile>(S, n, ti, tj, part, all_out);
}

// rowbest[x] = max over tile columns t of part[t][x]; 32 vertices per block,
// its 8 warps sharing the tile columns (a thread per vertex walking them all
// took 16 us at n = 8,192).  Also clears the candidate count and best delta.
static __global__ void __launch_bounds__(256) k_best_reduce(const unsigned long long* __restrict__ part, int n, int tiles,
                                                            unsigned long long* __restrict__ rowbest,
                                                            int* __restrict__ counters) {
    __shared__ unsigned long long s_k[8][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int x = blockIdx.x * 32 + lane;
    if (blockIdx.x == 0 && threadIdx.x < 2) counters[threadIdx.x] = 0;
    unsigned long long k = 0;
    if (x < n) {
#pragma unroll 4
        for (int t = wid; t < tiles; t += 8) k = kmax(k, part[(size_t)t * n + x]);
    }
    s_k[wid][lane] = k;
    __syncthreads();
    if (wid == 0 && x < n) {
#pragma unroll
        for (int w = 1; w < 8; w++) k = kmax(k, s_k[w][lane]);
        rowbest[x] = k;
    }
}

// ---------------------------------------------------------------------------
// Set commit (one CTA).  The rule is sequential over the sorted candidates:
//   * skip the pair if either vertex already moved in this sweep;
//   * otherwise its current delta is the sweep delta plus, for every G1 edge
//     from one of its vertices x to an already-moved vertex z, the change of
//     that edge's term between z's pre-move image (pold) and its image now;
//     a pair with at least one moved neighbour is the "re-verified" case
//     (counted, and limited by max_verify);
//   * commit iff the current delta is > 0.
// It is executed CG pairs at a time: the CTA makes one coalesced pass over
// the step's edge lists (entries spread evenly over all threads, so a hub
// pair does not stall the step), accumulating each pair's correction
// from moved neighbours (a flag check per entry; W2 is read only for moved
// neighbours) and noting which earlier pairs of the step it shares a vertex
// with or is G1-adjacent to.  For an entry whose neighbour belongs to an
// earlier pair i of the step, the scan also adds the change that pair i's
// swap would make to this pair's delta into cc[j][i] (each G1 edge has one
// endpoint outside the pair, so these changes add up).  Warp 0 then decides
// the pairs in order: a pair sharing a vertex with an earlier committed pair
// is skipped, a pair next to a moved vertex (an earlier step's, or an earlier
// committed pair of this step) is re-verified as its sweep delta plus those
// changes, and it commits iff that is > 0.  A pair's delta depends only on p
// at its vertices and their G1 neighbours, so every decision equals the
// one-at-a-time rule's, re-verification budget included, and no pair is
// scanned twice.
//
// Pairs per step of a batched instance's commit: as many as 16-bit marks hold.
// 8 took 200 steps where 16 take 100 (n = 7,681), 16.0 against 14.0 ms for three
// sweeps of 64 instances.
constexpr int kCGBatch = 16;

// 16-bit atomic OR in shared memory through the aligned 32-bit word.
__device__ __forceinline__ void atomicOr_u16(uint16_t* p, uint16_t v) {
    const size_t addr = reinterpret_cast<size_t>(p);
    unsigned* w = reinterpret_cast<unsigned*>(addr & ~(size_t)3);
    atomicOr(w, (unsigned)v << ((addr & 2) ? 16 : 0));
}

// The set commit of one instance; all 1024 threads of the block call it.
// smem: commit_group_smem(n) bytes of dynamic shared memory.
template <bool W16, int CG>
__device__ __forceinline__ void commit_group(const DevView<W16>& g, const unsigned long long* __restrict__ keys,
                                             int lim, int max_verify, CommitStats* __restrict__ st,
                                             unsigned char* smem) {
    typedef Ent<W16> EN;
    // shared: used[n] flags, then the matching and the pre-move images as
    // 16-bit ids (n <= 65535, so the "unmatched" value n fits)
    const int n = g.n;
    unsigned char* used = smem;
    uint16_t* p16 = reinterpret_cast<uint16_t*>(smem + ((n + 15) & ~15));
    uint16_t* q16 = p16 + ((n + 8) & ~7);
    uint16_t* mark = q16 + ((n + 8) & ~7);  // bit i set: vertex belongs to pair i of the step
    __shared__ int s_lo[CG], s_hi[CG], s_d0[CG];
    __shared__ int s_corr[CG], s_cnt[CG], s_pre[CG + 1];
    __shared__ unsigned s_imask[CG];   // earlier pairs of the step G1-adjacent to this one
    __shared__ unsigned s_share[CG];   // earlier pairs of the step sharing a vertex with this one
    __shared__ unsigned s_dead;         // pairs with a vertex already moved when the step starts
    __shared__ int s_inf[CG][8];       // la0, la, ia0, ia, lb0, lb, ib0, ib
    __shared__ int s_segpre[4 * CG + 1];  // the step's lists as segments 4j + k: prefix of their lengths
    __shared__ int s_segoff[4 * CG];      // first entry of segment 4j + k in ent1o (k even) or ent1i (k odd)
    __shared__ int s_n, s_k, s_scanned;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    __shared__ int s_cc[CG][CG];   // s_cc[j][i]: change of pair j's delta if earlier pair i commits
    for (int i = tid; i < n; i += blockDim.x) { used[i] = 0; p16[i] = (uint16_t)g.p[i]; mark[i] = 0; }
    for (int i = tid; i < CG * CG; i += blockDim.x) (&s_cc[0][0])[i] = 0;
    if (tid == 0) { s_n = 0; s_k = 0; s_scanned = 0; p16[n] = (uint16_t)n; }
    long long total = 0, entries = 0;
    int verified = 0, committed = 0, steps = 0;
    __syncthreads();
    for (;;) {
        // ---- warp 0: the next live candidates, then the
        //      per-pair list extents and their prefix (lane j = pair j) ----
        if (wid == 0) {
            int cnt = s_n, k = s_k, scanned = s_scanned;
            while (cnt < CG && k < lim) {
                const int idx = k + lane;
                const unsigned long long key = idx < lim ? keys[idx] : ~0ull;
                const bool valid = key != ~0ull;
                const int lo = valid ? (int)((key >> 16) & 0xffffu) : 0;
                const int hi = valid ? (int)(key & 0xffffu) : 0;
                const bool live = valid && !used[lo] && !used[hi];
                const unsigned vmask = __ballot_sync(0xffffffffu, valid);
                const unsigned lmask = __ballot_sync(0xffffffffu, live);
                const int room = CG - cnt;
                const int before = __popc(lmask & ((1u << lane) - 1u));
                const int nvalid = __popc(vmask);  // valid keys form a prefix
                int consumed = nvalid, took = __popc(lmask);
                if (took > room) {  // stop just before the (room+1)-th live candidate
                    const unsigned over = __ballot_sync(0xffffffffu, live && before == room);
                    consumed = __ffs(over) - 1;
                    took = room;
                }
                if (live && before < room) {
                    const int q = cnt + before;
                    s_lo[q] = lo; s_hi[q] = hi;
                    s_d0[q] = (int)(0x7fffffffu - (unsigned)(key >> 32));
                    int4 i0, i1;   // list extents
                    i0.x = g.off1o[lo]; i0.y = g.off1o[lo + 1] - i0.x;
                    i0.z = g.off1i[lo]; i0.w = g.off1i[lo + 1] - i0.z;
                    i1.x = g.off1o[hi]; i1.y = g.off1o[hi + 1] - i1.x;
                    i1.z = g.off1i[hi]; i1.w = g.off1i[hi + 1] - i1.z;
                    s_inf[q][0] = i0.x; s_inf[q][1] = i0.y; s_inf[q][2] = i0.z; s_inf[q][3] = i0.w;
                    s_inf[q][4] = i1.x; s_inf[q][5] = i1.y; s_inf[q][6] = i1.z; s_inf[q][7] = i1.w;
                }
                cnt += took;
                k += consumed;
                scanned += consumed;
                if (consumed == nvalid && nvalid < 32) { k = lim; break; }
            }
            __syncwarp();
            int len = 0;
            if (lane < cnt) {
                const int a = s_lo[lane], b = s_hi[lane];
                len = s_inf[lane][1] + s_inf[lane][3] + s_inf[lane][5] + s_inf[lane][7];
                s_corr[lane] = 0; s_cnt[lane] = 0; s_imask[lane] = 0;
                atomicOr_u16(&mark[a], (uint16_t)(1u << lane));
                atomicOr_u16(&mark[b], (uint16_t)(1u << lane));
            }
            __syncwarp();
            if (lane < cnt) {  // earlier pairs of the step that share a vertex: read off the marks
                const unsigned m = (unsigned)mark[s_lo[lane]] | (unsigned)mark[s_hi[lane]];
                s_share[lane] = m & ((1u << lane) - 1u);
            }
            int incl = len;  // inclusive prefix over lanes
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane < cnt) s_pre[lane + 1] = incl;
            __syncwarp();
            {   // segment table: segment 4j + k (a out, a in, b out, b in of pair j), 32 per pass
                int carry = 0;
                for (int h = 0; h < (4 * CG + 31) / 32; h++) {
                    const int seg = lane + 32 * h, j = seg >> 2, k = seg & 3;
                    const int slen = j < cnt ? s_inf[j][2 * k + 1] : 0;
                    int sincl = slen;
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, sincl, o);
                        if (lane >= o) sincl += y;
                    }
                    if (seg < 4 * CG) {
                        s_segpre[seg + 1] = carry + sincl;
                        s_segoff[seg] = j < cnt ? s_inf[j][2 * k] : 0;
                    }
                    carry += __shfl_sync(0xffffffffu, sincl, 31);
                }
                if (lane == 0) s_segpre[0] = 0;
            }
            const unsigned dead = __ballot_sync(0xffffffffu, lane < cnt && (used[s_lo[lane < cnt ? lane : 0]] | used[s_hi[lane < cnt ? lane : 0]]));
            if (lane == 0) {
                s_pre[0] = 0; s_dead = dead;
                s_n = cnt; s_k = k; s_scanned = scanned;
            }
            if (cnt) {
                const int tot = __shfl_sync(0xffffffffu, incl, cnt - 1);
                if (lane == 0) { entries += tot; steps++; }
            }
        } else {   // the other warps clear the step's conditional changes
            for (int q = tid - 32; q < CG * CG; q += blockDim.x - 32) (&s_cc[0][0])[q] = 0;
        }
        __syncthreads();
        const int cnt = s_n;
        if (cnt == 0) break;
        // ---- scan all pairs of the step, an entry per thread.  A moved neighbour x
        //      changes the pair's delta by what it would make of the edge now against
        //      before (into corr); a neighbour in earlier pairs i of the step by what
        //      each one's swap would change (x taking its partner's image, into
        //      cc[j][i]).  Both are the same difference between an image px and qx, so
        //      one loop serves them, with four earlier pairs' loads in flight: early in
        //      a descent a hub is in most pairs of a step. ----
        const int tot = s_pre[cnt], nseg = 4 * cnt;
        for (int base = 0; base < tot; base += blockDim.x) {
            const int e = base + tid;
            int j = -1, corr = 0, moved = 0;
            if (e < tot) {
                int lo = 0, hi = nseg;  // s_segpre[lo] <= e < s_segpre[hi]
                while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (s_segpre[mid] <= e) lo = mid; else hi = mid; }
                j = lo >> 2;
                const bool out = !(lo & 1);
                const typename EN::T en = ((lo & 1) ? g.ent1i : g.ent1o)[s_segoff[lo] + (e - s_segpre[lo])];
                const int x = EN::id(en), w = EN::w(en);
                const unsigned im = mark[x] & ((1u << j) - 1u);  // earlier pairs with vertex x
                if (im) atomicOr(&s_imask[j], im);
                const int a = s_lo[j], b = s_hi[j];
                unsigned rest = im;
                if (used[x]) { moved = 1; rest = 1u; }
                if (x == a || x == b) { moved = 0; rest = 0; }
                if (rest) {
                    // a takes p(b) and b takes p(a): the terms of b's edges have the opposite sign
                    const int pa = p16[(lo & 2) ? b : a], pb = p16[(lo & 2) ? a : b], qx = moved ? q16[x] : p16[x];
                    // out-edges: W2 rows of the images, in-edges: rows of the transpose
                    auto term = [&](int f, int z) { return out ? g.w2(f, z) : g.w2t(z, f); };
                    const int t0 = term(pb, qx), t1 = term(pa, qx);
                    while (rest) {
                        int i[4], v0[4], v1[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            i[u] = -1; v0[u] = 0; v1[u] = 0;
                            if (!rest) continue;
                            i[u] = __ffs(rest) - 1;
                            rest &= rest - 1;
                            const int px = p16[moved ? x : s_lo[i[u]] == x ? s_hi[i[u]] : s_lo[i[u]]];
                            v0[u] = term(pb, px);
                            v1[u] = term(pa, px);
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            if (i[u] < 0) continue;
                            const int c = (imin(w, v0[u]) - imin(w, v1[u])) - (imin(w, t0) - imin(w, t1));
                            if (moved) corr = c;
                            else if (c) atomicAdd(&s_cc[j][i[u]], c);
                        }
                    }
                }
            }
            // the warp's entries are mostly of one pair: one atomic for all of it
            const int j0 = __shfl_sync(0xffffffffu, j, 0);
            if (__all_sync(0xffffffffu, j == j0)) {
                moved = __reduce_add_sync(0xffffffffu, moved);
                corr = __reduce_add_sync(0xffffffffu, corr);
                if (lane || j0 < 0) { moved = 0; corr = 0; }
            }
            if (corr) atomicAdd(&s_corr[j], corr);
            if (moved) atomicAdd(&s_cnt[j], moved);
        }
        const int my_lo = tid < cnt ? s_lo[tid] : 0, my_hi = tid < cnt ? s_hi[tid] : 0;
        __syncthreads();
        // ---- clear the step's marks; decide in order in warp 0: lane j holds pair
        //      j's fields, every lane replays the same bitmask logic over the
        //      shuffled fields, then the lanes apply their own outcomes ----
        if (tid < cnt) { mark[my_lo] = 0; mark[my_hi] = 0; }
        if (wid == 0) {
            const bool in = lane < cnt;
            const unsigned share = in ? s_share[lane] : 0u, adj = in ? s_imask[lane] : 0u;
            const int moved = in ? s_cnt[lane] : 0, d0 = in ? s_d0[lane] : 0;
            int corr = in ? s_corr[lane] : 0;   // grows by cc[lane][i] when earlier pair i commits
            const int a = in ? s_lo[lane] : 0, b = in ? s_hi[lane] : 0;
            const unsigned dead = s_dead;
            unsigned cm = 0;
#pragma unroll
            for (int j = 0; j < CG; j++) {
                const unsigned sh_j = __shfl_sync(0xffffffffu, share, j);
                const unsigned ad_j = __shfl_sync(0xffffffffu, adj, j);
                const int mv_j = __shfl_sync(0xffffffffu, moved, j);
                const int co_j = __shfl_sync(0xffffffffu, corr, j);
                const int d0_j = __shfl_sync(0xffffffffu, d0, j);
                if (j >= cnt) continue;
                if (((dead >> j) & 1u) || (sh_j & cm)) continue;   // a vertex already moved: skip
                int d = d0_j;
                bool ok = true;
                if (mv_j > 0 || (ad_j & cm)) {                   // next to a moved vertex: re-verify
                    if (max_verify >= 0 && verified >= max_verify) ok = false;
                    else { verified++; d += co_j; }
                }
                if (ok && d > 0) {
                    cm |= 1u << j;
                    total += d;
                    committed++;
                    if (lane > j && lane < cnt) corr += s_cc[lane][j];
                }
            }
            __syncwarp();
            if ((cm >> lane) & 1u) {  // committed pairs share no vertex: apply in parallel
                const int fa = p16[a], fb = p16[b];
                q16[a] = (uint16_t)fa; q16[b] = (uint16_t)fb;
                p16[a] = (uint16_t)fb; p16[b] = (uint16_t)fa;
                if (fb < n) g.pinv[fb] = a;
                if (fa < n) g.pinv[fa] = b;
                used[a] = 1; used[b] = 1;
            }
            if (lane == 0) s_n = 0;
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += blockDim.x) g.p[i] = p16[i];
    if (tid == 0) {
        st->total_delta = total;
        st->scanned = s_scanned;
        st->verified = verified;
        st->committed = committed;
        st->steps = steps;
        st->entries = entries;
        st->carried = 0;   // every pair is decided in the step that scans it
    }
}

// Shared memory bytes of commit_group for n vertices (used flags, matching,
// pre-move images, step marks).
__host__ __device__ inline size_t commit_group_smem(int n) {
    return (size_t)((n + 15) & ~15) + 6 * (size_t)((n + 8) & ~7);
}

// Whether a sweep takes n: what a batched instance's commit keeps in a CTA's
// shared memory fits (n up to 32,615).  k_commit_sets needs less, and the 3-cycle
// and 4-set rounds, which commit with it too, take every n; for sweeps the bound
// stands because callers rely on the refusal.
inline bool sweep_takes(int n, size_t smem_optin) { return commit_group_smem(n) + 4096 <= smem_optin; }

}  // namespace bm
