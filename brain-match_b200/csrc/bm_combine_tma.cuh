// bm_combine_tma.cuh -- the sweep's pair combine with TMA-staged tiles.
//
// Same result as k_combine64 (bm_select.cuh): for every 64x64 tile (I,J),
// I <= J, of the profit matrix S, delta(a,b) = S[a][b] + S[b][a] - S[a][a]
// - S[b][b] and the best partner of every vertex inside the tile, written to
// the per-tile partial array that k_best_reduce folds.  The difference is how
// S reaches shared memory: a persistent CTA walks its share of the tile pairs
// and keeps kCmbStages pairs in flight, each pair's two 16 KB tiles
// (S[I][J] and S[J][I]) fetched by cp.async.bulk.tensor (TMA, the CTA's own
// shared memory, no multicast) onto one mbarrier with an expected byte count.
//
// A tile arrives as two 32-column boxes in the 128-byte swizzle.  A thread owns
// one vertex of the tile pair, a row (warps 0-3) or a column vertex, and walks
// 32 of its partners in ascending order: its own row four values per 16-byte
// read (eight lanes' rows fall into different banks), the partner's row one
// value across consecutive lanes.  Both are free of bank conflicts, and a best
// is a compare and two moves in registers.  One barrier per tile: it frees the
// stage and hands the two halves of every owner's partners to the merge.
//
// What bounds it: reading S once from HBM in 128-byte rows of boxes.  16 warps
// per CTA on dense tiles walked along diagonals, a shuffle per step for the
// column bests and packed 64-bit keys took 438 us at n = 18,524 (3.1 TB/s; now
// 312, 4.4 TB/s), and n not a multiple of 4 could not use TMA at all (n = 6,007:
// 90 us, now 39).
//
// Works at every n >= 64 (S's row pitch is a multiple of 16 bytes).  Every wait
// on a tile is bounded: when one runs out the CTA sets bit 4 of err, waits
// (bounded) for the copies it issued and returns, and the host reports
// BM_E_TIMEOUT.
#pragma once
#include <cstdint>
#include <climits>
#include <cuda.h>
#include "bm_kernels.cuh"

namespace bm {

constexpr int kCmbT = 64;                                // tile edge
constexpr int kCmbBox = 32;                              // columns of a box (128 bytes)
constexpr int kCmbStages = 2;                            // tile pairs in flight per CTA
constexpr int kCmbBoxBytes = kCmbT * kCmbBox * 4;        // 8 KB
constexpr int kCmbStageBytes = 4 * kCmbBoxBytes;         // S[I][J] and S[J][I], two boxes each
constexpr int kCmbThreads = 256;
constexpr int kCmbSmem = kCmbStages * kCmbStageBytes + 1024 + 64;   // + alignment + barriers
constexpr int kCmbErrBit = 4;

__device__ __forceinline__ uint32_t cmb_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool cmb_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool cmb_wait(uint32_t bar, uint32_t parity, int limit = 1 << 22) {
    for (int i = 0; i < limit; i++)
        if (cmb_try_wait(bar, parity)) return true;
    return false;
}

// Both tiles of a pair onto one mbarrier: boxes 0, 1 = rows a0.., columns b0..
// and b0 + 32..; boxes 2, 3 = rows b0.., columns a0.. and a0 + 32.. (x = column,
// y = row; x is a multiple of 32 elements, so every copy starts on a 128-byte
// boundary of its row).
__device__ __forceinline__ void cmb_issue(const CUtensorMap* tm, uint32_t dst, uint32_t bar, int a0, int b0) {
    // the stage's earlier reads (generic proxy) are ordered before the copy's writes
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(kCmbStageBytes) : "memory");
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int x = (q < 2 ? b0 : a0) + kCmbBox * (q & 1), y = q < 2 ? a0 : b0;
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            :: "r"(dst + q * kCmbBoxBytes), "l"(tm), "r"(x), "r"(y), "r"(bar) : "memory");
    }
}

// Place in the upper triangle of tiles, row-major: tile pair (ti, ti + off).
struct CmbPlace {
    int ti, off;
    __device__ __forceinline__ void skip(long long k, int tiles) {   // k pairs further
        long long o = off + k;
        while (ti < tiles && o >= tiles - ti) { o -= tiles - ti; ti++; }
        off = (int)o;
    }
};

static __global__ void __launch_bounds__(kCmbThreads, 3)
k_combine_tma(const __grid_constant__ CUtensorMap tm, const int* __restrict__ diag, int n, int tiles,
              unsigned long long* __restrict__ part, int* __restrict__ err, int stall) {
    extern __shared__ __align__(128) unsigned char cmb_raw[];
    const uint32_t raw = cmb_smem(cmb_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* basep = cmb_raw + (base - raw);
    const uint32_t bars = base + kCmbStages * kCmbStageBytes;
    __shared__ __align__(16) int s_diag[2][2 * kCmbT];                     // S[x][x] of the tile's rows, columns; by tile parity
    __shared__ int2 s_best[2][2][2][kCmbT];                  // (best without own diagonal, partner): parity, dir, half, owner
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    // warp: owners (row or column vertices, half of them), and the half of the partners it walks
    const int dir = wid >> 2, half = wid & 1, seg = (wid >> 1) & 1;
    const int o = 32 * half + lane;
    const int step = gridDim.x;
    CmbPlace at = {0, 0}, ahead = {0, 0};   // the tile pair at hand; the next to issue
    at.skip(blockIdx.x, tiles);
    ahead = at;
    auto diag_of = [&](const CmbPlace& p) {   // this thread's diagonal entry (tid < 128)
        const int x = tid < kCmbT ? p.ti * kCmbT + tid : (p.ti + p.off) * kCmbT + tid - kCmbT;
        return p.ti < tiles && x < n ? __ldg(&diag[x]) : 0;
    };
    if (tid == 0) {
        for (int s = 0; s < kCmbStages; s++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bars + 8 * s) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    for (int s = 0; s < kCmbStages; s++) {
        if (tid == 0 && ahead.ti < tiles)
            cmb_issue(&tm, base + s * kCmbStageBytes, bars + 8 * s, ahead.ti * kCmbT, (ahead.ti + ahead.off) * kCmbT);
        ahead.skip(step, tiles);
    }
    CmbPlace next = at;
    next.skip(step, tiles);
    int dnext = 0;
    if (tid < 2 * kCmbT) {
        s_diag[0][tid] = diag_of(at);
        dnext = diag_of(next);
    }
    __syncthreads();
    int it = 0;
    bool failed = false;
    for (; at.ti < tiles; it++) {
        const int s = it % kCmbStages, par = it & 1;
        const uint32_t phase = (uint32_t)((it / kCmbStages) & 1);
        const int ti = at.ti, tj = at.ti + at.off, a0 = ti * kCmbT, b0 = tj * kCmbT;
        bool ok = cmb_wait(bars + 8 * s, phase);
        // test hook (bm_test_stall): CTA 0's first tile also waits for the
        // stage's next phase, which no copy completes before it is issued
        if (ok && stall && blockIdx.x == 0 && it == 0) ok = cmb_wait(bars + 8 * s, phase ^ 1u, 1 << 12);
        const bool diagt = ti == tj;
        if (ok && !(diagt && dir)) {
            const unsigned char* st = basep + s * kCmbStageBytes;
            const unsigned char* own = st + (2 * dir + seg) * kCmbBoxBytes + o * 128;             // own row, partners' box
            const unsigned char* oth = st + (2 * (dir ^ 1) + half) * kCmbBoxBytes + 32 * seg * 128;   // partners' rows, own box
            const int* dP = s_diag[par] + (dir ? 0 : kCmbT) + 32 * seg;
            const int p0 = (dir ? a0 : b0) + 32 * seg;     // first partner's vertex
            int bd = INT_MIN, bi = -1;
            if (!diagt && p0 + 32 <= n) {
                bi = 0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int4 x = *reinterpret_cast<const int4*>(own + ((k ^ (o & 7)) << 4));
                    const int4 q = *reinterpret_cast<const int4*>(dP + 4 * k);
                    const int xs[4] = {x.x, x.y, x.z, x.w}, qs[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int c = 4 * k + e;
                        const int y = *reinterpret_cast<const int*>(oth + c * 128 + (((lane >> 2) ^ (c & 7)) << 4) + (lane & 3) * 4);
                        const int d = xs[e] + y - qs[e];
                        if (c == 0 || d > bd) { bd = d; bi = c; }
                    }
                }
            } else {
                for (int c = 0; c < 32 && p0 + c < n; c++) {
                    const int x = *reinterpret_cast<const int*>(own + (((c >> 2) ^ (o & 7)) << 4) + (c & 3) * 4);
                    const int y = *reinterpret_cast<const int*>(oth + c * 128 + (((lane >> 2) ^ (c & 7)) << 4) + (lane & 3) * 4);
                    const int d = x + y - dP[c];
                    if (!(diagt && 32 * seg + c == o) && (bi < 0 || d > bd)) { bd = d; bi = c; }
                }
            }
            s_best[par][dir][seg][o] = make_int2(bd, bi < 0 ? -1 : p0 + bi);
        }
        if (tid < 2 * kCmbT) s_diag[par ^ 1][tid] = dnext;
        // stage s is free, the halves' bests are complete; every thread leaves on a timeout
        if (!__syncthreads_and(ok)) { failed = true; break; }
        if (tid == 0 && ahead.ti < tiles)
            cmb_issue(&tm, base + s * kCmbStageBytes, bars + 8 * s, ahead.ti * kCmbT, (ahead.ti + ahead.off) * kCmbT);
        ahead.skip(step, tiles);
        if (tid < 2 * kCmbT) {
            const int d = tid / kCmbT, q = tid & (kCmbT - 1), x = (d ? b0 : a0) + q;
            if (x < n && !(d && diagt)) {   // a diagonal tile's rows already cover both orders
                int2 k = s_best[par][d][0][q];
                const int2 y = s_best[par][d][1][q];
                if (y.y >= 0 && (k.y < 0 || y.x > k.x)) k = y;   // ties to the lower half
                part[(size_t)(d ? ti : tj) * n + x] = k.y < 0 ? 0ull : pack_best(k.x - s_diag[par][d * kCmbT + q], k.y);
            }
            next.skip(step, tiles);
            dnext = diag_of(next);
        }
        at.skip(step, tiles);
        // s_best and s_diag of this parity are rewritten only after the next
        // tile's barrier, which every thread passes after the reads above
    }
    // on a timeout: wait (bounded) for the copies still in flight into this
    // CTA's shared memory before it exits
    if (tid == 0 && failed) {
        atomicOr(err, 1 << kCmbErrBit);
        for (int j = 0; j < kCmbStages; j++) {
            const int jt = it + j;
            if (at.ti < tiles) cmb_wait(bars + 8 * (jt % kCmbStages), (uint32_t)((jt / kCmbStages) & 1));
            at.skip(step, tiles);
        }
    }
}

// S[a][a] for every a (the combine reads it per tile row and column).
static __global__ void k_diag(const int* __restrict__ S, int n, int* __restrict__ diag) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a < n) diag[a] = S[(size_t)a * (s_pitch(n) + 1)];
}

}  // namespace bm
