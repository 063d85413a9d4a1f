// bm_mlp.cuh -- device code of the learned swap-proposal network.
//
// MLP 128 -> 256 -> 256 -> 1 (ReLU), bf16 weights and activations, fp32
// accumulation.  The two wide layers and every backward GEMM run through one
// tcgen05 kernel, C = A * B^T with A (M x K) and B (N x K) bf16 row-major
// (K-major) and C fp32, accumulated in TMEM (kind::f16, bf16 inputs); the same
// shared-memory staging and 128-byte swizzle as the hub GEMM.  The 256 -> 1
// head, bias/ReLU backward, loss and SGD are small CUDA-core kernels.
// Ranking many pairs uses a second, fused kernel (k_mlp_rank, below).
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include "bm_hub.cuh"

namespace bm {

constexpr int kMlpIn = 128, kMlpHid = 256;

// What the GEMM's epilogue does with C[M x N] = A[M x K] * B[N x K]^T.
struct GemmOut {
    const float* bias = nullptr;      // + bias[col]
    int relu = 0;                     // max(., 0)
    const float* mask = nullptr;      // M x N: 0 where mask <= 0
    float* C = nullptr;               // M x N fp32
    float* colsum = nullptr;          // N: += column sums
    __nv_bfloat16* Cb = nullptr;      // M x N bf16
    __nv_bfloat16* CbT = nullptr;     // N x M bf16, transposed
};

// M % 128 == 0, N % BN == 0, K % 64 == 0; N / BN * M / 128 CTAs along x (the
// other dimensions end at 65,535), a row tile's columns side by side.
// The network's GEMMs are small (1,024 x 256 x 256 for a training batch), so a
// launch is bound by its latency and by how many SMs it uses: 64 columns per
// CTA (32 CTAs per batch instead of 8 with whole rows), the four K-chunks of a
// layer all in flight, and the passes that followed the GEMMs -- ReLU' and
// bias gradient, transposes for the weight gradients -- done in the epilogue
// from registers (a GEMM 21 -> 9 us, one of the weight gradients 12; ReLU' 17 us
// and six transposes of 3.6 us gone; a step of 1,024 rows 178 -> 71 us of kernels).
constexpr int kMlpStages = 4;
template <int BN>
static __global__ void __launch_bounds__(kGemmThreads, 1)
k_gemm_bf16(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B, int M, int N, int K,
            GemmOut o, int* __restrict__ err, int stall) {
    constexpr int kStage = (kGemmM + BN) * kGemmKC;                   // bytes per stage
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) |  // f32 accum, bf16 x bf16
                                ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kGemmM >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t bars = base + kMlpStages * kStage;
    const uint32_t tslot = bars + 8 * kMlpStages;
    uint32_t* tslot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tslot - raw));
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    const int cols = N / BN, b0 = (blockIdx.x % cols) * BN, a0 = (blockIdx.x / cols) * kGemmM;
    const int KB = K * 2;                        // bytes per row
    const int KC = KB / kGemmKC;                 // 128-byte chunks
    const uint8_t* Ab = reinterpret_cast<const uint8_t*>(A);
    const uint8_t* Bb = reinterpret_cast<const uint8_t*>(B);

    if (wid == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(tslot), "r"(BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kMlpStages; s++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bars + 8 * s) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot_ptr;
    bool ok = true;

    auto load = [&](int st, int kc) {
        const uint32_t sA = base + st * kStage, sB = sA + kGemmM * kGemmKC;
        const size_t koff = (size_t)kc * kGemmKC;
        for (int i = tid; i < kGemmM * 8; i += kGemmThreads) {
            const int r = i >> 3, c = i & 7;
            cp_async16(sA + r * 128 + ((c ^ (r & 7)) << 4), Ab + (size_t)(a0 + r) * KB + koff + c * 16);
        }
        for (int i = tid; i < BN * 8; i += kGemmThreads) {
            const int r = i >> 3, c = i & 7;
            cp_async16(sB + r * 128 + ((c ^ (r & 7)) << 4), Bb + (size_t)(b0 + r) * KB + koff + c * 16);
        }
    };
    for (int s = 0; s < kMlpStages - 1; s++) {
        if (s < KC) load(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int kc = 0; kc < KC; kc++) {
        const int nxt = kc + kMlpStages - 1;
        if (nxt < KC) {
            if (kc >= 1) {
                const int prev = kc - 1;
                ok = ok && mbar_wait_bounded(bars + 8 * (prev % kMlpStages), (prev / kMlpStages) & 1, err);
            }
            load(nxt % kMlpStages, nxt);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group %0;" :: "n"(kMlpStages - 1) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0 && ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int st = kc % kMlpStages;
            const uint32_t sa = base + st * kStage, sb = sa + kGemmM * kGemmKC;
#pragma unroll
            for (int j = 0; j < kGemmKC / 32; j++) {  // 16 bf16 = 32 bytes of K per MMA
                const uint64_t da = umma_desc_sw128(sa + j * 32), db = umma_desc_sw128(sb + j * 32);
                const uint32_t acc = (kc > 0 || j > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    :: "r"(tmem), "l"(da), "l"(db), "r"(kIdesc), "r"(acc) : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         :: "r"(bars + 8 * st) : "memory");
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (KC > 0) {
        const int last = KC - 1;
        ok = ok && mbar_wait_bounded(bars + 8 * (last % kMlpStages), (last / kMlpStages) & 1, err);
        // test hook (bm_test_stall): the barrier's next phase never completes
        if (stall && blockIdx.x == 0)
            ok = ok && mbar_wait_bounded(bars + 8 * (last % kMlpStages), ((last / kMlpStages) + 1) & 1, err,
                                         kStallPolls);
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int row = a0 + wid * 32 + lane;
    for (int cb = 0; cb < BN / 32; cb++) {
        uint32_t r[32];
        const uint32_t taddr = tmem + ((uint32_t)(wid * 32) << 16) + (uint32_t)(cb * 32);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (!__all_sync(0xffffffffu, ok)) continue;
        const int c0 = b0 + cb * 32;
        float v[32];
#pragma unroll
        for (int q = 0; q < 32; q++) {
            float x = __uint_as_float(r[q]);
            if (o.bias) x += o.bias[c0 + q];
            if (o.relu) x = fmaxf(x, 0.f);
            v[q] = x;
        }
        if (o.mask) {
            const float4* m4 = reinterpret_cast<const float4*>(o.mask + (size_t)row * N + c0);
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const float4 m = m4[q];
                if (!(m.x > 0.f)) v[4 * q] = 0.f;
                if (!(m.y > 0.f)) v[4 * q + 1] = 0.f;
                if (!(m.z > 0.f)) v[4 * q + 2] = 0.f;
                if (!(m.w > 0.f)) v[4 * q + 3] = 0.f;
            }
        }
        if (o.C) {
            float4* d4 = reinterpret_cast<float4*>(o.C + (size_t)row * N + c0);
#pragma unroll
            for (int q = 0; q < 8; q++) d4[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        }
        if (o.Cb) {
            __nv_bfloat162* d2 = reinterpret_cast<__nv_bfloat162*>(o.Cb + (size_t)row * N + c0);
#pragma unroll
            for (int q = 0; q < 16; q++) d2[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
        }
        if (o.CbT) {   // a warp's 32 rows are consecutive: 64 bytes per column
#pragma unroll
            for (int q = 0; q < 32; q++) o.CbT[(size_t)(c0 + q) * M + row] = __float2bfloat16(v[q]);
        }
        if (o.colsum) {   // halving: lane q ends with column q
#pragma unroll
            for (int w = 16; w; w >>= 1) {
                const bool up = lane & w;
#pragma unroll
                for (int q = 0; q < w; q++) {
                    const float give = up ? v[q] : v[q + w], keep = up ? v[q + w] : v[q];
                    v[q] = keep + __shfl_xor_sync(0xffffffffu, give, w);
                }
            }
            atomicAdd(o.colsum + c0 + lane, v[0]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (wid == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(BN) : "memory");
}

template <int BN>
constexpr int gemm_bf16_smem() { return kMlpStages * (kGemmM + BN) * kGemmKC + 1024 + 256; }

// out[i] = bf16(x[i]) for a rows x kMlpIn matrix (zero rows from k on), and its
// transpose (ld = rows) if outT is given.  32 rows per block of 128 threads.
static __global__ void __launch_bounds__(kMlpIn) k_rows_bf16(const float* __restrict__ x, int k, int rows,
                                                             __nv_bfloat16* __restrict__ out,
                                                             __nv_bfloat16* __restrict__ outT) {
    const int c = threadIdx.x, r0 = blockIdx.x * 32;
    __align__(16) __nv_bfloat16 col[32];
#pragma unroll
    for (int r = 0; r < 32; r++) {
        col[r] = __float2bfloat16(r0 + r < k ? x[(size_t)(r0 + r) * kMlpIn + c] : 0.f);
        out[(size_t)(r0 + r) * kMlpIn + c] = col[r];
    }
    if (outT) {
        uint4* dst = reinterpret_cast<uint4*>(outT + (size_t)c * rows + r0);
#pragma unroll
        for (int q = 0; q < 4; q++) dst[q] = reinterpret_cast<const uint4*>(col)[q];
    }
}

// Head and loss: y = H2 . w3 + b3 (rows < Bv valid), dy = 2 (y - t) / Bv,
// dH2 = dy w3 masked by ReLU'(H2) (bf16, and its transpose), dw3 += H2^T dy,
// db3 += sum dy, db2 += column sums of dH2.  32 rows per block: warps take four
// rows' dot products each, then a thread per column walks the rows, so the
// column gradients cost an atomic per block and column (one per row and column
// before, 11 us, and a pass of its own for db2, 10 us).
static __global__ void __launch_bounds__(kMlpHid) k_head(const float* __restrict__ H2, int Bv, int Bpad,
                                                         const float* __restrict__ w3, const float* __restrict__ b3,
                                                         float* __restrict__ y, const float* __restrict__ target,
                                                         float* __restrict__ loss, __nv_bfloat16* __restrict__ dH2,
                                                         __nv_bfloat16* __restrict__ dH2T, float* __restrict__ dw3,
                                                         float* __restrict__ db3, float* __restrict__ db2) {
    __shared__ float s_dy[32], s_loss[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, r0 = blockIdx.x * 32;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int r = 4 * wid + q, row = r0 + r;
        const float* h = H2 + (size_t)row * kMlpHid;
        float s = 0.f;
#pragma unroll
        for (int c = lane; c < kMlpHid; c += 32) s += h[c] * w3[c];
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
            const float out = s + b3[0];
            if (y && row < Bv) y[row] = out;
            float dy = 0.f, l = 0.f;
            if (target && row < Bv) {
                const float d = out - target[row];
                dy = 2.f * d / (float)Bv;
                l = d * d / (float)Bv;
            }
            s_dy[r] = dy;
            s_loss[r] = l;
        }
    }
    if (!target) return;
    __syncthreads();
    if (wid == 0) {
        float l = s_loss[lane], d = s_dy[lane];
        for (int o = 16; o; o >>= 1) { l += __shfl_xor_sync(0xffffffffu, l, o); d += __shfl_xor_sync(0xffffffffu, d, o); }
        if (lane == 0) { atomicAdd(loss, l); atomicAdd(db3, d); }
    }
    const int c = tid;
    const float w = w3[c];
    float g3 = 0.f, g2 = 0.f;
    __align__(16) __nv_bfloat16 col[32];
#pragma unroll
    for (int r = 0; r < 32; r++) {
        const float hv = H2[(size_t)(r0 + r) * kMlpHid + c], dy = s_dy[r];
        col[r] = __float2bfloat16(hv > 0.f ? dy * w : 0.f);
        dH2[(size_t)(r0 + r) * kMlpHid + c] = col[r];
        if (dy != 0.f) g3 += hv * dy;   // a padded row's activation may be infinite: it adds nothing
        g2 += __bfloat162float(col[r]);
    }
    uint4* dst = reinterpret_cast<uint4*>(dH2T + (size_t)c * Bpad + r0);
#pragma unroll
    for (int q = 0; q < 4; q++) dst[q] = reinterpret_cast<const uint4*>(col)[q];
    atomicAdd(&dw3[c], g3);
    atomicAdd(&db2[c], g2);
}

// SGD on the fp32 master weights, refreshing the bf16 copies the GEMMs read
// (W1, W2 and W2's transpose): w -= lr * g, the product and the difference each
// rounded to nearest (no fused multiply-add), so the update is reproducible on
// any IEEE host.  With g == nullptr only the copies are refreshed.
static __global__ void k_sgd(float* __restrict__ w, const float* __restrict__ g, int count, float lr, int oW1, int oW2,
                             __nv_bfloat16* __restrict__ W1b, __nv_bfloat16* __restrict__ W2b,
                             __nv_bfloat16* __restrict__ W2Tb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float v = w[i];
    if (g) {
        v = __fsub_rn(v, __fmul_rn(lr, g[i]));
        w[i] = v;
    }
    const int j1 = i - oW1, j2 = i - oW2;
    if (j1 >= 0 && j1 < kMlpHid * kMlpIn) W1b[j1] = __float2bfloat16(v);
    if (j2 >= 0 && j2 < kMlpHid * kMlpHid) {
        const __nv_bfloat16 b = __float2bfloat16(v);
        W2b[j2] = b;
        W2Tb[(j2 % kMlpHid) * kMlpHid + j2 / kMlpHid] = b;
    }
}

// ---------------------------------------------------------------------------
// Ranking many pairs (inference), factorised.  The first layer is linear in
// the concatenated input x = [f1(a), f1(b), f2(p a), f2(p b)], so
// W1 x + b1 = U[a] + V[b] with per-vertex vectors
//   U[a] = b1 + W1[:, 0:32] f1(a) + W1[:, 64:96]  f2(p a)
//   V[b] =      W1[:, 32:64] f1(b) + W1[:, 96:128] f2(p b)
// (bf16-rounded weights and features, fp32 sums -- the values the GEMM path
// multiplies).  One persistent kernel then scores every pair: the CTA keeps
// W2 (bf16, 128 KB) resident in shared memory, builds each 128-pair A tile
// bf16(relu(U[a] + V[b])) directly in the swizzled operand layout, runs one
// 128 x 256 x 256 tcgen05 MMA into TMEM, and its epilogue applies b2, ReLU
// and the 256 -> 1 head, writing one float per pair.

constexpr int kFeatDim = 32;

// U and V for n vertices: block of 256 threads (one per hidden unit) over kUvRows
// vertices.  F1, F2: n x 32 fp32; W1b: 256 x 128 bf16; p: matching.  A thread
// holds its unit's 128 weights in registers; the block pays for loading them
// (64 KB) once per kUvRows vertices -- with 8 vertices and 2-byte loads the
// weights were the launch (145 us at n = 8,192; now 34).  Two vertices at a
// time: four independent chains of fused multiply-adds, each in column order.
constexpr int kUvRows = 32;
static __global__ void __launch_bounds__(256) k_uv(const float* __restrict__ F1, const float* __restrict__ F2,
                                                   const int* __restrict__ p, int n,
                                                   const __nv_bfloat16* __restrict__ W1b,
                                                   const float* __restrict__ b1, float* __restrict__ U,
                                                   float* __restrict__ V) {
    __shared__ __align__(16) float f[kUvRows][2][kFeatDim];  // per vertex: f1, f2(p), as bf16-rounded floats
    const int c = threadIdx.x;
    const int v0 = blockIdx.x * kUvRows;
    for (int i = c; i < kUvRows * 2 * kFeatDim; i += 256) {
        const int v = i / (2 * kFeatDim), k = i % (2 * kFeatDim), a = v0 + v;
        float x = 0.f;
        if (a < n) {
            if (k < kFeatDim) x = F1[(size_t)a * kFeatDim + k];
            else {
                const int img = p[a];
                x = img < n ? F2[(size_t)img * kFeatDim + (k - kFeatDim)] : 0.f;
            }
        }
        f[v][k < kFeatDim ? 0 : 1][k & (kFeatDim - 1)] = __bfloat162float(__float2bfloat16(x));
    }
    float w[4][kFeatDim];  // W1[c] in four 32-column quarters: f1(a), f1(b), f2(pa), f2(pb)
    {
        const uint4* w4 = reinterpret_cast<const uint4*>(W1b + (size_t)c * kMlpIn);
#pragma unroll
        for (int i = 0; i < kMlpIn / 8; i++) {
            const uint4 q = w4[i];
            const uint32_t r[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {   // bf16 -> float is a shift
                w[i >> 2][8 * (i & 3) + 2 * u] = __uint_as_float(r[u] << 16);
                w[i >> 2][8 * (i & 3) + 2 * u + 1] = __uint_as_float(r[u] & 0xffff0000u);
            }
        }
    }
    const float bias = b1[c];
    __syncthreads();
    for (int v = 0; v < kUvRows && v0 + v < n; v += 2) {
        float u[2] = {0.f, 0.f}, x[2] = {0.f, 0.f};
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int k = 0; k < kFeatDim; k += 4) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float4 q = *reinterpret_cast<const float4*>(&f[v + e][h][k]);
                    u[e] = fmaf(w[2 * h][k], q.x, u[e]);
                    x[e] = fmaf(w[2 * h + 1][k], q.x, x[e]);
                    u[e] = fmaf(w[2 * h][k + 1], q.y, u[e]);
                    x[e] = fmaf(w[2 * h + 1][k + 1], q.y, x[e]);
                    u[e] = fmaf(w[2 * h][k + 2], q.z, u[e]);
                    x[e] = fmaf(w[2 * h + 1][k + 2], q.z, x[e]);
                    u[e] = fmaf(w[2 * h][k + 3], q.w, u[e]);
                    x[e] = fmaf(w[2 * h + 1][k + 3], q.w, x[e]);
                }
            }
#pragma unroll
        for (int e = 0; e < 2; e++)
            if (v0 + v + e < n) {
                U[(size_t)(v0 + v + e) * kMlpHid + c] = u[e] + bias;
                V[(size_t)(v0 + v + e) * kMlpHid + c] = x[e];
            }
    }
}

constexpr int kRankBuilders = 512, kRankThreads = kRankBuilders + 128;   // 16 builder warps, 4 epilogue warps
constexpr int kRankRows = kGemmM / (kRankBuilders / 32);                  // rows a builder warp makes per tile
constexpr int kRankA = kGemmM * 512;          // A tile: 128 rows x 256 bf16 (4 k-blocks of 16 KB)
constexpr int kRankB = kMlpHid * 512;         // W2: 256 rows x 256 bf16 (4 k-blocks of 32 KB)
constexpr int kRankSmem = kRankA + kRankB + 2 * kMlpHid * 4 + 1024 + 256;

// y[i] = w3 . relu(W2 relu(U[pa i] + V[pb i]) + b2) + b3 for i < k.
// The builder warps make tile t + 1 and its MMA runs while the epilogue warps
// reduce tile t from the other half of TMEM (two 256-column accumulators), so a
// tile costs its build and MMA, not the epilogue too; the pairs are loaded a tile
// ahead and 16 warps build (246 -> 223 -> 174 us for 524,288 pairs at n = 8,192,
// 8.9 -> 6.3 us per tile of 128 pairs and SM).  Bound by the gathers of the
// build, 2 KB of fp32 U and V per pair.
// Every wait is bounded: after a timeout (err set) a thread waits no more, no
// further MMA is issued or accumulator read, and the warps run out their loops.
// STALL: the test hook's form, in a kernel of its own because the registers of
// this one are all taken (a run-time switch cost the learned sweep 1.7%).
template <bool STALL>
static __global__ void __launch_bounds__(kRankThreads, 1)
k_mlp_rank(const float* __restrict__ U, const float* __restrict__ V, const int* __restrict__ pa,
           const int* __restrict__ pb, long long k, const __nv_bfloat16* __restrict__ W2b,
           const float* __restrict__ b2, const float* __restrict__ w3, const float* __restrict__ b3,
           float* __restrict__ y, int* __restrict__ err) {
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kMlpHid >> 3) << 17) |
                                ((uint32_t)(kGemmM >> 4) << 24);
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    const uint32_t sA = base, sB = base + kRankA;
    float* sb2 = reinterpret_cast<float*>(smem_raw + (sB + kRankB - raw));
    float* sw3 = sb2 + kMlpHid;
    const uint32_t bars = sB + kRankB + 2 * kMlpHid * 4;   // mma[2]: tile in accumulator h done; free[2]: h reduced
    const uint32_t tslot = bars + 32;
    uint32_t* tslot_ptr = reinterpret_cast<uint32_t*>(smem_raw + (tslot - raw));
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    auto bar_mma = [&](int h) { return bars + 8 * h; };
    auto bar_free = [&](int h) { return bars + 16 + 8 * h; };

    if (wid == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(tslot), "r"(2 * kMlpHid) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int h = 0; h < 2; h++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar_mma(h)) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" :: "r"(bar_free(h)) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // W2 resident: row r (output unit), 16-byte chunk c of its 512 bytes
    const uint8_t* W2 = reinterpret_cast<const uint8_t*>(W2b);
    for (int i = tid; i < kMlpHid * 32; i += kRankThreads) {
        const int r = i >> 5, c = i & 31, kb = c >> 3, cc = c & 7;
        const uint4 v = *reinterpret_cast<const uint4*>(W2 + (size_t)r * 512 + c * 16);
        const uint32_t dst = sB + kb * (kMlpHid * 128) + r * 128 + ((cc ^ (r & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" :: "r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
    }
    for (int i = tid; i < kMlpHid; i += kRankThreads) { sb2[i] = b2[i]; sw3[i] = w3[i]; }
    const float bias3 = b3[0];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // W2, read by the tensor cores
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot_ptr;

    const long long tiles = (k + kGemmM - 1) / kGemmM;
    constexpr int limit = STALL ? kStallPolls : 1 << 22;   // polls of a wait
    int it = 0, issued = 0;   // tiles begun; tiles handed to the tensor cores (thread 0)
    bool ok = true;
    if (wid < kRankBuilders / 32) {
        int na = 0, nb = 0;
        {
            const long long i = (long long)blockIdx.x * kGemmM + wid * kRankRows + lane;
            if (lane < kRankRows && i < k) { na = pa[i]; nb = pb[i]; }
        }
        for (long long t = blockIdx.x; t < tiles; t += gridDim.x, it++) {
            const int h = it & 1;
            const long long row0 = t * kGemmM;
            // the previous tile's MMA has read A
            if (ok && it > 0) ok = mbar_wait_bounded(bar_mma(h ^ 1), ((it - 1) >> 1) & 1, err, limit);
            // A tile: warp w builds rows 8 w .. 8 w + 7 (four rows per pass, their
            // loads all issued before any store); lane = 16-byte chunk (8 units).
            // Lane q holds row q's pair, loaded a tile ahead.
            const int ca = na, cb = nb;
            const long long next = row0 + (long long)gridDim.x * kGemmM + wid * kRankRows + lane;
            if (lane < kRankRows && next < k) { na = pa[next]; nb = pb[next]; }
#pragma unroll
            for (int r0 = 0; r0 < kRankRows; r0 += 4) {
                float4 u[4][2], x[4][2];
                bool live[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int a = __shfl_sync(0xffffffffu, ca, r0 + q), b = __shfl_sync(0xffffffffu, cb, r0 + q);
                    live[q] = row0 + wid * kRankRows + r0 + q < k;
                    if (live[q]) {
                        const float4* u4 = reinterpret_cast<const float4*>(U + (size_t)a * kMlpHid + lane * 8);
                        const float4* v4 = reinterpret_cast<const float4*>(V + (size_t)b * kMlpHid + lane * 8);
                        u[q][0] = u4[0]; u[q][1] = u4[1]; x[q][0] = v4[0]; x[q][1] = v4[1];
                    }
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int r = wid * kRankRows + r0 + q;
                    uint4 out = make_uint4(0, 0, 0, 0);
                    if (live[q]) {
                        const float4 u0 = u[q][0], u1 = u[q][1], x0 = x[q][0], x1 = x[q][1];
                        __nv_bfloat162 h0 = __floats2bfloat162_rn(fmaxf(u0.x + x0.x, 0.f), fmaxf(u0.y + x0.y, 0.f));
                        __nv_bfloat162 h1 = __floats2bfloat162_rn(fmaxf(u0.z + x0.z, 0.f), fmaxf(u0.w + x0.w, 0.f));
                        __nv_bfloat162 h2 = __floats2bfloat162_rn(fmaxf(u1.x + x1.x, 0.f), fmaxf(u1.y + x1.y, 0.f));
                        __nv_bfloat162 h3 = __floats2bfloat162_rn(fmaxf(u1.z + x1.z, 0.f), fmaxf(u1.w + x1.w, 0.f));
                        out.x = *reinterpret_cast<uint32_t*>(&h0);
                        out.y = *reinterpret_cast<uint32_t*>(&h1);
                        out.z = *reinterpret_cast<uint32_t*>(&h2);
                        out.w = *reinterpret_cast<uint32_t*>(&h3);
                    }
                    const int kb = lane >> 3, cc = lane & 7;
                    const uint32_t dst = sA + kb * (kGemmM * 128) + r * 128 + ((cc ^ (r & 7)) << 4);
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" :: "r"(dst), "r"(out.x), "r"(out.y), "r"(out.z), "r"(out.w) : "memory");
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("bar.sync 1, %0;" :: "n"(kRankBuilders) : "memory");
            // the accumulator's previous tile has been reduced
            if (tid == 0 && ok && it >= 2) ok = mbar_wait_bounded(bar_free(h), ((it >> 1) - 1) & 1, err, limit);
            if (tid == 0 && ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int kb = 0; kb < 4; kb++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {  // 16 bf16 = 32 bytes of K per MMA
                        const uint64_t da = umma_desc_sw128(sA + kb * (kGemmM * 128) + j * 32);
                        const uint64_t db = umma_desc_sw128(sB + kb * (kMlpHid * 128) + j * 32);
                        const uint32_t acc = (kb | j) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                            :: "r"(tmem + h * kMlpHid), "l"(da), "l"(db), "r"(kIdesc), "r"(acc) : "memory");
                    }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             :: "r"(bar_mma(h)) : "memory");
                issued = it + 1;
            }
        }
        // the last MMA has finished before the CTA frees TMEM and leaves
        if (tid == 0 && issued > 0) mbar_wait_bounded(bar_mma((issued - 1) & 1), ((issued - 1) >> 1) & 1, err);
    } else {
        const int q4 = wid & 3;   // the TMEM lane quarter a warp may read
        for (long long t = blockIdx.x; t < tiles; t += gridDim.x, it++) {
            const int h = it & 1;
            bool here = ok && mbar_wait_bounded(bar_mma(h), (it >> 1) & 1, err, limit);
            // test hook (bm_test_stall): CTA 0's first tile also waits for the
            // accumulator's next tile, which needs this one reduced first
            if (here && STALL && blockIdx.x == 0 && it == 0) here = mbar_wait_bounded(bar_mma(h), 1, err, limit);
            ok = __all_sync(0xffffffffu, here);
            if (!ok) continue;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const long long i = t * kGemmM + q4 * 32 + lane;
            float acc = 0.f;
            for (int cb = 0; cb < kMlpHid / 32; cb++) {
                uint32_t r[32];
                const uint32_t taddr = tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)(h * kMlpHid + cb * 32);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                    "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                    "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                      "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                      "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int q = 0; q < 32; q++) {
                    const int c = cb * 32 + q;
                    acc = fmaf(fmaxf(__uint_as_float(r[q]) + sb2[c], 0.f), sw3[c], acc);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar_free(h)) : "memory");
            if (i < k) y[i] = acc + bias3;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (wid == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(2 * kMlpHid) : "memory");
}

}  // namespace bm
