// mlp.cu -- the learned surrogate's network: a multilayer perceptron
// (GELU hidden layers) trained and evaluated entirely on the GPU with
// hand-written kernels.  rfsyn has no learned component; this maps a scene's
// parameter vector to its tx -> rx transfer function.
//
// Kernels:
//   k_gemm      C[M,N] = op(A) op(B) on the tensor cores (BF16 operands,
//               mma.sync m16n8k16, FP32 accumulation), operands in either
//               layout, tiles staged by cp.async (four stages), fused
//               epilogues: bias + GELU (hidden layers, pre-activation kept in
//               FP32 for the backward pass), bias (output layer), GELU'
//               (backward through a hidden layer, dZ in FP32 and BF16), plain
//               FP32 (weight gradients);
//   k_gemm_tc   the same products and epilogues on tcgen05 (accumulators in
//               tensor memory), selectable; slower on this network's products;
//   k_mse       loss gradient 2 (out - y) / (M N), FP32 / BF16, per-block loss
//               partials (deterministic);
//   k_colsum    bias gradients as deterministic column sums of dZ;
//   k_adam      Adam over every parameter in one launch, with bias correction
//               and a cosine learning rate taken from the device step
//               counter; writes the BF16 weights used by the next step's
//               GEMMs and advances the counter;
//   k_gather    a training batch from the resident data set through a
//               per-epoch permutation and the device step counter.
// The transposed copies (weights, activations, dZ) exist only for k_gemm_tc,
// whose operands are both K-major.
// One training step (gather, forward, loss, backward, Adam) is captured in a
// CUDA graph and replayed; the weight and bias gradients run beside the chain
// of dX products on streams of their own.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "engine.h"
#include "overlap.cuh"

typedef __nv_bfloat16 bf16;
using rfb::grid_launch_next;
using rfb::grid_wait;
using rfb::launch_step;

namespace {

constexpr int GK = 64;      // K per stage
constexpr int GSTAGES = 4;  // stages of the ring

enum { EPI_HIDDEN = 0, EPI_OUT = 1, EPI_BWD_GELU = 2, EPI_F32 = 3 };

struct Epi {
    const float *bias;   // [N] (HIDDEN, OUT)
    float *f32;          // HIDDEN: pre-activation (or null); OUT: output; BWD_GELU: dZ; F32: C
    bf16 *b16;           // HIDDEN: GELU(pre); BWD_GELU: dZ
    bf16 *b16t;          // BWD_GELU: dZ^T ([N][M]), or null
    const float *pre;    // BWD_GELU: pre-activation of the layer whose output gradient this is
};

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

__device__ __forceinline__ void cp16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}

__device__ __forceinline__ void mma_bf16(float c[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                         unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16-byte chunk c of row r of a tile whose rows hold CH chunks: where it lies,
// so that the eight rows of an ldmatrix fall on different banks.
template <int CH>
__device__ __forceinline__ int swz(int r, int c) {
    return CH == 8 ? (c ^ (r & 7)) : (c ^ ((r >> 1) & 3));
}
template <bool TRANS>
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], unsigned addr) {
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr));
}

// C = op(A) op(B): A is [M][lda] (K contiguous), with TA [K][lda] (M
// contiguous); B is [N][ldb], with TB [K][ldb].  M, N multiples of the tile,
// K of 64, lda / ldb of 8.  BM x BN output tiles, four warps as 2 x 2.
//
// Bound by latency: a training step's products are 0.13 GFLOP, so what counts
// is how many CTAs there are and how far the loads run ahead.  32 x 32 tiles
// give 256 x 512 outputs 128 CTAs (64 x 64 tiles: 32 on 148 SMs), and three
// 64-deep stages are in flight while one is used: 4.2-7.2 us a product of
// the 256-row step, cold, against 6.6-17.1 us with 64 x 64 tiles, two 32-deep
// stages and scalar fragment loads; the whole step 0.19 -> 0.063 ms (calls of
// 200 steps) with the changes around it.  K runs in the same order in every tile, so the tile changes no
// result.  Operands in either layout save the transposed copies of weights,
// activations and gradients.
template <int EPI, bool TA, bool TB, int BM, int BN>
__global__ void __launch_bounds__(128) k_gemm(const bf16 *__restrict__ A, int lda, const bf16 *__restrict__ B, int ldb,
                                              int M, int N, int K, Epi epi) {
    constexpr int ACH = TA ? BM / 8 : GK / 8, BCH = TB ? BN / 8 : GK / 8;  // chunks of a row
    constexpr int AR = TA ? GK : BM, BR = TB ? GK : BN;                    // rows
    constexpr int MI = BM / 32, NI = BN / 16;                              // m16 and n8 tiles of a warp
    extern __shared__ __align__(128) unsigned char gsm[];
    grid_launch_next();
    grid_wait();
    const unsigned as = (unsigned)__cvta_generic_to_shared(gsm), bs = as + GSTAGES * BM * GK * 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * (BM / 2), wn = (warp & 1) * (BN / 2);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[MI][NI][4] = {};
    auto load = [&](int st, int k0) {
#pragma unroll
        for (int q = tid; q < AR * ACH; q += 128) {
            const int r = q / ACH, c = q % ACH;
            const bf16 *g = TA ? A + (size_t)(k0 + r) * lda + m0 + c * 8 : A + (size_t)(m0 + r) * lda + k0 + c * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                             as + st * BM * GK * 2 + (r * ACH + swz<ACH>(r, c)) * 16),
                         "l"(g));
        }
#pragma unroll
        for (int q = tid; q < BR * BCH; q += 128) {
            const int r = q / BCH, c = q % BCH;
            const bf16 *g = TB ? B + (size_t)(k0 + r) * ldb + n0 + c * 8 : B + (size_t)(n0 + r) * ldb + k0 + c * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                             bs + st * BN * GK * 2 + (r * BCH + swz<BCH>(r, c)) * 16),
                         "l"(g));
        }
    };
    const int nk = K / GK;
#pragma unroll
    for (int q = 0; q < GSTAGES - 1; q++) {
        if (q < nk) load(q, q * GK);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    for (int kt = 0; kt < nk; kt++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(GSTAGES - 2) : "memory");
        // stage kt has landed for every thread, and stage kt - 1 is used up
        __syncthreads();
        if (kt + GSTAGES - 1 < nk) load((kt + GSTAGES - 1) % GSTAGES, (kt + GSTAGES - 1) * GK);
        asm volatile("cp.async.commit_group;\n" ::);
        const unsigned at = as + (kt % GSTAGES) * BM * GK * 2, bt = bs + (kt % GSTAGES) * BN * GK * 2;
#pragma unroll
        for (int kk = 0; kk < GK; kk += 16) {
            unsigned a[MI][4], b[NI / 2][4];
#pragma unroll
            for (int mi = 0; mi < MI; mi++) {
                const int mr = wm + 16 * mi;
                const int r = TA ? kk + (lane & 7) + ((lane >> 4) << 3) : mr + (lane & 15);
                const int c = TA ? mr / 8 + ((lane >> 3) & 1) : kk / 8 + (lane >> 4);
                ldsm4<TA>(a[mi], at + (r * ACH + swz<ACH>(r, c)) * 16);
            }
#pragma unroll
            for (int nj = 0; nj < NI / 2; nj++) {
                const int nr = wn + 16 * nj;
                const int r = TB ? kk + (lane & 15) : nr + (lane & 7) + ((lane >> 4) << 3);
                const int c = TB ? nr / 8 + (lane >> 4) : kk / 8 + ((lane >> 3) & 1);
                ldsm4<TB>(b[nj], bt + (r * BCH + swz<BCH>(r, c)) * 16);
            }
#pragma unroll
            for (int mi = 0; mi < MI; mi++)
#pragma unroll
                for (int ni = 0; ni < NI; ni++)
                    mma_bf16(acc[mi][ni], a[mi][0], a[mi][1], a[mi][2], a[mi][3], b[ni / 2][2 * (ni & 1)],
                             b[ni / 2][2 * (ni & 1) + 1]);
        }
    }
    // epilogue: acc[mi][ni] covers rows r, r+8 and columns c, c+1
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mi = 0; mi < MI; mi++)
#pragma unroll
        for (int ni = 0; ni < NI; ni++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = m0 + wm + 16 * mi + g + 8 * h;
                const int c = n0 + wn + 8 * ni + 2 * t;
                float v0 = acc[mi][ni][2 * h], v1 = acc[mi][ni][2 * h + 1];
                const size_t o = (size_t)r * N + c;
                if (EPI == EPI_HIDDEN || EPI == EPI_OUT) {
                    v0 += epi.bias[c];
                    v1 += epi.bias[c + 1];
                    if (EPI == EPI_OUT || epi.f32) *reinterpret_cast<float2 *>(epi.f32 + o) = make_float2(v0, v1);
                    if (EPI == EPI_HIDDEN) {
                        __nv_bfloat162 p;
                        p.x = __float2bfloat16_rn(gelu(v0));
                        p.y = __float2bfloat16_rn(gelu(v1));
                        *reinterpret_cast<__nv_bfloat162 *>(epi.b16 + o) = p;
                    }
                } else if (EPI == EPI_BWD_GELU) {
                    v0 *= gelu_grad(epi.pre[o]);
                    v1 *= gelu_grad(epi.pre[o + 1]);
                    *reinterpret_cast<float2 *>(epi.f32 + o) = make_float2(v0, v1);
                    __nv_bfloat162 p;
                    p.x = __float2bfloat16_rn(v0);
                    p.y = __float2bfloat16_rn(v1);
                    *reinterpret_cast<__nv_bfloat162 *>(epi.b16 + o) = p;
                    if (epi.b16t) {
                        epi.b16t[(size_t)c * M + r] = p.x;
                        epi.b16t[(size_t)(c + 1) * M + r] = p.y;
                    }
                } else {
                    *reinterpret_cast<float2 *>(epi.f32 + o) = make_float2(v0, v1);
                }
            }
}

// ---- the same contraction on the 5th-generation tensor cores ----------------
// k_gemm_tc: C = A . B^T with one tcgen05.mma (M 128, N 32, K 16, BF16 in,
// FP32 accumulation in tensor memory) stream per CTA tile of 128 x 32.
// K is staged 64 at a time (one 128-byte row per tile row) by cp.async into
// a four-stage ring in the 128-byte-swizzled K-major layout the MMA's shared
// memory descriptors describe (16-byte chunk c of row r at chunk c ^ (r % 8)
// of the row, 8-row groups 1024 bytes apart).  One thread issues the four
// MMAs of a stage and commits them to the stage's mbarrier, which frees the
// stage for a later load; the last commit releases the accumulator, which
// eight warps read back (tcgen05.ld, warp w lanes 32 (w % 4) .. +31 = tile
// rows, columns 16 (w / 4) .. +15) into the same fused epilogues as
// k_gemm.  Every wait is bounded: on a timeout the CTA records it,
// waits (bounded) for its MMAs in flight, frees its tensor memory and
// returns.  Measured on the surrogate's network (54-512x4-512, one B200):
// a training step takes 0.182 ms at batch 256 against 0.068 ms on k_gemm, and
// 0.38 against 0.17 ms at batch 2048 -- products of at most 512 x 2048 x 512
// are latency-bound on staging their tiles, which this cp.async-fed form does
// no faster, and its operands need transposed copies -- so it runs only when
// asked for (RFSYN_FDTD_MLP_GEMM=tcgen05).
namespace tc {
// Tiles of 128 rows x BN columns (BN 32: more CTAs on these small products
// -- 128 x 128 tiles, fewer CTAs and fewer re-reads of A, measured slower
// even on 2048-row batches), K staged 64 at a time in a 4-stage ring filled
// three steps ahead (a refill waits for the MMAs of the step before, which
// take far less than a load)
constexpr int BM = 128, BK = 64, STAGES = 4, DIST = 3, THREADS = 256;
template <int BN>
struct Shape {
    static constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    static_assert(STAGE_BYTES % 1024 == 0 && A_BYTES % 1024 == 0, "swizzle atoms stay 1024-byte aligned");
    static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 64;  // tiles 1024-aligned, then barriers, TMEM address
    static constexpr uint32_t TMEM_COLS = BN;                     // FP32 accumulator: a column per output column
    // instruction descriptor: F32 accumulator, BF16 A and B, both K-major,
    // N >> 3 at bit 17, M >> 4 at bit 24
    static constexpr uint32_t IDESC =
        (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
};
constexpr long long WAIT = 2000000000LL;  // SM cycles, about a second
}  // namespace tc

__device__ __forceinline__ unsigned sm_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory descriptor of a K-major, 128-byte-swizzled operand tile at
// shared address `a`: start address >> 4, leading offset 16 bytes (unused
// with swizzling), stride offset 1024 bytes (one 8-row group), descriptor
// version 1, layout 2 (128-byte swizzle).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t a) {
    return (uint64_t)((a >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

__device__ __forceinline__ void tc_mbar_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(sm_addr(bar)));
}

__device__ __forceinline__ bool tc_mbar_wait(uint64_t *bar, unsigned parity) {
    const long long t0 = clock64();
    for (;;) {
        unsigned ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(sm_addr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > tc::WAIT) return false;
    }
}

template <int EPI>
__device__ __forceinline__ void epi_store(const Epi &epi, int M, int N, int r, int c, float v) {
    const size_t o = (size_t)r * N + c;
    if (EPI == EPI_HIDDEN || EPI == EPI_OUT) {
        v += epi.bias[c];
        if (EPI == EPI_OUT || epi.f32) epi.f32[o] = v;
        if (EPI == EPI_HIDDEN) epi.b16[o] = __float2bfloat16_rn(gelu(v));
    } else if (EPI == EPI_BWD_GELU) {
        v *= gelu_grad(epi.pre[o]);
        epi.f32[o] = v;
        const bf16 b = __float2bfloat16_rn(v);
        epi.b16[o] = b;
        epi.b16t[(size_t)c * M + r] = b;
    } else {
        epi.f32[o] = v;
    }
}

// C = A . B^T.  A: [M][lda], B: [N][ldb], BF16 row-major (K-major); M a
// multiple of 128, N of 32, K of 64, lda / ldb multiples of 8.
template <int EPI, int BN>
__global__ void __launch_bounds__(tc::THREADS) k_gemm_tc(const bf16 *__restrict__ A, int lda, const bf16 *__restrict__ B,
                                                 int ldb, int M, int N, int K, Epi epi, int *err) {
    using S = tc::Shape<BN>;
    extern __shared__ unsigned char tc_smem[];
    const unsigned pad = (1024u - (sm_addr(tc_smem) & 1023u)) & 1023u;
    unsigned char *tiles = tc_smem + pad;
    uint64_t *bar = reinterpret_cast<uint64_t *>(tiles + tc::STAGES * S::STAGE_BYTES);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar + tc::STAGES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * tc::BM, n0 = blockIdx.x * BN;
    if (tid == 0) {
        for (int s = 0; s < tc::STAGES; s++) tc_mbar_init(&bar[s]);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(sm_addr(tmem_slot)),
                     "r"(S::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    auto load = [&](int s, int k0) {
        unsigned char *as = tiles + s * S::STAGE_BYTES, *bs = as + S::A_BYTES;
        for (int q = tid; q < tc::BM * 8; q += tc::THREADS) {
            const int r = q >> 3, c = q & 7;
            cp16(as + r * 128 + ((c ^ (r & 7)) << 4), A + (size_t)(m0 + r) * lda + k0 + c * 8);
        }
        for (int q = tid; q < BN * 8; q += tc::THREADS) {
            const int r = q >> 3, c = q & 7;
            cp16(bs + r * 128 + ((c ^ (r & 7)) << 4), B + (size_t)(n0 + r) * ldb + k0 + c * 8);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    const int nk = K / tc::BK;
    bool failed = false;
    int committed = -1;  // the last K step whose MMAs were committed
    for (int p = 0; p < tc::DIST && p < nk; p++) load(p % tc::STAGES, p * tc::BK);
    for (int kt = 0; kt < nk; kt++) {
        const int s = kt % tc::STAGES, nxt = kt + tc::DIST;
        if (nxt < nk) {
            // stage nxt % STAGES was last read by the MMAs of step nxt - STAGES
            const int ns = nxt % tc::STAGES, prev = nxt - tc::STAGES;
            if (prev >= 0 && !tc_mbar_wait(&bar[ns], (prev / tc::STAGES) & 1)) failed = true;
            if (__syncthreads_or(failed)) break;
            load(ns, nxt * tc::BK);
        }
        // step kt's copies are complete once at most the copies of the steps
        // loaded after it are pending
        const int after = nk - 1 - kt < tc::DIST ? nk - 1 - kt : tc::DIST;
        static_assert(tc::DIST <= 3, "the waits below cover up to three later groups");
        if (after >= 3) asm volatile("cp.async.wait_group 3;\n" ::: "memory");
        else if (after == 2) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        else if (after == 1) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        // make them visible to the tensor core's (async-proxy) reads, then to
        // the issuing thread
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const uint32_t as = sm_addr(tiles + s * S::STAGE_BYTES), bs = as + S::A_BYTES;
#pragma unroll
            for (int kk = 0; kk < tc::BK / 16; kk++) {
                const uint64_t da = sw128_desc(as + 32 * kk), db = sw128_desc(bs + 32 * kk);
                const uint32_t acc = (kt | kk) ? 1u : 0u;
                asm volatile(
                    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(S::IDESC), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             sm_addr(&bar[s]))
                         : "memory");
        }
        committed = kt;
    }
    // the last commit covers every MMA this CTA issued; copies still in
    // flight (after an early exit) land before the shared memory is released
    if (committed >= 0 && !tc_mbar_wait(&bar[committed % tc::STAGES], (committed / tc::STAGES) & 1)) failed = true;
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (__syncthreads_or(failed)) {
        if (tid == 0) atomicExch(err, 1);
    } else {
        // warp w reads TMEM lanes 32 (w % 4) .. (the tile rows it may
        // access) and the BN / 2 columns of half w / 4, 16 at a time
        static_assert(tc::THREADS == 256 && BN % 32 == 0, "eight warps: four lane groups x two column halves");
        const int r = m0 + 32 * (warp & 3) + lane;  // TMEM lane = tile row
#pragma unroll
        for (int cc = (BN / 2) * (warp >> 2); cc < (BN / 2) * ((warp >> 2) + 1); cc += 16) {
            uint32_t v[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                "[%16];\n"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)cc));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int q = 0; q < 16; q++) epi_store<EPI>(epi, M, N, r, n0 + cc + q, __uint_as_float(v[q]));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(S::TMEM_COLS)
                     : "memory");
}

// Loss gradient of the mean squared error over M x N outputs; per-block
// partial sums of the squared error (fixed order: deterministic).
__global__ void k_mse(const float *out, const float *y, int M, int N, float *d32, bf16 *d16, bf16 *d16t,
                      float *partial) {
    __shared__ float red[256];
    grid_launch_next();
    grid_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float se = 0.f;
    if (i < M * N) {
        const float e = out[i] - y[i];
        se = e * e;
        const float gr = 2.0f * e / (float)(M * N);
        d32[i] = gr;
        const bf16 b = __float2bfloat16_rn(gr);
        d16[i] = b;
        if (d16t) {
            const int r = i / N, c = i - r * N;
            d16t[(size_t)c * M + r] = b;
        }
    }
    red[threadIdx.x] = se;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// Column sums of d [M][N] (bias gradients), one thread per column.
// Block of 32 columns x 8 warps: warp w sums rows w, w + 8, ... of its
// lane's column, then the eight partial sums are added in warp order (a
// fixed order: deterministic).
__global__ void __launch_bounds__(256) k_colsum(const float *d, int M, int N, float *out) {
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (c < N)
        for (int r = w; r < M; r += 8) s += d[(size_t)r * N + c];
    part[w][lane] = s;
    __syncthreads();
    if (w == 0 && c < N) {
        float t = part[0][lane];
        for (int q = 1; q < 8; q++) t += part[q][lane];
        out[c] = t;
    }
}

// One parameter array (a layer's weights or its bias).
struct AdamSeg {
    float *w, *m, *v;
    const float *g;
    bf16 *w16, *w16t;    // BF16 copies [rows][cols] (null for biases) and [cols][rows] (or null)
    int n, rows, cols;
};
struct AdamCfg {
    float lr0, beta1, beta2, eps;
    long long total_steps;
};

constexpr int ADAM_BLOCK = 1024;  // parameters of a block, four a thread

// Adam with bias correction over every parameter, learning rate lr0 * 0.5 (1
// + cos(pi s / S)); block b takes the parameters from blocks[b].y on of
// segs[blocks[b].x].  24 bytes a parameter move (and 2 of BF16), so one
// launch of 16-byte accesses takes the place of one per array with scalar
// ones: ten launches of 4.2-8.2 us, cold, for the 5-layer network, and two
// powf a parameter, before.  The last block to finish advances *step (steps
// done before this update), which every block has read by then.
__global__ void __launch_bounds__(256) k_adam(const AdamSeg *segs, const int2 *blocks, const AdamCfg *cfg, long long *step,
                                              int *done) {
    __shared__ float s_lr, s_c1, s_c2;
    grid_launch_next();
    grid_wait();
    const AdamCfg a = *cfg;
    if (threadIdx.x == 0) {
        const long long s = *step + 1;
        const float frac = (float)min(1.0, (double)(s - 1) / (double)max(1LL, a.total_steps));
        s_lr = a.lr0 * 0.5f * (1.0f + cospif(frac));
        s_c1 = 1.0f - powf(a.beta1, (float)s);
        s_c2 = 1.0f - powf(a.beta2, (float)s);
    }
    __syncthreads();
    const float lr = s_lr, c1 = s_c1, c2 = s_c2;
    const int2 b = blocks[blockIdx.x];
    const AdamSeg sg = segs[b.x];
    const int i = b.y + 4 * threadIdx.x;
    if (i < sg.n) {
        // aligned for the vector accesses also where they are kept in memory
        alignas(16) float g[4], m[4], v[4], w[4];
        alignas(8) bf16 h[4];
        *reinterpret_cast<float4 *>(g) = *reinterpret_cast<const float4 *>(sg.g + i);
        *reinterpret_cast<float4 *>(m) = *reinterpret_cast<const float4 *>(sg.m + i);
        *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(sg.v + i);
        *reinterpret_cast<float4 *>(w) = *reinterpret_cast<const float4 *>(sg.w + i);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            // the contractions nvcc chose for b m + (1 - b) g, written out so
            // that the update stays the same bit for bit
            m[q] = __fmaf_rn(1.0f - a.beta1, g[q], __fmul_rn(a.beta1, m[q]));
            v[q] = __fmaf_rn(__fmul_rn(1.0f - a.beta2, g[q]), g[q], __fmul_rn(a.beta2, v[q]));
            const float mh = m[q] / c1, vh = v[q] / c2;
            w[q] = w[q] - lr * mh / (sqrtf(vh) + a.eps);
            h[q] = __float2bfloat16_rn(w[q]);
        }
        *reinterpret_cast<float4 *>(sg.m + i) = *reinterpret_cast<const float4 *>(m);
        *reinterpret_cast<float4 *>(sg.v + i) = *reinterpret_cast<const float4 *>(v);
        *reinterpret_cast<float4 *>(sg.w + i) = *reinterpret_cast<const float4 *>(w);
        if (sg.w16) *reinterpret_cast<uint2 *>(sg.w16 + i) = *reinterpret_cast<const uint2 *>(h);
        if (sg.w16t) {
            const int r = i / sg.cols, c = i - r * sg.cols;  // four columns of one row (cols a multiple of 4)
#pragma unroll
            for (int q = 0; q < 4; q++) sg.w16t[(size_t)(c + q) * sg.rows + r] = h[q];
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(done, 1) == (int)gridDim.x - 1) {
            *done = 0;
            *step += 1;
        }
    }
}

// Batch of B rows from the resident set: row q of the batch is sample
// perm[(step * B + q) mod n]; X as BF16 [B][kin] and its transpose, Y FP32.
__global__ void k_gather(const bf16 *X, const float *Y, const int *perm, long long n, const long long *step, int B,
                         int kin, int nout, bf16 *xb, bf16 *xbt, float *yb) {
    grid_launch_next();
    const int q = blockIdx.x;
    grid_wait();
    const long long idx = perm[((*step) * B + q) % n];
    for (int c = threadIdx.x; c < kin; c += blockDim.x) {
        const bf16 v = X[idx * kin + c];
        xb[(size_t)q * kin + c] = v;
        if (xbt) xbt[(size_t)c * B + q] = v;
    }
    for (int c = threadIdx.x; c < nout; c += blockDim.x) yb[(size_t)q * nout + c] = Y[idx * nout + c];
}

__global__ void k_f2bf(const float *in, bf16 *out, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __float2bfloat16_rn(in[i]);
}

// Rows of X [n][n_in] FP32 into BF16 [n][kin] (zero padding).
__global__ void k_pack_x(const float *in, int n_in, bf16 *out, int kin, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * kin) return;
    const size_t r = i / kin;
    const int c = (int)(i - r * kin);
    out[i] = __float2bfloat16_rn(c < n_in ? in[r * n_in + c] : 0.f);
}

}  // namespace

extern unsigned long long rfb_launch_count(void);

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct Layer {
    int in, out;             // out x in weights
    float *w = nullptr, *b = nullptr, *mw = nullptr, *vw = nullptr, *mb = nullptr, *vb = nullptr;
    float *gw = nullptr, *gb = nullptr;
    bf16 *w16 = nullptr, *w16t = nullptr;
};

struct fdtd_b200_mlp {
    int n_in, kin, width, depth, n_out;
    std::vector<Layer> L;
    int bmax = 0;                          // batch buffers sized for this many rows
    std::vector<float *> pre;              // per hidden layer [B][width]
    std::vector<bf16 *> act, actt;         // per layer input: act[0] = x, act[l] = GELU(pre[l-1]); transposes
    float *out = nullptr, *y = nullptr, *partial = nullptr;
    // gradient at each layer's output, FP32 and BF16 (and transposed for the
    // tcgen05 products): one set a layer, as the weight gradients of a layer
    // run while the next ones are computed
    std::vector<float *> g32;
    std::vector<bf16 *> g16, g16t;
    float *xf = nullptr;                   // bmax FP32 input rows on their way to BF16
    void *batch_mem = nullptr, *param_mem = nullptr;  // the blocks of the batch and of the parameter arrays
    // resident training set
    bf16 *X = nullptr;
    float *Y = nullptr;
    int *perm = nullptr;
    size_t n_data = 0;
    long long *step = nullptr;
    cudaStream_t st = nullptr, st_w = nullptr, st_b = nullptr;  // main; weight and bias gradients
    std::vector<cudaEvent_t> ev_g;         // gradient of layer l ready
    cudaEvent_t ev_w = nullptr, ev_b = nullptr;
    cudaGraphExec_t graph = nullptr;       // a training step, for batches of graph_b
    int graph_b = 0;
    unsigned long long graph_l = 0, graph_tc = 0;  // launches a captured step makes, and those on tcgen05
    AdamCfg *cfg = nullptr;
    bool overlap = false;                  // launches are being captured as programmatic dependents
    AdamSeg *segs = nullptr;
    int2 *blocks = nullptr;
    int n_blocks = 0, *done = nullptr;
    unsigned long long launches = 0;
    // tensor-core products: enabled (the shared memory attribute was set),
    // their launches, and the device flag a timed-out wait sets
    int tc = 0;
    unsigned long long tc_launches = 0;
    int *d_err = nullptr;
};

typedef struct fdtd_b200_mlp fdtd_b200_mlp_t;

#define MCK(call)                                                                             \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) {                                                              \
            rfb_set_error("%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); \
            return -1;                                                                        \
        }                                                                                     \
    } while (0)

// Sub-arrays of one block, on 256-byte boundaries: a driver allocation costs
// up to milliseconds, whatever its size.
struct Arena {
    char *base;
    size_t used = 0;
    template <typename X>
    void take(X *&p, size_t n) {
        p = base ? reinterpret_cast<X *>(base + used) : nullptr;
        used += (n * sizeof(X) + 255) / 256 * 256;
    }
};

static void mlp_free_graph(fdtd_b200_mlp *m) {
    if (m->graph) cudaGraphExecDestroy(m->graph);
    m->graph = nullptr;
}

static void mlp_free_batch(fdtd_b200_mlp *m) {
    cudaFree(m->batch_mem);
    m->batch_mem = nullptr;
    mlp_free_graph(m);
    m->bmax = 0;
}

static size_t mlp_lay_batch(fdtd_b200_mlp *m, int B, char *base) {
    const int nl = (int)m->L.size();
    Arena a{base};
    m->pre.assign(nl - 1, nullptr);
    m->act.assign(nl, nullptr);
    m->actt.assign(nl, nullptr);
    m->g32.assign(nl, nullptr);
    m->g16.assign(nl, nullptr);
    m->g16t.assign(nl, nullptr);
    for (int l = 0; l < nl; l++) {
        const size_t ni = (size_t)B * m->L[l].in, no = (size_t)B * m->L[l].out;
        a.take(m->act[l], ni);
        a.take(m->g32[l], no);
        a.take(m->g16[l], no);
        if (m->tc) {
            a.take(m->actt[l], ni);
            a.take(m->g16t[l], no);
        }
        if (l < nl - 1) a.take(m->pre[l], no);
    }
    const size_t no = (size_t)B * m->n_out;
    a.take(m->out, no);
    a.take(m->y, no);
    a.take(m->partial, no / 256 + 1);
    a.take(m->xf, (size_t)B * m->n_in);
    return a.used;
}

static int mlp_batch_buffers(fdtd_b200_mlp *m, int B) {
    if (B <= m->bmax) return 0;
    mlp_free_batch(m);
    MCK(cudaMalloc(&m->batch_mem, mlp_lay_batch(m, B, nullptr)));
    mlp_lay_batch(m, B, static_cast<char *>(m->batch_mem));
    m->bmax = B;
    return 0;
}

// The network's products on k_gemm, or with RFSYN_FDTD_MLP_GEMM=tcgen05 on
// k_gemm_tc where both operands are K-major and the shapes fit its tiles (M a
// multiple of 128, N of 32, K of 64 -- every training-step product of the
// surrogate does).  64 x 64 tiles once they give every SM a CTA: half the
// operand re-reads of 32 x 32 tiles, which a smaller product needs for CTAs
// (256 x 512 outputs: 32 against 128).
template <int BM>
constexpr int gemm_smem() {
    return GSTAGES * 2 * BM * GK * (int)sizeof(bf16);
}
template <int EPI, bool TA = false, bool TB = false>
static void gemm(fdtd_b200_mlp *m, cudaStream_t st, const bf16 *A, int lda, const bf16 *B, int ldb, int M, int N, int K,
                 Epi epi) {
    if constexpr (!TA && !TB) {
        if (m->tc && M > 0 && N > 0 && K > 0 && M % tc::BM == 0 && N % 32 == 0 && K % tc::BK == 0 && lda % 8 == 0 &&
            ldb % 8 == 0) {
            dim3 grid(N / 32, M / tc::BM);
            k_gemm_tc<EPI, 32><<<grid, tc::THREADS, tc::Shape<32>::SMEM, st>>>(A, lda, B, ldb, M, N, K, epi, m->d_err);
            m->tc_launches++;
            m->launches++;
            return;
        }
    }
    // the products of the main stream's chain are programmatic dependents
    const bool overlap = m->overlap && st == m->st;
    if ((long long)(M / 64) * (N / 64) >= 148)
        launch_step(k_gemm<EPI, TA, TB, 64, 64>, dim3(N / 64, M / 64), dim3(128), gemm_smem<64>(), st, overlap, A, lda, B,
                    ldb, M, N, K, epi);
    else
        launch_step(k_gemm<EPI, TA, TB, 32, 32>, dim3(N / 32, M / 32), dim3(128), gemm_smem<32>(), st, overlap, A, lda, B,
                    ldb, M, N, K, epi);
    m->launches++;
}
template <int EPI, bool TA, bool TB>
static bool gemm_attr() {
    return cudaFuncSetAttribute(k_gemm<EPI, TA, TB, 64, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                gemm_smem<64>()) == cudaSuccess;
}
static bool gemm_attrs() {
    return gemm_attr<EPI_HIDDEN, false, false>() && gemm_attr<EPI_OUT, false, false>() &&
           gemm_attr<EPI_BWD_GELU, false, false>() && gemm_attr<EPI_BWD_GELU, false, true>() &&
           gemm_attr<EPI_F32, false, false>() && gemm_attr<EPI_F32, true, true>();
}

// The tensor-core products need more than 48 KB of shared memory.
template <int BN>
static bool tc_attrs() {
    const int sm = tc::Shape<BN>::SMEM;
    return cudaFuncSetAttribute(k_gemm_tc<EPI_HIDDEN, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) ==
               cudaSuccess &&
           cudaFuncSetAttribute(k_gemm_tc<EPI_OUT, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) ==
               cudaSuccess &&
           cudaFuncSetAttribute(k_gemm_tc<EPI_BWD_GELU, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) ==
               cudaSuccess &&
           cudaFuncSetAttribute(k_gemm_tc<EPI_F32, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) ==
               cudaSuccess;
}

// A timed-out wait in a tensor-core product, reported once per call.
static int mlp_check_err(fdtd_b200_mlp *m) {
    int e = 0;
    if (cudaMemcpy(&e, m->d_err, sizeof e, cudaMemcpyDeviceToHost) != cudaSuccess) {
        rfb_set_error("surrogate: reading the error flag failed");
        return -1;
    }
    if (e) {
        cudaMemset(m->d_err, 0, sizeof(int));
        rfb_set_error("surrogate: a tensor-core product's wait timed out");
        return -1;
    }
    return 0;
}

// Forward pass of B rows whose input is already in act[0]; the hidden
// pre-activations are kept when a backward pass follows.
static void mlp_forward(fdtd_b200_mlp *m, int B, bool keep) {
    const int nl = (int)m->L.size();
    for (int l = 0; l < nl; l++) {
        const Layer &ly = m->L[l];
        Epi e{};
        e.bias = ly.b;
        if (l < nl - 1) {
            e.f32 = keep ? m->pre[l] : nullptr;
            e.b16 = m->act[l + 1];
            gemm<EPI_HIDDEN>(m, m->st, m->act[l], ly.in, ly.w16, ly.in, B, ly.out, ly.in, e);
        } else {
            e.f32 = m->out;
            gemm<EPI_OUT>(m, m->st, m->act[l], ly.in, ly.w16, ly.in, B, ly.out, ly.in, e);
        }
    }
}

// Transposes of the hidden activations (B x width, BF16) for the weight
// gradients on the tcgen05 products: written by a small kernel.
__global__ void k_transpose_bf16(const bf16 *in, int rows, int cols, bf16 *out) {
    __shared__ bf16 tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        if (r0 + y < rows && c0 + threadIdx.x < cols) tile[y][threadIdx.x] = in[(size_t)(r0 + y) * cols + c0 + threadIdx.x];
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        if (c0 + y < cols && r0 + threadIdx.x < rows) out[(size_t)(c0 + y) * rows + r0 + threadIdx.x] = tile[threadIdx.x][y];
}

// Backward pass after the forward (the output gradient already in the last
// layer's buffers): weight and bias gradients of every layer.  The chain of
// dX products runs on the main stream; each layer's weight gradient and bias
// sums follow on two streams of their own as its gradient is ready, and the
// main stream waits for both at the end.
static int mlp_backward(fdtd_b200_mlp *m, int B) {
    const int nl = (int)m->L.size();
    if (m->tc)
        // transposes of the layer inputs (act[0]^T is written by the gather)
        for (int l = 1; l < nl; l++) {
            dim3 grid((m->L[l].in + 31) / 32, (B + 31) / 32);
            k_transpose_bf16<<<grid, dim3(32, 8), 0, m->st>>>(m->act[l], B, m->L[l].in, m->actt[l]);
            m->launches++;
        }
    for (int l = nl - 1; l >= 0; l--) {
        const Layer &ly = m->L[l];
        MCK(cudaEventRecord(m->ev_g[l], m->st));
        MCK(cudaStreamWaitEvent(m->st_w, m->ev_g[l], 0));
        MCK(cudaStreamWaitEvent(m->st_b, m->ev_g[l], 0));
        // dW = dZ^T . X: [out][in] from dZ [B][out] and X [B][in]
        Epi e{};
        e.f32 = ly.gw;
        if (m->tc) gemm<EPI_F32>(m, m->st_w, m->g16t[l], B, m->actt[l], B, ly.out, ly.in, B, e);
        else gemm<EPI_F32, true, true>(m, m->st_w, m->g16[l], ly.out, m->act[l], ly.in, ly.out, ly.in, B, e);
        k_colsum<<<(ly.out + 31) / 32, 256, 0, m->st_b>>>(m->g32[l], B, ly.out, ly.gb);
        m->launches++;
        if (l > 0) {
            // dX = dZ . W, W [out][in], times GELU' of the previous layer's
            // pre-activation
            Epi eb{};
            eb.f32 = m->g32[l - 1];
            eb.b16 = m->g16[l - 1];
            eb.b16t = m->g16t[l - 1];
            eb.pre = m->pre[l - 1];
            if (m->tc) gemm<EPI_BWD_GELU>(m, m->st, m->g16[l], ly.out, ly.w16t, ly.out, B, ly.in, ly.out, eb);
            else gemm<EPI_BWD_GELU, false, true>(m, m->st, m->g16[l], ly.out, ly.w16, ly.in, B, ly.in, ly.out, eb);
        }
    }
    MCK(cudaEventRecord(m->ev_w, m->st_w));
    MCK(cudaEventRecord(m->ev_b, m->st_b));
    MCK(cudaStreamWaitEvent(m->st, m->ev_w, 0));
    MCK(cudaStreamWaitEvent(m->st, m->ev_b, 0));
    return 0;
}

static void mlp_loss(fdtd_b200_mlp *m, int B) {
    const int n = B * m->n_out;
    launch_step(k_mse, dim3((n + 255) / 256), dim3(256), 0, m->st, m->overlap, m->out, m->y, B, m->n_out, m->g32.back(),
                m->g16.back(), m->g16t.back(), m->partial);
    m->launches++;
}

static void mlp_adam(fdtd_b200_mlp *m) {
    k_adam<<<m->n_blocks, 256, 0, m->st>>>(m->segs, m->blocks, m->cfg, m->step, m->done);
    m->launches++;
}

// The parameter arrays and blocks of k_adam.
static int mlp_adam_segs(fdtd_b200_mlp *m) {
    std::vector<AdamSeg> segs;
    std::vector<int2> blocks;
    for (Layer &ly : m->L) {
        segs.push_back(AdamSeg{ly.w, ly.mw, ly.vw, ly.gw, ly.w16, ly.w16t, ly.out * ly.in, ly.out, ly.in});
        segs.push_back(AdamSeg{ly.b, ly.mb, ly.vb, ly.gb, nullptr, nullptr, ly.out, 1, ly.out});
    }
    for (size_t q = 0; q < segs.size(); q++)
        for (int o = 0; o < segs[q].n; o += ADAM_BLOCK) blocks.push_back(make_int2((int)q, o));
    m->n_blocks = (int)blocks.size();
    MCK(cudaMalloc(&m->segs, segs.size() * sizeof(AdamSeg)));
    MCK(cudaMalloc(&m->blocks, blocks.size() * sizeof(int2)));
    MCK(cudaMalloc(&m->done, sizeof(int)));
    MCK(cudaMalloc(&m->cfg, sizeof(AdamCfg)));
    MCK(cudaMemcpy(m->segs, segs.data(), segs.size() * sizeof(AdamSeg), cudaMemcpyHostToDevice));
    MCK(cudaMemcpy(m->blocks, blocks.data(), blocks.size() * sizeof(int2), cudaMemcpyHostToDevice));
    MCK(cudaMemset(m->done, 0, sizeof(int)));
    return 0;
}

// BF16 copies (and transposes) of the FP32 master weights.
static int mlp_sync_bf16(fdtd_b200_mlp *m) {
    for (Layer &ly : m->L) {
        const size_t n = (size_t)ly.out * ly.in;
        k_f2bf<<<(unsigned)((n + 255) / 256), 256, 0, m->st>>>(ly.w, ly.w16, n);
        m->launches++;
        if (!m->tc) continue;
        dim3 grid((ly.in + 31) / 32, (ly.out + 31) / 32);
        k_transpose_bf16<<<grid, dim3(32, 8), 0, m->st>>>(ly.w16, ly.out, ly.in, ly.w16t);
        m->launches++;
    }
    MCK(cudaGetLastError());
    return 0;
}

extern "C" void fdtd_b200_mlp_destroy(fdtd_b200_mlp_t *m) {
    if (!m) return;
    if (m->st) cudaStreamSynchronize(m->st);
    mlp_free_batch(m);
    cudaFree(m->param_mem);
    cudaFree(m->X); cudaFree(m->Y); cudaFree(m->perm); cudaFree(m->step); cudaFree(m->d_err);
    cudaFree(m->segs); cudaFree(m->blocks); cudaFree(m->done); cudaFree(m->cfg);
    for (cudaEvent_t ev : m->ev_g) cudaEventDestroy(ev);
    if (m->ev_w) cudaEventDestroy(m->ev_w);
    if (m->ev_b) cudaEventDestroy(m->ev_b);
    for (cudaStream_t st : {m->st, m->st_w, m->st_b})
        if (st) cudaStreamDestroy(st);
    delete m;
}

// splitmix64: the initial weights' random stream
static uint64_t splitmix(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

extern "C" fdtd_b200_mlp_t *fdtd_b200_mlp_create(int n_in, int width, int depth, int n_out, uint64_t seed) {
    if (n_in < 1 || width < 64 || width % 64 || n_out < 64 || n_out % 64 || depth < 1 || n_in > 4096) {
        rfb_set_error("mlp: n_in >= 1, width and n_out multiples of 64, depth >= 1");
        return nullptr;
    }
    fdtd_b200_mlp *m = new fdtd_b200_mlp();
    m->n_in = n_in;
    m->kin = (n_in + 63) / 64 * 64;
    m->width = width;
    m->depth = depth;
    m->n_out = n_out;
    for (int l = 0; l <= depth; l++) {
        Layer ly;
        ly.in = l == 0 ? m->kin : width;
        ly.out = l == depth ? n_out : width;
        m->L.push_back(ly);
    }
    uint64_t rs = seed;
    auto fail = [&]() -> fdtd_b200_mlp_t * {
        fdtd_b200_mlp_destroy(m);
        return nullptr;
    };
    for (cudaStream_t *st : {&m->st, &m->st_w, &m->st_b})
        if (cudaStreamCreateWithFlags(st, cudaStreamNonBlocking) != cudaSuccess) return fail();
    m->ev_g.assign(depth + 1, nullptr);
    for (cudaEvent_t &ev : m->ev_g)
        if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return fail();
    if (cudaEventCreateWithFlags(&m->ev_w, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&m->ev_b, cudaEventDisableTiming) != cudaSuccess)
        return fail();
    if (!gemm_attrs()) {
        rfb_set_error("mlp: cannot configure the products' shared memory");
        return fail();
    }
    {
        // RFSYN_FDTD_MLP_GEMM=tcgen05 puts the products whose shapes fit on
        // k_gemm_tc; by default every product runs on k_gemm, which is
        // faster on this network's products at every batch measured (see
        // k_gemm_tc)
        const char *v = getenv("RFSYN_FDTD_MLP_GEMM");
        const bool want = v && !strcmp(v, "tcgen05");
        m->tc = want && tc_attrs<32>();
        if (want && !m->tc) {
            rfb_set_error("mlp: cannot configure the tensor-core products' shared memory");
            return fail();
        }
    }
    auto lay = [&](char *base) {
        Arena a{base};
        for (Layer &ly : m->L) {
            const size_t nw = (size_t)ly.out * ly.in;
            for (float **p : {&ly.w, &ly.mw, &ly.vw, &ly.gw}) a.take(*p, nw);
            for (float **p : {&ly.b, &ly.mb, &ly.vb, &ly.gb}) a.take(*p, (size_t)ly.out);
            a.take(ly.w16, nw);
            if (m->tc) a.take(ly.w16t, nw);
        }
        return a.used;
    };
    const size_t param_bytes = lay(nullptr);
    if (cudaMalloc(&m->param_mem, param_bytes) != cudaSuccess) return fail();
    if (cudaMemset(m->param_mem, 0, param_bytes) != cudaSuccess) return fail();
    lay(static_cast<char *>(m->param_mem));
    for (int l = 0; l <= depth; l++) {
        Layer &ly = m->L[l];
        const size_t nw = (size_t)ly.out * ly.in;
        // uniform(-lim, lim), lim = sqrt(6 / fan_in) (He); only the real inputs
        // of the first layer count, padded columns start at zero
        const int fan_in = l == 0 ? n_in : ly.in;
        const double lim = sqrt(6.0 / fan_in) * (l == depth ? 0.5 : 1.0);
        std::vector<float> w(nw, 0.f);
        for (int r = 0; r < ly.out; r++)
            for (int c = 0; c < ly.in; c++) {
                const double u = (double)(splitmix(rs) >> 11) * (1.0 / 9007199254740992.0);
                w[(size_t)r * ly.in + c] = (l == 0 && c >= n_in) ? 0.f : (float)((2.0 * u - 1.0) * lim);
            }
        if (cudaMemcpy(ly.w, w.data(), nw * 4, cudaMemcpyHostToDevice) != cudaSuccess) return fail();
    }
    if (cudaMalloc(&m->step, sizeof(long long)) != cudaSuccess) return fail();
    if (cudaMemset(m->step, 0, sizeof(long long)) != cudaSuccess) return fail();
    if (cudaMalloc(&m->d_err, sizeof(int)) != cudaSuccess) return fail();
    if (cudaMemset(m->d_err, 0, sizeof(int)) != cudaSuccess) return fail();
    if (mlp_adam_segs(m) != 0) return fail();
    if (mlp_sync_bf16(m) != 0) return fail();
    if (cudaStreamSynchronize(m->st) != cudaSuccess) return fail();
    return m;
}

extern "C" size_t fdtd_b200_mlp_n_params(const fdtd_b200_mlp_t *m) {
    size_t n = 0;
    for (const Layer &ly : m->L) n += (size_t)ly.out * ly.in + ly.out;
    return n;
}

// Parameters in layer order: W (out x in, row-major, first layer with its
// zero-padded input columns), then b.
extern "C" int fdtd_b200_mlp_get_params(fdtd_b200_mlp_t *m, float *out) {
    MCK(cudaStreamSynchronize(m->st));
    size_t o = 0;
    for (const Layer &ly : m->L) {
        const size_t nw = (size_t)ly.out * ly.in;
        MCK(cudaMemcpy(out + o, ly.w, nw * 4, cudaMemcpyDeviceToHost));
        o += nw;
        MCK(cudaMemcpy(out + o, ly.b, ly.out * 4, cudaMemcpyDeviceToHost));
        o += ly.out;
    }
    return 0;
}

extern "C" int fdtd_b200_mlp_set_params(fdtd_b200_mlp_t *m, const float *in) {
    MCK(cudaStreamSynchronize(m->st));
    size_t o = 0;
    for (const Layer &ly : m->L) {
        const size_t nw = (size_t)ly.out * ly.in;
        MCK(cudaMemcpy(ly.w, in + o, nw * 4, cudaMemcpyHostToDevice));
        o += nw;
        MCK(cudaMemcpy(ly.b, in + o, ly.out * 4, cudaMemcpyHostToDevice));
        o += ly.out;
    }
    return mlp_sync_bf16(m);
}

// Reads the gradients of the last backward pass in parameter layout.
static int mlp_read_grads(fdtd_b200_mlp *m, float *out) {
    MCK(cudaStreamSynchronize(m->st));
    size_t o = 0;
    for (const Layer &ly : m->L) {
        const size_t nw = (size_t)ly.out * ly.in;
        MCK(cudaMemcpy(out + o, ly.gw, nw * 4, cudaMemcpyDeviceToHost));
        o += nw;
        MCK(cudaMemcpy(out + o, ly.gb, ly.out * 4, cudaMemcpyDeviceToHost));
        o += ly.out;
    }
    return 0;
}

// n rows of host X as BF16 rows [n][kin] in dst through the FP32 rows xf
// (queued on the main stream; X may be reused once the stream has passed).
static int mlp_upload_x(fdtd_b200_mlp *m, const float *X, size_t n, bf16 *dst, float *xf) {
    MCK(cudaMemcpyAsync(xf, X, n * m->n_in * sizeof(float), cudaMemcpyHostToDevice, m->st));
    const size_t tot = n * m->kin;
    k_pack_x<<<(unsigned)((tot + 255) / 256), 256, 0, m->st>>>(xf, m->n_in, dst, m->kin, n);
    m->launches++;
    MCK(cudaGetLastError());
    return 0;
}

// One forward + backward pass on the given batch (B a multiple of 64):
// loss = mean squared error, grads in parameter layout.
extern "C" int fdtd_b200_mlp_grad(fdtd_b200_mlp_t *m, const float *X, const float *Y, int B, double *loss,
                                  float *grads) {
    if (B < 64 || B % 64) {
        rfb_set_error("mlp: batch must be a positive multiple of 64");
        return -1;
    }
    if (mlp_batch_buffers(m, B) != 0) return -1;
    if (mlp_upload_x(m, X, B, m->act[0], m->xf) != 0) return -1;
    if (m->tc) {
        dim3 grid((m->kin + 31) / 32, (B + 31) / 32);
        k_transpose_bf16<<<grid, dim3(32, 8), 0, m->st>>>(m->act[0], B, m->kin, m->actt[0]);
    }
    MCK(cudaMemcpyAsync(m->y, Y, (size_t)B * m->n_out * 4, cudaMemcpyHostToDevice, m->st));
    mlp_forward(m, B, true);
    mlp_loss(m, B);
    if (mlp_backward(m, B) != 0) return -1;
    MCK(cudaGetLastError());
    std::vector<float> part((size_t)B * m->n_out / 256 + 1);
    const int nb = (B * m->n_out + 255) / 256;
    MCK(cudaMemcpyAsync(part.data(), m->partial, nb * 4, cudaMemcpyDeviceToHost, m->st));
    if (mlp_read_grads(m, grads) != 0) return -1;
    if (mlp_check_err(m) != 0) return -1;
    double se = 0;
    for (int q = 0; q < nb; q++) se += part[q];
    if (loss) *loss = se / ((double)B * m->n_out);
    return 0;
}

extern "C" int fdtd_b200_mlp_set_data(fdtd_b200_mlp_t *m, const float *X, const float *Y, size_t n) {
    MCK(cudaStreamSynchronize(m->st));
    cudaFree(m->X);
    cudaFree(m->Y);
    cudaFree(m->perm);
    m->X = nullptr;
    m->Y = nullptr;
    m->perm = nullptr;
    m->n_data = 0;
    if (n == 0) return 0;
    MCK(cudaMalloc(&m->X, n * m->kin * sizeof(bf16)));
    MCK(cudaMalloc(&m->Y, n * m->n_out * sizeof(float)));
    MCK(cudaMalloc(&m->perm, n * sizeof(int)));
    {
        // the whole data set's staging is not kept
        float *xf = nullptr;
        MCK(cudaMalloc(&xf, n * m->n_in * sizeof(float)));
        const int rc = mlp_upload_x(m, X, n, m->X, xf);
        const cudaError_t e = cudaStreamSynchronize(m->st);
        cudaFree(xf);
        if (rc != 0) return -1;
        MCK(e);
    }
    MCK(cudaMemcpy(m->Y, Y, n * m->n_out * sizeof(float), cudaMemcpyHostToDevice));
    m->n_data = n;
    mlp_free_graph(m);
    return 0;
}

static int mlp_train_step(fdtd_b200_mlp *m, int B) {
    launch_step(k_gather, dim3(B), dim3(128), 0, m->st, false, m->X, m->Y, m->perm, (long long)m->n_data,
                m->step, B, m->kin, m->n_out, m->act[0], m->actt[0], m->y);
    m->launches++;
    mlp_forward(m, B, true);
    mlp_loss(m, B);
    if (mlp_backward(m, B) != 0) return -1;
    mlp_adam(m);
    return 0;
}

// Captures a training step.  The graph holds the batch buffers and the data
// set, not the schedule (cfg, step), so it serves every later call.  A graph
// of eight steps cost 2 ms more on a network's first call (8 steps of 64 rows:
// 1.31 against 3.3 ms) and gave little back: 200 steps of 256 rows take 12.6
// against 13.0 ms, of 64 rows 10.7 against 10.4, 43 steps of 64 rows on two
// layers of 128 1.30 against 1.23.
static int mlp_capture(fdtd_b200_mlp *m, int B) {
    cudaGraph_t g = nullptr;
    MCK(cudaStreamBeginCapture(m->st, cudaStreamCaptureModeThreadLocal));
    m->overlap = !m->tc;
    const unsigned long long l0 = m->launches, t0 = m->tc_launches;
    const int rc = mlp_train_step(m, B);
    m->overlap = false;
    // counted as they are replayed
    m->graph_l = m->launches - l0;
    m->graph_tc = m->tc_launches - t0;
    m->launches = l0;
    m->tc_launches = t0;
    const cudaError_t ce = cudaStreamEndCapture(m->st, &g);
    if (rc != 0 || ce != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        MCK(ce);
        return -1;
    }
    const cudaError_t e = cudaGraphInstantiate(&m->graph, g, 0);
    cudaGraphDestroy(g);
    MCK(e);
    return 0;
}

// `steps` Adam steps of batch B over the resident data set, sampled through a
// permutation that is reshuffled (seeded) every pass over the data; the
// learning rate follows lr0 * 0.5 (1 + cos(pi s / steps)).  Each step is a
// CUDA graph replay.  *final_loss: mean squared error of the last batch.
extern "C" int fdtd_b200_mlp_train(fdtd_b200_mlp_t *m, size_t steps, int B, double lr, double beta1, double beta2,
                                   double eps, uint64_t shuffle_seed, double *final_loss) {
    if (!m->n_data) {
        rfb_set_error("mlp: no training data (fdtd_b200_mlp_set_data)");
        return -1;
    }
    if (B < 64 || B % 64) {
        rfb_set_error("mlp: batch must be a positive multiple of 64");
        return -1;
    }
    if (mlp_batch_buffers(m, B) != 0) return -1;
    MCK(cudaMemsetAsync(m->step, 0, sizeof(long long), m->st));
    const AdamCfg cfg = {(float)lr, (float)beta1, (float)beta2, (float)eps, (long long)steps};
    MCK(cudaMemcpyAsync(m->cfg, &cfg, sizeof cfg, cudaMemcpyHostToDevice, m->st));
    // first and second moments restart
    for (Layer &ly : m->L) {
        MCK(cudaMemsetAsync(ly.mw, 0, (size_t)ly.out * ly.in * 4, m->st));
        MCK(cudaMemsetAsync(ly.vw, 0, (size_t)ly.out * ly.in * 4, m->st));
        MCK(cudaMemsetAsync(ly.mb, 0, ly.out * 4, m->st));
        MCK(cudaMemsetAsync(ly.vb, 0, ly.out * 4, m->st));
    }
    if (m->graph_b != B) mlp_free_graph(m);
    m->graph_b = B;
    const size_t per_pass = std::max<size_t>(1, m->n_data / B);
    std::vector<int> perm(m->n_data);
    uint64_t rs = shuffle_seed;
    size_t done = 0;
    while (done < steps) {
        // permutation of this pass (Fisher-Yates on splitmix64), drawn while
        // the pass before runs; the copy to the device queues behind its steps
        for (size_t q = 0; q < m->n_data; q++) perm[q] = (int)q;
        for (size_t q = m->n_data - 1; q > 0; q--) std::swap(perm[q], perm[splitmix(rs) % (q + 1)]);
        MCK(cudaMemcpyAsync(m->perm, perm.data(), m->n_data * sizeof(int), cudaMemcpyHostToDevice, m->st));
        const size_t run = std::min(per_pass, steps - done);
        if (!m->graph && mlp_capture(m, B) != 0) return -1;
        for (size_t s = 0; s < run; s++) {
            MCK(cudaGraphLaunch(m->graph, m->st));
            m->launches += m->graph_l;
            m->tc_launches += m->graph_tc;
        }
        done += run;
    }
    MCK(cudaStreamSynchronize(m->st));
    if (final_loss) {
        const int nb = (B * m->n_out + 255) / 256;
        std::vector<float> part(nb);
        MCK(cudaMemcpy(part.data(), m->partial, nb * 4, cudaMemcpyDeviceToHost));
        double se = 0;
        for (float v : part) se += v;
        *final_loss = se / ((double)B * m->n_out);
    }
    return mlp_check_err(m);
}

// Network outputs of n inputs (any n; evaluated in batches of up to 1024
// rows, queued one behind the other).
extern "C" int fdtd_b200_mlp_predict(fdtd_b200_mlp_t *m, const float *X, size_t n, float *Y) {
    const int B = 1024;
    if (mlp_batch_buffers(m, B) != 0) return -1;
    for (size_t r0 = 0; r0 < n; r0 += B) {
        const size_t rows = std::min<size_t>(B, n - r0);
        // rows padded to the tensor-core tile height (zero rows)
        const int Bp = (int)((rows + tc::BM - 1) / tc::BM * tc::BM);
        if (mlp_upload_x(m, X + r0 * m->n_in, rows, m->act[0], m->xf) != 0) return -1;
        if ((size_t)Bp > rows)
            MCK(cudaMemsetAsync(m->act[0] + rows * m->kin, 0, (Bp - rows) * m->kin * sizeof(bf16), m->st));
        mlp_forward(m, Bp, false);
        MCK(cudaGetLastError());
        MCK(cudaMemcpyAsync(Y + r0 * m->n_out, m->out, rows * m->n_out * sizeof(float), cudaMemcpyDeviceToHost,
                            m->st));
    }
    MCK(cudaStreamSynchronize(m->st));
    return mlp_check_err(m);
}

extern "C" unsigned long long fdtd_b200_mlp_launch_count(const fdtd_b200_mlp_t *m) { return m->launches; }

extern "C" unsigned long long fdtd_b200_mlp_tensor_core_launches(const fdtd_b200_mlp_t *m) { return m->tc_launches; }
