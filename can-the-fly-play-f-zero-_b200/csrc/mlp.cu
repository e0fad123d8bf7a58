// Kernels of the learned surrogate (include/flysurrogate.h): a BF16 tensor-core GEMM with fused
// epilogues (bias, GELU, GELU gradient, transposed copies for the backward pass), the Poisson
// negative log-likelihood, column sums (bias gradients), Adam, and FP32 -> BF16 conversion.
//
// Every GEMM of the MLP's training step is written as C = A * B^T with both operands stored
// K-contiguous (the forward pass keeps transposed copies of activations and weights for the
// backward pass), so one kernel serves them all. Three forms: k_gemm_tma (the default: tcgen05
// MMAs, accumulator in TMEM, operands by TMA with the 128-byte swizzle), k_gemm_tc (the same with
// cp.async staging, for operands TMA cannot describe) and k_gemm (warp-level BF16 m16n8k16 MMAs
// on 128 x 64 tiles from padded shared memory, kept as the comparison).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include <cstdint>

#include "../../include/flybrain.h"
#include "../../include/flysurrogate.h"
#include "chain.cuh"

namespace fb {
void set_last_error(const char* msg);
}

namespace {

constexpr int BM = 128, BN = 64, BK = 32, PADK = BK + 8;

// The surrogate's kernels are launched as a chain (chain.cuh). Between ordinary launches the drain, the
// launch and the set-up of the next kernel were 1-2 us of every 4: a training step of 4,096 goes
// from 158 to 134 us with the chain, a screen of 1,024 inputs from 41.8 to 33.6 us.
using fb::launch_chain;
using fb::pdl_chain;

__device__ __forceinline__ uint16_t f2bf(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z)
{
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * expf(-0.5f * z * z) * 0.39894228040143268f;
}

// 8 consecutive bf16 of row `row` from column k (zero outside [0, rows) x [0, K))
__device__ __forceinline__ void load8(const uint16_t* X, int row, int k, int rows, int K, int ld, uint16_t* dst)
{
    if (row < rows && k + 8 <= K) {
        *reinterpret_cast<uint4*>(dst) = __ldg(reinterpret_cast<const uint4*>(X + (int64_t)row * ld + k));
    } else {
#pragma unroll
        for (int u = 0; u < 8; u++) dst[u] = (row < rows && k + u < K) ? X[(int64_t)row * ld + k + u] : (uint16_t)0;
    }
}

__device__ __forceinline__ uint32_t lds32(const uint16_t* p) { return *reinterpret_cast<const uint32_t*>(p); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

struct Epi {
    int32_t mode, ldo, ldo_t;
    const float* bias;
    const float* zin;
    float* out_f32;
    uint16_t* out_bf16;
    uint16_t* out_bf16_t;
};

__device__ __forceinline__ void epilogue(const Epi& e, int M, int N, int i, int j, float v)
{
    if (i >= M || j >= N) return;
    const int64_t o = (int64_t)i * e.ldo + j;
    switch (e.mode) {
    case FS_EPI_F32: e.out_f32[o] = v; break;
    case FS_EPI_BIAS_F32: e.out_f32[o] = v + e.bias[j]; break;
    case FS_EPI_BIAS_GELU: {
        const float z = v + e.bias[j];
        e.out_f32[o] = z;
        const uint16_t h = f2bf(gelu(z));
        e.out_bf16[o] = h;
        if (e.out_bf16_t) e.out_bf16_t[(int64_t)j * e.ldo_t + i] = h;
        break;
    }
    default: {   // FS_EPI_GELU_GRAD
        const uint16_t d = f2bf(v * gelu_grad(e.zin[o]));
        e.out_bf16[o] = d;
        if (e.out_bf16_t) e.out_bf16_t[(int64_t)j * e.ldo_t + i] = d;
    }
    }
}

// Whether rows of `p` (row stride ld elements of `size` bytes) start on 16-byte boundaries
__device__ __forceinline__ bool rows16(const void* p, int32_t ld, int size)
{
    return (((uintptr_t)p | ((uintptr_t)ld * (uintptr_t)size)) & 15) == 0;
}

// The epilogue of 16 consecutive columns j .. j + 15 of row i. A thread holds a whole run of a row, so the row
// outputs go out as 16-byte stores; one element at a time, every store of a warp touched 32 rows and
// moved 4 bytes of a 32-byte sector (4096 x 512 x 1280 with GELU and transpose: 58.5 us, now 18.9). The
// transposed output is contiguous over the warp's rows.
__device__ __forceinline__ void epilogue16(const Epi& e, int M, int N, int i, int j, const float (&v)[16])
{
    const bool f32 = e.mode != FS_EPI_GELU_GRAD, half = e.mode == FS_EPI_BIAS_GELU || e.mode == FS_EPI_GELU_GRAD;
    const bool whole = j + 16 <= N && (!f32 || rows16(e.out_f32, e.ldo, 4)) && (!half || rows16(e.out_bf16, e.ldo, 2)) &&
                       (e.mode != FS_EPI_GELU_GRAD || rows16(e.zin, e.ldo, 4));
    if (i >= M) return;
    if (!whole) {
#pragma unroll
        for (int u = 0; u < 16; u++) epilogue(e, M, N, i, j + u, v[u]);
        return;
    }
    const int64_t o = (int64_t)i * e.ldo + j;
    float z[16];
    if (e.mode == FS_EPI_GELU_GRAD) {
#pragma unroll
        for (int u = 0; u < 16; u += 4) {
            const float4 q = *reinterpret_cast<const float4*>(e.zin + o + u);
            z[u] = q.x; z[u + 1] = q.y; z[u + 2] = q.z; z[u + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int u = 0; u < 16; u++) z[u] = e.mode == FS_EPI_F32 ? v[u] : v[u] + e.bias[j + u];
#pragma unroll
        for (int u = 0; u < 16; u += 4) *reinterpret_cast<float4*>(e.out_f32 + o + u) = make_float4(z[u], z[u + 1], z[u + 2], z[u + 3]);
    }
    if (!half) return;
    uint16_t h[16];
#pragma unroll
    for (int u = 0; u < 16; u++) h[u] = f2bf(e.mode == FS_EPI_BIAS_GELU ? gelu(z[u]) : v[u] * gelu_grad(z[u]));
#pragma unroll
    for (int u = 0; u < 16; u += 8) {
        uint4 q;
        q.x = (uint32_t)h[u] | ((uint32_t)h[u + 1] << 16);
        q.y = (uint32_t)h[u + 2] | ((uint32_t)h[u + 3] << 16);
        q.z = (uint32_t)h[u + 4] | ((uint32_t)h[u + 5] << 16);
        q.w = (uint32_t)h[u + 6] | ((uint32_t)h[u + 7] << 16);
        *reinterpret_cast<uint4*>(e.out_bf16 + o + u) = q;
    }
    if (e.out_bf16_t) {
#pragma unroll
        for (int u = 0; u < 16; u++) e.out_bf16_t[(int64_t)(j + u) * e.ldo_t + i] = h[u];
    }
}

__global__ void __launch_bounds__(256) k_gemm(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B, int M,
                                              int N, int K, int lda, int ldb, Epi e)
{
    __shared__ __align__(16) uint16_t As[BM][PADK];
    __shared__ __align__(16) uint16_t Bs[BN][PADK];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int wm = warp & 3, wn = warp >> 2;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += BK) {
        for (int c = tid; c < BM * 4; c += 256) load8(A, m0 + (c >> 2), k0 + (c & 3) * 8, M, K, lda, &As[c >> 2][(c & 3) * 8]);
        for (int c = tid; c < BN * 4; c += 256) load8(B, n0 + (c >> 2), k0 + (c & 3) * 8, N, K, ldb, &Bs[c >> 2][(c & 3) * 8]);
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk += 16) {
            uint32_t a[2][4], b[4][2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int r = wm * 32 + i * 16 + g;
                a[i][0] = lds32(&As[r][kk + 2 * t4]);
                a[i][1] = lds32(&As[r + 8][kk + 2 * t4]);
                a[i][2] = lds32(&As[r][kk + 2 * t4 + 8]);
                a[i][3] = lds32(&As[r + 8][kk + 2 * t4 + 8]);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int c = wn * 32 + j * 8 + g;
                b[j][0] = lds32(&Bs[c][kk + 2 * t4]);
                b[j][1] = lds32(&Bs[c][kk + 2 * t4 + 8]);
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) mma_bf16(acc[i][j], a[i], b[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = m0 + wm * 32 + i * 16 + g, c = n0 + wn * 32 + j * 8 + 2 * t4;
            epilogue(e, M, N, r, c, acc[i][j][0]);
            epilogue(e, M, N, r, c + 1, acc[i][j][1]);
            epilogue(e, M, N, r + 8, c, acc[i][j][2]);
            epilogue(e, M, N, r + 8, c + 1, acc[i][j][3]);
        }
}

// ---------------------------------------------------------------------------------------------
// The same GEMM on the 5th-generation tensor cores: tcgen05.mma (kind::f16, BF16 in, FP32
// accumulate) issued by one thread, operands in shared memory in the K-major no-swizzle
// core-matrix layout (8 rows x 16 bytes per core matrix), the 128 x BN accumulator in tensor memory
// (TMEM), read back with tcgen05.ld for the fused epilogue. Four shared-memory stages filled by
// cp.async: later K tiles load while the tensor cores work on the current one (a stage is
// refilled once tcgen05.commit's mbarrier shows its MMAs done).
// ---------------------------------------------------------------------------------------------
constexpr int TC_BM = 128, TC_BK = 64, TC_THREADS = 128, TC_STAGES = 4;
constexpr long long TC_WAIT_CYCLES = 4000000000LL;            // bounded waits (~2 s)

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, no swizzle; lbo = byte distance between the two 8-column
// halves of a K=16 slice, sbo = byte distance between 8-row groups
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);   // version 1, base offset 0, no swizzle
}

__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity)
{
    const long long t0 = clock64();
    uint32_t done = 0;
    while (!done) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (!done && clock64() - t0 > TC_WAIT_CYCLES) return false;
    }
    return true;
}

// 16-byte global -> shared copy without a register round trip (zero-filled outside the matrix)
__device__ __forceinline__ void cp_async16(void* dst, const uint16_t* X, int row, int k, int rows, int K, int ld)
{
    if (row < rows && k + 8 <= K) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(su32(dst)), "l"(X + (int64_t)row * ld + k)
                     : "memory");
    } else {
        uint16_t tmp[8];
#pragma unroll
        for (int u = 0; u < 8; u++) tmp[u] = (row < rows && k + u < K) ? X[(int64_t)row * ld + k + u] : (uint16_t)0;
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(tmp);
    }
}

template <int BN>
__global__ void __launch_bounds__(TC_THREADS) k_gemm_tc(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B,
                                                         int M, int N, int K, int lda, int ldb, Epi e)
{
    constexpr int A_BYTES = TC_BM * TC_BK * 2, B_BYTES = BN * TC_BK * 2, STAGE = A_BYTES + B_BYTES;
    constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
    extern __shared__ __align__(1024) uint8_t sm[];
    __shared__ __align__(8) uint64_t mbar[TC_STAGES];
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * BN;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&s_tmem)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < TC_STAGES; s++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&mbar[s])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    // instruction descriptor: FP32 accumulate (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 = 1),
    // both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
    const int nk = (K + TC_BK - 1) / TC_BK;
    // one K tile -> stage st: 16-byte chunks (row r, k-chunk kc) in the core-matrix layout
    auto load_tile = [&](int kt) {
        uint8_t* sa = sm + (kt % TC_STAGES) * STAGE;
        uint8_t* sb = sa + A_BYTES;
        const int k0 = kt * TC_BK;
        for (int c = tid; c < TC_BM * 8; c += TC_THREADS) {
            const int r = c >> 3, kc = c & 7;
            cp_async16(sa + (kc * TC_BM + r) * 16, A, m0 + r, k0 + kc * 8, M, K, lda);
        }
        for (int c = tid; c < BN * 8; c += TC_THREADS) {
            const int r = c >> 3, kc = c & 7;
            cp_async16(sb + (kc * BN + r) * 16, B, n0 + r, k0 + kc * 8, N, K, ldb);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    bool ok = true;
    for (int kt = 0; kt < TC_STAGES - 1; kt++) {
        if (kt < nk) load_tile(kt);
        else asm volatile("cp.async.commit_group;" ::: "memory");        // keep the group count uniform
    }
    for (int kt = 0; kt < nk; kt++) {
        const int st = kt % TC_STAGES;
        asm volatile("cp.async.wait_group %0;" ::"n"(TC_STAGES - 2) : "memory");   // tile kt has landed
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // generic writes -> tensor-core reads
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint8_t* sa = sm + st * STAGE;
            uint8_t* sb = sa + A_BYTES;
#pragma unroll
            for (int kk = 0; kk < TC_BK / 16; kk++) {
                const uint64_t ad = smem_desc(su32(sa) + kk * 2 * TC_BM * 16, TC_BM * 16, 128);
                const uint64_t bd = smem_desc(su32(sb) + kk * 2 * BN * 16, BN * 16, 128);
                const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             su32(&mbar[st]))
                         : "memory");
        }
        // refill the stage the previous tile used once its MMAs are done
        const int nxt = kt + TC_STAGES - 1;
        if (nxt < nk) {
            if (kt >= 1) {
                const int ps = (kt - 1) % TC_STAGES;
                ok = tc_wait(su32(&mbar[ps]), (uint32_t)(((kt - 1) / TC_STAGES) & 1)) && ok;
            }
            load_tile(nxt);
        } else {
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // the last commit covers every MMA issued before it
    ok = tc_wait(su32(&mbar[(nk - 1) % TC_STAGES]), (uint32_t)(((nk - 1) / TC_STAGES) & 1)) && ok;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // epilogue: warp w holds rows 32w..32w+31 (TMEM lanes), 16 columns per load
    const int row = m0 + warp * 32 + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 16) {
        uint32_t v[16];
        const uint32_t addr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(addr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (ok) {
#pragma unroll
            for (int j = 0; j < 16; j++) epilogue(e, M, N, row, n0 + c0 + j, __uint_as_float(v[j]));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// ---------------------------------------------------------------------------------------------
// The tcgen05 GEMM fed by the Tensor Memory Accelerator: one thread issues each K tile of A (128 rows)
// and B (BN rows) as two 2-D TMA loads (64 bf16 = 128 bytes of K per row, 128-byte swizzle, zeros
// outside the matrices) into a ring of TMA_STAGES shared-memory stages; one thread issues the
// tensor-core MMAs from swizzled K-major descriptors as each stage lands and releases the stage with
// tcgen05.commit; all eight warps then read the accumulator from TMEM for the epilogue. No cluster
// multicast anywhere. Every wait is bounded; after a timeout no result is written.
//
// Split K (gridDim.z = S > 1, launched as clusters of 1 x 1 x S blocks): block z of a cluster
// accumulates K tiles [z * nk / S, (z + 1) * nk / S) of the same output tile, writes its FP32
// partial to its own shared memory (the drained stage ring), and after a cluster barrier each block
// sums its 1/S share of the tile's rows over the S partials in the order z = 0 .. S-1 through
// distributed shared memory (ld.shared::cluster, 16 bytes a thread along a row: 512 x 1280 x 4096 in
// 16.8 us, element by element 24.8, down the columns 41), then applies the epilogue. The sum order is
// fixed, so a result depends on S and never on scheduling. A second cluster barrier keeps every block's
// shared memory alive until all reads end.
// ---------------------------------------------------------------------------------------------
constexpr int TMA_STAGES = 4;
constexpr int TMA_THREADS = 256;             // two warps per 32 TMEM lanes: each takes half of a tile's columns (the
                                             // same GEMM with one warp per 32 lanes: 20.9 us)
constexpr int MAX_SPLIT = 8;                 // portable cluster size

// generic-proxy accesses of shared memory after (or before) the tensor-core / TMA proxy's
__device__ __forceinline__ void fence_async_to_generic() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the shared-memory address `local` of this block, as seen in block `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t local, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ int ld_cluster_s32(uint32_t addr)
{
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// shared-memory descriptor, K-major with the 128-byte swizzle: 8-row atoms of 1024 bytes (SBO), the
// K offset inside the 128-byte row added to the start address (LBO unused: 16 bytes)
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFF) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t mbar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(mbar)
        : "memory");
}

template <int BN>
__global__ void __launch_bounds__(TMA_THREADS) k_gemm_tma(const __grid_constant__ CUtensorMap mapA,
                                                          const __grid_constant__ CUtensorMap mapB, int M, int N, int K,
                                                          Epi e)
{
    constexpr int A_BYTES = TC_BM * 128, B_BYTES = BN * 128, STAGE = A_BYTES + B_BYTES;
    static_assert(A_BYTES % 1024 == 0 && B_BYTES % 1024 == 0, "stages must keep 1024-byte alignment");
    constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
    extern __shared__ uint8_t dyn[];
    __shared__ __align__(8) uint64_t full[TMA_STAGES], empty[TMA_STAGES], done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_ok, s_issued, s_used;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * BN;
    const uint32_t base = (su32(dyn) + 1023u) & ~1023u;            // the swizzle needs 1024-byte atoms
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&s_tmem)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < TMA_STAGES; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&full[s])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&empty[s])) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&done)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_ok = 1;
        s_issued = 0;
        s_used = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    pdl_chain();                                      // (barriers and TMEM are set up beside the predecessor)
    const uint32_t tmem = s_tmem;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
    // this block's K tiles: all of them, or its share of a split (every share has at least one)
    const int S = (int)gridDim.z, z = S > 1 ? (int)cluster_rank() : 0;
    const int nk_all = (K + 63) / 64, kt0 = (int)((int64_t)z * nk_all / S);
    const int nk = (int)((int64_t)(z + 1) * nk_all / S) - kt0;
    if (tid == 0) {                                   // producer: the TMA loads
        int kt = 0;
        for (; kt < nk; kt++) {
            const int s = kt % TMA_STAGES;
            if (kt >= TMA_STAGES && !tc_wait(su32(&empty[s]), (uint32_t)((kt / TMA_STAGES - 1) & 1))) {
                s_ok = 0;
                break;
            }
            const uint32_t sa = base + s * STAGE;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(&full[s])), "r"(STAGE)
                         : "memory");
            tma_load_2d(sa, &mapA, (kt0 + kt) * 64, m0, su32(&full[s]));
            tma_load_2d(sa + A_BYTES, &mapB, (kt0 + kt) * 64, n0, su32(&full[s]));
        }
        s_issued = kt;
    } else if (tid == 32) {                           // the MMA issuer
        int kt = 0;
        for (; kt < nk; kt++) {
            const int s = kt % TMA_STAGES;
            if (!tc_wait(su32(&full[s]), (uint32_t)((kt / TMA_STAGES) & 1))) {
                s_ok = 0;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = base + s * STAGE, sb = sa + A_BYTES;
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {              // K = 16 per MMA: 32 bytes along the swizzled row
                const uint64_t ad = smem_desc_sw128(sa + kk * 32), bd = smem_desc_sw128(sb + kk * 32);
                const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                    ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             su32(&empty[s]))
                         : "memory");
        }
        s_used = kt;
        // the last commit covers every MMA issued before it
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(&done))
                     : "memory");
    }
    const bool fin = tc_wait(su32(&done), 0u);
    // loads still in flight after a timeout land before the stage ring is reused or the block
    // leaves (bounded)
    if (tid == 0)
        for (int kt = s_used; kt < s_issued; kt++) (void)tc_wait(su32(&full[kt % TMA_STAGES]), (uint32_t)((kt / TMA_STAGES) & 1));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    const bool ok = fin && s_ok != 0;
    const int trow = (warp & 3) * 32 + lane;          // this thread's row of the tile (its warp's TMEM lanes)
    constexpr int PSTR = BN + 4;                      // partial rows padded: eight lanes' 16 bytes hit all banks
    float* part = reinterpret_cast<float*>(dyn + (base - su32(dyn)));
    if (S > 1) fence_async_to_generic();
    constexpr int HALF = BN >= 32 ? BN / 2 : BN;
    const int c_first = (warp >> 2) * HALF;
#pragma unroll 1
    for (int c0 = c_first; c0 < min(BN, c_first + HALF); c0 += 16) {
        uint32_t v[16];
        const uint32_t addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(addr));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (S > 1) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
                *reinterpret_cast<float4*>(part + trow * PSTR + c0 + j) =
                    make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
        } else if (ok) {
            float f[16];
#pragma unroll
            for (int j = 0; j < 16; j++) f[j] = __uint_as_float(v[j]);
            epilogue16(e, M, N, m0 + trow, n0 + c0, f);
        }
    }
    if (S > 1) {
        if (tid == 0) s_ok = ok ? 1 : 0;
        cluster_sync_all();                           // every partial is written and visible
        bool all_ok = true;
        for (int r = 0; r < S; r++) all_ok = all_ok && ld_cluster_s32(map_rank(su32(&s_ok), (uint32_t)r)) != 0;
        // this block's share of the tile's rows, four columns per thread and consecutive threads on consecutive
        // columns (remote shared memory is read in whole lines); plain outputs go out as they are summed, the
        // others pass through this block's own partial to the unsplit epilogue's rows
        const int r_lo = z * TC_BM / S, r_hi = (z + 1) * TC_BM / S;
        const bool plain = e.mode == FS_EPI_F32 || e.mode == FS_EPI_BIAS_F32;
        const bool wide = plain && rows16(e.out_f32, e.ldo, 4);
        const uint32_t pbase = su32(part);
        for (int q4 = tid; q4 < (r_hi - r_lo) * (BN / 4); q4 += TMA_THREADS) {
            const int r = r_lo + q4 / (BN / 4), c = q4 % (BN / 4) * 4;
            const uint32_t off = pbase + (uint32_t)(r * PSTR + c) * 4u;
            float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
            for (int q = 0; q < S; q++) {
                const float4 x = ld_cluster_f32x4(map_rank(off, (uint32_t)q));
                acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
            }
            const int i = m0 + r, j = n0 + c;
            if (!plain) {
                *reinterpret_cast<float4*>(part + r * PSTR + c) = acc;
            } else if (all_ok && wide && i < M && j + 4 <= N) {
                if (e.mode == FS_EPI_BIAS_F32) {
                    acc.x += e.bias[j]; acc.y += e.bias[j + 1]; acc.z += e.bias[j + 2]; acc.w += e.bias[j + 3];
                }
                *reinterpret_cast<float4*>(e.out_f32 + (int64_t)i * e.ldo + j) = acc;
            } else if (all_ok) {
                epilogue(e, M, N, i, j, acc.x);
                epilogue(e, M, N, i, j + 1, acc.y);
                epilogue(e, M, N, i, j + 2, acc.z);
                epilogue(e, M, N, i, j + 3, acc.w);
            }
        }
        if (!plain) {
            __syncthreads();
            for (int run = tid; run < (r_hi - r_lo) * (BN / 16); run += TMA_THREADS) {
                const int r = r_lo + run % (r_hi - r_lo), c = run / (r_hi - r_lo) * 16;
                float acc[16];
#pragma unroll
                for (int u = 0; u < 16; u += 4) {
                    const float4 x = *reinterpret_cast<const float4*>(part + r * PSTR + c + u);
                    acc[u] = x.x; acc[u + 1] = x.y; acc[u + 2] = x.z; acc[u + 3] = x.w;
                }
                if (all_ok) epilogue16(e, M, N, m0 + r, n0 + c, acc);
            }
        }
        cluster_sync_all();                           // no block leaves while another reads its partial
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

__global__ void k_poisson(const float* z, const float* y, int M, int D, double* loss, uint16_t* dz, int ldd, uint16_t* dz_t)
{
    pdl_chain();
    __shared__ double part[8];
    double s = 0.0;
    const int64_t total = (int64_t)M * D;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < total; p += (int64_t)gridDim.x * blockDim.x) {
        const float zz = z[p], yy = y[p];
        const float ez = expf(zz);
        s += (double)ez - (double)yy * (double)zz;
        const uint16_t d = f2bf((ez - yy) / (float)M);
        const int64_t m = p / D, k = p - m * D;
        dz[m * ldd + k] = d;
        if (dz_t) dz_t[k * M + m] = d;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += part[w];
        atomicAdd(loss, t);
    }
}

// Column sums of several matrices in one launch: a cluster of S blocks per 32 columns of one of them, block z
// of it over rows [z M / S, (z + 1) M / S) with its 32 warps on interleaved rows (lanes on consecutive
// columns); the warps' partials, then the blocks' (through distributed shared memory), added in a fixed
// order. The bias gradients of the three layers: 5.6 us each on their own.
struct ColsumList {
    struct { const uint16_t* x; float* grad; int32_t n, ld, first; } m[FS_LIST_MAX];    // first: its first block of columns
    int32_t count, rows;
};
__global__ void __launch_bounds__(1024) k_colsum(const ColsumList L)
{
    pdl_chain();
    __shared__ float part[32][33];
    __shared__ float tot[32];
    int which = 0;
#pragma unroll
    for (int i = 1; i < FS_LIST_MAX; i++)
        if (i < L.count && (int)blockIdx.x >= L.m[i].first) which = i;
    const uint16_t* X = L.m[which].x;
    const int N = L.m[which].n, ld = L.m[which].ld, M = L.rows;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, j = ((int)blockIdx.x - L.m[which].first) * 32 + lane;
    const int S = (int)gridDim.y, z = S > 1 ? (int)cluster_rank() : 0;
    const int r0 = (int)((int64_t)z * M / S), r1 = (int)((int64_t)(z + 1) * M / S);
    float s = 0.0f;
    if (j < N) {
#pragma unroll 8
        for (int i = r0 + w; i < r1; i += 32) s += __bfloat162float(__ushort_as_bfloat16(X[(int64_t)i * ld + j]));
    }
    part[w][lane] = s;
    __syncthreads();
    if (w == 0) {
        float t = 0.0f;
        for (int q = 0; q < 32; q++) t += part[q][lane];
        tot[lane] = t;
    }
    if (S > 1) cluster_sync_all();
    else __syncthreads();
    if (z == 0 && w == 0 && j < N) {
        float t = 0.0f;
        for (int q = 0; q < S; q++) t += S > 1 ? ld_cluster_f32(map_rank(su32(&tot[lane]), (uint32_t)q)) : tot[lane];
        L.m[which].grad[j] = t;
    }
    if (S > 1) cluster_sync_all();                    // no block leaves while block 0 reads its sums
}

// Adam on one element (weight, gradient, moments; the moments and the weight updated); returns the new weight
__device__ __forceinline__ float adam_one(float& w, float gg, float& m, float& v, float lr, float b1, float b2, float eps,
                                          float c1, float c2)
{
    const float mm = b1 * m + (1.0f - b1) * gg;
    const float vv = b2 * v + (1.0f - b2) * gg * gg;
    m = mm;
    v = vv;
    w = w - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    return w;
}

// Adam on several parameters in one launch, in 32 x 32 tiles (block 32 x 8) of each rows x cols parameter (a
// run of elements: rows of 1,024); a weight's transposed bf16 copy is written through shared memory so that both copies
// are stored along rows. Six launches of 2 - 6 us each on their own.
struct AdamList {
    struct { float *w, *m, *v; const float* g; uint16_t *wb, *wbt; int64_t n; int32_t rows, cols, ldt, first, across; } p[FS_LIST_MAX];
    int32_t count;
};
__global__ void __launch_bounds__(256) k_adam(const AdamList A, float lr, float b1, float b2, float eps, float c1, float c2)
{
    pdl_chain();
    __shared__ uint16_t tile[32][34];
    int which = 0;
#pragma unroll
    for (int i = 1; i < FS_LIST_MAX; i++)
        if (i < A.count && (int)blockIdx.x >= A.p[i].first) which = i;
    const auto& P = A.p[which];
    const int t = (int)blockIdx.x - P.first;
    const int64_t c0 = (int64_t)(t % P.across) * 32, r0 = (int64_t)(t / P.across) * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    float w[4], g[4], m[4], v[4];                      // four rows per thread, their loads in flight together
    bool in[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int64_t r = r0 + ty + 8 * u, c = c0 + tx, p = r * P.cols + c;
        in[u] = r < P.rows && c < P.cols && p < P.n;   // (a run's last row may be short)
        if (in[u]) {
            w[u] = P.w[p];
            g[u] = P.g[p];
            m[u] = P.m[p];
            v[u] = P.v[p];
        }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (!in[u]) continue;
        const int64_t p = (r0 + ty + 8 * u) * P.cols + c0 + tx;
        const uint16_t h = f2bf(adam_one(w[u], g[u], m[u], v[u], lr, b1, b2, eps, c1, c2));
        P.w[p] = w[u];
        P.m[p] = m[u];
        P.v[p] = v[u];
        if (P.wb) P.wb[p] = h;
        tile[ty + 8 * u][tx] = h;
    }
    if (!P.wbt) return;                                // (the same for the whole block)
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
        const int64_t c = c0 + k, r = r0 + tx;
        if (r < P.rows && c < P.cols) P.wbt[c * P.ldt + r] = tile[tx][k];
    }
}

__global__ void k_to_bf16(const float* x, int64_t n, uint16_t* out)
{
    pdl_chain();
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
        out[p] = f2bf(x[p]);
}

// FP32 -> bf16 of a rows x cols matrix in 32 x 32 tiles (block 32 x 8): the plain copy (when `out`)
// and the transposed one, both stored along rows
__global__ void k_to_bf16_t(const float* x, uint16_t* out, uint16_t* out_t, int rows, int cols, int ldt)
{
    pdl_chain();
    __shared__ uint16_t tile[32][34];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32, tx = threadIdx.x, ty = threadIdx.y;
    for (int k = ty; k < 32; k += 8) {
        const int r = r0 + k, c = c0 + tx;
        if (r < rows && c < cols) {
            const int64_t p = (int64_t)r * cols + c;
            const uint16_t h = f2bf(x[p]);
            if (out) out[p] = h;
            tile[k][tx] = h;
        }
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
        const int c = c0 + k, r = r0 + tx;
        if (r < rows && c < cols) out_t[(int64_t)c * ldt + r] = tile[tx][k];
    }
}

// The same in 64 x 64 tiles with 16-byte loads and 8-byte stores of both copies (block 256; cols and ldt
// multiples of 4, every base aligned): 4096 x 1280 in 9 us, element by element 18.6. Bound by memory.
__global__ void __launch_bounds__(256) k_to_bf16_t4(const float* x, uint16_t* out, uint16_t* out_t, int rows, int cols, int ldt)
{
    pdl_chain();
    __shared__ __align__(8) uint16_t tile[64][64 + 4]; // [column][row], read four rows (8 bytes) at a time
    const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64, lane = threadIdx.x & 15, w = threadIdx.x >> 4;
    float4 q[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int r = r0 + w + 16 * u, c = c0 + 4 * lane;
        q[u] = r < rows && c < cols ? *reinterpret_cast<const float4*>(x + (int64_t)r * cols + c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int k = w + 16 * u, r = r0 + k, c = c0 + 4 * lane;
        const uint16_t h[4] = {f2bf(q[u].x), f2bf(q[u].y), f2bf(q[u].z), f2bf(q[u].w)};
        if (out && r < rows && c < cols)
            *reinterpret_cast<uint2*>(out + (int64_t)r * cols + c) =
                make_uint2((uint32_t)h[0] | ((uint32_t)h[1] << 16), (uint32_t)h[2] | ((uint32_t)h[3] << 16));
#pragma unroll
        for (int i = 0; i < 4; i++) tile[4 * lane + i][k] = h[i];
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int k = w + 16 * u, c = c0 + k, r = r0 + 4 * lane;
        if (c >= cols) continue;
        uint16_t* to = out_t + (int64_t)c * ldt + r;
        if (r + 4 <= rows) {
            *reinterpret_cast<uint2*>(to) = *reinterpret_cast<const uint2*>(&tile[k][4 * lane]);
        } else {
            for (int i = 0; i < 4 && r + i < rows; i++) to[i] = tile[k][4 * lane + i];
        }
    }
}

int g_gemm_kind = FS_GEMM_TCGEN05_TMA;

int fail(const char* msg)
{
    fb::set_last_error(msg);
    return FB_ERR_ARG;
}

int cuda_status()
{
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return FB_OK;
    fb::set_last_error(cudaGetErrorString(e));
    return FB_ERR_CUDA;
}

template <int BN>
int launch_tc(const uint16_t* A, const uint16_t* B, int M, int N, int K, int lda, int ldb, const Epi& e, cudaStream_t st)
{
    constexpr int smem = TC_STAGES * (TC_BM * TC_BK * 2 + BN * TC_BK * 2);
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_gemm_tc<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return cuda_status();
        attr = true;
    }
    dim3 grid((N + BN - 1) / BN, (M + TC_BM - 1) / TC_BM);
    k_gemm_tc<BN><<<grid, TC_THREADS, smem, st>>>(A, B, M, N, K, lda, ldb, e);
    return cuda_status();
}

// A K-contiguous bf16 matrix (rows x K, row stride ld) as a TMA tensor map: boxes of 64 x box_rows
// elements with the 128-byte swizzle. False when the driver entry point is missing or rejects it.
bool tensor_map(CUtensorMap* map, const uint16_t* X, int rows, int K, int ld, int box_rows)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", (void**)&encode, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            encode = nullptr;
        (void)cudaGetLastError();
    }
    if (!encode || ((uintptr_t)X & 15) || ld % 8) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(X), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int g_gemm_split = MAX_SPLIT;

// K split of a TMA GEMM: enough blocks to fill the SMs at `per_sm` blocks each (the kernel's
// shared-memory occupancy), at least eight 64-deep K tiles per block (below that the cluster
// reduction costs more than the split saves), at most the set limit
int split_for(int tiles, int K, int per_sm)
{
    if (g_gemm_split <= 1) return 1;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
        (void)cudaGetLastError();
        sms = 148;
    }
    const int nk = (K + 63) / 64;
    return std::max(1, std::min({g_gemm_split, (per_sm * sms) / std::max(tiles, 1), nk / 8}));
}

// 1: launched; 0: not eligible for TMA (the caller falls back); negative: an error code
template <int BN>
int launch_tma(const uint16_t* A, const uint16_t* B, int M, int N, int K, int lda, int ldb, const Epi& e, cudaStream_t st)
{
    CUtensorMap ma, mb;
    if (!tensor_map(&ma, A, M, K, lda, TC_BM) || !tensor_map(&mb, B, N, K, ldb, BN)) return 0;
    constexpr int smem = TMA_STAGES * (TC_BM * 128 + BN * 128) + 1024;
    static_assert(TC_BM * (BN + 4) * 4 <= TMA_STAGES * (TC_BM * 128 + BN * 128), "split-K partials fit the stage ring");
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_gemm_tma<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return -cuda_status();
        attr = true;
    }
    const unsigned gx = (N + BN - 1) / BN, gy = (M + TC_BM - 1) / TC_BM;
    const int S = split_for((int)(gx * gy), K, smem * 2 <= 227 * 1024 ? 2 : 1);
    if (launch_chain(k_gemm_tma<BN>, dim3(gx, gy, (unsigned)S), dim3(TMA_THREADS), smem, st, 1u, (unsigned)S, ma, mb, M, N, K, e) !=
        cudaSuccess)
        return -cuda_status();
    const int rc = cuda_status();
    return rc == FB_OK ? 1 : -rc;
}

unsigned blocks_for(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16)); }

}  // namespace

extern "C" int fs_gemm(const uint16_t* A, const uint16_t* B, int32_t M, int32_t N, int32_t K, int32_t lda, int32_t ldb,
                       int32_t epi, const float* bias, const float* zin, float* out_f32, uint16_t* out_bf16,
                       uint16_t* out_bf16_t, int32_t ldo, int32_t ldo_t, void* stream)
{
    if (!A || !B || M <= 0 || N <= 0 || K <= 0) return fail("fs_gemm: bad operands");
    if (lda % 8 || ldb % 8 || lda < K || ldb < K) return fail("fs_gemm: lda, ldb must be multiples of 8 and >= K");
    if (epi < FS_EPI_F32 || epi > FS_EPI_GELU_GRAD) return fail("fs_gemm: unknown epilogue");
    if ((epi == FS_EPI_F32 || epi == FS_EPI_BIAS_F32 || epi == FS_EPI_BIAS_GELU) && !out_f32)
        return fail("fs_gemm: out_f32 needed");
    if ((epi == FS_EPI_BIAS_F32 || epi == FS_EPI_BIAS_GELU) && !bias) return fail("fs_gemm: bias needed");
    if ((epi == FS_EPI_BIAS_GELU || epi == FS_EPI_GELU_GRAD) && !out_bf16) return fail("fs_gemm: out_bf16 needed");
    if (epi == FS_EPI_GELU_GRAD && !zin) return fail("fs_gemm: zin needed");
    Epi e{epi, ldo, ldo_t, bias, zin, out_f32, out_bf16, out_bf16_t};
    cudaStream_t st = (cudaStream_t)stream;
    if (g_gemm_kind == FS_GEMM_TCGEN05_TMA) {
        const int rc = N <= 16 ? launch_tma<16>(A, B, M, N, K, lda, ldb, e, st) : launch_tma<64>(A, B, M, N, K, lda, ldb, e, st);
        if (rc != 0) return rc > 0 ? FB_OK : -rc;
    }
    if (g_gemm_kind == FS_GEMM_TCGEN05 || g_gemm_kind == FS_GEMM_TCGEN05_TMA) {
        if (N <= 16) return launch_tc<16>(A, B, M, N, K, lda, ldb, e, st);
        return launch_tc<64>(A, B, M, N, K, lda, ldb, e, st);
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    k_gemm<<<grid, 256, 0, st>>>(A, B, M, N, K, lda, ldb, e);
    return cuda_status();
}

extern "C" int fs_gemm_kind(int32_t kind)
{
    if (kind != FS_GEMM_MMA_SYNC && kind != FS_GEMM_TCGEN05 && kind != FS_GEMM_TCGEN05_TMA && kind != -1)
        return fail("fs_gemm_kind: unknown kind");
    const int old = g_gemm_kind;
    if (kind >= 0) g_gemm_kind = kind;
    return old;
}

extern "C" int fs_gemm_split(int32_t max_split)
{
    if (max_split == 0 || max_split < -1 || max_split > MAX_SPLIT) return -fail("fs_gemm_split: 1 .. 8, or -1 to keep");
    const int old = g_gemm_split;
    if (max_split > 0) g_gemm_split = max_split;
    return old;
}

extern "C" int fs_poisson_nll(const float* z, const float* y, int32_t M, int32_t D, double* loss_sum, uint16_t* dz,
                              int32_t ldd, uint16_t* dz_t, void* stream)
{
    if (!z || !y || !loss_sum || !dz || M <= 0 || D <= 0 || ldd < D) return fail("fs_poisson_nll: bad arguments");
    launch_chain(k_poisson, blocks_for((int64_t)M * D), 256, 0, (cudaStream_t)stream, 1, 1, z, y, M, D, loss_sum, dz, ldd, dz_t);
    return cuda_status();
}

extern "C" int fs_colsum_list(const fs_colsum_item* items, int32_t count, int32_t M, void* stream)
{
    if (!items || count <= 0 || count > FS_LIST_MAX || M <= 0) return fail("fs_colsum: bad arguments");
    ColsumList L{};
    L.count = count;
    L.rows = M;
    int blocks = 0;
    for (int i = 0; i < count; i++) {
        const fs_colsum_item& it = items[i];
        if (!it.X || !it.grad || it.N <= 0 || it.ld < it.N) return fail("fs_colsum: bad arguments");
        L.m[i].x = it.X; L.m[i].grad = it.grad; L.m[i].n = it.N; L.m[i].ld = it.ld; L.m[i].first = blocks;
        blocks += (it.N + 31) / 32;
    }
    const int S = std::min(MAX_SPLIT, std::max(1, M / 256));    // >= 8 rows per warp
    launch_chain(k_colsum, dim3((unsigned)blocks, (unsigned)S), dim3(1024), 0, (cudaStream_t)stream, (unsigned)S, 1, L);
    return cuda_status();
}

extern "C" int fs_colsum(const uint16_t* X, int32_t M, int32_t N, int32_t ld, float* grad, void* stream)
{
    const fs_colsum_item it{X, grad, N, ld};
    return fs_colsum_list(&it, 1, M, stream);
}

extern "C" int fs_adam_list(const fs_adam_item* items, int32_t count, float lr, float beta1, float beta2, float eps, int32_t t,
                            void* stream)
{
    if (!items || count <= 0 || count > FS_LIST_MAX || t < 1) return fail("fs_adam: bad arguments");
    AdamList A{};
    A.count = count;
    int64_t blocks = 0;
    for (int i = 0; i < count; i++) {
        const fs_adam_item& it = items[i];
        if (!it.w || !it.grad || !it.m || !it.v || it.n <= 0) return fail("fs_adam: bad arguments");
        if (it.w_bf16_t && (it.rows <= 0 || it.cols <= 0 || it.rows > 65535 * 32 || (int64_t)it.rows * it.cols != it.n || it.ldt < it.rows))
            return fail("fs_adam: the transposed copy needs 0 < rows <= 2097120, rows * cols == n and ldt >= rows");
        auto& p = A.p[i];
        p.w = it.w; p.m = it.m; p.v = it.v; p.g = it.grad; p.wb = it.w_bf16; p.wbt = it.w_bf16_t;
        p.n = it.n;
        if ((it.n + 1023) / 1024 > INT32_MAX) return fail("fs_adam: too many elements");
        p.cols = it.w_bf16_t ? it.cols : (int32_t)std::min<int64_t>(it.n, 1024);
        p.rows = it.w_bf16_t ? it.rows : (int32_t)((it.n + p.cols - 1) / p.cols);
        p.ldt = it.ldt;
        p.across = (p.cols + 31) / 32;
        p.first = (int32_t)blocks;
        blocks += (int64_t)p.across * ((p.rows + 31) / 32);
        if (blocks > INT32_MAX) return fail("fs_adam: too many elements");
    }
    const float c1 = 1.0f - powf(beta1, (float)t), c2 = 1.0f - powf(beta2, (float)t);
    launch_chain(k_adam, dim3((unsigned)blocks), dim3(32, 8), 0, (cudaStream_t)stream, 1, 1, A, lr, beta1, beta2, eps, c1, c2);
    return cuda_status();
}

extern "C" int fs_adam(float* w, const float* grad, float* m, float* v, int64_t n, float lr, float beta1, float beta2,
                       float eps, int32_t t, uint16_t* w_bf16, uint16_t* w_bf16_t, int32_t rows, int32_t cols,
                       int32_t ldt, void* stream)
{
    const fs_adam_item it{w, grad, m, v, w_bf16, w_bf16_t, n, rows, cols, ldt};
    return fs_adam_list(&it, 1, lr, beta1, beta2, eps, t, stream);
}

extern "C" int fs_to_bf16(const float* x, int64_t n, uint16_t* out, uint16_t* out_t, int32_t rows, int32_t cols,
                          int32_t ldt, void* stream)
{
    if (!x || n <= 0 || (!out && !out_t)) return fail("fs_to_bf16: bad arguments");
    if (out_t && (rows <= 0 || cols <= 0 || rows > 65535 * 32 || (int64_t)rows * cols != n || ldt < rows))
        return fail("fs_to_bf16: the transposed copy needs 0 < rows <= 2097120, rows * cols == n and ldt >= rows");
    if (out_t && cols % 4 == 0 && ldt % 4 == 0 && (((uintptr_t)x & 15) | ((uintptr_t)out & 7) | ((uintptr_t)out_t & 7)) == 0) {
        const dim3 grid((unsigned)((cols + 63) / 64), (unsigned)((rows + 63) / 64));
        launch_chain(k_to_bf16_t4, grid, dim3(256), 0, (cudaStream_t)stream, 1, 1, x, out, out_t, rows, cols, ldt);
    } else if (out_t) {
        const dim3 grid((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32));
        launch_chain(k_to_bf16_t, grid, dim3(32, 8), 0, (cudaStream_t)stream, 1, 1, x, out, out_t, rows, cols, ldt);
    } else {
        launch_chain(k_to_bf16, blocks_for(n), 256, 0, (cudaStream_t)stream, 1, 1, x, n, out);
    }
    return cuda_status();
}
