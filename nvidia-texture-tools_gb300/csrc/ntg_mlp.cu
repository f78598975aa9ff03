// The learned endpoint proposal's network on the 5th-generation tensor cores: an MLP
// 48 -> 256 -> 256 -> 8 (GELU, tanh form; BF16 weights and activations, FP32 accumulation) trained
// with Adam.
// Inputs are a block's 16 texels x RGB; outputs 0-5 are the two endpoints of the block's cluster
// fit, output 6 the fit's log-error (used to decide when the pruned search falls back to the full
// one), output 7 is unused. No counterpart in the reference.
//
// Training runs in two kernels: k_mlp_train takes a tile of 128 rows forward and back through all layers
// (weights in shared memory, accumulators in TMEM), and k_mlp_grads multiplies what it left in memory into the weight
// gradients. Inference is k_mlp_infer. The unfused forward pass and ntg_gemm_bf16 use a plain product,
// k_gemm: D[M x N] = A[M x K] * B[N x K]^T with both operands K-major BF16, staged by the CTA's threads into shared memory in the canonical no-swizzle layout
// (8-row x 16-byte core matrices), multiplied by tcgen05.mma (kind::f16, M = 128) issued by one
// thread into a TMEM accumulator, double-buffered with an mbarrier per stage that the MMA's
// tcgen05.commit arrives on. The epilogue reads the accumulator back with tcgen05.ld (thread t owns
// row t) and applies bias + GELU. Every wait is bounded (a poll count the
// host sets per network, ntg_mlp_set_wait_limit): on timeout the kernel records an error, waits (with
// the default limit) for the tensor-core work it has already issued, frees its TMEM and returns.
#include <cuda_bf16.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <random>
#include <string>
#include <vector>

#include "ntg.h"
#include "ntg_async.cuh"
#include "ntg_internal.h"

namespace ntg {
namespace mlp {

constexpr int IN = 48, HID = 256, OUT = 8, OUTP = 16;  // OUTP: output rows padded for the MMA's N
constexpr int BM = 128, BK = 64;                       // CTA tile rows, K chunk
constexpr uint32_t LBO = 128, SBO = 1024;              // K-direction and row-group core-matrix strides

enum Epi { EPI_F32 = 0, EPI_GELU = 1 };

struct GemmArgs {
    const __nv_bfloat16 *A;  // [M x K], row stride lda (elements)
    const __nv_bfloat16 *B;  // [N x K], row stride ldb
    int lda, ldb, M, N, K;
    int epi;
    const float *bias;       // [N] or null
    float *C;                // fp32 [M x N] (ldc), or null
    int ldc;
    __nv_bfloat16 *H;        // bf16 [M x N] (ldh), or null
    int ldh;
    int *status;             // set to a non-zero code when a wait gives up
    int polls;               // polls of each wait before it gives up
};

// ---- PTX wrappers (tcgen05, mbarrier) ----

// Shared-memory matrix descriptor: start address, leading (K) and stride (row-group) byte offsets,
// the fixed 0b001 field at bits 46-48, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t sbo = SBO) {
    uint64_t d = (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)((LBO >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, N and M.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Polls of a wait by default, and of the drain after a wait gave up: the MMAs already issued
// still write the TMEM accumulator, so they must finish before it is freed.
constexpr int kWaitPolls = 1 << 22;

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// The same without the wait, into raw registers, and the wait that makes them valid (it names them, so that no use moves
// above it): several loads in flight.
__device__ __forceinline__ void tmem_ld16_start(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16_finish(uint32_t (&r)[16], float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// GELU in its tanh form (Hendrycks & Gimpel, "Gaussian Error Linear Units", 2016):
// gelu(z) = z / 2 (1 + tanh(sqrt(2 / pi) (z + 0.044715 z^3))), with the hardware tanh
// (tanh.approx.f32, about 2^-11 relative error, below the BF16 rounding of the activations), and its
// derivative for training. The network is defined with this activation, in training, inference and
// the oracle alike.
__device__ __forceinline__ float tanh_hw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
constexpr float GELU_S = 0.7978845608028654f;  // sqrt(2 / pi)
constexpr float GELU_C = 0.044715f;
__device__ __forceinline__ float gelu(float z) {
    const float t = tanh_hw(GELU_S * (z + GELU_C * (z * z * z)));
    return 0.5f * z * (1.0f + t);
}
__device__ __forceinline__ float gelu_grad(float z) {
    const float z2 = z * z;
    const float t = tanh_hw(GELU_S * (z + GELU_C * (z2 * z)));
    return 0.5f * (1.0f + t) + 0.5f * z * (1.0f - t * t) * GELU_S * (1.0f + 3.0f * GELU_C * z2);
}

// Copies rows [r0, r0 + rows) x K-chunk [k0, k0 + BK) of a K-major matrix into the canonical
// layout at `dst` (rows beyond `nrows` or columns beyond K read as zero).
__device__ __forceinline__ void stage_tile(uint8_t *dst, const __nv_bfloat16 *src, int ld, int r0, int nrows, int rows,
                                           int k0, int K) {
    const int pieces = rows * (BK / 8);  // 16-byte pieces
    for (int p = threadIdx.x; p < pieces; p += blockDim.x) {
        const int rr = p & 7, kc = (p >> 3) & 7, rg = p >> 6;  // row in core matrix, K chunk, row group
        const int r = rg * 8 + rr, k = k0 + kc * 8;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r0 + r < nrows && k < K) v = *reinterpret_cast<const uint4 *>(src + (size_t)(r0 + r) * ld + k);
        *reinterpret_cast<uint4 *>(dst + rg * SBO + kc * LBO + rr * 16) = v;
    }
}

template <int BN>
__global__ void __launch_bounds__(128) k_gemm(GemmArgs g) {
    constexpr int TMEM_COLS = BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
    constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2;
    constexpr uint32_t IDESC = idesc_bf16(BM, BN);
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bars[3];
    __shared__ uint32_t tmem_base;
    uint8_t *a_st[2] = {smem, smem + A_BYTES + B_BYTES};
    uint8_t *b_st[2] = {smem + A_BYTES, smem + 2 * A_BYTES + B_BYTES};
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int chunks = (g.K + BK - 1) / BK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == 0) tmem_alloc(&tmem_base, TMEM_COLS);
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_init(&bars[2], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    int committed = -1;  // last chunk whose MMAs were issued and committed

    for (int c = 0; c < chunks && ok; c++) {
        const int s = c & 1;
        if (c >= 2) {  // the MMAs of chunk c-2 read this stage; the CTA agrees on the outcome
            ok = __syncthreads_and(mbar_wait(&bars[s], ((c - 2) >> 1) & 1, g.polls)) != 0;
            if (!ok) break;
        }
        const int k0 = c * BK;
        stage_tile(a_st[s], g.A, g.lda, m0, g.M, BM, k0, g.K);
        stage_tile(b_st[s], g.B, g.ldb, n0, g.N, BN, k0, g.K);
        fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(a_st[s]), b0 = smem_u32(b_st[s]);
#pragma unroll
            for (int j = 0; j < BK / 16; j++)
                mma_bf16(tmem, smem_desc(a0 + j * 2 * LBO), smem_desc(b0 + j * 2 * LBO), IDESC, (c > 0 || j > 0) ? 1u : 0u);
            mma_commit(&bars[s]);
        }
        committed = c;
    }
    // all MMAs done: the last chunk's commit completes after every earlier one
    if (ok && chunks > 0) ok = __syncthreads_and(mbar_wait(&bars[(chunks - 1) & 1], ((chunks - 1) >> 1) & 1, g.polls)) != 0;
    if (!ok) {
        if (g.status && threadIdx.x == 0) atomicExch(g.status, 1);
        // drain: the last commit's barrier completes once every MMA issued so far has finished
        if (committed >= 0) __syncthreads_and(mbar_wait(&bars[committed & 1], (committed >> 1) & 1, kWaitPolls));
    }
    tc_fence_after();

    if (ok) {
        const int row = warp * 32 + lane, m = m0 + row;
        const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            float v[16];
            if (chunks > 0) tmem_ld16(lane_addr + c0, v);
            else
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = 0.0f;
            if (m >= g.M) continue;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int n = n0 + c0 + i;
                if (n >= g.N) break;
                float x = v[i];
                if (g.bias) x += g.bias[n];
                if (g.C) g.C[(size_t)m * g.ldc + n] = x;
                if (g.H) g.H[(size_t)m * g.ldh + n] = __float2bfloat16_rn(g.epi == EPI_GELU ? gelu(x) : x);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, TMEM_COLS);
}

size_t gemm_smem(int bn) { return 2 * (size_t)(BM * BK * 2 + bn * BK * 2) + 1024; }

template <int BN>
int launch_gemm_t(const GemmArgs &g, cudaStream_t s) {
    static std::atomic<unsigned long long> configured{0};
    const size_t sm = gemm_smem(BN);
    if (first_use_on_device(configured)) cudaFuncSetAttribute(k_gemm<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    dim3 grid((g.M + BM - 1) / BM, (g.N + BN - 1) / BN);
    k_gemm<BN><<<grid, 128, sm, s>>>(g);
    return launch_status();
}

// Picks the N tile (16, 48, 64 or 256 columns) for the product's N.
int launch_gemm(const GemmArgs &g, cudaStream_t s) {
    if (g.K % 8 || g.lda % 8 || g.ldb % 8) return NTG_ERROR_INVALID_INPUT;
    if (g.N <= 16) return launch_gemm_t<16>(g, s);
    if (g.N <= 48) return launch_gemm_t<48>(g, s);
    if (g.N <= 64) return launch_gemm_t<64>(g, s);
    return launch_gemm_t<256>(g, s);
}

// ---- elementwise kernels ----

// fp32 -> bf16
__global__ void k_to_bf16(const float *__restrict__ x, long long n, __nv_bfloat16 *__restrict__ y) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = __float2bfloat16_rn(x[i]);
}

// Parameter layout (flat fp32): W1 [HID x IN], b1 [HID], W2 [HID x HID], b2 [HID], W3 [OUT x HID], b3 [OUT].
constexpr size_t OFF_W1 = 0, OFF_B1 = OFF_W1 + (size_t)HID * IN, OFF_W2 = OFF_B1 + HID, OFF_B2 = OFF_W2 + (size_t)HID * HID,
                 OFF_W3 = OFF_B2 + HID, OFF_B3 = OFF_W3 + (size_t)OUT * HID, NPARAM = OFF_B3 + OUT;

__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       int n, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// BF16 operand copies of the weights: W1 [HID x IN], W2 [HID x HID], W2^T, W3 padded [OUTP x HID],
// W3^T [HID x OUTP]; biases as fp32 (b3 padded to OUTP).
__global__ void k_refresh(const float *__restrict__ p, __nv_bfloat16 *__restrict__ w1, __nv_bfloat16 *__restrict__ w2,
                          __nv_bfloat16 *__restrict__ w2t, __nv_bfloat16 *__restrict__ w3, __nv_bfloat16 *__restrict__ w3t,
                          float *__restrict__ b3p) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < HID * HID; i += gridDim.x * blockDim.x) {
        const int r = i / HID, c = i % HID;
        const __nv_bfloat16 b = __float2bfloat16_rn(p[OFF_W2 + i]);
        w2[i] = b;
        w2t[(size_t)c * HID + r] = b;
        if (i < HID * IN) w1[i] = __float2bfloat16_rn(p[OFF_W1 + i]);
        if (i < OUTP * HID) {
            const int o = i / HID, j = i % HID;
            const __nv_bfloat16 q = o < OUT ? __float2bfloat16_rn(p[OFF_W3 + (size_t)o * HID + j]) : __float2bfloat16_rn(0.0f);
            w3[i] = q;
            w3t[(size_t)j * OUTP + o] = q;
        }
        if (i < OUTP) b3p[i] = i < OUT ? p[OFF_B3 + i] : 0.0f;
    }
}

// ---- fused inference: the whole network per 128-row tile, on one CTA per SM ----
// The weights stay in shared memory for the kernel's lifetime (canonical layout, whole K per
// operand: row group stride = K / 8 x 128 bytes); a tile's activations go X -> TMEM -> GELU -> the
// same shared-memory operand buffer -> TMEM -> ... so nothing but x and y touches global memory.
// TMEM: layer 1 in columns [0, 256), layer 2 in [256, 512), layer 3 in [0, 16).
constexpr uint32_t SBO_IN = IN / 8 * 128, SBO_HID = HID / 8 * 128;
constexpr size_t F_W1 = 0, F_W2 = F_W1 + (size_t)HID * IN * 2, F_W3 = F_W2 + (size_t)HID * HID * 2,
                 F_ACT = F_W3 + (size_t)OUTP * HID * 2, F_BIAS = F_ACT + (size_t)BM * HID * 2,
                 F_BYTES = F_BIAS + (size_t)(HID + HID + OUTP) * 4;

// Writes 8 bf16 (16 bytes) at row r, K chunk kc of a canonical operand with row-group stride sbo.
__device__ __forceinline__ void put8(uint8_t *base, uint32_t sbo, int r, int kc, uint4 v) {
    *reinterpret_cast<uint4 *>(base + (r >> 3) * sbo + kc * LBO + (r & 7) * 16) = v;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Copies a bf16 row-major [rows x K] matrix from global memory into the canonical layout; eight consecutive threads
// write the eight rows of a core matrix (one 128-byte run: no bank conflicts), the next eight its neighbour along K.
__device__ void load_operand(uint8_t *dst, const __nv_bfloat16 *src, int rows, int K) {
    const int chunks = K / 8;
    for (int p = threadIdx.x; p < rows * chunks; p += blockDim.x) {
        const int g = p >> 3, kc = g % chunks, r = (g / chunks) * 8 + (p & 7);
        put8(dst, (uint32_t)chunks * LBO, r, kc, *reinterpret_cast<const uint4 *>(src + (size_t)r * K + kc * 8));
    }
}

// The same, asynchronously (cp.async, generic proxy): complete after async_wait<later groups> and a barrier.
__device__ __forceinline__ void load_operand_async(uint8_t *dst, const __nv_bfloat16 *src, int rows, int K) {
    const int chunks = K / 8;
    for (int p = threadIdx.x; p < rows * chunks; p += blockDim.x) {
        const int g = p >> 3, kc = g % chunks, r = (g / chunks) * 8 + (p & 7);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + (r >> 3) * (uint32_t)chunks * LBO + kc * LBO + (r & 7) * 16)),
                     "l"(src + (size_t)r * K + kc * 8)
                     : "memory");
    }
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LATER>
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LATER) : "memory"); }

// Bias + GELU of this thread's quarter (64 columns from c_begin) of its row's accumulator, into its
// row of the activation operand.
__device__ __forceinline__ void hidden_epilogue(uint32_t lane_addr, const float *bias, uint8_t *act, int row, int c_begin) {
#pragma unroll 1
    for (int c0 = c_begin; c0 < c_begin + HID / 4; c0 += 16) {
        float v[16];
        tmem_ld16(lane_addr + c0, v);
        uint32_t p[8];
#pragma unroll
        for (int i = 0; i < 8; i++) p[i] = pack_bf16(gelu(v[2 * i] + bias[c0 + 2 * i]), gelu(v[2 * i + 1] + bias[c0 + 2 * i + 1]));
        put8(act, SBO_HID, row, c0 / 8, make_uint4(p[0], p[1], p[2], p[3]));
        put8(act, SBO_HID, row, c0 / 8 + 1, make_uint4(p[4], p[5], p[6], p[7]));
    }
}

__global__ void __launch_bounds__(512, 1) k_mlp_infer(const __nv_bfloat16 *__restrict__ w1, const __nv_bfloat16 *__restrict__ w2,
                                                       const __nv_bfloat16 *__restrict__ w3, const float *__restrict__ b1,
                                                       const float *__restrict__ b2, const float *__restrict__ b3,
                                                       const float *__restrict__ x, long long rows, float *__restrict__ y,
                                                       int *status, int polls) {
    extern __shared__ __align__(16) uint8_t smem[];  // 226 KB of the 227 KB a CTA may have
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_base;
    uint8_t *sw1 = smem + F_W1, *sw2 = smem + F_W2, *sw3 = smem + F_W3, *act = smem + F_ACT;
    float *sb = reinterpret_cast<float *>(smem + F_BIAS);
    // 16 warps: thread t owns row t % 128 (TMEM lane: warp t / 32 reads lane quarter (t / 32) % 4) and
    // quarter t / 128 of its columns
    const int warp = threadIdx.x >> 5, row = threadIdx.x & 127, quarter = threadIdx.x >> 7;
    if (warp == 0) tmem_alloc(&tmem_base, 512);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    load_operand(sw1, w1, HID, IN);
    load_operand(sw2, w2, HID, HID);
    load_operand(sw3, w3, OUTP, HID);
    for (int i = threadIdx.x; i < HID; i += blockDim.x) { sb[i] = b1[i]; sb[HID + i] = b2[i]; }
    if (threadIdx.x < OUTP) sb[2 * HID + threadIdx.x] = b3[threadIdx.x];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base, lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t a_act = smem_u32(act), a_w1 = smem_u32(sw1), a_w2 = smem_u32(sw2), a_w3 = smem_u32(sw3);
    uint32_t phase = 0;
    bool ok = true;
    const long long tiles = (rows + BM - 1) / BM;
    // X of the next tile is loaded into registers while the current tile is in the tensor cores and
    // the epilogues (quarters 0 and 1: half a row each, rows past the end are zero)
    constexpr int XC = IN / 16;  // 8-element chunks per half row
    float4 xr[2 * XC];
    auto load_x = [&](long long tile) {
        const long long r = tile * BM + row;
#pragma unroll
        for (int k = 0; k < XC; k++) {
            const int kc = quarter * XC + k;
            xr[2 * k] = xr[2 * k + 1] = make_float4(0, 0, 0, 0);
            if (quarter < 2 && tile < tiles && r < rows) {
                xr[2 * k] = *reinterpret_cast<const float4 *>(x + r * IN + kc * 8);
                xr[2 * k + 1] = *reinterpret_cast<const float4 *>(x + r * IN + kc * 8 + 4);
            }
        }
    };
    load_x(blockIdx.x);
    for (long long tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const long long r = tile * BM + row;
        if (quarter < 2) {
#pragma unroll
            for (int k = 0; k < XC; k++) {
                const float4 a = xr[2 * k], b = xr[2 * k + 1];
                put8(act, SBO_IN, row, quarter * XC + k,
                     make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w)));
            }
        }
#pragma unroll 1
        for (int layer = 0; layer < 3 && ok; layer++) {
            fence_async_smem();
            tc_fence_before();
            __syncthreads();
            if (threadIdx.x == 0) {
                tc_fence_after();
                if (layer == 0) {
#pragma unroll
                    for (int j = 0; j < IN / 16; j++)
                        mma_bf16(tmem, smem_desc(a_act + j * 2 * LBO, SBO_IN), smem_desc(a_w1 + j * 2 * LBO, SBO_IN),
                                 idesc_bf16(BM, HID), j > 0);
                } else if (layer == 1) {
#pragma unroll 4
                    for (int j = 0; j < HID / 16; j++)
                        mma_bf16(tmem + HID, smem_desc(a_act + j * 2 * LBO, SBO_HID), smem_desc(a_w2 + j * 2 * LBO, SBO_HID),
                                 idesc_bf16(BM, HID), j > 0);
                } else {
#pragma unroll 4
                    for (int j = 0; j < HID / 16; j++)
                        mma_bf16(tmem, smem_desc(a_act + j * 2 * LBO, SBO_HID), smem_desc(a_w3 + j * 2 * LBO, SBO_HID),
                                 idesc_bf16(BM, OUTP), j > 0);
                }
                mma_commit(&bar);
            }
            ok = __syncthreads_and(mbar_wait(&bar, phase & 1, polls)) != 0;
            // gave up: drain this layer's MMAs (they write the accumulator) before TMEM is freed
            if (!ok) __syncthreads_and(mbar_wait(&bar, phase & 1, kWaitPolls));
            phase++;
            tc_fence_after();
            if (!ok) break;
            if (layer == 0) load_x(tile + gridDim.x);  // layer 1 has read this tile's X
            if (layer < 2) {
                hidden_epilogue(lane_addr + (layer == 0 ? 0u : (uint32_t)HID), sb + layer * HID, act, row, quarter * (HID / 4));
            } else if (quarter == 0) {
                float v[16];
                tmem_ld16(lane_addr, v);
                if (r < rows) {
                    float4 *o = reinterpret_cast<float4 *>(y + r * OUTP);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        o[q] = make_float4(v[4 * q] + sb[2 * HID + 4 * q], v[4 * q + 1] + sb[2 * HID + 4 * q + 1],
                                           v[4 * q + 2] + sb[2 * HID + 4 * q + 2], v[4 * q + 3] + sb[2 * HID + 4 * q + 3]);
                }
            }
        }
    }
    if (!ok && status && threadIdx.x == 0) atomicExch(status, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---- training: forward and backward of a 128-row tile in one kernel ----
// The layers run as in k_mlp_infer, and back: Y -> dY -> dZ2 -> dZ1, with Z2 kept in TMEM (columns [256, 512)) for its
// GELU', Z1 as FP32 in global memory (the TMEM columns of layer 1 are needed again), and the W2^T operand
// loaded over W2 once layer 2 is done. What the weight gradients need goes to memory row-major in BF16, once;
// bias gradients and the loss are summed in FP32 and added up with atomics. Bound by the four epilogues of 128 x 256
// (tanh, conversions, shared-memory stores) on the batch's tiles, one CTA each, four warps a scheduler: 54 us at
// batch 8192, and 18 for k_mlp_grads, where forward and backward as nine products, each writing its results element
// by element and in two layouts, with their column sums and conversions took 840.
struct TrainArgs {
    const __nv_bfloat16 *w1, *w2, *w2t, *w3, *w3t;
    const float *b1, *b2, *b3, *wout, *x, *t;
    int batch;
    float *z1;                                 // [batch x HID]
    __nv_bfloat16 *h1, *h2, *dz1, *dz2, *dyb;  // [batch x HID], dyb [batch x OUTP]
    float *g, *loss;
    int *status;
    int polls;
    bool aligned;  // x lies on a 16-byte boundary
};
constexpr size_t T_DY = F_W1, T_W3T = T_DY + (size_t)BM * OUTP * 2, T_DB = T_W3T + (size_t)HID * OUTP * 2;  // over W1
static_assert(T_DB + 2 * HID * 4 <= F_W2, "the operands that replace W1 fit its place");

// Sums over the warp's 32 lanes of 16 values each: lane l gets the sum of value (l >> 1).
__device__ __forceinline__ float warp_sum16(float (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8; n >= 1; n >>= 1) {  // lanes 2n apart exchange halves of what they still hold
        const bool up = (lane & (2 * n)) != 0;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float keep = up ? v[n + i] : v[i], send = up ? v[i] : v[n + i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// 16 values as BF16: into the activation operand (when act is given) and 32 bytes of a row in global memory.
__device__ __forceinline__ void put_bf16(const float (&v)[16], uint8_t *act, int row, int c0, __nv_bfloat16 *dst, bool live) {
    uint32_t p[8];
#pragma unroll
    for (int i = 0; i < 8; i++) p[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
    const uint4 lo = make_uint4(p[0], p[1], p[2], p[3]), hi = make_uint4(p[4], p[5], p[6], p[7]);
    if (act) {
        put8(act, SBO_HID, row, c0 / 8, lo);
        put8(act, SBO_HID, row, c0 / 8 + 1, hi);
    }
    if (live) {
        reinterpret_cast<uint4 *>(dst)[0] = lo;
        reinterpret_cast<uint4 *>(dst)[1] = hi;
    }
}

__global__ void __launch_bounds__(512, 1) k_mlp_train(TrainArgs g) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t bar;
    __shared__ uint32_t tmem_base;
    uint8_t *const act = smem + F_ACT, *const dyop = smem + T_DY;
    float *const sb = reinterpret_cast<float *>(smem + F_BIAS), *const db = reinterpret_cast<float *>(smem + T_DB);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = threadIdx.x & 127, quarter = threadIdx.x >> 7;
    if (warp == 0) tmem_alloc(&tmem_base, 512);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < HID; i += blockDim.x) { sb[i] = g.b1[i]; sb[HID + i] = g.b2[i]; }
    if (threadIdx.x < OUTP) sb[2 * HID + threadIdx.x] = g.b3[threadIdx.x];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base, lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t a_act = smem_u32(act), a_w1 = smem_u32(smem + F_W1), a_w2 = smem_u32(smem + F_W2), a_w3 = smem_u32(smem + F_W3);
    const uint32_t a_dy = smem_u32(dyop), a_w3t = smem_u32(smem + T_W3T);
    constexpr uint32_t SBO_OUT = OUTP / 8 * 128;
    uint32_t phase = 0;
    bool ok = true;
    // acc[128 x N] = A * B^T over `steps` 16-element steps of K; every thread returns once it is in TMEM
    auto product = [&](uint32_t acc, uint32_t a, uint32_t a_sbo, uint32_t b, uint32_t b_sbo, int steps, uint32_t idesc) {
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");  // the epilogue's last load ahead
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
            for (int j = 0; j < steps; j++) mma_bf16(acc, smem_desc(a + j * 2 * LBO, a_sbo), smem_desc(b + j * 2 * LBO, b_sbo), idesc, j > 0);
            mma_commit(&bar);
        }
        ok = __syncthreads_and(mbar_wait(&bar, phase & 1, g.polls)) != 0;
        // gave up: drain the MMAs (they write the accumulator) before TMEM is freed
        if (!ok) __syncthreads_and(mbar_wait(&bar, phase & 1, kWaitPolls));
        phase++;
        tc_fence_after();
        return ok;
    };
    const int tiles = (g.batch + BM - 1) / BM, c_begin = quarter * (HID / 4);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int r = tile * BM + row;
        const bool live = r < g.batch;
        const size_t rh = (size_t)r * HID;
        load_operand_async(smem + F_W1, g.w1, HID, IN);
        async_commit();
        load_operand_async(smem + F_W2, g.w2, HID, HID);
        load_operand_async(smem + F_W3, g.w3, OUTP, HID);
        async_commit();
        if (quarter < 2) {
#pragma unroll
            for (int k = 0; k < IN / 16; k++) {
                const int kc = quarter * (IN / 16) + k;
                float4 a = make_float4(0, 0, 0, 0), b = a;
                const float *const p = g.x + (size_t)r * IN + kc * 8;
                if (live && g.aligned) {
                    a = *reinterpret_cast<const float4 *>(p);
                    b = *reinterpret_cast<const float4 *>(p + 4);
                } else if (live) {
                    a = make_float4(p[0], p[1], p[2], p[3]);
                    b = make_float4(p[4], p[5], p[6], p[7]);
                }
                put8(act, SBO_IN, row, kc, make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w)));
            }
        }
        async_wait<1>();
        if (!product(tmem, a_act, SBO_IN, a_w1, SBO_IN, IN / 16, idesc_bf16(BM, HID))) break;
        // Z1 -> H1; in each epilogue the next 16 columns are on their way while these are worked on
        uint32_t raw[16];
        tmem_ld16_start(lane_addr + c_begin, raw);
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_begin + HID / 4; c0 += 16) {
            float v[16];
            tmem_ld16_finish(raw, v);
            tmem_ld16_start(lane_addr + (c0 + 16 < c_begin + HID / 4 ? c0 + 16 : c0), raw);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] += sb[c0 + i];
            if (live)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    reinterpret_cast<float4 *>(g.z1 + rh + c0)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = gelu(v[i]);
            put_bf16(v, act, row, c0, g.h1 + rh + c0, live);
        }
        // W1 is done with: its place takes W3^T and the bias sums (dY follows)
        async_wait<0>();
        load_operand_async(smem + T_W3T, g.w3t, HID, OUTP);
        for (int i = threadIdx.x; i < 2 * HID; i += blockDim.x) db[i] = 0.0f;
        if (!product(tmem + HID, a_act, SBO_HID, a_w2, SBO_HID, HID / 16, idesc_bf16(BM, HID))) break;
        load_operand_async(smem + F_W2, g.w2t, HID, HID);  // beside the epilogue
        async_commit();
        // Z2 -> H2
        tmem_ld16_start(lane_addr + HID + c_begin, raw);
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_begin + HID / 4; c0 += 16) {
            float v[16];
            tmem_ld16_finish(raw, v);
            tmem_ld16_start(lane_addr + HID + (c0 + 16 < c_begin + HID / 4 ? c0 + 16 : c0), raw);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = gelu(v[i] + sb[HID + c0 + i]);
            put_bf16(v, act, row, c0, g.h2 + rh + c0, live);
        }
        if (!product(tmem, a_act, SBO_HID, a_w3, SBO_HID, HID / 16, idesc_bf16(BM, OUTP))) break;
        // Y -> loss, dY = 2 w (Y - T) / (batch OUT)
        if (quarter == 0) {
            float v[16], part = 0.0f;
            tmem_ld16(lane_addr, v);
#pragma unroll
            for (int c = 0; c < 16; c++) {
                float d = 0.0f;
                if (c < OUT && live) {
                    const float e = v[c] + sb[2 * HID + c] - g.t[(size_t)r * OUT + c];
                    const float w = g.wout[c] / (float)(g.batch * OUT);
                    part += w * e * e;
                    d = 2.0f * w * e;
                }
                v[c] = d;
            }
            const uint4 lo = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
            const uint4 zero = make_uint4(0, 0, 0, 0);
            put8(dyop, SBO_OUT, row, 0, lo);
            put8(dyop, SBO_OUT, row, 1, zero);
            if (live) {
                reinterpret_cast<uint4 *>(g.dyb + (size_t)r * OUTP)[0] = lo;
                reinterpret_cast<uint4 *>(g.dyb + (size_t)r * OUTP)[1] = zero;
            }
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            if (lane == 0) atomicAdd(g.loss, part);
            const float s = warp_sum16(v);
            if ((lane & 1) == 0 && (lane >> 1) < OUT) atomicAdd(g.g + OFF_B3 + (lane >> 1), s);
        }
        async_wait<0>();
        if (!product(tmem, a_dy, SBO_OUT, a_w3t, SBO_OUT, 1, idesc_bf16(BM, HID))) break;
        // dZ2 = (dY W3) gelu'(Z2)
        uint32_t raw2[16];
        tmem_ld16_start(lane_addr + c_begin, raw);
        tmem_ld16_start(lane_addr + HID + c_begin, raw2);
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_begin + HID / 4; c0 += 16) {
            float v[16], z[16];
            tmem_ld16_finish(raw, v);
            tmem_ld16_finish(raw2, z);
            const int next = c0 + 16 < c_begin + HID / 4 ? c0 + 16 : c0;
            tmem_ld16_start(lane_addr + next, raw);
            tmem_ld16_start(lane_addr + HID + next, raw2);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = live ? v[i] * gelu_grad(z[i] + sb[HID + c0 + i]) : 0.0f;
            put_bf16(v, act, row, c0, g.dz2 + rh + c0, live);
            const float s = warp_sum16(v);
            if ((lane & 1) == 0) atomicAdd(&db[HID + c0 + (lane >> 1)], s);
        }
        if (!product(tmem, a_act, SBO_HID, a_w2, SBO_HID, HID / 16, idesc_bf16(BM, HID))) break;
        // dZ1 = (dZ2 W2) gelu'(Z1)
        float4 ahead[4];
        auto fetch_z1 = [&](int c) {
#pragma unroll
            for (int i = 0; i < 4; i++) ahead[i] = live ? reinterpret_cast<const float4 *>(g.z1 + rh + c)[i] : make_float4(0, 0, 0, 0);
        };
        fetch_z1(c_begin);
        tmem_ld16_start(lane_addr + c_begin, raw);
#pragma unroll 1
        for (int c0 = c_begin; c0 < c_begin + HID / 4; c0 += 16) {
            float v[16], z[16];
            tmem_ld16_finish(raw, v);
#pragma unroll
            for (int i = 0; i < 4; i++) { z[4 * i] = ahead[i].x; z[4 * i + 1] = ahead[i].y; z[4 * i + 2] = ahead[i].z; z[4 * i + 3] = ahead[i].w; }
            const int next = c0 + 16 < c_begin + HID / 4 ? c0 + 16 : c0;
            tmem_ld16_start(lane_addr + next, raw);
            fetch_z1(next);
#pragma unroll
            for (int i = 0; i < 16; i++) v[i] = live ? v[i] * gelu_grad(z[i]) : 0.0f;
            put_bf16(v, nullptr, row, c0, g.dz1 + rh + c0, live);
            const float s = warp_sum16(v);
            if ((lane & 1) == 0) atomicAdd(&db[c0 + (lane >> 1)], s);
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        __syncthreads();
        if (threadIdx.x < HID) {
            atomicAdd(g.g + OFF_B1 + threadIdx.x, db[threadIdx.x]);
            atomicAdd(g.g + OFF_B2 + threadIdx.x, db[HID + threadIdx.x]);
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }
    async_wait<0>();
    if (!ok && threadIdx.x == 0) atomicExch(g.status, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---- training: the weight gradients ----
// dW2 = dZ2^T H1, dW1 = dZ1^T X, dW3 = dY^T H2: products over the batch, split into runs of GRAD_K rows (blockIdx.x);
// blockIdx.y: dW2, dW1 and dW3^T, the upper and the lower 128 of their 256 rows. The operands lie row-major with the batch
// outermost, so staging turns them: a thread reads two columns of eight batch rows and writes them as two 16-byte
// runs along K. The sums go to the flat gradient with four-wide atomics.
// Bound by the latency of the staging loads: 18 us at batch 8192 with 512 threads a CTA, 25 with 256.
constexpr int GRAD_K = 256, GRAD_N = 256, GRAD_THREADS = 512;
constexpr size_t GRAD_STAGE = (size_t)(BM + GRAD_N) * BK * 2;

// Columns [c0, c0 + cols) of rows [k0, k0 + BK) (below `rows`) of a row-major matrix, as the K-major operand of `cols` rows.
template <int cols, typename T>
__device__ __forceinline__ void stage_turned(uint8_t *dst, const T *src, int ld, int c0, int k0, int rows) {
#pragma unroll 4
    for (int p = threadIdx.x; p < cols / 2 * (BK / 8); p += GRAD_THREADS) {
        const int c = 2 * (p % (cols / 2)), kc = p / (cols / 2);
        uint32_t v[8];  // columns c and c + 1 of eight rows
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int k = k0 + kc * 8 + i;
            v[i] = 0;
            if (k < rows) {
                if constexpr (sizeof(T) == 2) {
                    v[i] = *reinterpret_cast<const uint32_t *>(src + (size_t)k * ld + c0 + c);
                } else {
                    const float *const p = src + (size_t)k * ld + c0 + c;
                    v[i] = pack_bf16(p[0], p[1]);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = c + h;
            const unsigned sel = h ? 0x7632u : 0x5410u;
            *reinterpret_cast<uint4 *>(dst + (m >> 3) * SBO + kc * LBO + (m & 7) * 16) =
                make_uint4(__byte_perm(v[0], v[1], sel), __byte_perm(v[2], v[3], sel), __byte_perm(v[4], v[5], sel), __byte_perm(v[6], v[7], sel));
        }
    }
}

__global__ void __launch_bounds__(GRAD_THREADS, 2) k_mlp_grads(TrainArgs g) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tmem_base;
    const int job = blockIdx.y >> 1, m0 = (blockIdx.y & 1) * BM;
    const int kbeg = blockIdx.x * GRAD_K, kend = min(g.batch, kbeg + GRAD_K), chunks = (kend - kbeg + BK - 1) / BK;
    const int n = job == 0 ? HID : (job == 1 ? IN : OUTP);
    const uint32_t idesc = job == 0 ? idesc_bf16(BM, HID) : (job == 1 ? idesc_bf16(BM, IN) : idesc_bf16(BM, OUTP));
    const __nv_bfloat16 *const a = job == 0 ? g.dz2 : (job == 1 ? g.dz1 : g.h2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) tmem_alloc(&tmem_base, GRAD_N);
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    bool ok = true;
    int committed = -1;
    for (int c = 0; c < chunks; c++) {
        const int s = c & 1;
        if (c >= 2) {  // the MMAs of chunk c - 2 read this stage
            ok = __syncthreads_and(mbar_wait(&bars[s], ((c - 2) >> 1) & 1, g.polls)) != 0;
            if (!ok) break;
        }
        uint8_t *const as = smem + s * GRAD_STAGE, *const bs = as + (size_t)BM * BK * 2;
        const int k0 = kbeg + c * BK;
        stage_turned<BM>(as, a, HID, m0, k0, kend);
        if (job == 0) stage_turned<HID>(bs, g.h1, HID, 0, k0, kend);
        else if (job == 1) stage_turned<IN>(bs, g.x, IN, 0, k0, kend);
        else stage_turned<OUTP>(bs, g.dyb, OUTP, 0, k0, kend);
        fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(as), b0 = smem_u32(bs);
#pragma unroll
            for (int j = 0; j < BK / 16; j++)
                mma_bf16(tmem, smem_desc(a0 + j * 2 * LBO), smem_desc(b0 + j * 2 * LBO), idesc, (c > 0 || j > 0) ? 1u : 0u);
            mma_commit(&bars[s]);
        }
        committed = c;
    }
    if (ok) ok = __syncthreads_and(mbar_wait(&bars[committed & 1], (committed >> 1) & 1, g.polls)) != 0;
    if (!ok) {
        if (threadIdx.x == 0) atomicExch(g.status, 1);
        // drain: the last commit's barrier completes once every MMA issued so far has finished
        __syncthreads_and(mbar_wait(&bars[committed & 1], (committed >> 1) & 1, kWaitPolls));
    }
    tc_fence_after();
    if (ok) {
        const int m = m0 + (warp & 3) * 32 + lane;
        const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        // the warps of each quarter of the CTA take every fourth run of 16 columns
#pragma unroll 1
        for (int c0 = 16 * (warp >> 2); c0 < n; c0 += 4 * GRAD_THREADS / 32) {
            float v[16];
            tmem_ld16(lane_addr + c0, v);
            if (job == 2) {  // dW3^T: rows are W3's columns
#pragma unroll
                for (int i = 0; i < OUT; i++) atomicAdd(g.g + OFF_W3 + (size_t)i * HID + m, v[i]);
            } else {
                float4 *const o = reinterpret_cast<float4 *>(g.g + (job == 0 ? OFF_W2 + (size_t)m * HID : OFF_W1 + (size_t)m * IN) + c0);
#pragma unroll
                for (int i = 0; i < 4; i++) atomicAdd(o + i, make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, GRAD_N);
}

int grid_of(long long n) { return (int)std::min<long long>(152LL * 8, std::max<long long>(1, (n + 255) / 256)); }

}  // namespace mlp
}  // namespace ntg

using namespace ntg;
using namespace ntg::mlp;

struct ntg_mlp {
    int device = 0;
    int cap = 0;      // batch capacity of the activation buffers
    int step = 0;     // Adam steps taken
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // flat params, grads, Adam moments
    __nv_bfloat16 *w1 = nullptr, *w2 = nullptr, *w2t = nullptr, *w3 = nullptr, *w3t = nullptr;
    float *b3p = nullptr, *wout = nullptr, *loss = nullptr;
    int *status = nullptr;
    int polls = kWaitPolls;  // polls of each tensor-core wait before it gives up
    // activations and gradients, batch `cap`
    __nv_bfloat16 *xb = nullptr, *h1 = nullptr, *h2 = nullptr, *dyb = nullptr, *dz2 = nullptr, *dz1 = nullptr;
    float *z1 = nullptr, *y = nullptr;
    std::vector<void *> owned, act;

    ~ntg_mlp() {
        cudaSetDevice(device);
        for (void *q : act) cudaFree(q);
        for (void *q : owned) cudaFree(q);
    }
};

namespace {

int mlp_fail(int code, const std::string &msg) {
    set_last_error(msg);
    return code;
}

#define MLP_CUDA(call)                                                                   \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess) return mlp_fail(NTG_ERROR_CUDA, std::string(#call ": ") + cudaGetErrorString(e_)); \
    } while (0)

#define MLP_LAUNCH(call)                                                                                \
    do {                                                                                                \
        int r_ = (call);                                                                                \
        if (r_ != 0) return r_ >= kLaunchErrorBase ? mlp_fail(NTG_ERROR_CUDA, std::string(#call ": ") +     \
                                                               cudaGetErrorString((cudaError_t)(r_ - kLaunchErrorBase))) \
                                                   : mlp_fail(r_, #call);                               \
    } while (0)

template <typename T>
int dalloc(std::vector<void *> &list, T **p, size_t n) {
    MLP_CUDA(cudaMalloc((void **)p, n * sizeof(T)));
    list.push_back(*p);
    return NTG_OK;
}

int ensure_batch(ntg_mlp *m, int batch) {
    if (batch <= m->cap) return NTG_OK;
    for (void *q : m->act) cudaFree(q);
    m->act.clear();
    const size_t B = (size_t)batch;
    auto &L = m->act;
    m->cap = 0;
    if (dalloc(L, &m->xb, B * IN) || dalloc(L, &m->h1, B * HID) || dalloc(L, &m->h2, B * HID) || dalloc(L, &m->dyb, B * OUTP) ||
        dalloc(L, &m->dz2, B * HID) || dalloc(L, &m->dz1, B * HID) || dalloc(L, &m->z1, B * HID) || dalloc(L, &m->y, B * OUTP))
        return NTG_ERROR_CUDA;
    m->cap = batch;
    return NTG_OK;
}

GemmArgs gemm(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, int M, int N, int K, int epi, int *status,
              int polls = kWaitPolls) {
    GemmArgs g;
    std::memset(&g, 0, sizeof g);
    g.A = A; g.lda = lda; g.B = B; g.ldb = ldb; g.M = M; g.N = N; g.K = K; g.epi = epi; g.status = status;
    g.polls = polls;
    return g;
}

// The unfused forward pass: X -> H1 -> H2 -> Y [batch x OUTP], one product each.
int forward(ntg_mlp *m, const float *d_x, int batch, cudaStream_t s) {
    k_to_bf16<<<grid_of((long long)batch * IN), 256, 0, s>>>(d_x, (long long)batch * IN, m->xb);
    MLP_LAUNCH(launch_status());
    GemmArgs g = gemm(m->xb, IN, m->w1, IN, batch, HID, IN, EPI_GELU, m->status, m->polls);
    g.bias = m->p + OFF_B1; g.H = m->h1; g.ldh = HID;
    MLP_LAUNCH(launch_gemm(g, s));
    g = gemm(m->h1, HID, m->w2, HID, batch, HID, HID, EPI_GELU, m->status, m->polls);
    g.bias = m->p + OFF_B2; g.H = m->h2; g.ldh = HID;
    MLP_LAUNCH(launch_gemm(g, s));
    g = gemm(m->h2, HID, m->w3, HID, batch, OUTP, HID, EPI_F32, m->status, m->polls);
    g.bias = m->b3p; g.C = m->y; g.ldc = OUTP;
    MLP_LAUNCH(launch_gemm(g, s));
    return NTG_OK;
}

// Forward and backward: the batch's loss into m->loss, its gradient into the flat vector m->g.
int backprop(ntg_mlp *m, const float *d_x, const float *d_t, int batch, cudaStream_t s) {
    if (batch % 8) return mlp_fail(NTG_ERROR_INVALID_INPUT, "training batches are multiples of 8");
    static std::atomic<unsigned long long> configured{0};
    if (first_use_on_device(configured)) {
        cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F_BYTES);
        cudaFuncSetAttribute(k_mlp_grads, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * GRAD_STAGE));
    }
    TrainArgs g;
    g.w1 = m->w1; g.w2 = m->w2; g.w2t = m->w2t; g.w3 = m->w3; g.w3t = m->w3t;
    g.b1 = m->p + OFF_B1; g.b2 = m->p + OFF_B2; g.b3 = m->b3p; g.wout = m->wout; g.x = d_x; g.t = d_t;
    g.batch = batch;
    g.aligned = reinterpret_cast<uintptr_t>(d_x) % 16 == 0;
    g.z1 = m->z1; g.h1 = m->h1; g.h2 = m->h2; g.dz1 = m->dz1; g.dz2 = m->dz2; g.dyb = m->dyb;
    g.g = m->g; g.loss = m->loss; g.status = m->status; g.polls = m->polls;
    MLP_CUDA(cudaMemsetAsync(m->g, 0, (NPARAM + 1) * sizeof(float), s));
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
    k_mlp_train<<<std::min((batch + BM - 1) / BM, std::max(1, sms)), 512, F_BYTES, s>>>(g);
    MLP_LAUNCH(launch_status());
    k_mlp_grads<<<dim3((batch + GRAD_K - 1) / GRAD_K, 6), GRAD_THREADS, 2 * GRAD_STAGE, s>>>(g);
    MLP_LAUNCH(launch_status());
    return NTG_OK;
}

int refresh(ntg_mlp *m, cudaStream_t s) {
    k_refresh<<<grid_of(HID * HID), 256, 0, s>>>(m->p, m->w1, m->w2, m->w2t, m->w3, m->w3t, m->b3p);
    MLP_LAUNCH(launch_status());
    return NTG_OK;
}

int check_status(ntg_mlp *m, cudaStream_t s) {
    int st = 0;
    MLP_CUDA(cudaMemcpyAsync(&st, m->status, sizeof st, cudaMemcpyDeviceToHost, s));
    MLP_CUDA(cudaStreamSynchronize(s));
    if (st) return mlp_fail(NTG_ERROR_CUDA, "tensor-core wait timed out");
    return NTG_OK;
}

}  // namespace

namespace ntg {
// Forward pass for callers inside the library (the learned encoder): x fp32 [batch x 48] ->
// y fp32 [batch x 16].
int mlp_forward_device(ntg_mlp *m, const float *d_x, long long rows, float *d_y, cudaStream_t s) {
    if (!m || !d_x || !d_y || rows <= 0) return NTG_ERROR_INVALID_INPUT;
    static std::atomic<unsigned long long> configured{0};
    if (first_use_on_device(configured))
        cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F_BYTES);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
    const long long tiles = (rows + BM - 1) / BM;
    const int grid = (int)std::min<long long>(tiles, std::max(1, sms));
    k_mlp_infer<<<grid, 512, F_BYTES, s>>>(m->w1, m->w2, m->w3, m->p + OFF_B1, m->p + OFF_B2, m->b3p, d_x, rows, d_y,
                                           m->status, m->polls);
    MLP_LAUNCH(launch_status());
    return NTG_OK;
}
}  // namespace ntg

extern "C" {

int ntg_mlp_create(int device, unsigned long long seed, ntg_mlp **out) {
    if (!out) return mlp_fail(NTG_ERROR_INVALID_INPUT, "null output");
    MLP_CUDA(cudaSetDevice(device));
    std::unique_ptr<ntg_mlp> m(new ntg_mlp);
    m->device = device;
    auto &L = m->owned;
    if (dalloc(L, &m->p, NPARAM) || dalloc(L, &m->g, NPARAM + 2) || dalloc(L, &m->m, NPARAM) || dalloc(L, &m->v, NPARAM) ||
        dalloc(L, &m->w1, (size_t)HID * IN) || dalloc(L, &m->w2, (size_t)HID * HID) || dalloc(L, &m->w2t, (size_t)HID * HID) ||
        dalloc(L, &m->w3, (size_t)OUTP * HID) || dalloc(L, &m->w3t, (size_t)HID * OUTP) || dalloc(L, &m->b3p, OUTP) ||
        dalloc(L, &m->wout, OUT))
        return NTG_ERROR_CUDA;
    m->loss = m->g + NPARAM;  // zeroed with the gradient, read together with the status
    m->status = reinterpret_cast<int *>(m->g + NPARAM + 1);
    // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights and biases, seeded
    std::vector<float> p(NPARAM);
    std::mt19937_64 rng(seed);
    auto fill = [&](size_t off, size_t n, int fan_in) {
        std::uniform_real_distribution<float> u(-1.0f / std::sqrt((float)fan_in), 1.0f / std::sqrt((float)fan_in));
        for (size_t i = 0; i < n; i++) p[off + i] = u(rng);
    };
    fill(OFF_W1, (size_t)HID * IN, IN); fill(OFF_B1, HID, IN);
    fill(OFF_W2, (size_t)HID * HID, HID); fill(OFF_B2, HID, HID);
    fill(OFF_W3, (size_t)OUT * HID, HID); fill(OFF_B3, OUT, HID);
    const float wout[OUT] = {1, 1, 1, 1, 1, 0.25f, 0, 0};
    MLP_CUDA(cudaMemcpy(m->p, p.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice));
    MLP_CUDA(cudaMemset(m->m, 0, NPARAM * sizeof(float)));
    MLP_CUDA(cudaMemset(m->v, 0, NPARAM * sizeof(float)));
    MLP_CUDA(cudaMemset(m->status, 0, sizeof(int)));
    MLP_CUDA(cudaMemcpy(m->wout, wout, sizeof wout, cudaMemcpyHostToDevice));
    int r = refresh(m.get(), nullptr);
    if (r) return r;
    MLP_CUDA(cudaDeviceSynchronize());
    *out = m.release();
    return NTG_OK;
}

int ntg_mlp_destroy(ntg_mlp *m) {
    delete m;
    return NTG_OK;
}

int ntg_mlp_param_count(void) { return (int)NPARAM; }

int ntg_mlp_get_params(ntg_mlp *m, float *h_params) {
    if (!m || !h_params) return mlp_fail(NTG_ERROR_INVALID_INPUT, "bad arguments");
    MLP_CUDA(cudaSetDevice(m->device));
    MLP_CUDA(cudaMemcpy(h_params, m->p, NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    return NTG_OK;
}

int ntg_mlp_set_params(ntg_mlp *m, const float *h_params) {
    if (!m || !h_params) return mlp_fail(NTG_ERROR_INVALID_INPUT, "bad arguments");
    MLP_CUDA(cudaSetDevice(m->device));
    MLP_CUDA(cudaMemcpy(m->p, h_params, NPARAM * sizeof(float), cudaMemcpyHostToDevice));
    int r = refresh(m, nullptr);
    if (r) return r;
    MLP_CUDA(cudaDeviceSynchronize());
    return NTG_OK;
}

int ntg_mlp_infer(ntg_mlp *m, const float *d_x, int batch, float *d_y, void *stream) {
    if (!m || !d_x || !d_y || batch <= 0) return mlp_fail(NTG_ERROR_INVALID_INPUT, "bad arguments");
    MLP_CUDA(cudaSetDevice(m->device));
    return mlp_forward_device(m, d_x, batch, d_y, (cudaStream_t)stream);
}

// The unfused forward pass (three k_gemm launches), for testing.
int ntg_mlp_infer_unfused(ntg_mlp *m, const float *d_x, int batch, float *d_y, void *stream) {
    if (!m || !d_x || !d_y || batch <= 0) return mlp_fail(NTG_ERROR_INVALID_INPUT, "bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    int r = ensure_batch(m, batch);
    if (!r) r = forward(m, d_x, batch, s);
    if (r) return r;
    MLP_CUDA(cudaMemcpyAsync(d_y, m->y, sizeof(float) * batch * OUTP, cudaMemcpyDeviceToDevice, s));
    return NTG_OK;
}

int ntg_mlp_gradients(ntg_mlp *m, const float *d_x, const float *d_t, int batch, float *d_grads, float *h_loss,
                      void *stream) {
    if (!m || !d_x || !d_t || batch <= 0) return mlp_fail(NTG_ERROR_INVALID_INPUT, "bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    int r = ensure_batch(m, batch);
    if (!r) r = backprop(m, d_x, d_t, batch, s);
    if (r) return r;
    if (d_grads) MLP_CUDA(cudaMemcpyAsync(d_grads, m->g, NPARAM * sizeof(float), cudaMemcpyDeviceToDevice, s));
    struct { float loss; int status; } h;
    MLP_CUDA(cudaMemcpyAsync(&h, m->loss, sizeof h, cudaMemcpyDeviceToHost, s));
    MLP_CUDA(cudaStreamSynchronize(s));
    if (h_loss) *h_loss = h.loss;
    return h.status ? mlp_fail(NTG_ERROR_CUDA, "tensor-core wait timed out") : NTG_OK;
}

int ntg_mlp_train_step(ntg_mlp *m, const float *d_x, const float *d_t, int batch, float lr, float *d_loss, void *stream) {
    if (!m || !d_x || !d_t || batch <= 0) return mlp_fail(NTG_ERROR_INVALID_INPUT, "bad arguments");
    cudaStream_t s = (cudaStream_t)stream;
    int r = ensure_batch(m, batch);
    if (!r) r = backprop(m, d_x, d_t, batch, s);
    if (r) return r;
    m->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, (float)m->step), c2 = 1.0f - std::pow(b2, (float)m->step);
    k_adam<<<grid_of(NPARAM), 256, 0, s>>>(m->p, m->g, m->m, m->v, (int)NPARAM, lr, b1, b2, 1e-8f, c1, c2);
    MLP_LAUNCH(launch_status());
    r = refresh(m, s);
    if (r) return r;
    if (d_loss) MLP_CUDA(cudaMemcpyAsync(d_loss, m->loss, sizeof(float), cudaMemcpyDeviceToDevice, s));
    return NTG_OK;
}

int ntg_mlp_status(ntg_mlp *m) {
    if (!m) return mlp_fail(NTG_ERROR_INVALID_INPUT, "null network");
    MLP_CUDA(cudaSetDevice(m->device));
    return check_status(m, nullptr);
}

int ntg_mlp_set_wait_limit(ntg_mlp *m, int polls) {
    if (!m) return mlp_fail(NTG_ERROR_INVALID_INPUT, "null network");
    MLP_CUDA(cudaSetDevice(m->device));
    MLP_CUDA(cudaDeviceSynchronize());
    m->polls = polls < 0 ? kWaitPolls : polls;
    MLP_CUDA(cudaMemset(m->status, 0, sizeof(int)));
    MLP_CUDA(cudaDeviceSynchronize());
    return NTG_OK;
}

int ntg_gemm_bf16(const void *d_a, const void *d_b, int M, int N, int K, float *d_c, void *stream) {
    if (!d_a || !d_b || !d_c || M <= 0 || N <= 0 || K <= 0) return mlp_fail(NTG_ERROR_INVALID_INPUT, "bad arguments");
    GemmArgs g = gemm((const __nv_bfloat16 *)d_a, K, (const __nv_bfloat16 *)d_b, K, M, N, K, EPI_F32, nullptr);
    g.C = d_c; g.ldc = N;
    MLP_LAUNCH(launch_gemm(g, (cudaStream_t)stream));
    return NTG_OK;
}

}  // extern "C"
