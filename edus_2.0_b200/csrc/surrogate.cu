// Learned HSEX surrogate: a multilayer perceptron trained on the GPU by its
// own forward and backward kernels (no reference counterpart).
//
// Network: n_in -> H -> H -> H -> n_out, GELU after each hidden layer, linear
// output.  Weights are kept in FP32 (the optimiser's master copy) and in BF16
// (what the tensor cores multiply); activations are FP32 and are rounded to
// BF16 as the operand of the next product; every product accumulates in FP32
// in tensor memory (tcgen05.mma kind::f16, 128 x 128 tiles).  Loss: mean squared error over the
// batch and the outputs.  Optimiser: Adam.
//
// Layouts: a batch of B samples is row-major [B][features]; a weight matrix is
// row-major [in][out].  All batch buffers passed to the entry points are
// device pointers.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>
#include "../../include/edus_gpu.h"

namespace {

constexpr int kLayers = 4;  // three hidden layers and the output layer

// ---------------------------------------------------------------------------
// C[M][N] (+)= op(A)[M][K] op(B)[K][N] on the 5th-generation tensor cores
// (tcgen05.mma kind::f16, BF16 operands, FP32 accumulator in tensor memory).
// A(i, k) = A[i * a_rs + k * a_cs], B(k, j) = B[k * b_rs + j * b_cs] (BF16), so
// a transposed operand is only a change of strides.
//
// A CTA of 4 warps owns a 128 x 128 tile of C, accumulated in 128 TMEM columns
// (lane = row, column = output column).  K runs in chunks of 64: the 128 threads
// gather A's 128 x 64 and B's 64 x 128 chunk from global memory (strided,
// out-of-range rows, columns and K read as zero) into shared memory in the
// K-major, non-swizzled layout of the tensor-core operand descriptors: 8 rows x
// 16 bytes per core matrix, core matrices of one 8-row group contiguous along K
// (leading byte offset 128 B), 8-row groups 1024 B apart (stride byte offset).
// One thread issues the chunk's four 128 x 128 x 16 MMAs and commits them to an
// mbarrier, which every thread waits on (bounded) before the next chunk
// overwrites the operands.  Epilogue: each warp reads its 32 TMEM lanes
// (tcgen05.ld 32x32b, 8 columns at a time), adds the bias, writes C.
constexpr int UM = 128, UN = 128, UK = 64;
constexpr int TM = UM, TN = UN;
// instruction descriptor: FP32 accumulator, BF16 A and B, both K-major, N, M
constexpr unsigned kUmmaIdesc =
    (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(UN >> 3) << 17) | ((unsigned)(UM >> 4) << 24);

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// shared-memory operand descriptor (K-major, no swizzle, descriptor version 1)
__device__ __forceinline__ unsigned long long umma_desc(const void* p) {
    return (unsigned long long)((smem_addr(p) >> 4) & 0x3FFFu) | ((unsigned long long)(128u >> 4) << 16) |
           ((unsigned long long)(1024u >> 4) << 32) | (1ull << 46);
}

// element offset of (row r, k) of a 64-wide K chunk in the core-matrix layout
__device__ __forceinline__ int umma_off(int r, int k) { return (r >> 3) * 512 + (k >> 3) * 64 + (r & 7) * 8 + (k & 7); }

__device__ __forceinline__ bool mbar_wait_parity(unsigned long long* bar, unsigned parity, int limit) {
    for (int i = 0; i < limit; ++i) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

constexpr int kMlpPolls = 1 << 22;
// False if the wait ran out after `polls`; what was waited for is then awaited
// once more (bounded), so that no copy or product of this CTA is in flight when
// the caller reports the failure and goes on.
__device__ __forceinline__ bool mbar_wait_drain(unsigned long long* bar, unsigned parity, int polls) {
    if (mbar_wait_parity(bar, parity, polls)) return true;
    mbar_wait_parity(bar, parity, kMlpPolls);
    return false;
}

__global__ void __launch_bounds__(128) gemm_bf16_kernel(int M, int N, int K, const __nv_bfloat16* __restrict__ A,
                                                       long long a_rs, long long a_cs,
                                                       const __nv_bfloat16* __restrict__ B, long long b_rs,
                                                       long long b_cs, float* __restrict__ C, int ldc,
                                                       const float* __restrict__ bias, int accumulate,
                                                       int* __restrict__ status, int polls) {
    __shared__ __align__(1024) __nv_bfloat16 As[UM * UK];  // 16 KB
    __shared__ __align__(1024) __nv_bfloat16 Bs[UN * UK];  // 16 KB
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ unsigned tmem_slot;
    const int m0 = blockIdx.y * UM, n0 = blockIdx.x * UN;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_slot)),
                     "r"(UN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_addr(&mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem = tmem_slot;
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    unsigned phase = 0;
    bool ok = true;
    for (int k0 = 0; k0 < K; k0 += UK) {
        for (int e = threadIdx.x; e < UM * UK; e += blockDim.x) {
            const int r = e / UK, k = e - (e / UK) * UK;
            const int gi = m0 + r, gk = k0 + k;
            As[umma_off(r, k)] = (gi < M && gk < K) ? A[gi * a_rs + gk * a_cs] : zero;
        }
        for (int e = threadIdx.x; e < UN * UK; e += blockDim.x) {
            const int c = e / UK, k = e - (e / UK) * UK;
            const int gj = n0 + c, gk = k0 + k;
            Bs[umma_off(c, k)] = (gj < N && gk < K) ? B[gk * b_rs + gj * b_cs] : zero;
        }
        // the operands were written by the generic proxy; the tensor core reads them by the async proxy
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int st = 0; st < UK / 16; ++st) {
                const unsigned long long da = umma_desc(As + st * 128);  // two core matrices = 16 of K
                const unsigned long long db = umma_desc(Bs + st * 128);
                const unsigned accum = (k0 > 0 || st > 0) ? 1u : 0u;
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(kUmmaIdesc), "r"(accum)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_addr(&mbar))
                         : "memory");
        }
        // the MMAs have read the operands (and written TMEM) once the phase completes
        if (!mbar_wait_drain(&mbar, phase, polls)) ok = false;  // give up: report, skip the rest
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
    }
    if (!ok && threadIdx.x == 0 && status) atomicOr(status, 1);
    // epilogue: TMEM lanes 32 warp .. 32 warp + 31 are this warp's rows
    const int row = m0 + warp * 32 + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < (ok ? UN : 0); c0 += 8) {
        unsigned v[8];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
            : "r"(tmem + ((unsigned)(warp * 32) << 16) + (unsigned)c0));
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        if (row < M) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int col = n0 + c0 + j;
                if (col < N) {
                    float x = __uint_as_float(v[j]);
                    if (bias) x += bias[col];
                    float* dst = C + (long long)row * ldc + col;
                    *dst = accumulate ? *dst + x : x;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(UN) : "memory");
}

// ---------------------------------------------------------------------------
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

// a = GELU(z) (FP32) and its BF16 copy
__global__ void gelu_kernel(const float* __restrict__ z, float* __restrict__ a, __nv_bfloat16* __restrict__ ab,
                            long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = gelu(z[i]);
        a[i] = v;
        ab[i] = __float2bfloat16(v);
    }
}
__global__ void to_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ xb, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        xb[i] = __float2bfloat16(x[i]);
}
// dz = da * GELU'(z), and its BF16 copy
__global__ void gelu_back_kernel(const float* __restrict__ da, const float* __restrict__ z, float* __restrict__ dz,
                                 __nv_bfloat16* __restrict__ dzb, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float v = da[i] * gelu_grad(z[i]);
        dz[i] = v;
        dzb[i] = __float2bfloat16(v);
    }
}
// dy = 2 (y - t) / n_total, and the loss (mean of squares; one atomic per block)
__global__ void mse_kernel(const float* __restrict__ y, const float* __restrict__ t, float* __restrict__ dy,
                           __nv_bfloat16* __restrict__ dyb, long long n, float scale, float* __restrict__ loss) {
    __shared__ float red[256];
    float s = 0.f;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float d = y[i] - t[i];
        s += d * d;
        const float g = 2.f * d * scale;
        dy[i] = g;
        dyb[i] = __float2bfloat16(g);
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0] * scale);
}
// db[j] = sum_i dz[i][j]
__global__ void colsum_kernel(const float* __restrict__ dz, float* __restrict__ db, int rows, int cols) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols) return;
    float s = 0.f;
    for (int i = 0; i < rows; ++i) s += dz[(long long)i * cols + j];
    db[j] = s;
}
// An update leaves weights and moments alone when a wait ran out in the kernels
// that made its gradients (or in an earlier step's, not reported yet): status
// stays set until the host reads it, and `skipped` counts the training steps
// that were left out, which the host takes back from its step count.
// `status` is read beside the operands, which the kernel waits for anyway.
__device__ __forceinline__ bool update_skipped(int status, int* skipped, bool training) {
    if (!status) return false;
    if (training && blockIdx.x == 0 && threadIdx.x == 0) ++*skipped;
    return true;
}

// Adam on the FP32 master weights, refreshing their BF16 copy
__global__ void adam_kernel(float* __restrict__ w, __nv_bfloat16* __restrict__ wb, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, long long n, float lr, float b1, float b2,
                            float eps, float c1, float c2, const int* __restrict__ status, int* __restrict__ skipped) {
    if (update_skipped(*status, skipped, true)) return;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        wb[i] = __float2bfloat16(wi);
    }
}

// ---------------------------------------------------------------------------
// Networks of hidden width 128 (what the surrogate uses; other widths run the
// kernels above): the whole forward and backward chain of 128 batch rows in a
// cluster of four CTAs, all weight and bias gradients in a second launch (each a
// contraction over the whole batch, not split), Adam and the weights' BF16 blocks in
// a third.
//
// Layer by layer through global memory this step was bound by its launches and
// by serial work, not by arithmetic: the weight gradients contract over the
// batch, so each was one CTA walking 4096 rows (0.88 ms a layer), and the
// column sums were one thread a column (0.23 ms); 4096 x 259 -> 254 took
// 4.05 ms a training step.  Here activations never leave the SM between
// layers (shared memory as BF16 operands, tensor memory as FP32
// pre-activations), and each layer's gradient is spread over the SMs by tiles and
// column groups.
//
// Operand blocks.  Activations, gradients and weights are 128 x 128 BF16 blocks
// (32 KB) of 8 x 8 core matrices (128 B).  Gradients and weights: element (r, c)
// at (r >> 3) * 1024 + (c >> 3) * 64 + (r & 7) * 8 + (c & 7).  Read with c along K
// this is the K-major operand layout (core matrices 128 B apart along K, 2048 B
// along the rows); read with r along K it is the MN-major layout of the
// transposed matrix.  Activations: four column groups of 32, each laid out that
// way (512 B between row groups), so that a group is contiguous.  One copy of
// each block therefore serves both products it enters: an activation block (r =
// batch row, c = feature) is the row operand of the forward product and, by
// column groups, the column operand of the weight gradient; a weight block (r =
// output, c = input) is used as it is forward and transposed backward.  Blocks
// move between global and shared memory by bulk copies.
constexpr int kBlk = 128 * 128;            // elements of a block
constexpr unsigned kBlkBytes = kBlk * 2u;  // 32 KB
constexpr int kGrp = 128 * 32;             // elements of an activation block's column group
constexpr int kRing = 3;                   // weight blocks in flight
constexpr int kActs = 3;                   // activation blocks in shared memory
constexpr size_t kRowsSmem = (size_t)(kRing + kActs) * kBlkBytes + 1024;
constexpr int kDwStages = 5;
constexpr unsigned kDwStage = kBlkBytes + kGrp * 2u;  // a dz block and an activation column group
constexpr size_t kDwSmem = (size_t)kDwStages * kDwStage + 1024;
constexpr unsigned kBiasStage = 128 * 32 * 4;  // 128 rows x 32 outputs of dz in FP32

__device__ __forceinline__ int blk_off(int r, int c) { return (r >> 3) * 1024 + (c >> 3) * 64 + (r & 7) * 8 + (c & 7); }
__device__ __forceinline__ int act_off(int r, int c) {
    return (c >> 5) * kGrp + (r >> 3) * 256 + ((c >> 3) & 3) * 64 + (r & 7) * 8 + (c & 7);
}

// operand descriptor: `kcore` bytes between core matrices along K, `mncore` along the rows
__device__ __forceinline__ unsigned long long op_desc(const void* p, unsigned kcore, unsigned mncore) {
    return (unsigned long long)((smem_addr(p) >> 4) & 0x3FFFu) | ((unsigned long long)(kcore >> 4) << 16) |
           ((unsigned long long)(mncore >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void mma_k16(unsigned tmem, unsigned long long da, unsigned long long db, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate ? 1u : 0u)
        : "memory");
}
constexpr unsigned kTransA = 1u << 15, kTransB = 1u << 16;

// acc[out 128][in 32] (+)= dz^T act over 128 batch rows: both operands MN-major
__device__ __forceinline__ void dw_mma(const __nv_bfloat16* dz, const __nv_bfloat16* act, unsigned tmem, bool accumulate) {
    constexpr unsigned idesc =
        (1u << 4) | (1u << 7) | (1u << 10) | kTransA | kTransB | ((32u >> 3) << 17) | ((unsigned)(UM >> 4) << 24);
#pragma unroll
    for (int st = 0; st < 8; ++st)
        mma_k16(tmem, op_desc(dz + st * 2048, 2048, 128), op_desc(act + st * 512, 512, 128), idesc,
                accumulate || st > 0);
}
__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ void bar_init1(unsigned long long* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_addr(bar)) : "memory");
}
// block global -> shared, completion on bar (which takes one arrival per copy)
__device__ __forceinline__ void blk_load(void* dst, const void* src, unsigned long long* bar, unsigned bytes = kBlkBytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(reinterpret_cast<unsigned long long>(src)), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld16(float* v, unsigned addr) {
    unsigned u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
        "[%16];\n"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
          "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(u[i]);
}
__device__ __forceinline__ void tmem_ld8(float* v, unsigned addr) {
    unsigned u[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(u[i]);
}

struct MlpRowsArgs {
    int B, n_in, n_out, KT, NT;
    const float* x;            // [B][n_in]
    const float* t;            // [B][n_out] (TRAIN)
    float* y;                  // [B][n_out] (forward only)
    const __nv_bfloat16* wp;   // weight blocks: layer 0 by input block, layers 1, 2, output layer by output block
    const float* bias[4];
    __nv_bfloat16* act;        // [row block][KT + 3]: x blocks, a1, a2, a3 (TRAIN)
    __nv_bfloat16* dz;         // [row block][3 + NT]: dz of layers 0, 1, 2 and of the output blocks (TRAIN)
    float* dzf;                // [row block][3 + NT][4 column groups][128][32]: dz in FP32 (TRAIN)
    float* lossp;              // [row block][4] (TRAIN)
    float scale;               // 1 / (B n_out)
    int* status;
    int polls;                 // limit of every wait
};

constexpr int kTeam = 4;  // CTAs of a row block, a column group each

__device__ __forceinline__ unsigned peer_addr(const void* p, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_addr(p)), "r"(rank));
    return r;
}
// every thread of the team, with what each wrote to shared memory (its own and
// the peers') before it
__device__ __forceinline__ void team_sync() {
    asm volatile("fence.proxy.async.shared::cluster;\n" ::: "memory");
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cluster;\n" ::: "memory");
}

// 128 batch rows through the network and, with TRAIN, back, by a cluster of four
// CTAs.  CTA j computes columns 32 j .. 32 j + 31 of every 128-wide layer block: its
// share of the products (N = 32), of GELU and its derivative (erff and expf, the
// largest part of the time: one CTA a row block, 4096 rows on 32 SMs, took 84 us;
// four, 42 us) and of the loads and stores.  It writes its columns of an
// activation or gradient block into all four CTAs' shared memory, so each holds
// the whole block as the operand of its next product; one cluster barrier a
// product orders this.  Buffers rotate: when a CTA writes block i it has passed
// the barrier of block i - 1, so every CTA's product of block i - 2 is done and the
// buffer of block i - 3 is free.
//
// 16 warps; a thread owns one row (32 (warp & 3) + lane, its tensor-memory lane)
// and 8 columns of the group, 32 bytes of each FP32 row it reads or writes.
// Tensor-memory columns: the pre-activations of the hidden layers at 0, 32, 64,
// the output block at 96; backward, the gradient of a layer's activations takes
// the columns of the layer above it.  Every wait is bounded; one that runs out
// is drained (mbar_wait_drain), sets *status and tells the team (`failed`, by the
// parity of the next barrier, so that all four leave at the same one).
template <bool TRAIN>
__global__ void __cluster_dims__(kTeam, 1, 1) __launch_bounds__(512, 1) mlp_rows_kernel(MlpRowsArgs a) {
    extern __shared__ unsigned char mraw[];
    __shared__ __align__(8) unsigned long long full[kRing], mma_bar, rel_bar;
    __shared__ unsigned tmem_slot;
    __shared__ int failed[2];
    __shared__ float red[16];
    __nv_bfloat16* act = (__nv_bfloat16*)(((unsigned long long)mraw + 1023) & ~1023ull);
    __nv_bfloat16* ring = act + kActs * kBlk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x & (kTeam - 1), rb = blockIdx.x / kTeam;
    const int row = (warp & 3) * 32 + lane, sub = (warp >> 2) * 8, col0 = rank * 32 + sub;
    const long long grow = (long long)rb * 128 + row;
    const bool live = grow < a.B;
    const int KT = a.KT, NT = a.NT;
    const int nqf = KT + 2 + NT, nq = TRAIN ? nqf + NT + 2 : nqf;
    constexpr unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((32u >> 3) << 17) | ((unsigned)(UM >> 4) << 24);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_slot)),
                     "r"(128)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    int issued = 0;  // thread 0: weight blocks requested
    // weight block of product q (forward layers, then backward from the output);
    // forward this CTA needs the block's 32 output rows only
    auto prefetch = [&](int q) {
        if (q >= nq) return;
        __nv_bfloat16* dst = ring + (q % kRing) * kBlk;
        if (q < nqf) {
            blk_load(dst + rank * 4096, a.wp + (size_t)q * kBlk + rank * 4096, &full[q % kRing], kBlkBytes / kTeam);
        } else {
            const int p = q - nqf;
            blk_load(dst, a.wp + (size_t)(p < NT ? KT + 2 + p : (p == NT ? KT + 1 : KT)) * kBlk, &full[q % kRing]);
        }
        issued = q + 1;
    };
    if (tid == 0) {
        failed[0] = failed[1] = 0;
        for (int i = 0; i < kRing; ++i) bar_init1(&full[i]);
        bar_init1(&mma_bar);
        bar_init1(&rel_bar);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        for (int q = 0; q < kRing; ++q) prefetch(q);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    team_sync();  // the peers' shared memory may be written from here on
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem = tmem_slot;
    const unsigned lanes = tmem + ((unsigned)((warp & 3) * 32) << 16) + sub;

    int nsync = 0;  // team barriers passed in product()
    auto tell_failed = [&]() {
        for (int r = 0; r < kTeam; ++r)
            asm volatile("st.shared::cluster.u32 [%0], %1;\n" ::"r"(peer_addr(&failed[(nsync + 1) & 1], r)), "r"(1) : "memory");
    };
    // 8 columns of this thread's row, rounded to BF16, into the block's buffer of all four CTAs
    auto put8 = [&](int buf, bool activation, const float* v) {
        __nv_bfloat162 p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        const uint4 u = *reinterpret_cast<uint4*>(p);
        const __nv_bfloat16* d = act + buf * kBlk + (activation ? act_off(row, col0) : blk_off(row, col0));
#pragma unroll
        for (int r = 0; r < kTeam; ++r)
            asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(peer_addr(d, r)), "r"(u.x), "r"(u.y),
                         "r"(u.z), "r"(u.w)
                         : "memory");
    };
    // this thread's 8 FP32 of a dz block, for the bias gradients
    auto put_dzf = [&](int slot, const float* v) {
        float* d = a.dzf + ((((size_t)rb * (3 + NT) + slot) * 4 + rank) * 128 + row) * 32 + sub;
        *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(d + 4) = make_float4(v[4], v[5], v[6], v[7]);
    };
    // the team's barrier after a block is written; false: leave (all four CTAs do)
    auto block_ready = [&]() {
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        // stores older than the last one have left their buffers
        if (TRAIN && tid == 0) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
        team_sync();
        ++nsync;
        return *(volatile int*)&failed[nsync & 1] == 0;
    };
    // a quarter of a block in shared memory to global memory: an activation
    // block's column group, or a gradient block's 32 rows (8 KB either way)
    auto store_share = [&](__nv_bfloat16* dst, int buf) {
        const __nv_bfloat16* src = act + buf * kBlk + rank * (kBlk / kTeam);
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(
                         reinterpret_cast<unsigned long long>(dst + rank * (kBlk / kTeam))),
                     "r"(smem_addr(src)), "r"(kBlkBytes / kTeam)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
    };
    // product q: the block in buffer `buf` times the weight block, into tensor-memory column `col`
    auto product = [&](int q, int buf, bool forward, unsigned col, bool accumulate) {
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (!mbar_wait_drain(&full[q % kRing], (unsigned)((q / kRing) & 1), a.polls)) tell_failed();
            const __nv_bfloat16* A = act + buf * kBlk;
            const __nv_bfloat16* W = ring + (q % kRing) * kBlk;
#pragma unroll
            for (int st = 0; st < 8; ++st) {  // K = 16 each
                if (forward)
                    mma_k16(tmem + col, op_desc(A + (st >> 1) * kGrp + (st & 1) * 128, 128, 512),
                            op_desc(W + rank * 4096 + st * 128, 128, 2048), idesc, accumulate || st > 0);
                else
                    mma_k16(tmem + col, op_desc(A + st * 128, 128, 2048), op_desc(W + rank * 256 + st * 2048, 2048, 128),
                            idesc | kTransB, accumulate || st > 0);
            }
            mma_commit(&mma_bar);
        }
    };
    // product q is done; its weight block's slot is refilled
    auto finished = [&](int q) {
        const bool ok = mbar_wait_drain(&mma_bar, (unsigned)(q & 1), a.polls);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (!ok) tell_failed();
        __syncthreads();
        if (tid == 0) prefetch(q + kRing);
        __syncwarp();
    };
    __nv_bfloat16* keep_act = TRAIN ? a.act + (size_t)rb * (KT + 3) * kBlk : nullptr;
    __nv_bfloat16* keep_dz = TRAIN ? a.dz + (size_t)rb * (3 + NT) * kBlk : nullptr;
    auto load8 = [&](const float* src, int width, int c, float* v) {  // 8 of this thread's row; zeros past the ends
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = (live && c + i < width) ? __ldg(src + grow * width + c + i) : 0.f;
    };

    // activation block i sits in buffer i % kActs
    int q = 0, i = 0;
    bool ok = true;
    float v[8], z[8];
    load8(a.x, a.n_in, col0, v);
    for (int kt = 0; ok && kt < KT; ++kt, ++i, ++q) {
        put8(i % kActs, true, v);
        if (kt + 1 < KT) load8(a.x, a.n_in, (kt + 1) * 128 + col0, v);
        if (!(ok = block_ready())) break;
        product(q, i % kActs, true, 0, kt > 0);
        if (TRAIN && tid == 0) store_share(keep_act + (size_t)kt * kBlk, i % kActs);
        finished(q);
    }
    for (int l = 0; ok && l < 3; ++l, ++i) {
        tmem_ld8(v, lanes + l * 32);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = gelu(v[j] + __ldg(&a.bias[l][col0 + j]));
        put8(i % kActs, true, v);
        if (!(ok = block_ready())) break;
        if (TRAIN && tid == 0) store_share(keep_act + (size_t)(KT + l) * kBlk, i % kActs);
        if (l < 2) {
            product(q, i % kActs, true, (l + 1) * 32, false);
            finished(q++);
        }
    }
    const int b3 = i - 1;  // a3's block
    float loss = 0.f;
    for (int nt = 0; ok && nt < NT; ++nt) {
        const int col = nt * 128 + col0;
        if (TRAIN) load8(a.t, a.n_out, col, z);
        product(q, b3 % kActs, true, 96, false);
        finished(q++);
        tmem_ld8(v, lanes + 96);
        if (!TRAIN) {
            // the next product overwrites these columns
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (live && col + j < a.n_out) a.y[grow * a.n_out + col + j] = v[j] + __ldg(&a.bias[3][col + j]);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const bool on = live && col + j < a.n_out;
                const float d = on ? v[j] + __ldg(&a.bias[3][col + j]) - z[j] : 0.f;
                loss += d * d;
                v[j] = 2.f * d * a.scale;
            }
            // output blocks take turns in the two buffers that a3 leaves
            const int buf = (b3 + 1 + (nt & 1)) % kActs;
            if (nt >= 2) {
                // the block before last has left its buffer in every CTA
                if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
                team_sync();
            }
            put8(buf, false, v);
            if (!(ok = block_ready())) break;
            if (tid == 0) store_share(keep_dz + (size_t)(3 + nt) * kBlk, buf);
            put_dzf(3 + nt, v);
        }
    }
    if (TRAIN) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, s);
        if (lane == 0) red[warp] = loss;
        __syncthreads();
        if (tid == 0) {
            float s = 0.f;
            for (int w = 0; w < 16; ++w) s += red[w];
            a.lossp[rb * kTeam + rank] = s * a.scale;
        }
        // gradient of a3: sum over the output blocks of dz_out W^T (column 96; more
        // than two blocks are read back from global memory)
        if (NT > 2) {
            if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");  // the blocks are written
            asm volatile("fence.proxy.async.global;\n" ::: "memory");
            team_sync();
            asm volatile("fence.proxy.async.global;\n" ::: "memory");
        }
        for (int nt = 0; ok && nt < NT; ++nt) {
            const int buf = (b3 + 1 + (nt & 1)) % kActs;
            if (NT > 2) {
                if (tid == 0) {
                    blk_load(act + buf * kBlk, keep_dz + (size_t)(3 + nt) * kBlk, &rel_bar);
                    if (!mbar_wait_drain(&rel_bar, (unsigned)(nt & 1), a.polls)) tell_failed();
                }
                __syncthreads();
            }
            product(q, buf, false, 96, nt > 0);
            finished(q++);
        }
        // the next blocks' buffers: a3's, then the output blocks'
        i = b3 + 3;
        for (int l = 2; ok && l >= 0; --l, ++i) {
            // dz_l = da * GELU'(z_l)
            tmem_ld8(v, lanes + (l + 1) * 32);
            tmem_ld8(z, lanes + l * 32);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] *= gelu_grad(z[j] + __ldg(&a.bias[l][col0 + j]));
            if (l == 2) {
                // every CTA's products and stores of the buffers written from here on are done
                if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                team_sync();
            }
            put8(i % kActs, false, v);
            if (!(ok = block_ready())) break;
            if (l > 0) product(q, i % kActs, false, l * 32, false);
            if (tid == 0) store_share(keep_dz + (size_t)l * kBlk, i % kActs);
            put_dzf(l, v);
            if (l > 0) finished(q++);
        }
    }
    if (tid == 0) {
        if (!ok) {
            atomicOr(a.status, 1);
            // weight blocks still in flight land before the CTA ends
            for (int j = issued - 1; j >= 0 && j >= issued - kRing; --j)
                mbar_wait_parity(&full[j % kRing], (unsigned)((j / kRing) & 1), kMlpPolls);
        }
        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    team_sync();  // no peer writes this CTA's shared memory any more
    if (tid == 0 && (failed[0] | failed[1])) atomicOr(a.status, 1);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(128) : "memory");
}

// Weight gradients: CTA (tile, group) contracts over the whole batch in row
// order, grad[tile][c][r] = sum over rows of act(row, c) dz(row, r), for 32 of
// the tile's 128 inputs c (r = output, c = input of one layer's 128 x 128 tile).
// The batch is not split: the sums are those of one accumulator that walks the
// rows, at 40 KB a row block, which five stages of copies keep flowing.
//
// blockIdx.x past the tiles: the bias gradients of 32 outputs (slot of dz, column
// group blockIdx.y), one lane an output, summed in row order; 16 KB a row block.
__global__ void __launch_bounds__(128, 1) mlp_dw_kernel(const __nv_bfloat16* __restrict__ act,
                                                        const __nv_bfloat16* __restrict__ dz,
                                                        const float* __restrict__ dzf, int KT, int NT, int nrb, int B,
                                                        float* __restrict__ grad, float* __restrict__ bgrad,
                                                        int* __restrict__ status, int polls) {
    extern __shared__ unsigned char mraw[];
    __shared__ __align__(8) unsigned long long full[kDwStages], read[kDwStages], done;
    __shared__ unsigned tmem_slot;
    unsigned char* buf = (unsigned char*)(((unsigned long long)mraw + 1023) & ~1023ull);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x, grp = blockIdx.y;
    if (tile >= KT + 2 + NT) {
        if (warp) return;
        const int slot = tile - (KT + 2 + NT);
        if (lane == 0) {
            for (int i = 0; i < kDwStages; ++i) bar_init1(&full[i]);
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
        __syncwarp();
        auto load = [&](int i) {
            blk_load(buf + (size_t)(i % kDwStages) * kBiasStage,
                     dzf + (((size_t)i * (3 + NT) + slot) * 4 + grp) * (128 * 32), &full[i % kDwStages], kBiasStage);
        };
        int loaded = 0;
        if (lane == 0)
            for (; loaded < nrb && loaded < kDwStages; ++loaded) load(loaded);
        float sum = 0.f;
        bool ok = true;
        int i = 0;
        for (; ok && i < nrb; ++i) {
            ok = __all_sync(0xffffffffu, mbar_wait_parity(&full[i % kDwStages], (unsigned)((i / kDwStages) & 1), polls));
            if (!ok) break;
            const float* d = (const float*)(buf + (size_t)(i % kDwStages) * kBiasStage) + lane;
            const int rows = min(128, B - i * 128);
            int r = 0;
            for (; r + 32 <= rows; r += 32) {
                float x[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) x[j] = d[(r + j) * 32];
#pragma unroll
                for (int j = 0; j < 32; ++j) sum += x[j];
            }
            for (; r < rows; ++r) sum += d[r * 32];
            __syncwarp();
            if (lane == 0 && loaded < nrb) load(loaded++);
        }
        if (ok) bgrad[slot * 128 + grp * 32 + lane] = sum;
        else if (lane == 0) {
            atomicOr(status, 1);
            for (int j = i; j < loaded; ++j)
                mbar_wait_parity(&full[j % kDwStages], (unsigned)((j / kDwStages) & 1), kMlpPolls);
        }
        return;
    }
    const int ablk = tile < KT + 2 ? tile : KT + 2;
    const int zblk = tile < KT ? 0 : (tile < KT + 2 ? tile - KT + 1 : 3 + tile - KT - 2);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&tmem_slot)),
                     "r"(32)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < kDwStages; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;\n" ::"r"(smem_addr(&full[i])) : "memory");
            bar_init1(&read[i]);
        }
        bar_init1(&done);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem = tmem_slot;
    bool ok = true;
    if (tid == 0) {
        auto load = [&](int i) {
            unsigned char* d = buf + (size_t)(i % kDwStages) * kDwStage;
            blk_load(d, dz + ((size_t)i * (3 + NT) + zblk) * kBlk, &full[i % kDwStages]);
            blk_load(d + kBlkBytes, act + ((size_t)i * (KT + 3) + ablk) * kBlk + grp * kGrp, &full[i % kDwStages],
                     kGrp * 2u);
        };
        int loaded = 0, used = 0;
        for (; loaded < nrb && loaded < kDwStages; ++loaded) load(loaded);
        for (; ok && used < nrb; ++used) {
            const int i = used;
            ok = mbar_wait_parity(&full[i % kDwStages], (unsigned)((i / kDwStages) & 1), polls);
            if (!ok) break;
            const __nv_bfloat16* d = (const __nv_bfloat16*)(buf + (size_t)(i % kDwStages) * kDwStage);
            dw_mma(d, d + kBlk, tmem, i > 0);
            mma_commit(&read[i % kDwStages]);
            // the stage that the previous row block has left takes a new one
            if (i >= 1 && loaded < nrb) {
                ok = mbar_wait_parity(&read[(i - 1) % kDwStages], (unsigned)(((i - 1) / kDwStages) & 1), polls);
                if (ok) load(loaded++);
            }
        }
        if (!ok) {
            for (int j = used; j < loaded; ++j)  // no copy may land after the CTA ends
                mbar_wait_parity(&full[j % kDwStages], (unsigned)((j / kDwStages) & 1), kMlpPolls);
        }
        mma_commit(&done);
    }
    ok = mbar_wait_drain(&done, 0, polls) && ok;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (__syncthreads_or(!ok)) {
        if (tid == 0) atomicOr(status, 1);
    } else {
        // lane = output, tensor-memory column = input: each column is a coalesced row of the tile
        float* dst = grad + (size_t)tile * kBlk + (size_t)grp * 32 * 128 + warp * 32 + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < 32; c0 += 16) {
            float v[16];
            tmem_ld16(v, tmem + ((unsigned)(warp * 32) << 16) + c0);
#pragma unroll
            for (int i = 0; i < 16; ++i) dst[(c0 + i) * 128] = v[i];
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(32) : "memory");
}

// Where parameter i lives: layer, weight (input k, output n) or bias (k = -1).
struct MlpShape {
    int n_in, n_out, KT, NT;
    long long woff[4], boff[4];
    long long nparams;
};
__device__ __forceinline__ void mlp_locate(const MlpShape& s, long long i, int& l, int& k, int& n) {
    l = i < s.woff[1] ? 0 : (i < s.woff[2] ? 1 : (i < s.woff[3] ? 2 : 3));
    const long long wo = l == 0 ? s.woff[0] : (l == 1 ? s.woff[1] : (l == 2 ? s.woff[2] : s.woff[3]));
    const long long bo = l == 0 ? s.boff[0] : (l == 1 ? s.boff[1] : (l == 2 ? s.boff[2] : s.boff[3]));
    const int out = l < 3 ? 128 : s.n_out;
    if (i >= bo) {
        k = -1;
        n = (int)(i - bo);
    } else {
        const int e = (int)(i - wo);
        k = e / out;
        n = e - k * out;
    }
}
// block index of weight (l, k, n) and its row (output) and column (input) there
__device__ __forceinline__ int mlp_block(const MlpShape& s, int l, int k, int n, int& r, int& c) {
    r = n & 127;
    c = k & 127;
    return l == 0 ? (k >> 7) : (l < 3 ? s.KT + l - 1 : s.KT + 2 + (n >> 7));
}

// BF16 weight blocks from the FP32 parameters (padding stays zero from the allocation)
__global__ void mlp_pack_kernel(MlpShape s, const float* __restrict__ w, __nv_bfloat16* __restrict__ wp) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < s.nparams; i += (long long)gridDim.x * blockDim.x) {
        int l, k, n, r, c;
        mlp_locate(s, i, l, k, n);
        if (k < 0) continue;
        const int b = mlp_block(s, l, k, n, r, c);
        wp[(size_t)b * kBlk + blk_off(r, c)] = __float2bfloat16(w[i]);
    }
}

// The gradients in parameter order and, with lr > 0, the Adam update of the
// master weights and their BF16 blocks.  Blocks 0 .. 8 tiles - 1: a thread takes
// eight inputs of one output of a weight tile, so its BF16 weights are one 16-byte
// row of a core matrix and neighbouring threads read neighbouring outputs (one
// parameter a thread, with 2-byte stores into the blocks, took 18 us for 99 k
// parameters; this way 8).  The next blocks: a thread per bias; the last sums the loss.
struct AdamArgs {
    float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ void adam_step(const AdamArgs& ad, float g, float* w, float* m, float* v) {
    const float mi = ad.b1 * *m + (1.f - ad.b1) * g;
    const float vi = ad.b2 * *v + (1.f - ad.b2) * g * g;
    *m = mi;
    *v = vi;
    *w = *w - ad.lr * (mi / ad.c1) / (sqrtf(vi / ad.c2) + ad.eps);
}
__global__ void __launch_bounds__(256) mlp_update_kernel(MlpShape s, const float* __restrict__ dw,
                                                         const float* __restrict__ bgrad,
                                                         const float* __restrict__ lossp, int nloss,
                                                         float* __restrict__ grads, float* __restrict__ w,
                                                         __nv_bfloat16* __restrict__ wp, float* __restrict__ m,
                                                         float* __restrict__ v, float* __restrict__ loss, AdamArgs ad,
                                                         const int* __restrict__ status, int* __restrict__ skipped) {
    const int ran_out = *status;
    const bool training = ad.lr > 0.f;
    const int tiles = s.KT + 2 + s.NT;
    if ((int)blockIdx.x < 8 * tiles) {
        const int tile = blockIdx.x >> 3;
        const int r = threadIdx.x & 127, c0 = ((blockIdx.x & 7) * 2 + (threadIdx.x >> 7)) * 8;
        const int l = tile < s.KT ? 0 : (tile < s.KT + 2 ? tile - s.KT + 1 : 3);
        const int k0 = (l == 0 ? tile * 128 : 0) + c0, n = (l == 3 ? (tile - s.KT - 2) * 128 : 0) + r;
        const int in = l == 0 ? s.n_in : 128, out = l == 3 ? s.n_out : 128;
        if (n >= out) return;
        const long long wo = l == 0 ? s.woff[0] : (l == 1 ? s.woff[1] : (l == 2 ? s.woff[2] : s.woff[3]));
        float g[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = dw[(size_t)tile * kBlk + (c0 + j) * 128 + r];
        float wi[8], mi[8], vi[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            wi[j] = mi[j] = vi[j] = 0.f;
            if (training && k0 + j < in) {
                const long long i = wo + (long long)(k0 + j) * out + n;
                wi[j] = w[i];
                mi[j] = m[i];
                vi[j] = v[i];
            }
        }
        if (update_skipped(ran_out, skipped, training)) return;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j >= in) continue;
            const long long i = wo + (long long)(k0 + j) * out + n;
            grads[i] = g[j];
            if (training) {
                adam_step(ad, g[j], wi + j, mi + j, vi + j);
                w[i] = wi[j];
                m[i] = mi[j];
                v[i] = vi[j];
            }
        }
        if (training) {
            __nv_bfloat162 p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = __floats2bfloat162_rn(wi[2 * j], wi[2 * j + 1]);
            *reinterpret_cast<uint4*>(wp + (size_t)tile * kBlk + blk_off(r, c0)) = *reinterpret_cast<uint4*>(p);
        }
        return;
    }
    if (blockIdx.x == gridDim.x - 1) {
        if (threadIdx.x >= 32) return;
        float t = 0.f;
        for (int i = threadIdx.x; i < nloss; i += 32) t += lossp[i];
        if (ran_out) return;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) *loss = t;
        return;
    }
    const int q = ((int)blockIdx.x - 8 * tiles) * 256 + threadIdx.x;
    if (q >= 384 + s.n_out) return;
    const int l = min(q >> 7, 3), n = q - l * 128;
    const long long i = (l == 0 ? s.boff[0] : (l == 1 ? s.boff[1] : (l == 2 ? s.boff[2] : s.boff[3]))) + n;
    const float g = bgrad[q];
    if (ran_out) return;
    grads[i] = g;
    if (training) adam_step(ad, g, w + i, m + i, v + i);
}

int grid1(long long n) { return (int)std::min<long long>((n + 255) / 256, 148LL * 8); }

}  // namespace

struct edus_mlp {
    int dims[kLayers + 1] = {0};  // n_in, H, H, H, n_out
    int device = 0;
    std::string err;
    long long nparams = 0;
    float* params = nullptr;      // FP32 master: W0 b0 W1 b1 W2 b2 W3 b3
    float* grads = nullptr;
    float* m = nullptr;
    float* v = nullptr;
    __nv_bfloat16* wbf = nullptr;  // BF16 copy (same offsets as params); the 128-wide form has wp instead
    long long woff[kLayers] = {0}, boff[kLayers] = {0};
    int step = 0;
    // activations for a batch of up to `cap` samples
    int cap = 0;
    float* z[kLayers] = {nullptr};  // pre-activations [B][dims[l+1]]
    float* a[kLayers] = {nullptr};  // GELU of the hidden pre-activations
    __nv_bfloat16* ab[kLayers + 1] = {nullptr};  // BF16 operands: ab[0] = x, ab[l] = a[l-1]
    float* da = nullptr;
    float* dz = nullptr;
    __nv_bfloat16* dzb = nullptr;
    float* loss = nullptr;
    int* status = nullptr;  // the word after loss: set when a bounded wait in a kernel ran out
    int* skipped = nullptr; // the next word: training steps left out since (update_skipped)
    struct Report {
        float loss;
        int status, skipped;
    }* report = nullptr;    // pinned: the three words, read back in one copy
    int polls = kMlpPolls;  // edus_mlp_set_wait_limit
    cudaStream_t stream = nullptr;
    // hidden width 128: weight blocks, and per 128-row block the operands of the weight gradients
    bool blocks = false;
    MlpShape shape{};
    __nv_bfloat16* wp = nullptr;
    int cap_rb = 0;               // row blocks the buffers below hold
    __nv_bfloat16* actb = nullptr;
    __nv_bfloat16* dzblk = nullptr;
    float* dzf = nullptr;
    float* bgrad = nullptr;
    float* lossp = nullptr;
    float* dw = nullptr;          // [tiles][in 128][out 128] weight gradients
};

namespace {

thread_local std::string g_mlp_create_error;

int mfail(edus_mlp* m, int code, const std::string& msg) {
    if (m) m->err = msg;
    else g_mlp_create_error = msg;
    return code;
}
#define MCU(m, call)                                                                                              \
    do {                                                                                                          \
        cudaError_t e_ = (call);                                                                                  \
        if (e_ != cudaSuccess) return mfail(m, EDUS_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// Wait for the stream's work; its loss, and a report (cleared) of a wait that ran out.
int mlp_finish(edus_mlp* m, float* loss_host) {
    MCU(m, cudaMemcpyAsync(m->report, m->loss, sizeof(*m->report), cudaMemcpyDeviceToHost, m->stream));
    MCU(m, cudaStreamSynchronize(m->stream));
    if (loss_host) *loss_host = m->report->loss;
    if (m->report->status) {
        // every step since the wait ran out was left out, those before a new set of parameters among them
        m->step = std::max(0, m->step - m->report->skipped);
        MCU(m, cudaMemset(m->status, 0, 2 * sizeof(int)));
        return mfail(m, EDUS_ERR_TIMEOUT,
                     "a bounded wait of a network kernel ran out; training steps left out, weights as before them: " +
                         std::to_string(m->report->skipped));
    }
    return EDUS_OK;
}

// Buffers of the 128-wide path for B rows.
int ensure_blocks(edus_mlp* m, int B) {
    const int nrb = (B + 127) / 128;
    if (nrb <= m->cap_rb) return EDUS_OK;
    const int KT = m->shape.KT, NT = m->shape.NT;
    MCU(m, cudaStreamSynchronize(m->stream));
    for (void* p : {(void*)m->actb, (void*)m->dzblk, (void*)m->dzf, (void*)m->lossp}) cudaFree(p);
    m->actb = m->dzblk = nullptr;
    m->dzf = m->lossp = nullptr;
    m->cap_rb = 0;
    MCU(m, cudaMalloc((void**)&m->actb, (size_t)nrb * (KT + 3) * kBlkBytes));
    MCU(m, cudaMalloc((void**)&m->dzblk, (size_t)nrb * (3 + NT) * kBlkBytes));
    MCU(m, cudaMalloc((void**)&m->dzf, (size_t)nrb * (3 + NT) * kBlk * sizeof(float)));
    MCU(m, cudaMalloc((void**)&m->lossp, (size_t)nrb * kTeam * sizeof(float)));
    if (!m->dw) MCU(m, cudaMalloc((void**)&m->dw, (size_t)(KT + 2 + NT) * kBlk * sizeof(float)));
    if (!m->bgrad) MCU(m, cudaMalloc((void**)&m->bgrad, (size_t)(3 + NT) * 128 * sizeof(float)));
    m->cap_rb = nrb;
    return EDUS_OK;
}

MlpRowsArgs rows_args(edus_mlp* m, int B, const float* x, const float* t, float* y) {
    MlpRowsArgs a{};
    a.B = B;
    a.n_in = m->shape.n_in;
    a.n_out = m->shape.n_out;
    a.KT = m->shape.KT;
    a.NT = m->shape.NT;
    a.x = x;
    a.t = t;
    a.y = y;
    a.wp = m->wp;
    for (int l = 0; l < kLayers; ++l) a.bias[l] = m->params + m->boff[l];
    a.act = m->actb;
    a.dz = m->dzblk;
    a.dzf = m->dzf;
    a.lossp = m->lossp;
    a.scale = 1.f / (float)((long long)B * a.n_out);
    a.status = m->status;
    a.polls = m->polls;
    return a;
}

// Loss and gradients of the batch and, with lr > 0, an Adam step.
int blocks_backward(edus_mlp* m, int B, const float* x, const float* t, float lr, float c1, float c2) {
    int rc;
    if ((rc = ensure_blocks(m, B))) return rc;
    const int nrb = (B + 127) / 128, tiles = m->shape.KT + 2 + m->shape.NT;
    mlp_rows_kernel<true><<<kTeam * nrb, 512, kRowsSmem, m->stream>>>(rows_args(m, B, x, t, nullptr));
    mlp_dw_kernel<<<dim3(tiles + 3 + m->shape.NT, 4), 128, kDwSmem, m->stream>>>(
        m->actb, m->dzblk, m->dzf, m->shape.KT, m->shape.NT, nrb, B, m->dw, m->bgrad, m->status, m->polls);
    mlp_update_kernel<<<8 * tiles + (384 + m->shape.n_out + 255) / 256 + 1, 256, 0, m->stream>>>(
        m->shape, m->dw, m->bgrad, m->lossp, kTeam * nrb, m->grads, m->params, m->wp, m->m, m->v, m->loss,
        AdamArgs{lr, 0.9f, 0.999f, 1e-8f, c1, c2}, m->status, m->skipped);
    MCU(m, cudaGetLastError());
    return EDUS_OK;
}

void gemm(edus_mlp* mm, int M, int N, int K, const __nv_bfloat16* A, long long a_rs, long long a_cs,
          const __nv_bfloat16* B, long long b_rs, long long b_cs, float* C, int ldc, const float* bias) {
    dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
    gemm_bf16_kernel<<<grid, 128, 0, mm->stream>>>(M, N, K, A, a_rs, a_cs, B, b_rs, b_cs, C, ldc, bias, 0,
                                                   mm->status, mm->polls);
}

int ensure_cap(edus_mlp* m, int B) {
    if (B <= m->cap) return EDUS_OK;
    for (int l = 0; l < kLayers; ++l) {
        cudaFree(m->z[l]);
        cudaFree(m->a[l]);
        m->z[l] = m->a[l] = nullptr;
    }
    for (int l = 0; l <= kLayers; ++l) {
        cudaFree(m->ab[l]);
        m->ab[l] = nullptr;
    }
    cudaFree(m->da);
    cudaFree(m->dz);
    cudaFree(m->dzb);
    m->da = m->dz = nullptr;
    m->dzb = nullptr;
    m->cap = 0;
    int wmax = 0;
    for (int l = 0; l <= kLayers; ++l) wmax = std::max(wmax, m->dims[l]);
    for (int l = 0; l < kLayers; ++l) {
        MCU(m, cudaMalloc((void**)&m->z[l], (size_t)B * m->dims[l + 1] * sizeof(float)));
        MCU(m, cudaMalloc((void**)&m->a[l], (size_t)B * m->dims[l + 1] * sizeof(float)));
    }
    for (int l = 0; l <= kLayers; ++l)
        MCU(m, cudaMalloc((void**)&m->ab[l], (size_t)B * m->dims[l] * sizeof(__nv_bfloat16)));
    MCU(m, cudaMalloc((void**)&m->da, (size_t)B * wmax * sizeof(float)));
    MCU(m, cudaMalloc((void**)&m->dz, (size_t)B * wmax * sizeof(float)));
    MCU(m, cudaMalloc((void**)&m->dzb, (size_t)B * wmax * sizeof(__nv_bfloat16)));
    m->cap = B;
    return EDUS_OK;
}

// forward pass of B samples x (device FP32 [B][n_in]); output in z[kLayers-1]
void forward(edus_mlp* m, int B, const float* x) {
    to_bf16_kernel<<<grid1((long long)B * m->dims[0]), 256, 0, m->stream>>>(x, m->ab[0], (long long)B * m->dims[0]);
    for (int l = 0; l < kLayers; ++l) {
        const int in = m->dims[l], out = m->dims[l + 1];
        gemm(m, B, out, in, m->ab[l], in, 1, m->wbf + m->woff[l], out, 1, m->z[l], out, m->params + m->boff[l]);
        if (l < kLayers - 1)
            gelu_kernel<<<grid1((long long)B * out), 256, 0, m->stream>>>(m->z[l], m->a[l], m->ab[l + 1],
                                                                          (long long)B * out);
    }
}

// gradients of the mean squared error into m->grads (the loss into m->loss)
void backward(edus_mlp* m, int B, const float* target) {
    const int nout = m->dims[kLayers];
    const long long n = (long long)B * nout;
    cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream);
    mse_kernel<<<grid1(n), 256, 0, m->stream>>>(m->z[kLayers - 1], target, m->dz, m->dzb, n, 1.f / (float)n, m->loss);
    for (int l = kLayers - 1; l >= 0; --l) {
        const int in = m->dims[l], out = m->dims[l + 1];
        // dW = a_{l-1}^T dz : [in][B] x [B][out]
        gemm(m, in, out, B, m->ab[l], 1, in, m->dzb, out, 1, m->grads + m->woff[l], out, nullptr);
        colsum_kernel<<<(out + 127) / 128, 128, 0, m->stream>>>(m->dz, m->grads + m->boff[l], B, out);
        if (l == 0) break;
        // da_{l-1} = dz W^T : [B][out] x [out][in]
        gemm(m, B, in, out, m->dzb, out, 1, m->wbf + m->woff[l], 1, out, m->da, in, nullptr);
        gelu_back_kernel<<<grid1((long long)B * in), 256, 0, m->stream>>>(m->da, m->z[l - 1], m->dz, m->dzb,
                                                                          (long long)B * in);
    }
}

}  // namespace

extern "C" {

int edus_mlp_create(int n_in, int n_hidden, int n_out, unsigned long long seed, int device, edus_mlp** out) {
    if (!out || n_in < 1 || n_hidden < 1 || n_out < 1) return mfail(nullptr, EDUS_ERR_ARG, "bad MLP sizes");
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) return mfail(nullptr, EDUS_ERR_CUDA, "cudaSetDevice failed");
    edus_mlp* m = new edus_mlp();
    m->device = device;
    m->dims[0] = n_in;
    for (int l = 1; l < kLayers; ++l) m->dims[l] = n_hidden;
    m->dims[kLayers] = n_out;
    long long off = 0;
    for (int l = 0; l < kLayers; ++l) {
        m->woff[l] = off;
        off += (long long)m->dims[l] * m->dims[l + 1];
        m->boff[l] = off;
        off += m->dims[l + 1];
    }
    m->nparams = off;
    m->blocks = n_hidden == 128;
    if (m->blocks) {
        m->shape.n_in = n_in;
        m->shape.n_out = n_out;
        m->shape.KT = (n_in + 127) / 128;
        m->shape.NT = (n_out + 127) / 128;
        m->shape.nparams = off;
        for (int l = 0; l < kLayers; ++l) {
            m->shape.woff[l] = m->woff[l];
            m->shape.boff[l] = m->boff[l];
        }
        const size_t wb = (size_t)(m->shape.KT + 2 + m->shape.NT) * kBlkBytes;
        if (cudaMalloc((void**)&m->wp, wb) != cudaSuccess || cudaMemset(m->wp, 0, wb) != cudaSuccess ||
            cudaFuncSetAttribute(mlp_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmem) != cudaSuccess ||
            cudaFuncSetAttribute(mlp_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmem) != cudaSuccess ||
            cudaFuncSetAttribute(mlp_dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDwSmem) != cudaSuccess) {
            edus_mlp_destroy(m);
            return mfail(nullptr, EDUS_ERR_NOMEM, "MLP weight block set-up failed");
        }
    }
    // a blocking stream: ordered after the legacy stream, where callers prepare their batches
    if (cudaStreamCreate(&m->stream) != cudaSuccess ||
        cudaMalloc((void**)&m->params, off * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void**)&m->grads, off * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void**)&m->m, off * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void**)&m->v, off * sizeof(float)) != cudaSuccess ||
        (!m->blocks && cudaMalloc((void**)&m->wbf, off * sizeof(__nv_bfloat16)) != cudaSuccess) ||
        cudaMalloc((void**)&m->loss, sizeof(*m->report)) != cudaSuccess ||
        cudaMallocHost((void**)&m->report, sizeof(*m->report)) != cudaSuccess ||
        cudaMemset(m->loss, 0, sizeof(*m->report)) != cudaSuccess) {
        edus_mlp_destroy(m);
        return mfail(nullptr, EDUS_ERR_NOMEM, "MLP device allocation failed");
    }
    m->status = (int*)(m->loss + 1);
    m->skipped = m->status + 1;
    // uniform initialisation scaled by the fan-in (seeded LCG), zero biases
    std::vector<float> p(off, 0.f);
    unsigned long long s = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto uni = [&]() {
        s = s * 6364136223846793005ULL + 1442695040888963407ULL;
        return ((s >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0;
    };
    for (int l = 0; l < kLayers; ++l) {
        const double a = std::sqrt(3.0 / m->dims[l]) * (l < kLayers - 1 ? std::sqrt(2.0) : 1.0);
        for (long long i = 0; i < (long long)m->dims[l] * m->dims[l + 1]; ++i) p[m->woff[l] + i] = (float)(a * uni());
    }
    const int rc = edus_mlp_set_params(m, p.data());
    if (rc) {
        g_mlp_create_error = m->err;
        edus_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return EDUS_OK;
}

int edus_mlp_destroy(edus_mlp* m) {
    if (!m) return EDUS_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->params);
    cudaFree(m->grads);
    cudaFree(m->m);
    cudaFree(m->v);
    cudaFree(m->wbf);
    cudaFree(m->loss);
    if (m->report) cudaFreeHost(m->report);
    for (void* p : {(void*)m->wp, (void*)m->actb, (void*)m->dzblk, (void*)m->dzf, (void*)m->bgrad, (void*)m->lossp, (void*)m->dw})
        cudaFree(p);
    for (int l = 0; l < kLayers; ++l) {
        cudaFree(m->z[l]);
        cudaFree(m->a[l]);
    }
    for (int l = 0; l <= kLayers; ++l) cudaFree(m->ab[l]);
    cudaFree(m->da);
    cudaFree(m->dz);
    cudaFree(m->dzb);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return EDUS_OK;
}

const char* edus_mlp_last_error(const edus_mlp* m) { return m ? m->err.c_str() : g_mlp_create_error.c_str(); }

long long edus_mlp_param_count(const edus_mlp* m) { return m ? m->nparams : 0; }

int edus_mlp_set_params(edus_mlp* m, const float* host) {
    if (!m || !host) return EDUS_ERR_ARG;
    MCU(m, cudaSetDevice(m->device));
    MCU(m, cudaMemcpyAsync(m->params, host, m->nparams * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    if (m->blocks) mlp_pack_kernel<<<grid1(m->nparams), 256, 0, m->stream>>>(m->shape, m->params, m->wp);
    else to_bf16_kernel<<<grid1(m->nparams), 256, 0, m->stream>>>(m->params, m->wbf, m->nparams);
    MCU(m, cudaMemsetAsync(m->m, 0, m->nparams * sizeof(float), m->stream));
    MCU(m, cudaMemsetAsync(m->v, 0, m->nparams * sizeof(float), m->stream));
    m->step = 0;
    MCU(m, cudaStreamSynchronize(m->stream));
    return EDUS_OK;
}

int edus_mlp_set_wait_limit(edus_mlp* m, int polls) {
    if (!m) return EDUS_ERR_ARG;
    m->polls = polls < 0 ? kMlpPolls : polls;
    return EDUS_OK;
}

int edus_mlp_get_params(edus_mlp* m, float* host) {
    if (!m || !host) return EDUS_ERR_ARG;
    MCU(m, cudaSetDevice(m->device));
    MCU(m, cudaMemcpyAsync(host, m->params, m->nparams * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    return mlp_finish(m, nullptr);
}

int edus_mlp_forward(edus_mlp* m, int batch, const float* x, float* y) {
    if (!m || !x || !y || batch < 1) return EDUS_ERR_ARG;
    MCU(m, cudaSetDevice(m->device));
    int rc;
    if (m->blocks) {
        mlp_rows_kernel<false><<<kTeam * ((batch + 127) / 128), 512, kRowsSmem, m->stream>>>(
            rows_args(m, batch, x, nullptr, y));
    } else {
        if ((rc = ensure_cap(m, batch))) return rc;
        forward(m, batch, x);
        MCU(m, cudaMemcpyAsync(y, m->z[kLayers - 1], (size_t)batch * m->dims[kLayers] * sizeof(float),
                               cudaMemcpyDeviceToDevice, m->stream));
    }
    MCU(m, cudaGetLastError());
    return mlp_finish(m, nullptr);
}

int edus_mlp_gradients(edus_mlp* m, int batch, const float* x, const float* target, float* grads_host,
                       float* loss_host) {
    if (!m || !x || !target || batch < 1) return EDUS_ERR_ARG;
    MCU(m, cudaSetDevice(m->device));
    int rc;
    if (m->blocks) {
        if ((rc = blocks_backward(m, batch, x, target, 0.f, 1.f, 1.f))) return rc;
    } else {
        if ((rc = ensure_cap(m, batch))) return rc;
        forward(m, batch, x);
        backward(m, batch, target);
    }
    MCU(m, cudaGetLastError());
    if (grads_host)
        MCU(m, cudaMemcpyAsync(grads_host, m->grads, m->nparams * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    return mlp_finish(m, loss_host);
}

int edus_mlp_train_step(edus_mlp* m, int batch, const float* x, const float* target, float lr, float* loss_host) {
    if (!m || !x || !target || batch < 1 || !(lr > 0.f)) return EDUS_ERR_ARG;
    MCU(m, cudaSetDevice(m->device));
    int rc;
    if ((rc = m->blocks ? ensure_blocks(m, batch) : ensure_cap(m, batch))) return rc;
    m->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)m->step), c2 = 1.f - std::pow(b2, (float)m->step);
    if (m->blocks) {
        if ((rc = blocks_backward(m, batch, x, target, lr, c1, c2))) return rc;
    } else {
        forward(m, batch, x);
        backward(m, batch, target);
        adam_kernel<<<grid1(m->nparams), 256, 0, m->stream>>>(m->params, m->wbf, m->grads, m->m, m->v, m->nparams, lr,
                                                              b1, b2, 1e-8f, c1, c2, m->status, m->skipped);
    }
    MCU(m, cudaGetLastError());
    return loss_host ? mlp_finish(m, loss_host) : EDUS_OK;
}

}  // extern "C"
