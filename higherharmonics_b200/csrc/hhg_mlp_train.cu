// hhg_mlp_train.cu -- training of the step-size proposer on the tensor cores.
//
// Every GEMM of the forward and backward pass is a 128-row tile on the
// 5th-generation tensor cores: operands staged by the CTA's threads into
// shared memory in the canonical K-major layout without swizzle (8-row x
// 16-byte core matrices), one elected thread issues tcgen05.mma (kind::f16,
// BF16 inputs, FP32 accumulation in tensor memory) for each K = 16 slice,
// tcgen05.commit arrives on an mbarrier, and each warp reads its 32
// accumulator rows back with tcgen05.ld.  All waits are bounded; on a
// timeout the kernel raises an error flag, waits (bounded) for the MMAs it
// issued, frees its tensor memory and returns.
//
//   forward     Z_l = H_{l-1} W_l^T + b_l,  H_l = SiLU(Z_l)        (M = rows, N = 64)
//   output      y = H_3 w_4 + b_4, loss = mean (y - T)^2           (CUDA cores, 64 -> 1)
//   data grad   dH_{l-1} = dZ_l W_l,  dZ_{l-1} = dH_{l-1} SiLU'(Z_{l-1})  (N = 64)
//   weight grad dW_l = dZ_l^T H_{l-1} over the tile's 128 rows, M padded to 128
//   Adam on FP32 master weights, then BF16 copies [n][k] and [k][n].
//
// One kernel carries a tile through all of it (mlp_step_kernel); the
// optimiser is the only other launch of a step.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/hhg_gpu.h"
#include "hhg_device.cuh"

namespace {

using bf16 = __nv_bfloat16;
constexpr int kH = hhg::kMlpH;          // 64
constexpr int kIn = hhg::kMlpIn;        // 8
constexpr int kInPad = hhg::kMlpInPad;  // 16
constexpr int kRows = 128;              // rows per tile (M)
constexpr long long kSpin = 1ll << 24;  // bounded mbarrier polls

// FP32 master parameters on the device (the first layer's inputs padded to 16)
constexpr int kOffW1 = 0;                      // [64][16]
constexpr int kOffB1 = kOffW1 + kH * kInPad;   // [64]
constexpr int kOffW2 = kOffB1 + kH;            // [64][64]
constexpr int kOffB2 = kOffW2 + kH * kH;
constexpr int kOffW3 = kOffB2 + kH;            // [64][64]
constexpr int kOffB3 = kOffW3 + kH * kH;
constexpr int kOffW4 = kOffB3 + kH;            // [64]
constexpr int kOffB4 = kOffW4 + kH;            // [1]
constexpr int kNMaster = kOffB4 + 1;
// the ABI layout of hhg_mlp::params (first layer unpadded)
constexpr int aW1 = 0, aB1 = aW1 + kH * kIn, aW2 = aB1 + kH, aB2 = aW2 + kH * kH, aW3 = aB2 + kH,
              aB3 = aW3 + kH * kH, aW4 = aB3 + kH, aB4 = aW4 + kH;
static_assert(aB4 + 1 == HHG_MLP_N_PARAMS, "hhg_mlp parameter layout");

// ---------------------------------------------------------------------------
// tcgen05 / mbarrier primitives (PTX ISA 8.7, sm_100a)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor, K-major, no swizzle: start, leading byte
// offset (between the two 8-element K chunks of a K = 16 slice), stride byte
// offset (between 8-row groups), version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor: D f32, A/B bf16, both K-major, M = 128, N.
__host__ __device__ constexpr uint32_t umma_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void umma_commit(uint64_t *mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :
                 : "r"(smem_u32(mbar))
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t *mbar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" : : "r"(smem_u32(mbar)), "r"(count) : "memory");
}

// Bounded wait for phase `parity`; true when it completed.
__device__ __forceinline__ bool mbar_wait(uint64_t *mbar, uint32_t parity) {
    const uint32_t a = smem_u32(mbar);
    for (long long it = 0; it < kSpin; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, int ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :
                 : "r"(smem_u32(dst_smem)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, int ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" : : "r"(taddr), "r"(ncols) : "memory");
}

// 32 lanes x 8 consecutive FP32 columns starting at taddr (one warp).
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// The reverse of tmem_ld8 (the caller orders it before later reads).
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :
                 : "r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])),
                   "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])),
                   "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
                 : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Byte offset of element (row, k) in a canonical K-major no-swizzle tile with
// `rows` rows: core matrix (row / 8, k / 8) at ((k / 8) * rows / 8 + row / 8) *
// 128, row (row % 8) at 16 B, element (k % 8) at 2 B.  LBO (next K chunk) =
// rows * 16, SBO (next row group) = 128.
__device__ __forceinline__ uint32_t kmaj_off(int row, int k, int rows) {
    return (uint32_t)((((k >> 3) * (rows >> 3) + (row >> 3)) << 7) + ((row & 7) << 4) + ((k & 7) << 1));
}

// SiLU(z) = z / (1 + e^-z) and SiLU'(z) = s (1 + z (1 - s)), s = 1 / (1 + e^-z)
__device__ __forceinline__ float silu_f(float z, float &ds) {
    const float d = 1.0f + __expf(-z), s = __frcp_rn(d);
    ds = s * (1.0f + z * (1.0f - s));
    return z / d;
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// Records -> standardised BF16 inputs X [n x 16] and FP32 targets.
struct Norm {
    float mu[kIn], isig[kIn];
    float out_mu, out_isig;
};
__global__ void mlp_prepare_kernel(const float *rec, int stride, long long n, const Norm nm, bf16 *X,
                                   float *T) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *r = rec + i * stride;
#pragma unroll
    for (int c = 0; c < kInPad; ++c)
        X[i * kInPad + c] = __float2bfloat16_rn(c < kIn ? (r[c] - nm.mu[c]) * nm.isig[c] : 0.0f);
    T[i] = (r[kIn] - nm.out_mu) * nm.out_isig;
}

// The BF16 copies of the weights that the tensor cores read: W [out][in] for
// the forward products, W^T [in][out] for the data gradients.
struct Weights {
    bf16 w1[kH * kInPad], w2[kH * kH], w2t[kH * kH], w3[kH * kH], w3t[kH * kH];
};

__device__ __forceinline__ void store_bf16(Weights *W, int i, float p) {
    const bf16 v = __float2bfloat16_rn(p);
    if (i < kOffB1) {
        W->w1[i - kOffW1] = v;
    } else if (i >= kOffW2 && i < kOffB2) {
        const int q = i - kOffW2;
        W->w2[q] = v;
        W->w2t[(q % kH) * kH + q / kH] = v;
    } else if (i >= kOffW3 && i < kOffB3) {
        const int q = i - kOffW3;
        W->w3[q] = v;
        W->w3t[(q % kH) * kH + q / kH] = v;
    }
}

__global__ void to_bf16_kernel(const float *P, Weights *W) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kNMaster) store_bf16(W, i, P[i]);
}

// ---------------------------------------------------------------------------
// One pass over a batch: forward, output layer, loss and (GRAD) the whole
// backward pass, or (!GRAD) the predicted levels.
//
// A batch of 4096 rows is 0.2 GFLOP: what bounds a training step is not the
// tensor cores but the number of dependent launches and round trips through
// memory.  As one kernel per layer and direction, with the activations and
// pre-activations in global memory and the batch sums in shared-memory
// atomics, a step took 12 launches and ~450 us.  Here a CTA carries its
// 128-row tiles through every layer: the pre-activations, and from the forward
// pass on the SiLU' that the backward pass needs, stay in tensor memory, the
// activations in shared memory in the two orders the products read them in
// (K-major by unit for the next layer, K-major by row for the weight
// gradient), the weight gradients accumulate in tensor memory over the CTA's
// tiles, and each CTA leaves one row of partial sums that the optimiser adds
// in a fixed order: 2 launches a step, and a run is reproducible bit for bit.
//
// 512 threads: the four warps w, w + 4, ... share the accumulator lanes (rows)
// 32 (w mod 4) .. + 31 and take 16 columns each.  The element-wise work is one
// chain of exponential, reciprocal and stores per value: with 8 warps and the
// column loops unrolled the kernel waited for instructions and latencies (42
// us a launch at 4096 rows, 15 % issue); 16 warps over rolled loops of 8
// columns take 23 us (cold caches), the optimiser 6 us.
// ---------------------------------------------------------------------------
constexpr int kStepThreads = 512;
constexpr int kColParts = kStepThreads / kRows;  // threads a row
// tensor-memory columns
constexpr int kColZ1 = 0, kColDH = 192, kColW1 = 256, kTmemCols = 512;  // Z and dW: 64 a layer

struct StepSmem {
    // A operands [128 rows][K] and B operands [N rows][K] of the products
    alignas(128) unsigned char x[kRows * kInPad * 2];     // A: X, K = inputs
    alignas(128) unsigned char xt[kInPad * kRows * 2];    // B: X^T, K = rows
    alignas(128) unsigned char h1[kRows * kH * 2], h2[kRows * kH * 2];     // A, K = units
    alignas(128) unsigned char h1t[kH * kRows * 2], h2t[kH * kRows * 2];   // B, K = rows
    alignas(128) unsigned char h3t[kH * kRows * 2];       // H3^T, read by the dw4 sums
    alignas(128) unsigned char dz[kRows * kH * 2];        // A: dZ, K = units
    alignas(128) unsigned char dzt[kRows * kRows * 2];    // A: dZ^T, units 64 .. 127 zero, K = rows
    alignas(128) unsigned char w1[kH * kInPad * 2], w2[kH * kH * 2], w3[kH * kH * 2];
    alignas(128) unsigned char w2t[kH * kH * 2], w3t[kH * kH * 2];
    float b[3][kH], w4[kH];
    float y[kRows], gy[kRows], t[kRows];
    float dw4[kH], db[3][kH], red[2][kStepThreads / 32];
    uint64_t mbar;
    uint32_t taddr;
};

// [N][K] BF16 matrix in global memory -> canonical K-major tile, 16 bytes a thread.
template <int N, int K>
__device__ __forceinline__ void stage_weights(unsigned char *dst, const bf16 *src) {
    for (int c = threadIdx.x; c < N * K / 8; c += kStepThreads) {
        const int row = c / (K / 8), kc = c % (K / 8);
        *reinterpret_cast<uint4 *>(dst + kmaj_off(row, 8 * kc, N)) =
            *reinterpret_cast<const uint4 *>(src + row * K + 8 * kc);
    }
}

// Issue the K / 16 MMAs of one product (A: 128 x K, B: N x K, canonical) into
// the columns at taddr (one thread).
__device__ __forceinline__ void issue_product(const unsigned char *sA, const unsigned char *sB, int K,
                                              int N, uint32_t taddr, bool accumulate) {
    const uint32_t a0 = smem_u32(sA), b0 = smem_u32(sB);
    const uint32_t idesc = umma_idesc(N);
#pragma unroll 1
    for (int ks = 0; ks < K / 16; ++ks) {
        // K slice ks = chunks 2ks, 2ks+1
        const uint64_t da = umma_desc(a0 + (uint32_t)(2 * ks) * (kRows * 16), kRows * 16, 128);
        const uint64_t db = umma_desc(b0 + (uint32_t)(2 * ks) * (N * 16), N * 16, 128);
        umma_f16(taddr, da, db, idesc, (accumulate || ks > 0) ? 1u : 0u);
    }
}

// The CTA's shared-memory operands and tensor-memory reads before this point
// are visible to the products thread 0 issues after it.
__device__ __forceinline__ void before_products() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Eight values of a row, columns col .. col + 7, into a K-major [128][64]
// tile (kmaj, unless null) and transposed into a [rows_t][128] tile (K = rows).
__device__ __forceinline__ void put8(unsigned char *kmaj, unsigned char *trans, int rows_t, int row,
                                     int col, const float *v) {
    uint4 w;
    __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&w);
#pragma unroll
    for (int c = 0; c < 4; ++c) p[c] = __floats2bfloat162_rn(v[2 * c], v[2 * c + 1]);
    if (kmaj) *reinterpret_cast<uint4 *>(kmaj + kmaj_off(row, col, kRows)) = w;
    const bf16 *e = reinterpret_cast<const bf16 *>(&w);
    unsigned char *t = trans + kmaj_off(col, row, rows_t);  // col is a multiple of 8: 16 bytes a unit
#pragma unroll
    for (int c = 0; c < 8; ++c) *reinterpret_cast<bf16 *>(t + 16 * c) = e[c];
}

// Sum over the tile's rows of unit u of a [rows_t][128] K-major tile (times
// gy with GY): eight threads a unit, 16 rows each.
template <bool GY>
__device__ __forceinline__ float unit_sum(const StepSmem &S, const unsigned char *tile, int rows_t) {
    const int u = threadIdx.x >> 3, part = threadIdx.x & 7;
    float acc = 0.0f;
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
        const int r0 = 16 * part + 8 * q;
        const uint4 w = *reinterpret_cast<const uint4 *>(tile + kmaj_off(u, r0, rows_t));
        const bf16 *e = reinterpret_cast<const bf16 *>(&w);
#pragma unroll
        for (int c = 0; c < 8; ++c) acc += GY ? S.gy[r0 + c] * __bfloat162float(e[c]) : __bfloat162float(e[c]);
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    acc += __shfl_xor_sync(0xffffffffu, acc, 4);
    return acc;
}

// perm: row i of the batch is row perm[i] of X and T (null: row i).  part:
// one row of kPartStride floats per CTA, the gradient in the master layout and
// the loss after it.  The output layer's weights are rounded to BF16 as in
// inference; targets are standardised; loss = mean (y - T)^2.
constexpr int kPartStride = (kNMaster + 1 + 31) / 32 * 32;  // partial rows start on 128 bytes
template <bool GRAD>
__global__ void __launch_bounds__(kStepThreads) mlp_step_kernel(const bf16 *X, const float *T,
                                                                const int *perm, long long n,
                                                                const Weights *W, const float *P,
                                                                float *part, float out_mu,
                                                                float out_sigma, float *y_out,
                                                                int *err) {
    extern __shared__ __align__(128) unsigned char step_dyn[];
    StepSmem &S = *reinterpret_cast<StepSmem *>(step_dyn);
    const int tid = threadIdx.x, lane = tid & 31, wq = (tid >> 5) & 3, quarter = tid >> 7;
    const int row = 32 * wq + lane;
    stage_weights<kH, kInPad>(S.w1, W->w1);
    stage_weights<kH, kH>(S.w2, W->w2);
    stage_weights<kH, kH>(S.w3, W->w3);
    if (GRAD) {
        stage_weights<kH, kH>(S.w2t, W->w2t);
        stage_weights<kH, kH>(S.w3t, W->w3t);
        // dZ^T's units 64 .. 127 and X^T's padding stay zero
        for (int i = tid; i < kRows * kRows * 2 / 16; i += kStepThreads)
            reinterpret_cast<uint4 *>(S.dzt)[i] = make_uint4(0u, 0u, 0u, 0u);
        for (int i = tid; i < kInPad * kRows * 2 / 16; i += kStepThreads)
            reinterpret_cast<uint4 *>(S.xt)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (tid < kH) {
        S.b[0][tid] = P[kOffB1 + tid];
        S.b[1][tid] = P[kOffB2 + tid];
        S.b[2][tid] = P[kOffB3 + tid];
        S.w4[tid] = __bfloat162float(__float2bfloat16_rn(P[kOffW4 + tid]));
        S.dw4[tid] = S.db[0][tid] = S.db[1][tid] = S.db[2][tid] = 0.0f;
    }
    const float b4 = P[kOffB4];
    if (tid == 0) mbar_init(&S.mbar, 1);
    if (tid < 32) tmem_alloc(&S.taddr, kTmemCols);
    before_products();
    const uint32_t tm = S.taddr;
    const uint32_t trow = tm + ((uint32_t)(32 * wq) << 16) + 16 * quarter;  // this thread's row and columns
    const long long tiles = (n + kRows - 1) / kRows;
    uint32_t phase = 0;
    bool ok = true;
    float loss = 0.0f, db4 = 0.0f;
    // waits for the products committed last; false for every thread of the CTA on a timeout
    auto wait = [&]() {
        const bool w = mbar_wait(&S.mbar, phase & 1u);
        ++phase;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return __syncthreads_and(w) != 0;
    };
    bool first = true;
    for (long long tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x, first = false) {
        const long long g = tile * kRows + row;
        if (quarter == 0) {
            uint4 a = make_uint4(0u, 0u, 0u, 0u), c = a;
            float t = 0.0f;
            if (g < n) {
                const long long r = perm ? perm[g] : g;
                const uint4 *src = reinterpret_cast<const uint4 *>(X + r * kInPad);
                a = src[0];
                c = src[1];
                if (GRAD) t = T[r];
            }
            *reinterpret_cast<uint4 *>(S.x + kmaj_off(row, 0, kRows)) = a;
            *reinterpret_cast<uint4 *>(S.x + kmaj_off(row, 8, kRows)) = c;
            S.t[row] = t;
            if (GRAD) {
                const bf16 *e = reinterpret_cast<const bf16 *>(&a);  // columns 8 .. 15 are padding
#pragma unroll
                for (int u = 0; u < kIn; ++u)
                    *reinterpret_cast<bf16 *>(S.xt + kmaj_off(u, row, kInPad)) = e[u];
            }
        }
        // the hidden layers: Z_l stays in tensor memory, H_l goes to shared memory
#pragma unroll 1
        for (int l = 0; l < 3; ++l) {
            before_products();
            if (tid == 0) {
                issue_product(l == 0 ? S.x : l == 1 ? S.h1 : S.h2, l == 0 ? S.w1 : l == 1 ? S.w2 : S.w3,
                              l == 0 ? kInPad : kH, kH, tm + kColZ1 + kH * l, false);
                umma_commit(&S.mbar);
            }
            if (!(ok = wait())) break;
            unsigned char *h = l == 0 ? S.h1 : l == 1 ? S.h2 : nullptr;
            unsigned char *ht = l == 0 ? S.h1t : l == 1 ? S.h2t : S.h3t;
#pragma unroll 1
            for (int q = 0; q < 2; ++q) {
                const int col = 16 * quarter + 8 * q;
                float v[8], ds[8];
                tmem_ld8(trow + kColZ1 + kH * l + 8 * q, v);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    v[c] = silu_f(v[c] + S.b[l][col + c], ds[c]);
                }
                if (GRAD) tmem_st8(trow + kColZ1 + kH * l + 8 * q, ds);
                put8(h, ht, kH, row, col, v);
            }
        }
        if (!ok) break;
        // the output layer: the row's dot product in the order of the columns,
        // handed on from quarter to quarter
#pragma unroll 1
        for (int qd = 0; qd < kColParts; ++qd) {
            if (quarter == qd) {
                float ys = qd == 0 ? b4 : S.y[row];
#pragma unroll
                for (int c = 0; c < kH / kColParts; ++c) {
                    const int col = (kH / kColParts) * qd + c;
                    ys += __bfloat162float(*reinterpret_cast<const bf16 *>(S.h3t + kmaj_off(col, row, kH))) * S.w4[col];
                }
                S.y[row] = ys;
            }
            __syncthreads();
        }
        const float y = S.y[row];
        if constexpr (!GRAD) {
            if (quarter == 0 && g < n) y_out[g] = y * out_sigma + out_mu;
        } else {
            const float d = g < n ? y - S.t[row] : 0.0f;
            const float gy = 2.0f * d / (float)n;
            if (quarter == 0) {
                S.gy[row] = gy;
                loss += d * d / (float)n;
                db4 += gy;
            }
            // dZ_l, then the products it enters: the weight gradient of layer
            // l and the data gradient of layer l - 1
#pragma unroll 1
            for (int l = 2; l >= 0; --l) {
#pragma unroll 1
                for (int q = 0; q < 2; ++q) {
                    const int col = 16 * quarter + 8 * q;
                    float ds[8], v[8];
                    tmem_ld8(trow + kColZ1 + kH * l + 8 * q, ds);
                    if (l < 2) tmem_ld8(trow + kColDH + 8 * q, v);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        v[c] = (l == 2 ? gy * S.w4[col + c] : v[c]) * ds[c];
                    put8(l > 0 ? S.dz : nullptr, S.dzt, kRows, row, col, v);
                }
                before_products();
                if (tid == 0) {
                    if (l > 0) issue_product(S.dz, l == 2 ? S.w3t : S.w2t, kH, kH, tm + kColDH, false);
                    issue_product(S.dzt, l == 2 ? S.h2t : l == 1 ? S.h1t : S.xt, kRows, l > 0 ? kH : kInPad,
                                  tm + kColW1 + kH * l, !first);
                    umma_commit(&S.mbar);
                }
                // while they run: the column sums on the CUDA cores
                if (l == 2) {
                    const float dw4 = unit_sum<true>(S, S.h3t, kH);
                    if ((lane & 7) == 0) S.dw4[tid >> 3] += dw4;
                }
                const float db = unit_sum<false>(S, S.dzt, kRows);
                if ((lane & 7) == 0) S.db[l][tid >> 3] += db;
                if (!(ok = wait())) break;
            }
        }
    }
    if constexpr (GRAD) {
        if (ok) {
            float *out = part + (size_t)blockIdx.x * kPartStride;
            // weight gradients: accumulator lane = output unit (64 real), columns = inputs
            if (wq < 2) {
#pragma unroll 1
                for (int q = 0; q < 6; ++q) {
                    const int l = q >> 1, col = 16 * quarter + 8 * (q & 1), width = l == 0 ? kInPad : kH;
                    float v[8];
                    tmem_ld8(trow + kColW1 + kH * l + 8 * (q & 1), v);
                    if (col < width) {
                        float *o = out + (l == 0 ? kOffW1 : l == 1 ? kOffW2 : kOffW3) + row * width + col;
                        *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
                        *reinterpret_cast<float4 *>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
                    }
                }
            }
            for (int o = 16; o >= 1; o >>= 1) {
                loss += __shfl_xor_sync(0xffffffffu, loss, o);
                db4 += __shfl_xor_sync(0xffffffffu, db4, o);
            }
            if (lane == 0) {
                S.red[0][tid >> 5] = loss;
                S.red[1][tid >> 5] = db4;
            }
            __syncthreads();
            if (tid < kH) {
                out[kOffW4 + tid] = S.dw4[tid];
                out[kOffB1 + tid] = S.db[0][tid];
                out[kOffB2 + tid] = S.db[1][tid];
                out[kOffB3 + tid] = S.db[2][tid];
            }
            if (tid == 0) {
                float l = 0.0f, b = 0.0f;
                for (int w = 0; w < 4; ++w) l += S.red[0][w], b += S.red[1][w];  // quarter 0's warps
                out[kOffB4] = b;
                out[kNMaster] = l;
            }
        }
    }
    if (!ok) {
        // the MMAs may still be in flight: one more bounded wait before freeing
        if (tid == 0) atomicExch(err, 1);
        mbar_wait(&S.mbar, (phase + 1u) & 1u);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid < 32) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_dealloc(tm, kTmemCols);
    }
}

// Warp-level inference of the integration kernel on raw feature records.
__global__ void __launch_bounds__(hhg::kBlockThreads) mlp_infer_kernel(const hhg::MlpPacked *net,
                                                                       const float *rec, int stride,
                                                                       long long n, float *out) {
    extern __shared__ __align__(16) unsigned char dyn[];
    bf16 *stage = reinterpret_cast<bf16 *>(dyn);
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long i = (blockIdx.x * (long long)hhg::kWarpsPerBlock + wib) * 32 + lane;
    float f[kIn];
#pragma unroll
    for (int c = 0; c < kIn; ++c) f[c] = i < n ? rec[i * stride + c] : 0.0f;
    const float T = hhg::mlp_warp_infer(net, f, stage + wib * hhg::kMlpWarpStage);
    if (i < n) out[i] = T;
}

// Gradient (and loss) = the CTAs' partial rows added in CTA order.
__device__ __forceinline__ float sum_partials(const float *part, int rows, int i) {
    float g = 0.0f;
#pragma unroll 8
    for (int c = 0; c < rows; ++c) g += part[(size_t)c * kPartStride + i];
    return g;
}

__global__ void gradient_kernel(const float *part, int rows, float *g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= kNMaster) g[i] = sum_partials(part, rows, i);
}

// Adam on the FP32 master parameters from the batch's partial gradients, then
// the BF16 copies; the thread after the last parameter adds loss_scale x the
// batch loss to *loss.
__global__ void adam_kernel(float *p, const float *part, int rows, float *m, float *v, Weights *W,
                            float lr, float b1, float b2, float eps, float bc1, float bc2,
                            float *loss, float loss_scale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > kNMaster) return;
    const float gi = sum_partials(part, rows, i);
    if (i == kNMaster) {
        *loss += gi * loss_scale;
        return;
    }
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float w = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    p[i] = w;
    store_bf16(W, i, w);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace hhg {
// hhg_mlp (ABI) -> the packed BF16 device network of the integration kernel.
void pack_mlp(const hhg_mlp &net, MlpPacked *out) {
    std::memset(out, 0, sizeof *out);
    const float *p = net.params;
    for (int o = 0; o < kH; ++o) {
        for (int i = 0; i < kIn; ++i) out->w1[o][i] = __float2bfloat16_rn(p[aW1 + o * kIn + i]);
        for (int i = kIn; i < kInPad; ++i) out->w1[o][i] = __float2bfloat16_rn(0.0f);
        for (int i = 0; i < kH; ++i) {
            out->w2[o][i] = __float2bfloat16_rn(p[aW2 + o * kH + i]);
            out->w3[o][i] = __float2bfloat16_rn(p[aW3 + o * kH + i]);
        }
        out->b1[o] = p[aB1 + o];
        out->b2[o] = p[aB2 + o];
        out->b3[o] = p[aB3 + o];
    }
    for (int r = 0; r < kMlpOutPad; ++r)
        for (int i = 0; i < kH; ++i) out->w4[r][i] = __float2bfloat16_rn(r == 0 ? p[aW4 + i] : 0.0f);
    out->b4 = p[aB4];
    out->out_mu = net.out_mu;
    out->out_sigma = net.out_sigma;
    out->level_margin = net.level_margin;
    for (int c = 0; c < kIn; ++c) {
        out->in_mu[c] = net.in_mu[c];
        out->in_isig[c] = net.in_isig[c];
    }
}
}  // namespace hhg

namespace {
void abi_to_master(const float *a, float *m) {
    std::memset(m, 0, sizeof(float) * kNMaster);
    for (int o = 0; o < kH; ++o)
        for (int i = 0; i < kIn; ++i) m[kOffW1 + o * kInPad + i] = a[aW1 + o * kIn + i];
    std::memcpy(m + kOffB1, a + aB1, sizeof(float) * kH);
    std::memcpy(m + kOffW2, a + aW2, sizeof(float) * (kH * kH + kH + kH * kH + kH + kH + 1));
}

void master_to_abi(const float *m, float *a) {
    for (int o = 0; o < kH; ++o)
        for (int i = 0; i < kIn; ++i) a[aW1 + o * kIn + i] = m[kOffW1 + o * kInPad + i];
    std::memcpy(a + aB1, m + kOffB1, sizeof(float) * kH);
    std::memcpy(a + aW2, m + kOffW2, sizeof(float) * (kH * kH + kH + kH * kH + kH + kH + 1));
}

Norm make_norm(const hhg_mlp &net) {
    Norm nm{};
    for (int c = 0; c < kIn; ++c) {
        nm.mu[c] = net.in_mu[c];
        nm.isig[c] = net.in_isig[c];
    }
    nm.out_mu = net.out_mu;
    nm.out_isig = 1.0f / net.out_sigma;
    return nm;
}

uint64_t splitmix64(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Device buffers of one training / evaluation session: slices of one
// allocation (one for each cost 1.0 ms of cudaMalloc and 0.9 ms of cudaFree a
// call at 262144 records), sized by a first pass over the same requests and freed on scope exit.
struct Session {
    unsigned char *base = nullptr;
    size_t used = 0;
    template <typename T>
    void alloc(T *&p, size_t n) {
        p = base ? reinterpret_cast<T *>(base + used) : nullptr;
        used += (n * sizeof(T) + 255) / 256 * 256;
    }
    // `request` names every buffer of the session; it runs twice
    template <class F>
    cudaError_t build(F request) {
        request();
        const cudaError_t e = cudaMalloc(&base, used);
        if (e != cudaSuccess) return e;
        used = 0;
        request();
        return cudaSuccess;
    }
    ~Session() { cudaFree(base); }
};

// Parameters, their BF16 copies and the partial gradients of one session.
struct Net {
    float *P = nullptr, *m = nullptr, *v = nullptr, *part = nullptr;
    Weights *W = nullptr;
    int *err = nullptr;
    int max_ctas = 1;
    cudaError_t init(bool grad) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&max_ctas, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = grad ? cudaFuncSetAttribute(mlp_step_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)sizeof(StepSmem))
                     : cudaFuncSetAttribute(mlp_step_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)sizeof(StepSmem));
        return e;
    }
    // grad_rows: rows of a gradient batch (0: no gradients); one row of partial
    // sums per CTA of its launch (a row for every SM is 5 MB, mapped and unmapped
    // on each call: 0.73 ms instead of 0.09 for the gradient of 100 records)
    void request(Session &S, long long grad_rows, bool optimiser) {
        S.alloc(P, kNMaster);
        if (optimiser) {
            S.alloc(m, kNMaster);
            S.alloc(v, kNMaster);
        }
        if (grad_rows > 0) S.alloc(part, (size_t)ctas(grad_rows) * kPartStride);
        S.alloc(W, 1);
        S.alloc(err, 1);
    }
    // one CTA per SM at most (the step's shared and tensor memory)
    int ctas(long long n) const {
        return (int)std::min<long long>((n + kRows - 1) / kRows, max_ctas);
    }
    void weights_bf16(cudaStream_t s) const {
        to_bf16_kernel<<<(kNMaster + 255) / 256, 256, 0, s>>>(P, W);
    }
    void gradients(const bf16 *X, const float *T, const int *perm, long long n, cudaStream_t s) const {
        mlp_step_kernel<true><<<ctas(n), kStepThreads, sizeof(StepSmem), s>>>(X, T, perm, n, W, P, part,
                                                                              0.0f, 1.0f, nullptr, err);
    }
    void predict(const bf16 *X, long long n, float out_mu, float out_sigma, float *y, cudaStream_t s) const {
        mlp_step_kernel<false><<<ctas(n), kStepThreads, sizeof(StepSmem), s>>>(
            X, nullptr, nullptr, n, W, P, nullptr, out_mu, out_sigma, y, err);
    }
};

hhg_status fail(hhg_status st, const char *what, cudaError_t e, std::string *msg) {
    if (msg) *msg = std::string(what) + (e != cudaSuccess ? std::string(": ") + cudaGetErrorString(e) : "");
    return st;
}

bool check_net(const hhg_mlp *net) {
    if (!net || !(net->out_sigma > 0.0f) || !std::isfinite(net->out_sigma)) return false;
    for (int c = 0; c < kIn; ++c)
        if (!std::isfinite(net->in_mu[c]) || !std::isfinite(net->in_isig[c])) return false;
    return true;
}
}  // namespace

// Internal entry points used by the C ABI (hhg_gpu.cu owns the context).
namespace hhg {
hhg_status mlp_train_impl(cudaStream_t s, const float *records, int64_t n, const hhg_train_opts &o,
                          hhg_mlp *net, float *epoch_loss, double *train_ms, std::string *msg) {
    if (!records || !net || n < kRows) return fail(HHG_BAD_CONFIG, "need at least 128 records and a network", cudaSuccess, msg);
    if (!check_net(net)) return fail(HHG_BAD_CONFIG, "network standardisation not set (hhg_mlp_init)", cudaSuccess, msg);
    if (o.epochs < 1 || o.batch < kRows || o.batch % kRows != 0 || !(o.lr > 0.0f))
        return fail(HHG_BAD_CONFIG, "epochs >= 1, batch a multiple of 128, lr > 0", cudaSuccess, msg);
    if (n > (int64_t)1 << 30) return fail(HHG_BAD_CONFIG, "at most 2^30 records", cudaSuccess, msg);
    const long long B = std::min<long long>(o.batch, n / kRows * kRows);
    const long long nb = n / B;
    Session S;
    Net W;
    float *d_rec = nullptr, *T = nullptr, *d_loss = nullptr;
    bf16 *X = nullptr;
    int *perm = nullptr;
    cudaError_t e = W.init(true);
    if (e == cudaSuccess)
        e = S.build([&] {
            W.request(S, B, true);
            S.alloc(d_rec, (size_t)n * HHG_HIST_FIELDS);
            S.alloc(X, (size_t)n * kInPad);
            S.alloc(T, (size_t)n);
            S.alloc(perm, (size_t)n);
            S.alloc(d_loss, (size_t)o.epochs);
        });
    if (e != cudaSuccess) return fail(HHG_CUDA_ERROR, "alloc training buffers", e, msg);
    std::vector<float> master(kNMaster);
    abi_to_master(net->params, master.data());
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEventCreate(&ev0);
    cudaEventCreate(&ev1);
    cudaEventRecord(ev0, s);
    cudaMemcpyAsync(d_rec, records, sizeof(float) * n * HHG_HIST_FIELDS, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(W.P, master.data(), sizeof(float) * kNMaster, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(W.m, 0, sizeof(float) * kNMaster, s);
    cudaMemsetAsync(W.v, 0, sizeof(float) * kNMaster, s);
    cudaMemsetAsync(W.err, 0, sizeof(int), s);
    cudaMemsetAsync(d_loss, 0, sizeof(float) * o.epochs, s);
    mlp_prepare_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_rec, HHG_HIST_FIELDS, n, make_norm(*net), X, T);
    W.weights_bf16(s);
    std::vector<int> hp(n);
    for (long long i = 0; i < n; ++i) hp[i] = (int)i;
    uint64_t rng = o.seed;
    const double total = (double)o.epochs * nb;
    long long step = 0;
    for (int ep = 0; ep < o.epochs; ++ep) {
        for (long long i = n - 1; i > 0; --i) std::swap(hp[i], hp[splitmix64(rng) % (uint64_t)(i + 1)]);
        if ((e = cudaMemcpyAsync(perm, hp.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s)) != cudaSuccess)
            return fail(HHG_CUDA_ERROR, "upload batch order", e, msg);
        for (long long b = 0; b < nb; ++b, ++step) {
            W.gradients(X, T, perm + b * B, B, s);
            const double t = (double)(step + 1);
            const double lr = o.lr_final + 0.5 * (o.lr - o.lr_final) * (1.0 + std::cos(M_PI * step / total));
            adam_kernel<<<(kNMaster + 1 + 127) / 128, 128, 0, s>>>(
                W.P, W.part, W.ctas(B), W.m, W.v, W.W, (float)lr, o.beta1, o.beta2, o.eps,
                (float)(1.0 - std::pow((double)o.beta1, t)), (float)(1.0 - std::pow((double)o.beta2, t)),
                d_loss + ep, 1.0f / (float)nb);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return fail(HHG_CUDA_ERROR, "training launch", e, msg);
    }
    cudaEventRecord(ev1, s);
    int h_err = 0;
    std::vector<float> h_loss(o.epochs);
    cudaMemcpyAsync(master.data(), W.P, sizeof(float) * kNMaster, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&h_err, W.err, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(h_loss.data(), d_loss, sizeof(float) * o.epochs, cudaMemcpyDeviceToHost, s);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(HHG_CUDA_ERROR, "training", e, msg);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    if (h_err) return fail(HHG_CUDA_ERROR, "tensor-core completion wait timed out", cudaSuccess, msg);
    for (float v : master)
        if (!std::isfinite(v)) return fail(HHG_NONFINITE, "training diverged (non-finite weights)", cudaSuccess, msg);
    master_to_abi(master.data(), net->params);
    if (epoch_loss) std::memcpy(epoch_loss, h_loss.data(), sizeof(float) * o.epochs);
    if (train_ms) *train_ms = ms;
    return HHG_OK;
}

hhg_status mlp_gradients_impl(cudaStream_t s, const float *records, int64_t n, const hhg_mlp *net,
                              float *grad_out, float *loss_out, std::string *msg) {
    if (!records || !net || !grad_out || n < 1 || n > (int64_t)1 << 20)
        return fail(HHG_BAD_CONFIG, "1 <= n_records <= 2^20, network and output required", cudaSuccess, msg);
    if (!check_net(net)) return fail(HHG_BAD_CONFIG, "network standardisation not set", cudaSuccess, msg);
    Session S;
    Net W;
    float *d_rec = nullptr, *T = nullptr, *G = nullptr;  // G: the gradient and the loss
    bf16 *X = nullptr;
    cudaError_t e = W.init(true);
    if (e == cudaSuccess)
        e = S.build([&] {
            W.request(S, n, false);
            S.alloc(d_rec, (size_t)n * HHG_HIST_FIELDS);
            S.alloc(X, (size_t)n * kInPad);
            S.alloc(T, (size_t)n);
            S.alloc(G, kNMaster + 1);
        });
    if (e != cudaSuccess) return fail(HHG_CUDA_ERROR, "alloc buffers", e, msg);
    std::vector<float> master(kNMaster + 1);
    abi_to_master(net->params, master.data());
    cudaMemcpyAsync(d_rec, records, sizeof(float) * n * HHG_HIST_FIELDS, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(W.P, master.data(), sizeof(float) * kNMaster, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(W.err, 0, sizeof(int), s);
    mlp_prepare_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_rec, HHG_HIST_FIELDS, n, make_norm(*net), X, T);
    W.weights_bf16(s);
    W.gradients(X, T, nullptr, n, s);
    gradient_kernel<<<(kNMaster + 1 + 127) / 128, 128, 0, s>>>(W.part, W.ctas(n), G);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(HHG_CUDA_ERROR, "gradient launch", e, msg);
    int h_err = 0;
    cudaMemcpyAsync(master.data(), G, sizeof(float) * (kNMaster + 1), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&h_err, W.err, sizeof(int), cudaMemcpyDeviceToHost, s);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(HHG_CUDA_ERROR, "gradients", e, msg);
    if (h_err) return fail(HHG_CUDA_ERROR, "tensor-core completion wait timed out", cudaSuccess, msg);
    master_to_abi(master.data(), grad_out);
    if (loss_out) *loss_out = master[kNMaster];
    return HHG_OK;
}

hhg_status mlp_predict_impl(cudaStream_t s, const float *records, int64_t n, const hhg_mlp *net,
                            int path, float *out, std::string *msg) {
    if (!records || !net || !out || n < 1 || n > (int64_t)1 << 24 || (path != 0 && path != 1))
        return fail(HHG_BAD_CONFIG, "1 <= n_records <= 2^24, path 0 or 1", cudaSuccess, msg);
    if (!check_net(net)) return fail(HHG_BAD_CONFIG, "network standardisation not set", cudaSuccess, msg);
    Session S;
    Net W;
    float *d_rec = nullptr, *d_out = nullptr, *T = nullptr;
    bf16 *X = nullptr;
    MlpPacked *d_net = nullptr;
    cudaError_t e = path == 1 ? W.init(false) : cudaSuccess;
    if (e == cudaSuccess)
        e = S.build([&] {
            S.alloc(d_rec, (size_t)n * HHG_HIST_FIELDS);
            S.alloc(d_out, (size_t)n);
            if (path == 0) {
                S.alloc(d_net, 1);
            } else {
                W.request(S, 0, false);
                S.alloc(X, (size_t)n * kInPad);
                S.alloc(T, (size_t)n);
            }
        });
    if (e != cudaSuccess) return fail(HHG_CUDA_ERROR, "alloc buffers", e, msg);
    cudaMemcpyAsync(d_rec, records, sizeof(float) * n * HHG_HIST_FIELDS, cudaMemcpyHostToDevice, s);
    int h_err = 0;
    if (path == 0) {
        MlpPacked h;
        pack_mlp(*net, &h);
        cudaMemcpyAsync(d_net, &h, sizeof h, cudaMemcpyHostToDevice, s);
        const long long rows_per_cta = 32LL * kWarpsPerBlock;
        mlp_infer_kernel<<<(unsigned)((n + rows_per_cta - 1) / rows_per_cta), kBlockThreads, mlp_smem_bytes(), s>>>(
            d_net, d_rec, HHG_HIST_FIELDS, n, d_out);
        // the packed copy must outlive the kernel: synchronise before the session frees it
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(HHG_CUDA_ERROR, "inference", e, msg);
    } else {
        std::vector<float> master(kNMaster);
        abi_to_master(net->params, master.data());
        cudaMemcpyAsync(W.P, master.data(), sizeof(float) * kNMaster, cudaMemcpyHostToDevice, s);
        cudaMemsetAsync(W.err, 0, sizeof(int), s);
        mlp_prepare_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d_rec, HHG_HIST_FIELDS, n, make_norm(*net), X, T);
        W.weights_bf16(s);
        W.predict(X, n, net->out_mu, net->out_sigma, d_out, s);
        cudaMemcpyAsync(&h_err, W.err, sizeof(int), cudaMemcpyDeviceToHost, s);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return fail(HHG_CUDA_ERROR, "predict launch", e, msg);
    cudaMemcpyAsync(out, d_out, sizeof(float) * n, cudaMemcpyDeviceToHost, s);
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fail(HHG_CUDA_ERROR, "predict", e, msg);
    if (h_err) return fail(HHG_CUDA_ERROR, "tensor-core completion wait timed out", cudaSuccess, msg);
    return HHG_OK;
}
}  // namespace hhg

extern "C" {

void hhg_default_train_opts(hhg_train_opts *o) {
    if (!o) return;
    std::memset(o, 0, sizeof *o);
    o->epochs = 30;
    o->batch = 4096;
    o->lr = 2e-3f;
    o->beta1 = 0.9f;
    o->beta2 = 0.999f;
    o->eps = 1e-8f;
    o->lr_final = 1e-4f;
    o->seed = 1;
}

hhg_status hhg_mlp_init(uint64_t seed, const float *records, int64_t n, hhg_mlp *net) {
    if (!net) return HHG_BAD_CONFIG;
    std::memset(net, 0, sizeof *net);
    uint64_t s = seed;
    auto uni = [&](float bound) {
        const double u = (double)(splitmix64(s) >> 11) * (1.0 / 9007199254740992.0);
        return (float)((2.0 * u - 1.0) * bound);
    };
    float *p = net->params;
    const float b_in = 1.0f / std::sqrt((float)kIn), b_h = 1.0f / std::sqrt((float)kH);
    for (int i = 0; i < kH * kIn; ++i) p[aW1 + i] = uni(b_in);
    for (int i = 0; i < kH; ++i) p[aB1 + i] = uni(b_in);
    for (int i = 0; i < kH * kH; ++i) p[aW2 + i] = uni(b_h);
    for (int i = 0; i < kH; ++i) p[aB2 + i] = uni(b_h);
    for (int i = 0; i < kH * kH; ++i) p[aW3 + i] = uni(b_h);
    for (int i = 0; i < kH; ++i) p[aB3 + i] = uni(b_h);
    for (int i = 0; i < kH; ++i) p[aW4 + i] = uni(b_h);
    p[aB4] = 0.0f;
    for (int c = 0; c < kIn; ++c) {
        net->in_mu[c] = 0.0f;
        net->in_isig[c] = 1.0f;
    }
    net->out_mu = 0.0f;
    net->out_sigma = 1.0f;
    net->level_margin = -0.5f;
    if (records && n > 1) {
        double sum[kIn + 1] = {}, sq[kIn + 1] = {};
        for (int64_t r = 0; r < n; ++r)
            for (int c = 0; c <= kIn; ++c) {
                const double v = records[r * HHG_HIST_FIELDS + c];
                sum[c] += v;
                sq[c] += v * v;
            }
        for (int c = 0; c <= kIn; ++c) {
            const double mu = sum[c] / n;
            const double var = std::max(sq[c] / n - mu * mu, 0.0);
            const double sd = std::sqrt(var);
            if (c < kIn) {
                net->in_mu[c] = (float)mu;
                net->in_isig[c] = sd > 1e-12 ? (float)(1.0 / sd) : 1.0f;
            } else {
                net->out_mu = (float)mu;
                net->out_sigma = (float)std::max(sd, 1e-3);
            }
        }
    }
    return HHG_OK;
}

}  // extern "C"
